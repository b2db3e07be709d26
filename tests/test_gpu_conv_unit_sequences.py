"""The surrogate's convolutions over the sequences of work units that large grids give a CTA: whole units,
then several whose last line is their only one (edges of 497 and more), units of one line throughout, and
short last units.  Unit length and CTAs are set, so that a small grid has them.  The layers against
PyTorch's fp32 convolution of the same stored bf16 input, to one bf16 unit; the gradient of a training pair
against autograd.  A wait that gives up is reported by the next sync."""
import numpy as np
import pytest

import test_gpu_surrogate as ts
import test_gpu_surrogate_train as tt

pytestmark = pytest.mark.gpu

# (edge, lines per unit, CTAs); 130: two x tiles
UNITS = [(17, 16, 1), (17, 16, 3), (17, 1, 5), (18, 16, 2), (17, 2, 4), (33, 16, 8), (130, 3, 20)]


@pytest.mark.parametrize("N,lines,ctas", UNITS)
def test_layers_over_unit_sequences(N, lines, ctas):
    w = ts.random_weights(12)
    Ws = ts.layer_params(w)
    with ts.make_sim(N, 4, cells=200) as sim:
        sim.surrogate_load(0, w, 50, 0.1, 1.0)
        sim.debug_conv_units(lines, ctas)
        sim.surrogate_run_layers(0, 1)
        x, h = sim.surrogate_read(0, 0)[:3], sim.surrogate_read(0, 1)
        ts.assert_bf16_close(h, np.maximum(ts.conv(x, Ws[0], N), 0), "input layer")
        sim.surrogate_run_layers(0, 2)
        t = sim.surrogate_read(0, 2)
        ts.assert_bf16_close(t, np.maximum(ts.conv(h, Ws[1], N), 0), "inner layer")
        sim.surrogate_run_layers(0, 3)
        ts.assert_bf16_close(sim.surrogate_read(0, 1), h + ts.conv(t, Ws[2], N), "residual layer")
        sim.surrogate_run_layers(0, 10)
        whole = sim.surrogate_read(0, 3)
        sim.sync()
        sim.debug_conv_units()
        sim.surrogate_run_layers(0, 10)
        np.testing.assert_array_equal(whole.view(np.uint32), sim.surrogate_read(0, 3).view(np.uint32))


@pytest.mark.parametrize("N,lines,ctas", UNITS)
def test_gradient_over_unit_sequences(N, lines, ctas):
    w = tt.random_weights(5)
    with tt.make_sim(N, 3, cells=200) as sim:
        sim.surrogate_train_init(0, w, 5, 0.1)
        sim.debug_conv_units(lines, ctas)
        p = sim.field(0)
        loss = sim.surrogate_train_pair(0, 0.0)
        grad, y, x = sim.surrogate_train_read(0, 1), sim.surrogate_train_read(0, 2), sim.surrogate_read(0, 0)[:3]
        sim.sync()
    tloss, tgrad = tt.torch_grads(w, x, p, y, N)
    assert abs(loss - tloss) <= 1e-3 * tloss
    for name, sl in tt.layer_slices():
        a, r = grad[sl].astype(np.float64), tgrad[sl].astype(np.float64)
        rel = np.linalg.norm(a - r) / max(np.linalg.norm(r), 1e-30)
        assert rel < 2e-2, (name, rel)  # the stored gradient planes are bf16
