"""The surrogate's convolutions at the edges of their work units: 16 output lines along z to a unit (one
line, a whole unit, one line more) and 128 voxels to an x tile (a tile, one voxel more), against
PyTorch's fp32 convolution of the same stored bf16 input, to one bf16 unit (the fp32 sums differ in
order only), and a training pair's gradient across the same edges against autograd."""
import numpy as np
import pytest

import test_gpu_surrogate as ts
import test_gpu_surrogate_train as tt

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [8, 16, 17, 33, 128, 129])
def test_layers_at_unit_edges(N):
    w = ts.random_weights(11)
    Ws = ts.layer_params(w)
    with ts.make_sim(N, 4, cells=200) as sim:
        sim.surrogate_load(0, w, 50, 0.1, 1.0)
        sim.surrogate_run_layers(0, 1)
        x, h = sim.surrogate_read(0, 0)[:3], sim.surrogate_read(0, 1)
        ts.assert_bf16_close(h, np.maximum(ts.conv(x, Ws[0], N), 0), "input layer")
        sim.surrogate_run_layers(0, 2)
        t = sim.surrogate_read(0, 2)
        ts.assert_bf16_close(t, np.maximum(ts.conv(h, Ws[1], N), 0), "inner layer")
        sim.surrogate_run_layers(0, 3)
        ts.assert_bf16_close(sim.surrogate_read(0, 1), h + ts.conv(t, Ws[2], N), "residual layer")


@pytest.mark.parametrize("N", [17, 33, 129])
def test_gradient_at_unit_edges(N):
    w = tt.random_weights(5)
    with tt.make_sim(N, 3, cells=200) as sim:
        sim.surrogate_train_init(0, w, 5, 0.1)
        p = sim.field(0)
        loss = sim.surrogate_train_pair(0, 0.0)
        grad, y, x = sim.surrogate_train_read(0, 1), sim.surrogate_train_read(0, 2), sim.surrogate_read(0, 0)[:3]
    tloss, tgrad = tt.torch_grads(w, x, p, y, N)
    assert abs(loss - tloss) <= 1e-3 * tloss
    for name, sl in tt.layer_slices():
        a, r = grad[sl].astype(np.float64), tgrad[sl].astype(np.float64)
        rel = np.linalg.norm(a - r) / max(np.linalg.norm(r), 1e-30)
        assert rel < 2e-2, (name, rel)  # the stored gradient planes are bf16, as in the larger tests
