"""Groups of the plane sweeps that are redone on the exact chain because a quotient was not the exact one, often:
fields that start at 0 beside a boundary value, where little diffusion takes the values through the
subnormal numbers.  Against the oracle's IEEE divisions: equal bits well above the subnormal
numbers, a few units in the last place and of 2^-149 below; and at a cost of the order of a substep without."""
import numpy as np
import pytest

import oracle_lib as ol

pytestmark = pytest.mark.gpu

gb = pytest.importorskip("gell_b200")


# (grids whose middle the boundary value's decay does not reach)
@pytest.mark.parametrize("N,D", [(33, 10.0), (64, 10.0), (97, 10.0), (131, 10.0), (64, 100.0), (97, 100.0), (131, 100.0),
                                 (97, 1e3), (131, 1e3)])
def test_fields_that_fall_through_the_subnormal_numbers(N, D):
    f, b = np.zeros(N ** 3, np.float32), 38.0
    with gb.Simulation(voxel_num=N, voxel_length=10.0, max_cell_num=16) as sim:
        sim.add_substrate(gb.Substrate(boundary=b, diffusion=D, decay=0.1, uptake=-10.0, init=0.0))
        sim.set_field(0, f)
        sim.PreLOD()
        sim.LODsolver(3)
        got = sim.field(0)
    E, F = ol.mesh_init(N, 10.0, D, 0.1, 0.01)
    want = np.asarray(ol.lod_substeps(f, np.zeros(N ** 3, np.float32), E, F, N, 0.01, b, 3), np.float32).reshape(-1)
    assert (np.abs(want) < 1.2e-38).any() and (want != 0).any()
    large = np.abs(want) > 1e-30
    np.testing.assert_array_equal(got[large].view(np.uint32), want[large].view(np.uint32))
    # below: the residuals that correct a quotient lose bits; at most 16 units passed along nine sweeps
    gap = np.abs(got.astype(np.float64) - want.astype(np.float64))
    assert (gap <= 16 * (np.abs(want.astype(np.float64)) * 2.0 ** -23 + 2.0 ** -149)).all()


def test_redone_groups_cost_no_more_than_the_sweeps():
    """200^3: ten substeps with every group redone (the option) within 2.4 times those without (2.6 times when the
    redone elements went one a turn)."""
    import torch
    with gb.Simulation(voxel_num=200, voxel_length=10.0, max_cell_num=16) as sim:
        stream = torch.cuda.Stream()
        sim.set_stream(stream)
        sim.add_substrate(gb.oxygen())
        sim.PreLOD()

        def best():
            out = []
            for _ in range(12):
                a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                a.record(stream)
                sim.LODsolver(10)
                b.record(stream)
                b.synchronize()
                out.append(a.elapsed_time(b))
            return min(out)

        plain = best()
        sim.set_exact_chain(True)
        redone = best()
    assert redone < 2.4 * plain, (redone, plain)
