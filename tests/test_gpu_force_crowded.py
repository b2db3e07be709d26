"""The thread-per-cell force kernel where bins are crowded: lists that fill up in some lanes of a warp and not
in others, warps that compute the forces in the walk from its start (more accepted candidates than a list
holds, by estimate), and populations in which both kinds sit side by side, against the oracle bit for bit;
and the cost of a crowded population, which is of the order of its accepted pairs."""
import numpy as np
import pytest

import oracle_lib as ol
from cases import ball_cells
from test_gpu_mech import raw

pytestmark = pytest.mark.gpu

gb = pytest.importorskip("gell_b200")


def crowd(N, parts, seed):
    """[(cells, radius as a fraction of the grid)]: balls in one another's middle."""
    c = np.concatenate([ball_cells(N, 10.0, n, seed + k, radius_frac=f, outside=0) for k, (n, f) in enumerate(parts)])
    return c[np.random.Generator(np.random.Philox(seed)).permutation(len(c))]


# 24 accepted candidates lie at about 3 cells to a bin
@pytest.mark.parametrize("N,parts,over", [
    (48, [(49000, 0.40)], {}),                 # 1.7 to a bin: some lanes' lists fill up
    (48, [(49000, 0.33)], {}),                 # 3: half of them
    (48, [(49000, 0.24)], {}),                 # 8: the walk computes
    (48, [(49000, 0.15)], {}),                 # 31
    (48, [(20000, 0.10), (30000, 0.45)], {}),  # a crowd of 43 to a bin inside 0.7 to a bin
    (48, [(49000, 0.33)], {"ra_ratio": 1.3}),
    (48, [(20000, 0.10), (30000, 0.45)], {"ra_ratio": 0.9}),
    (48, [(49000, 0.24)], {"cc_max_dist": 4.0}),
    (24, [(49000, 0.40)], {"voxel_length": 20.0}),
])
def test_crowded_bins_bit_exact_vs_oracle(N, parts, over):
    length = over.get("voxel_length", 10.0)
    cells = crowd(N, parts, 9)
    cells["pos"] *= np.float32(length / 10.0)
    oc = cells.copy()
    ol.fm_update(oc, ol.params(N=N, len=length, cap=65536, **{k: v for k, v in over.items() if k != "voxel_length"}))
    with gb.Simulation(**{"voxel_num": N, "voxel_length": length, "max_cell_num": 65536, **over}) as sim:
        sim.import_cells(cells)
        sim.FM_update()
        np.testing.assert_array_equal(raw(sim.export_cells()), raw(oc))


def test_a_crowd_costs_what_its_pairs_cost():
    """100,000 cells at 12 to a bin against 0.8 to a bin: 15 times the candidates, 6 times the time (16 times
    where a lane that has filled its list works it off by itself)."""
    def seconds(frac):
        cells = ball_cells(64, 10.0, 100000, 3, radius_frac=frac, outside=0)
        with gb.Simulation(voxel_num=64, voxel_length=10.0, max_cell_num=len(cells)) as sim:
            best = 1e9
            for _ in range(8):
                sim.import_cells(cells)
                sim.sync()
                sim.profile(True)
                sim.profile_read(True)
                sim.FM_update()
                sim.sync()
                r = sim.profile_read(True)
                sim.profile(False)
                best = min(best, r["k_force_move"][1])
            return best

    crowded, normal = seconds(0.195), seconds(0.49)
    assert crowded < 12 * normal, (crowded, normal)
