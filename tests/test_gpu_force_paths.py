"""The two force kernels (a warp per cell up to 48,000 cells, a thread per cell beyond) against the oracle,
bit for bit, where they can go wrong: more than 32 candidates to a cell (a second round of the warp's
lanes), more than 16 accepted ones (a full list of the thread's walk), one cell more than the rule's line,
a last block that is not full, cutoff ratios that are and are not floats, and a first cutoff that
accepts nothing."""
import numpy as np
import pytest

import oracle_lib as ol
from cases import ball_cells
from test_gpu_mech import raw

pytestmark = pytest.mark.gpu

gb = pytest.importorskip("gell_b200")


@pytest.mark.parametrize("N,n,frac,over", [
    (32, 1, 0.35, {}),
    (32, 33, 0.05, {}),
    (32, 3001, 0.12, {}),
    (32, 3001, 0.12, {"ra_ratio": 1.3}),
    (32, 3001, 0.12, {"cc_max_dist": 0.0}),
    (48, 48000, 0.45, {}),
    (48, 48001, 0.45, {}),
    (48, 48001, 0.33, {"ra_ratio": 1.3}),
    (48, 48001, 0.33, {"cc_max_dist": 4.0}),
])
def test_force_paths_bit_exact_vs_oracle(N, n, frac, over):
    cells = ball_cells(N, 10.0, n, 7, radius_frac=frac, outside=min(8, n // 4))
    oc = cells.copy()
    ol.fm_update(oc, ol.params(N=N, len=10.0, cap=65536, **over))
    with gb.Simulation(voxel_num=N, voxel_length=10.0, max_cell_num=65536, **over) as sim:
        sim.import_cells(cells)
        sim.FM_update()
        np.testing.assert_array_equal(raw(sim.export_cells()), raw(oc))
