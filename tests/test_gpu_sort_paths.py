"""The sort's forms at their edges, against the oracle's stable sort: one CTA up to 6,144 cells (one cell, a
warp, a round of 1,024 and one more, the largest, one more), tiles of 4,096 with the counts of up to 32 tiles
added in the scatter, or scanned by a launch of their own beyond; one to three passes of up to 10 bits."""
import numpy as np
import pytest

import oracle_lib as ol
from cases import ball_cells
from test_gpu_mech import raw

pytestmark = pytest.mark.gpu

gb = pytest.importorskip("gell_b200")


@pytest.mark.parametrize("N,n", [(4, 33), (9, 1), (20, 32), (32, 1024), (32, 1025), (100, 6144), (100, 6145),
                                 (33, 8192), (60, 8193), (130, 131072), (130, 131073), (300, 135169)])
def test_sort_forms_bit_exact_vs_oracle(N, n):
    cells = ball_cells(N, 10.0, n, 11, radius_frac=0.45, outside=min(8, n // 4))
    oc = cells.copy()
    P = dict(N=N, len=10.0, cap=150000)
    okeys, operm, os_, oe = ol.fm_update(oc, ol.params(**P))
    with gb.Simulation(voxel_num=N, voxel_length=10.0, max_cell_num=150000) as sim:
        sim.import_cells(cells)
        sim.FM_update()
        np.testing.assert_array_equal(sim.dump_keys(), okeys)
        np.testing.assert_array_equal(sim.dump_perm(), operm)
        s, e = sim.dump_se()
        np.testing.assert_array_equal(s, os_)
        np.testing.assert_array_equal(e, oe)
        np.testing.assert_array_equal(raw(sim.export_cells()), raw(oc))


@pytest.mark.parametrize("batched", [False, True])
def test_ensemble_sorts_small_and_large_members_together(batched):
    def members():
        out = []
        for N, n in [(20, 500), (32, 6144), (40, 6145), (100, 140000)]:
            sim = gb.Simulation(voxel_num=N, voxel_length=10.0, max_cell_num=150000)
            sim.add_substrate(gb.oxygen())
            sim.import_cells(ball_cells(N, 10.0, n, n, radius_frac=0.45))
            out.append(sim)
        return out

    alone, together = members(), members()
    for m in alone:
        for _ in range(3):
            m.mechanics_step(2)
    with gb.Ensemble(together) as ens:
        ens.set_batched(batched)
        ens.run_mechanics(3, 2)
        ens.sync()
    for a, b in zip(alone, together):
        np.testing.assert_array_equal(raw(a.export_cells()), raw(b.export_cells()))
        np.testing.assert_array_equal(a.dump_keys(), b.dump_keys())
        a.close()
        b.close()
