"""The line-tile sweeps where they are what runs: ensembles with a member of edge 225 to 256, whose batched
substeps go over one list of every member's line tiles (small and odd ones and two substrates among them), and
substrate streams with padded rows, on grids above the plane sweeps' edge and below it by option."""
import numpy as np
import pytest

from cases import one_per_voxel
from test_gpu_ensemble import member, raw

pytestmark = pytest.mark.gpu

gb = pytest.importorskip("gell_b200")


@pytest.mark.parametrize("edges", [(37, 100, 230, 64), (225, 256, 251), (32, 131, 256, 48, 225)])
def test_batched_line_tiles_match_members_stepped_alone(edges):
    def make():
        ms = [member(i, N, 20 * N) for i, N in enumerate(edges)]
        ms[1].add_substrate(gb.drug())
        return ms

    alone, together = make(), make()
    with gb.Ensemble(together) as ens:
        ens.configure(branches=2, sweep_warps=0)
        ens.set_batched(True)
        for a in alone:
            for _ in range(5):
                a.mechanics_step(3)
        ens.run_mechanics(5, 3)
        for a, b in zip(alone, together):
            a.CellBirth_kernel()
            b.CellBirth_kernel()
        for a in alone:
            for _ in range(2):
                a.mechanics_step(3)
        ens.run_mechanics(2, 3)
        ens.sync()
    for a, b in zip(alone, together):
        assert a.count() == b.count()
        np.testing.assert_array_equal(raw(a.export_cells()), raw(b.export_cells()))
        np.testing.assert_array_equal(a.field(0).view(np.uint32), b.field(0).view(np.uint32))
    np.testing.assert_array_equal(alone[1].field(1).view(np.uint32), together[1].field(1).view(np.uint32))
    for m in alone + together:
        m.close()


@pytest.mark.parametrize("N,ring", [(131, 0), (97, 0), (225, -1), (259, -1), (429, -1)])
def test_substrate_streams_with_padded_rows(N, ring):
    cells = one_per_voxel(N, 10.0, seed=N + 31, lo=N // 3, hi=N // 3 + N // 8)
    field = np.random.Generator(np.random.Philox(N)).uniform(10.0, 38.0, N ** 3).astype(np.float32)
    out = []
    for streams in (False, True):
        with gb.Simulation(voxel_num=N, voxel_length=10.0, max_cell_num=len(cells) + 1024) as sim:
            sim.add_substrate(gb.oxygen())
            sim.add_substrate(gb.drug())
            sim.set_sweep_ring(ring)
            sim.set_lod_streams(streams)
            sim.set_field(0, field)
            sim.set_field(1, field * np.float32(0.03))
            sim.import_cells(cells)
            sim.PreLOD()
            sim.LODsolver(3)
            sim.LODsolver(1)
            out.append((sim.field(0).view(np.uint32), sim.field(1).view(np.uint32)))
    for sub in range(2):
        np.testing.assert_array_equal(out[0][sub], out[1][sub])
