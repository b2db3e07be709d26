"""Birth and death at the edges of their blocks (256 and 1,024 cells: one less, whole, one more, and more
blocks than a block has threads to add their counts), where slots come from the counts before a block:
death against a stable compaction, birth's slots against the oracle."""
import numpy as np
import pytest

import oracle_lib as ol
from test_gpu_pd import eventful_cells, o2_field, raw

pytestmark = pytest.mark.gpu

gb = pytest.importorskip("gell_b200")


@pytest.mark.parametrize("n", [1, 3, 255, 257, 1023, 1024, 1025, 4097, 1050626])
def test_death_at_block_edges(n):
    cells = eventful_cells(64, 10.0, n, 5)
    cells["sign"] = np.random.Generator(np.random.Philox(n)).random(n) < 0.7
    with gb.Simulation(voxel_num=64, voxel_length=10.0, max_cell_num=n + 1) as sim:
        sim.import_cells(cells)
        left = cells[cells["sign"] != 0]
        assert sim.CellDeath_kernel() == len(left)
        np.testing.assert_array_equal(raw(sim.export_cells()), raw(left))


@pytest.mark.parametrize("n,cap", [(1, 64), (255, 4096), (257, 4096), (1023, 4096), (1024, 4096), (1025, 1100), (270001, 500000)])
def test_birth_slots_at_block_edges(n, cap):
    N, length = 32, 10.0
    cells = eventful_cells(N, length, n, 6)
    field = o2_field(N, 7)
    oc = np.concatenate([cells, gb.empty_cells(cap)])[:cap].copy()
    on = ol.birth_philox(oc, n, ol.params(N=N, len=length, cap=cap), field, 11, 0)
    with gb.Simulation(voxel_num=N, voxel_length=length, max_cell_num=cap, rng_mode=gb.GELL_RNG_PHILOX, seed=11) as sim:
        sim.add_substrate(gb.oxygen())
        sim.set_field(0, field)
        sim.import_cells(cells)
        assert sim.CellBirth_kernel() == on
        out = sim.export_cells()
    for f in ("sign", "phase", "V", "Vf", "Vcs", "Vns", "cell_clock"):
        np.testing.assert_array_equal(out[f], oc[f][:on])
    np.testing.assert_allclose(out["pos"], oc["pos"][:on], rtol=1e-6, atol=1e-4)  # CUDA's sinf, acosf and pow


def test_counts_of_many_contexts_side_by_side():
    """The counts come back through words shared by all contexts, 64 to a page: more contexts than a page has
    words, destroyed and created again in between, each with its own number of live cells."""
    def make(k):
        cells = eventful_cells(8, 10.0, 300 + k, k)
        cells["sign"] = 0
        cells["sign"][:2 + k] = 1
        sim = gb.Simulation(voxel_num=8, voxel_length=10.0, max_cell_num=512)
        sim.import_cells(cells)
        return sim

    sims = {k: make(k) for k in range(70)}
    for k in range(0, 70, 3):
        sims.pop(k).close()
    for k in range(0, 70, 6):
        sims[k] = make(k)
    for k in sorted(sims, reverse=True):
        assert sims[k].CellDeath_kernel() == 2 + k
        sims.pop(k).close()
