"""Birth and death of so many cells that the blocks' counts are scanned by launches of their own (4,096 counts:
of 256 cells for birth, of 1,024 for death): one count fewer, the first that is, a last block and a last group
of 1,024 counts that are not full, no marked cell and only marked ones; death against a stable compaction,
birth's slots against the oracle."""
import numpy as np
import pytest

import oracle_lib as ol
from test_gpu_pd import eventful_cells, o2_field, raw

pytestmark = pytest.mark.gpu

gb = pytest.importorskip("gell_b200")


@pytest.mark.parametrize("n,live", [(4095 * 1024, 0.7), (4095 * 1024 + 1, 0.7), (4097 * 1024 - 3, 0.3),
                                    (5 * 1024 * 1024 + 700, 0.99), (4500000, 0.0), (4500000, 1.0)])
def test_death_of_many_cells(n, live):
    cells = np.tile(eventful_cells(64, 10.0, 50000, 5), n // 50000 + 1)[:n]
    cells["cell_clock"] = np.arange(n) % 16777216  # so that no two neighbours are alike
    cells["sign"] = np.random.Generator(np.random.Philox(n)).random(n) < live
    with gb.Simulation(voxel_num=64, voxel_length=10.0, max_cell_num=n + 1, rng_mode=gb.GELL_RNG_PHILOX) as sim:
        sim.import_cells(cells)
        left = cells[cells["sign"] != 0]
        before = sim.launch_count()
        assert sim.CellDeath_kernel() == len(left)
        assert sim.launch_count() - before == (2 if n <= 4095 * 1024 else 4)
        np.testing.assert_array_equal(raw(sim.export_cells()), raw(left))


@pytest.mark.parametrize("n,room", [(4095 * 256, 300000), (4095 * 256 + 1, 300000), (4097 * 256 - 3, 1000), (1400000, 500000)])
def test_birth_slots_of_many_cells(n, room):
    N, length, cap = 32, 10.0, n + room
    cells = eventful_cells(N, length, n, 6)
    field = o2_field(N, 7)
    oc = np.concatenate([cells, gb.empty_cells(room)])
    on = ol.birth_philox(oc, n, ol.params(N=N, len=length, cap=cap), field, 11, 0)
    with gb.Simulation(voxel_num=N, voxel_length=length, max_cell_num=cap, rng_mode=gb.GELL_RNG_PHILOX, seed=11) as sim:
        sim.add_substrate(gb.oxygen())
        sim.set_field(0, field)
        sim.import_cells(cells)
        before = sim.launch_count()
        assert sim.CellBirth_kernel() == on
        assert sim.launch_count() - before == (2 if n <= 4095 * 256 else 4)
        out = sim.export_cells()
    for f in ("sign", "phase", "V", "Vf", "Vcs", "Vns", "cell_clock"):
        np.testing.assert_array_equal(out[f], oc[f][:on])
    np.testing.assert_allclose(out["pos"], oc["pos"][:on], rtol=1e-6, atol=1e-4)  # CUDA's sinf, acosf and pow
