"""The plane sweeps (grid edges up to 224, the default there): an xy-plane per CTA swept along x and y in
shared memory, then the z sweep one line tile per warp.

The edges below are those of the boxes of 32 the kernels cut a plane into (one box, a box and one
element, a whole last box), the smallest grid, the largest plane and the first edge past it, each with
two substrates, uptake in the boundary layers too, and several substeps.  Fields must equal the
oracle's (include/LODkernel.cuh:24-136) bit for bit up to the size it finishes in seconds, and the
line-tile kernels' at every size."""
import numpy as np
import pytest

import oracle_lib as ol
from cases import one_per_voxel, random_field

pytestmark = pytest.mark.gpu

gb = pytest.importorskip("gell_b200")


def run(N, cells, field, k, ring, exact=False):
    with gb.Simulation(voxel_num=N, voxel_length=10.0, max_cell_num=max(1024, len(cells))) as sim:
        sim.add_substrate(gb.oxygen())
        sim.add_substrate(gb.drug())
        sim.set_sweep_ring(ring)
        sim.set_exact_chain(exact)
        sim.set_field(0, field)
        sim.set_field(1, field * np.float32(0.03))
        sim.import_cells(cells)
        sim.PreLOD()
        sim.LODsolver(k)
        return sim.field(0).view(np.uint32), sim.field(1).view(np.uint32)


@pytest.mark.parametrize("N", [4, 5, 31, 32, 33, 36, 64, 65, 97, 128, 129, 131, 160, 223, 224, 225])
def test_plane_sweeps_bit_exact(N):
    # one cell per voxel of a block that starts in the boundary layers
    cells = one_per_voxel(N, 10.0, seed=N, lo=1, hi=max(2, N // 3))
    field = random_field(N, seed=N + 1)
    got = run(N, cells, field, 3, -1)
    for other in (run(N, cells, field, 3, 0), run(N, cells, field, 3, -1, exact=True)):
        for a, b in zip(got, other):
            np.testing.assert_array_equal(a, b)
    if N > 131:
        return
    for a, s, f in zip(got, (gb.oxygen(), gb.drug()), (field, field * np.float32(0.03))):
        rate = ol.prelod(cells, N, 10.0, s.uptake)
        E, F = ol.mesh_init(N, 10.0, s.diffusion, s.decay, 0.01)
        want = ol.lod_substeps(f, rate, E, F, N, 0.01, s.boundary, 3)
        np.testing.assert_array_equal(a, np.asarray(want, np.float32).reshape(-1).view(np.uint32))


def test_batched_planes_of_many_members():
    """More members of one edge than one batched launch takes, and a member of another edge."""
    edges = [8] * 130 + [40]

    def members():
        out = []
        for i, N in enumerate(edges):
            sim = gb.Simulation(voxel_num=N, voxel_length=10.0, max_cell_num=64, rng_mode=gb.GELL_RNG_PHILOX)
            sim.add_substrate(gb.oxygen())
            sim.set_field(0, random_field(N, seed=i))
            sim.import_cells(one_per_voxel(N, 10.0, seed=i, lo=2, hi=4))
            out.append(sim)
        return out

    alone, together = members(), members()
    for m in alone:
        for _ in range(3):
            m.mechanics_step(2)
    with gb.Ensemble(together) as ens:
        ens.set_batched(True)
        ens.configure(branches=4)
        ens.run_mechanics(3, 2)
        ens.sync()
    for a, b in zip(alone, together):
        np.testing.assert_array_equal(a.field(0).view(np.uint32), b.field(0).view(np.uint32))
        a.close()
        b.close()
