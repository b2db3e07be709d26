"""What the ensemble's tuner tries: two steps for each branch count (1, 2, 4 .. all members) with the members'
own sweeps and with the batched ones, and two widths more only where a member's grid is swept in line tiles,
which is what the width belongs to."""
import pytest

from test_gpu_ensemble import member

pytestmark = pytest.mark.gpu

gb = pytest.importorskip("gell_b200")


@pytest.mark.parametrize("edges,ring,variants", [((32, 40, 48, 56, 64), -1, 2), ((32, 40, 48, 56, 64), 0, 4), ((32, 225), -1, 4)])
def test_widths_are_tried_where_they_exist(edges, ring, variants):
    ms = [member(i, N, 500) for i, N in enumerate(edges)]
    for m in ms:
        m.set_sweep_ring(ring)
    branch_counts = {2: 2, 5: 4}[len(edges)]
    with gb.Ensemble(ms) as ens:
        taken, branches, warps = ens.tune(1)
        ens.sync()
    assert taken == 1 + 2 * branch_counts * variants
    assert 1 <= branches <= len(edges) and (warps == 0 if variants == 2 else warps in (0, 1, 2))
    for m in ms:
        m.close()
