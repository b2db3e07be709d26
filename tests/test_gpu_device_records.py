"""Cell records and fields in device memory (gell_cells_import / _export, gell_field_import / _export with
on_device): the block edges of the record kernels, an address that is not 16-byte aligned, and fields
whose pitched rows are wider than the dense ones.  The records must come back byte for byte (padding
zero) and the fields bit for bit."""
import ctypes

import numpy as np
import pytest

from cases import ball_cells, random_field

pytestmark = pytest.mark.gpu

gb = pytest.importorskip("gell_b200")
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n", [1, 255, 256, 257, 1000])
@pytest.mark.parametrize("offset", [0, 4])
def test_records_round_trip(n, offset):
    c = ball_cells(24, 10.0, max(n, 8), seed=n, phases=True)[:n].copy()
    rng = np.random.Generator(np.random.Philox(n))
    c["force"] = rng.normal(0, 1, (n, 3)).astype(np.float32)
    raw = torch.zeros(n * 72 + 16, dtype=torch.uint8, device="cuda")
    back = torch.full_like(raw, 0xAB)
    raw[offset:offset + n * 72] = torch.from_numpy(c.view(np.uint8).reshape(-1).copy()).cuda()
    torch.cuda.synchronize()
    with gb.Simulation(voxel_num=24, voxel_length=10.0, max_cell_num=n) as sim:
        sim.import_cells(raw[offset:offset + n * 72], on_device=True)
        assert sim.export_cells_device(back[offset:offset + n * 72]) == n
        sim.sync()
        got = back.cpu().numpy()
        assert got[offset:offset + n * 72].tobytes() == c.tobytes()
        assert (got[:offset] == 0xAB).all() and (got[offset + n * 72:] == 0xAB).all()
        assert sim.export_cells().tobytes() == c.tobytes()


@pytest.mark.parametrize("N", [4, 5, 32, 131, 258])
@pytest.mark.parametrize("offset", [0, 1])
def test_field_round_trip(N, offset):
    f = random_field(N, seed=N)
    d = torch.zeros(N ** 3 + 8, device="cuda")
    back = torch.full_like(d, -7.0)
    d[offset:offset + N ** 3] = torch.from_numpy(f).cuda()
    torch.cuda.synchronize()
    with gb.Simulation(voxel_num=N, voxel_length=10.0, max_cell_num=8) as sim:
        sim.add_substrate(gb.oxygen())
        for call, t in ((sim.lib.gell_field_import, d), (sim.lib.gell_field_export, back)):
            assert call(sim.h, 0, ctypes.c_void_p(t[offset:].data_ptr()), 1) == 0
        sim.sync()
        got = back.cpu().numpy()
        assert np.array_equal(got[offset:offset + N ** 3], f)
        assert (got[:offset] == -7.0).all() and (got[offset + N ** 3:] == -7.0).all()
        assert np.array_equal(sim.field(0), f)
