"""fv2d_residual_noalloc with more than 2^30 cells (most without faces: the entry bounds the faces, not the
cells): every cell's residual is written, once."""
import ctypes

import pytest

from conftest import bits_equal
from test_gpu_noalloc_sizes import make_case, oracle
from test_zz_no_alloc import NoallocMesh, device_mesh, perturbed_state

pytestmark = pytest.mark.gpu


def test_cells_beyond_2_30(pkg, orc):
    torch = pytest.importorskip("torch")
    n_all = (1 << 30) + 1027
    if torch.cuda.mem_get_info()[0] < 110 << 30:
        pytest.skip("needs 82 GB of device memory")
    grid = pkg.meshgen.channel_bump_quads(17, 9)
    case = make_case(pkg, "SLIP_WALL", "FREESTREAM")
    m, keep = device_mesh(pkg, torch, grid, case)
    n = grid.num_cells
    q = perturbed_state(case, n, seed=2)
    off = torch.empty(n_all + 1, dtype=torch.int32, device="cuda")
    off[: n + 1] = keep["off"]
    off[n + 1:] = keep["off"][-1]
    vol = torch.ones(n_all, dtype=torch.float64, device="cuda")
    vol[:n] = keep["vol"]
    wide = torch.empty(4, n_all, dtype=torch.float64, device="cuda")
    wide[:, :n] = torch.from_numpy(q.reshape(4, n)).cuda()
    r = torch.full_like(wide, float("nan"))
    m.num_cells, m.cell_face_offsets, m.cell_vol = n_all, off.data_ptr(), vol.data_ptr()
    fn = pkg.library().fv2d_residual_noalloc
    fn.restype = ctypes.c_int
    fn.argtypes = [ctypes.POINTER(NoallocMesh), ctypes.POINTER(pkg.Case), ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p]
    cs = pkg.case_from_dict(case)
    torch.cuda.synchronize()
    assert fn(ctypes.byref(m), ctypes.byref(cs), wide.data_ptr(), r.data_ptr(), None) == 0
    torch.cuda.synchronize()
    got = r[:, :n].cpu().numpy().reshape(-1)
    assert bits_equal(got, oracle(orc, grid, case, q))
    left = [int((r[j, n:] != 0.0).sum()) for j in range(4)]   # (numbers: a failure prints no large tensor)
    assert left == [0, 0, 0, 0]
    del off, vol, wide, r
    torch.cuda.empty_cache()
