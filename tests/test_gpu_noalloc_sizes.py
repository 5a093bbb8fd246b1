"""fv2d_residual_noalloc over its range, against the CPU oracle bit for bit: on both sides of the size from
which the cells' primitives have a pass of their own (24,000 faces), every boundary type, partial last
blocks, in place (r = q), and with more cells than the cell scratch holds (cells without faces)."""
import ctypes

import numpy as np
import pytest

from conftest import bits_equal
from test_zz_no_alloc import NoallocMesh, device_mesh, perturbed_state

pytestmark = pytest.mark.gpu


def call(pkg, torch, m, case, q, in_place=False):
    fn = pkg.library().fv2d_residual_noalloc
    fn.restype = ctypes.c_int
    fn.argtypes = [ctypes.POINTER(NoallocMesh), ctypes.POINTER(pkg.Case), ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p]
    q_dev = torch.from_numpy(q).cuda()
    r_dev = q_dev if in_place else torch.full_like(q_dev, float("nan"))
    cs = pkg.case_from_dict(case)
    assert fn(ctypes.byref(m), ctypes.byref(cs), q_dev.data_ptr(), r_dev.data_ptr(), None) == 0
    torch.cuda.synchronize()
    return r_dev.cpu().numpy()


def oracle(orc, grid, case, q):
    o = orc.Oracle("port", grid=grid, case=case)
    o.set_state(q)
    o.stage()
    return o.get(orc.RES)


def make_case(pkg, bc1, bc2):
    return dict(pkg.meshgen.DEFAULT_CASE, solution_poly_order=0, limiter="NONE", BC1=bc1, BC2=bc2,
                u=pkg.meshgen.mach_speed(0.5), v=-7.0)


@pytest.mark.parametrize("bc1,bc2", [("SLIP_WALL", "FREESTREAM"), ("NO_SLIP_WALL", "EXTRAPOLATION")])
@pytest.mark.parametrize("nx,ny", [(3, 3), (17, 9), (118, 100), (119, 100)])   # 23,818 and 24,019 faces
def test_sizes(pkg, orc, nx, ny, bc1, bc2):
    torch = pytest.importorskip("torch")
    grid = pkg.meshgen.channel_bump_quads(nx, ny)
    case = make_case(pkg, bc1, bc2)
    m, keep = device_mesh(pkg, torch, grid, case)
    q = perturbed_state(case, grid.num_cells, seed=nx)
    want = oracle(orc, grid, case, q)
    assert bits_equal(call(pkg, torch, m, case, q), want)
    assert bits_equal(call(pkg, torch, m, case, q, in_place=True), want)


@pytest.mark.parametrize("nx,ny", [(118, 100), (130, 100)])
def test_more_cells_than_the_cell_scratch(pkg, orc, nx, ny):
    torch = pytest.importorskip("torch")
    grid = pkg.meshgen.channel_bump_quads(nx, ny)
    case = make_case(pkg, "SLIP_WALL", "FREESTREAM")
    m, keep = device_mesh(pkg, torch, grid, case)
    n, pad = grid.num_cells, 180000
    q = perturbed_state(case, n, seed=5)
    off = torch.cat([keep["off"], keep["off"][-1:].expand(pad)]).contiguous()
    vol = torch.cat([keep["vol"], torch.ones(pad, dtype=torch.float64, device="cuda")])
    m.num_cells, m.cell_face_offsets, m.cell_vol = n + pad, off.data_ptr(), vol.data_ptr()
    wide = np.concatenate([np.concatenate([part, np.ones(pad)]) for part in q.reshape(4, n)])
    r = call(pkg, torch, m, case, wide).reshape(4, n + pad)
    assert bits_equal(r[:, :n].reshape(-1), oracle(orc, grid, case, q))
    assert np.all(r[:, n:] == 0.0)
