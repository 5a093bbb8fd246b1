"""fv2d_residual_noalloc on states of any kind: zero, subnormal, huge, infinite and NaN components beside ordinary
ones give what the CPU oracle gives, bit for bit (a NaN is a NaN)."""
import numpy as np
import pytest

from conftest import bits_equal
from test_gpu_noalloc_sizes import call, make_case, oracle
from test_zz_no_alloc import device_mesh, perturbed_state

pytestmark = pytest.mark.gpu

TINY = 5e-324
CASES = {
    "infinite energy": (3, [np.inf, -np.inf]),
    "zero energy": (3, [0.0, -0.0]),
    "huge energy": (3, [1e300, 1e305, 1.7e308]),
    "zero density": (0, [0.0, -0.0]),
    "subnormal density": (0, [TINY, 1e-310, 2.2250738585072014e-308]),
    "small density": (0, [1e-250, 1e-120, 1e-61, 1e-60]),
    "huge density": (0, [1e60, 1e61, 1e250, np.inf]),
    "negative density": (0, [-1.2, -1e-300]),
    "subnormal momentum": (1, [TINY, -1e-310, 1e-308]),
    "small momentum": (2, [1e-300, -1e-290, 1e-160, 1e-61, 1e-60]),
    "signed zero momentum": (2, [0.0, -0.0]),
    "huge momentum": (1, [1e60, 1e61, -1e160, 1e300]),
    "not a number": (1, [np.nan]),
    "density not a number": (0, [np.nan]),
    "vacuum": (0, [0.0, -0.0]),   # with every other component zero
}


@pytest.mark.parametrize("bc1,bc2", [("SLIP_WALL", "FREESTREAM"), ("NO_SLIP_WALL", "EXTRAPOLATION")])
@pytest.mark.parametrize("still", [False, True])   # True: no momentum in the planted cells, so that P stays positive
@pytest.mark.parametrize("name", CASES)
@pytest.mark.parametrize("nx,ny", [(40, 30), (130, 100)])   # without and with the cells' own pass
def test_operands_outside_the_ordinary_range(pkg, orc, nx, ny, name, still, bc1, bc2):
    torch = pytest.importorskip("torch")
    grid = pkg.meshgen.channel_bump_quads(nx, ny)
    case = make_case(pkg, bc1, bc2)
    m, keep = device_mesh(pkg, torch, grid, case)
    n = grid.num_cells
    q = perturbed_state(case, n, seed=3).reshape(4, n)
    j, values = CASES[name]
    at = np.random.default_rng(1).permutation(n)[: n // 10]   # boundary cells and neighbours of each other among them
    if still:
        q[1:3, at] = 0.0
    if name == "vacuum":
        q[:, at] = 0.0
    q[j, at] = np.resize(values, at.size)
    q = np.ascontiguousarray(q.reshape(-1))
    with np.errstate(all="ignore"):
        want = oracle(orc, grid, case, q)
    got = call(pkg, torch, m, case, q)
    bad = np.isnan(want)
    assert np.array_equal(bad, np.isnan(got))
    assert bits_equal(got[~bad], want[~bad])
