"""A state handed over in page-locked memory is taken before the call returns: the caller may write its buffer
at once, also when earlier work of the solve is still running."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["FP64", "FP32"])
@pytest.mark.parametrize("call", ["load_state", "set_state"])
@pytest.mark.parametrize("nx,ny,busy", [(24, 12, 40), (600, 300, 4)])
def test_pinned_state_may_be_overwritten_after_the_call(pkg, nx, ny, busy, call, precision):
    torch = pytest.importorskip("torch")
    mg = pkg.meshgen
    case = dict(mg.DEFAULT_CASE, u=mg.mach_speed(0.4), BC1="SLIP_WALL", BC2="FREESTREAM", CFL=0.5)
    s = pkg.Solver(mg.channel_bump_quads(nx, ny), case, precision=getattr(pkg, precision))
    q = s.get_state()
    q *= 1.0 + 1e-3 * np.random.default_rng(7).random(q.size)
    host = torch.empty(q.size, dtype=torch.float64, pin_memory=True)
    a = host.numpy()
    for _ in range(5):
        s.step(busy)   # still running when the state is handed over
        a[:] = q
        getattr(s, call)(a)
        a[:] = -1.0
        got = s.get_state()
        # the FP32 engine keeps a state as a pair of floats (48 bits)
        np.testing.assert_allclose(got, q, rtol=0 if precision == "FP64" else 2.0 ** -47, atol=0)
    s.close()


@pytest.mark.parametrize("precision", ["FP64", "FP32"])
def test_threads_fetch_solves_of_one_batch(pkg, precision):
    """Several threads read different solves of a batch back at once, each into its own array."""
    import concurrent.futures as cf

    mg = pkg.meshgen
    grids = [mg.channel_bump_quads(2 * n, n) for n in (8, 40, 150, 31, 90, 12)]   # 128 to 45,000 cells
    b = pkg.Batch(sum(g.num_cells for g in grids) + 4096, sum(g.num_faces for g in grids) + 4096, len(grids),
                  precision=getattr(pkg, precision))
    ids = [b.add(g, dict(mg.DEFAULT_CASE, u=mg.mach_speed(0.3 + 0.05 * i), BC1="SLIP_WALL", BC2="FREESTREAM", CFL=0.5))
           for i, g in enumerate(grids)]
    b.step(5)
    want = [b.get_state(i) for i in ids]
    with cf.ThreadPoolExecutor(8) as pool:
        for _ in range(10):
            got = list(pool.map(b.get_state, ids * 4))
            for k, q in enumerate(got):
                assert np.array_equal(q, want[k % len(ids)]), f"solve {k % len(ids)}"
    b.close()
