"""A caller that captures a handle's own stream in a CUDA graph: replays advance the solve exactly as the calls
would, and the handle goes on afterwards."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def options(pkg, order, eqn="EULER"):
    mg = pkg.meshgen
    return dict(mg.DEFAULT_CASE, solution_poly_order=order, eqn=eqn, limiter="SQUEEZE" if order else "NONE", CFL=0.5,
                u=mg.mach_speed(0.4), BC1="SLIP_WALL", BC2="FREESTREAM", time_step_type="GLOBAL")


def captured(torch, stream, fn):
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=torch.cuda.ExternalStream(stream), capture_error_mode="thread_local"):
        fn()
    return g


@pytest.mark.parametrize("order", [1, 0])
@pytest.mark.parametrize("nx,ny", [(32, 16), (100, 50)])
def test_captured_solver_steps(pkg, nx, ny, order):
    torch = pytest.importorskip("torch")
    grid = pkg.meshgen.channel_bump_quads(nx, ny)
    a, b = (pkg.Solver(grid, options(pkg, order), precision=pkg.FP32) for _ in range(2))
    for s in (a, b):
        s.step(4)
        s.synchronize()
    g = captured(torch, a.stream(), lambda: a.step(3))
    for _ in range(3):
        g.replay()
    torch.cuda.synchronize()
    b.step(9)
    assert np.array_equal(a.get_state(), b.get_state())
    a.step(5)   # the handle's own launches again
    b.step(5)
    assert np.array_equal(a.get_state(), b.get_state())
    assert np.array_equal(a.residual_norm(), b.residual_norm())


def test_captured_batch_steps(pkg):
    torch = pytest.importorskip("torch")
    grid = pkg.meshgen.channel_bump_quads(40, 20)
    a, b = (pkg.Batch(4 * grid.num_cells, 4 * grid.num_faces + 256, 4) for _ in range(2))
    ids = [[x.add(grid, options(pkg, o)) for o in (1, 0, 1)] for x in (a, b)]
    for x in (a, b):
        x.step(2)
        x.synchronize()
    g = captured(torch, a.stream(), lambda: a.step(2))
    for _ in range(2):
        g.replay()
    torch.cuda.synchronize()
    a.step(3)
    b.step(7)
    for i, j in zip(*ids):
        assert np.array_equal(a.get_state(i), b.get_state(j))


@pytest.mark.parametrize("order", [1, 0])
def test_solves_join_and_leave_between_replays(pkg, order):
    """The graph takes the tile list from device memory: a larger solve admitted after the capture is advanced
    by the replays, one removed is not."""
    torch = pytest.importorskip("torch")
    small, large = pkg.meshgen.channel_bump_quads(24, 12), pkg.meshgen.channel_bump_quads(120, 60)
    a, b = (pkg.Batch(16384, 36000, 4) for _ in range(2))
    first = [x.add(small, options(pkg, order)) for x in (a, b)]
    for x in (a, b):
        x.step(1)
        x.synchronize()
    g = captured(torch, a.stream(), lambda: a.step(2))
    joined = [x.add(large, options(pkg, order)) for x in (a, b)]
    for x in (a, b):
        x.step(1)
        x.synchronize()
    for _ in range(2):
        g.replay()
    torch.cuda.synchronize()
    b.step(4)
    for i, j in (first, joined):
        assert np.array_equal(a.get_state(i), b.get_state(j))
    for x, i in zip((a, b), first):
        x.remove(i)
    g.replay()
    torch.cuda.synchronize()
    b.step(2)
    assert np.array_equal(a.get_state(joined[0]), b.get_state(joined[1]))
