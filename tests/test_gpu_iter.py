"""The FP32 engine's whole-iteration kernel (a solve whose tiles are all resident at once: step()) against
its stage kernels (stage(), which larger solves use): the same bits, at the edges of the tile sizes
(one tile, a last tile of one cell, two and three tiles per SM), for every equation, limiter, time step
and wall, from the freestream and from a restart, and across mixed calls."""
import numpy as np
import pytest

from conftest import bits_equal, wheels_grid

pytestmark = pytest.mark.gpu

FIELDS = (0, 1, 2, 3, 4, 5)   # Qbar, Q*, residual, dt, both gradients


def case_of(pkg, **kw):
    mg = pkg.meshgen
    return dict(dict(mg.DEFAULT_CASE, limiter="SQUEEZE", time_step_type="LOCAL", CFL=0.4, u=mg.mach_speed(0.4), v=9.0), **kw)


def state(grid, case, seed):
    n = grid.num_cells
    rng = np.random.default_rng(seed)
    rho = case["rho"] * (1 + 0.02 * rng.standard_normal(n))
    u, v = case["u"] * (1 + 0.02 * rng.standard_normal(n)), 5.0 * rng.standard_normal(n)
    P = case["P"] * (1 + 0.02 * rng.standard_normal(n))
    return np.concatenate([rho, rho * u, rho * v, P / (case["gamma"] - 1) + 0.5 * rho * (u * u + v * v)])


def both(pkg, grid, case, q, iterations=3):
    out = []
    for whole in (True, False):
        s = pkg.Solver(grid, case, precision=pkg.FP32)
        if q is not None:
            s.set_state(q)
        if whole:
            s.step(iterations)
        else:
            s.stage(3 * iterations)
        out.append([s.get(f) for f in FIELDS])
        s.stage(2)          # a partial iteration on top of either, finished by step()
        s.step(2)
        out[-1].append(s.get_state())
        s.close()
    return out


@pytest.mark.parametrize("eqn,dt,order,limiter,wall", [
    ("EULER", "GLOBAL", 1, "SQUEEZE", "SLIP_WALL"), ("NS", "LOCAL", 1, "SQUEEZE", "NO_SLIP_WALL"),
    ("NS", "GLOBAL", 1, "NONE", "SLIP_WALL"), ("EULER", "LOCAL", 0, "NONE", "EXTRAPOLATION")])
@pytest.mark.parametrize("nx,ny", [(5, 4), (13, 5), (64, 64), (139, 70)])
def test_whole_iterations_equal_stages(pkg, nx, ny, eqn, dt, order, limiter, wall):
    grid = pkg.meshgen.channel_bump_quads(nx, ny)
    case = case_of(pkg, eqn=eqn, time_step_type=dt, solution_poly_order=order, limiter=limiter, BC1=wall,
                   mu=0.01 if eqn == "NS" else 0.0)
    for q in (None, state(grid, case, 3)):
        a, b = both(pkg, grid, case, q)
        for x, y in zip(a, b):
            assert bits_equal(x, y)


@pytest.mark.parametrize("cells", [9000, 30000, 76000, 84000])   # 64-cell tiles; two, two and three tiles per SM
def test_whole_iterations_equal_stages_polygons(pkg, cells):
    grid = pkg.meshgen.voronoi_bump_channel(cells, seed=3)
    case = case_of(pkg, eqn="NS", mu=0.02, BC1="NO_SLIP_WALL")
    a, b = both(pkg, grid, case, state(grid, case, 4), 2)
    for x, y in zip(a, b):
        assert bits_equal(x, y)


def test_whole_iterations_many_sided_cells(pkg):
    grid = wheels_grid(pkg)
    case = case_of(pkg, eqn="EULER", time_step_type="GLOBAL")
    a, b = both(pkg, grid, case, None)
    for x, y in zip(a, b):
        assert bits_equal(x, y)


def test_long_step_splits_into_launches(pkg):
    """step() cuts a long run into launches of 256 iterations: the same as one iteration at a time."""
    grid = pkg.meshgen.channel_bump_quads(40, 10)
    case = case_of(pkg, eqn="EULER", time_step_type="GLOBAL")
    a, b = (pkg.Solver(grid, case, precision=pkg.FP32) for _ in range(2))
    a.step(517)
    for _ in range(517):
        b.step(1)
    assert bits_equal(a.get_state(), b.get_state())
    a.close()
    b.close()


def test_batch_with_removed_solves(pkg):
    """Empty tile slots (a removed solve's) only take part in the barriers."""
    cases = [(pkg.meshgen.channel_bump_quads(n, 12), case_of(pkg, eqn="EULER")) for n in (40, 9, 70)]
    b = pkg.Batch(20000, 60000, 4, precision=pkg.FP32)
    ids = [b.add(g, c) for g, c in cases]
    b.step(3)
    b.remove(ids[1])
    b.step(4)
    for i in (0, 2):
        s = pkg.Solver(*cases[i], precision=pkg.FP32)
        s.stage(21)
        assert bits_equal(b.get_state(ids[i]), s.get_state())
        s.close()
    b.close()


def test_handles_of_different_plans_in_turn(pkg):
    """A handle with larger tiles steps after one with smaller tiles was planned (and the other way
    round): each handle's launches have its own shared-memory size."""
    big = pkg.meshgen.voronoi_bump_channel(76000, seed=3)
    small = pkg.meshgen.channel_bump_quads(13, 5)
    case = case_of(pkg, eqn="EULER")
    a, b = (pkg.Solver(g, case, precision=pkg.FP32) for g in (big, small))
    for s in (a, b, a, b):
        s.step(1)
    for s, g in ((a, big), (b, small)):
        t = pkg.Solver(g, case, precision=pkg.FP32)
        t.stage(6)
        assert bits_equal(s.get_state(), t.get_state())
        t.close()
        s.close()


@pytest.mark.parametrize("timing", [False, True])   # whole-iteration kernel, stage kernels
def test_batch_states_between_iterations(pkg, timing):
    """get_state() between iterations (it works in rows that the next iteration writes first) leaves the
    run as it is, for first- and second-order solves, and returns the freestream of a solve not yet stepped."""
    cases = [(pkg.meshgen.channel_bump_quads(31, 12), case_of(pkg, eqn="EULER")),
             (pkg.meshgen.voronoi_bump_channel(5000, seed=2), case_of(pkg, eqn="NS", mu=0.02, BC1="NO_SLIP_WALL")),
             (pkg.meshgen.channel_bump_quads(9, 30), case_of(pkg, eqn="EULER", solution_poly_order=0, limiter="NONE"))]
    b = pkg.Batch(20000, 60000, 4, precision=pkg.FP32)
    b.set_kernel_timing(timing)
    ids = [b.add(g, c) for g, c in cases]
    solvers = [pkg.Solver(g, c, precision=pkg.FP32) for g, c in cases]
    for n in (0, 1, 3, 2):
        b.step(n)
        for i, s in zip(ids, solvers):
            s.step(n)
            assert bits_equal(b.get_state(i), s.get_state())
    for s in solvers:
        s.close()
    b.close()
