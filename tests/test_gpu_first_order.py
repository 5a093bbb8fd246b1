"""The FP32 engine's first-order stage kernel (every solve of the launch is first order) against the
general stage kernel (the same solves beside a second-order one): the same bits, at the edges of the
tiles (part of one tile, a last tile of one cell, many-sided cells), for every wall and time step,
while second-order solves join and leave."""
import numpy as np
import pytest

from conftest import bits_equal, wheels_grid

pytestmark = pytest.mark.gpu


def case_of(pkg, **kw):
    mg = pkg.meshgen
    return dict(dict(mg.DEFAULT_CASE, solution_poly_order=0, limiter="NONE", time_step_type="LOCAL", CFL=0.4,
                     u=mg.mach_speed(0.4), v=9.0), **kw)


def grids(pkg):
    mg = pkg.meshgen
    return [mg.channel_bump_quads(5, 4), mg.channel_bump_quads(257, 1), mg.channel_bump_quads(64, 32),
            mg.voronoi_bump_channel(6000, seed=3), wheels_grid(pkg)]


def run(pkg, solves, second, iterations):
    """The solves in one batch, by stage kernels (kernel timing on), beside a second-order one from
    iteration second[0] to second[1]."""
    b = pkg.Batch(40000, 120000, 8, precision=pkg.FP32)
    b.set_kernel_timing(True)
    ids = [b.add(g, c) for g, c in solves]
    extra = None
    for i in range(iterations):
        if i == second[0]:
            extra = b.add(pkg.meshgen.channel_bump_quads(20, 9), case_of(pkg, solution_poly_order=1, limiter="SQUEEZE"))
        if i == second[1]:
            b.remove(extra)
        b.step(1)
    norms = b.norms()
    out = [b.get_state(i) for i in ids] + [norms[i][0] for i in ids]
    b.close()
    return out


@pytest.mark.parametrize("eqn,dt,wall", [("EULER", "GLOBAL", "SLIP_WALL"), ("NS", "LOCAL", "NO_SLIP_WALL"),
                                         ("EULER", "LOCAL", "EXTRAPOLATION")])
def test_first_order_kernel_equals_general_kernel(pkg, eqn, dt, wall):
    case = case_of(pkg, eqn=eqn, time_step_type=dt, BC1=wall, mu=0.01 if eqn == "NS" else 0.0)
    # (a mesh of one row of cells has wall faces numbered past its cells, which a no-slip wall refuses)
    solves = [(g, case) for i, g in enumerate(grids(pkg)) if i != 1 or wall != "NO_SLIP_WALL"]
    first = run(pkg, solves, (-1, -1), 6)
    general = run(pkg, solves, (0, -1), 6)
    mixed = run(pkg, solves, (2, 4), 6)
    for x, y, z in zip(first, general, mixed):
        assert np.all(np.isfinite(x)) and bits_equal(x, y) and bits_equal(x, z)


def test_first_order_restart_mid_iteration(pkg):
    """stage() kept in step with step() from a state, the residual kept, and a restart inside an iteration."""
    grid = pkg.meshgen.voronoi_bump_channel(9000, seed=5)
    case = case_of(pkg, eqn="EULER", time_step_type="GLOBAL")
    a, b = (pkg.Solver(grid, case, precision=pkg.FP32) for _ in range(2))
    q = a.get_state() * 1.01
    a.stage(2)
    for s in (a, b):
        s.set_store_residual(True)     # step() by stage kernels
        s.set_state(q)
    a.step(3)
    b.stage(9)
    for f in (0, 1, 2, 3):
        assert bits_equal(a.get(f), b.get(f))
    assert np.array_equal(a.residual_norm(), b.residual_norm())
    a.close()
    b.close()
