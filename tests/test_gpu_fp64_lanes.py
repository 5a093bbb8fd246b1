"""The FP64 engine's lane-parallel passes against the CPU oracle, bit for bit (signed zeros included), on
both sides of the two-lanes-per-face rule (64 faces per SM) and where the limiter's extremes, zero factors
and wall ghosts meet: uniform flow beside walls, every wall type, first order, random and restarted states."""
import numpy as np
import pytest

from conftest import bits_equal, wheels_grid

pytestmark = pytest.mark.gpu


def check(pkg, orc, grid, case, q, stages):
    gpu = pkg.Solver(grid, case, precision=pkg.FP64)
    gpu.set_store_residual(True)
    ref = orc.Oracle("port", grid=grid, case=case)
    if q is not None:
        gpu.set_state(q)
        ref.set_state(q)
    for s in range(stages):
        gpu.stage()
        ref.stage()
        assert bits_equal(gpu.get(2), ref.get(orc.RES)), f"residual, stage {s}"
        assert bits_equal(gpu.get(3), ref.get(orc.DT)), f"dt, stage {s}"
        if case["solution_poly_order"] and s % 3 == 0:
            assert bits_equal(gpu.get(4), ref.get(orc.QBAR_GRAD)), f"gradient, stage {s}"
        assert bits_equal(gpu.get(0 if s % 3 == 2 else 1), ref.get(orc.QBAR if s % 3 == 2 else orc.QSTAR)), f"state, stage {s}"
    gpu.close()


def state(grid, case, seed, noise):
    n = grid.num_cells
    rng = np.random.default_rng(seed)
    rho = case["rho"] * (1 + noise * rng.standard_normal(n))
    u, v = case["u"] * (1 + noise * rng.standard_normal(n)), 100 * noise * rng.standard_normal(n)
    P = case["P"] * (1 + noise * rng.standard_normal(n))
    v[: n // 3] = -0.0      # uniform patches and negative zeros
    rho[: n // 3], u[: n // 3], P[: n // 3] = case["rho"], case["u"], case["P"]
    return np.concatenate([rho, rho * u, rho * v, P / (case["gamma"] - 1) + 0.5 * rho * (u * u + v * v)])


@pytest.mark.parametrize("eqn,order,limiter,wall,far", [
    ("EULER", 1, "SQUEEZE", "SLIP_WALL", "FREESTREAM"), ("NS", 1, "SQUEEZE", "NO_SLIP_WALL", "EXTRAPOLATION"),
    ("NS", 1, "NONE", "SLIP_WALL", "FREESTREAM"), ("NS", 0, "NONE", "NO_SLIP_WALL", "FREESTREAM"),
    ("EULER", 0, "NONE", "EXTRAPOLATION", "SLIP_WALL")])
@pytest.mark.parametrize("shape", [(3, 3), (40, 12), (69, 69), (70, 70)])   # 9,660 and 9,940 faces: either side of the rule on 152 SMs
def test_lane_passes_match_oracle(pkg, orc, shape, eqn, order, limiter, wall, far):
    mg = pkg.meshgen
    grid = mg.channel_bump_quads(*shape)
    case = dict(mg.DEFAULT_CASE, eqn=eqn, solution_poly_order=order, limiter=limiter, BC1=wall, BC2=far, CFL=0.3,
                mu=0.05 if eqn == "NS" else 0.0, u=mg.mach_speed(0.4), v=-3.0,
                time_step_type="GLOBAL" if wall == "SLIP_WALL" else "LOCAL")
    for q in (None, state(grid, case, 7, 0.01)):
        check(pkg, orc, grid, case, q, 7)


@pytest.mark.parametrize("cells", [1500, 6000])
def test_lane_passes_polygons_match_oracle(pkg, orc, cells):
    mg = pkg.meshgen
    grid = mg.voronoi_bump_channel(cells, seed=8)
    case = dict(mg.DEFAULT_CASE, eqn="NS", mu=0.05, limiter="SQUEEZE", BC1="NO_SLIP_WALL", CFL=0.3, time_step_type="LOCAL",
                u=mg.mach_speed(0.4), v=-3.0)
    for q in (None, state(grid, case, 9, 0.02)):
        check(pkg, orc, grid, case, q, 7)


def test_lane_passes_many_sided_cells(pkg, orc):
    grid = wheels_grid(pkg)
    case = dict(pkg.meshgen.DEFAULT_CASE, eqn="EULER", limiter="SQUEEZE", time_step_type="GLOBAL", CFL=0.5,
                u=pkg.meshgen.mach_speed(0.4), v=5.0)
    check(pkg, orc, grid, case, state(grid, case, 11, 0.01), 6)


def test_graph_replays_match_stages(pkg):
    """step() (captured launches, programmatic for a small solve) and stage() give the same bits."""
    mg = pkg.meshgen
    for shape in ((24, 9), (100, 60)):
        grid = mg.channel_bump_quads(*shape)
        case = dict(mg.DEFAULT_CASE, eqn="EULER", limiter="SQUEEZE", time_step_type="GLOBAL", CFL=0.6, u=mg.mach_speed(0.5))
        a, b = (pkg.Solver(grid, case, precision=pkg.FP64) for _ in range(2))
        a.step(40)
        b.stage(120)
        for f in (0, 1, 2, 3, 4, 5):
            assert bits_equal(a.get(f), b.get(f))
        a.close()
        b.close()
