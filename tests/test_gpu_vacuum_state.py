"""A restart state with a cell of no mass, momentum and energy: 0/0 is NaN in the reference, so a first-order step
from it, or one whose face states are the cell's own, is non-physical.  The FP64 engine gives what the CPU oracle
gives stage by stage, bit for bit (a NaN is a NaN), and reports it where the oracle's states are non-physical."""
import numpy as np
import pytest

from conftest import bits_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cell", ["first", "middle"])
@pytest.mark.parametrize("nx,ny", [(24, 12), (150, 75)])   # two lanes per face, and one thread
@pytest.mark.parametrize("eqn,order", [("EULER", 1), ("NS", 1), ("EULER", 0), ("NS", 0)])
def test_vacuum_cell(pkg, orc, eqn, order, nx, ny, cell):
    mg = pkg.meshgen
    case = dict(mg.DEFAULT_CASE, eqn=eqn, solution_poly_order=order, limiter="NONE", u=mg.mach_speed(0.4), mu=1e-3,
                BC1="NO_SLIP_WALL" if eqn == "NS" else "SLIP_WALL", BC2="FREESTREAM", CFL=0.5, time_step_type="LOCAL")
    grid = mg.channel_bump_quads(nx, ny)
    s = pkg.Solver(grid, case, precision=pkg.FP64)
    q = s.get_state().reshape(4, -1)
    q[:, 0 if cell == "first" else q.shape[1] // 2] = 0.0
    q = np.ascontiguousarray(q.reshape(-1))
    ref = orc.Oracle("port", grid=grid, case=case)
    ref.set_state(q)
    s.set_state(q)
    bad = False
    for stage in range(3):
        s.stage()
        ref.stage()
        try:
            s.synchronize()
            reported = False
        except pkg.Fv2dError as e:
            assert "non-physical" in str(e)
            reported = True
        want = ref.get(orc.QBAR if stage == 2 else orc.QSTAR)
        w = want.reshape(4, -1)
        bad = bad or not bool(np.all((w[0] > 0) & (w[3] > 0)))
        assert reported == bad, f"stage {stage}"
        if bad:
            break   # a state is not read back through a reported one
        got = s.get_state() if stage == 2 else s.get(1)
        assert bits_equal(got, want), f"stage {stage}"
    if order == 0:
        assert bad
    s.close()
