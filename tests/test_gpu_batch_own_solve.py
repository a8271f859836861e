"""GPU: a problem of a batch solved on its own between the batch's steps (batch.problem(pid).solve).
The residual at the end of that solve starts the problem's next correction with that solve's
smoothing, the batch's step goes on with the batch's: u and r equal those of a refinement solver
taken through the same solves."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (omega, sweeps) of the solve in between; the batch uses the default omega and 2 sweeps
BETWEEN = [(-1.0, 2), (-1.0, 1), (0.6, 2), (-1.0, 0)]


@pytest.mark.parametrize("cycle", ["Vcycle", "Fcycle"])
@pytest.mark.parametrize("rlx", ["JACOBI", "GAUSSSEIDEL"])
@pytest.mark.parametrize("omega,ns", BETWEEN)
def test_own_solve_between_steps(mgp_mod, gpu_ready, omega, ns, rlx, cycle):
    m = mgp_mod
    dims, levels, h = (33, 17, 33), 3, 1 / 32
    bc = (0, 0, 1, 0, 0, 0)
    rx = getattr(m, rlx)
    e = m.Solver(dims, levels, h, bc, m.FULLWEIGHTING, rx, m.F64, 1, 1, 0.0, flags=m.FLAG_REFINE_F32)
    b = m.Batch(m.FULLWEIGHTING, rx, m.F32, cycle, 2, max_problems=2)
    pid = b.add(dims, levels, h, bc)
    other = b.add((17, 17, 17), 3, 1 / 16)
    p = b.problem(pid)
    p.set_iteration_limits(1, 1, 0.0)
    rng = np.random.default_rng(3)
    f = rng.uniform(-1, 1, size=e.level[0].pad)
    faces = [rng.uniform(-1, 1, size=e.level[0].face_shape[fc]) for fc in range(6)]
    for s in (e, p):
        s.upload("f", f)
        for fc in range(6):
            s.upload_face(fc, faces[fc])
        s.write_bc(0)
    b.problem(other).upload("f", rng.uniform(-1, 1, size=b.problem(other).level[0].pad))
    b.step()
    e.solve(cycle, 2)
    for _ in range(2):
        p.solve(cycle, ns, omega)
        e.solve(cycle, ns, omega)
        b.step()
        e.solve(cycle, 2)
        assert np.array_equal(e.download("u"), p.download("u"))
    b.solve(0.0, 2)
    for _ in range(2):
        e.solve(cycle, 2)
    for name in ("u", "r"):
        assert np.array_equal(e.download(name), p.download(name)), name
    e.close()
    b.close()
