"""GPU: the refinement residual that also writes the correction's first sweep.  A refinement solver
takes that sweep from the residual pass, a batch sweeps the zero guess itself: the same problem
gives the same bits both ways, for Jacobi and red-black smoothing, odd and even smoothing counts,
FP32 and FP64 corrections, Dirichlet and Neumann faces, last vectors full and half-filled."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [((65, 33, 33), 4, (0, 0, 0, 0, 0, 0)), ((33, 65, 17), 3, (1, 1, 1, 0, 1, 1)), ((129, 65, 65), 4, (0, 0, 1, 1, 0, 0))]


@pytest.mark.parametrize("ns", [1, 2, 3])
@pytest.mark.parametrize("inner", ["f32", "f64"])
@pytest.mark.parametrize("rlx", ["jacobi", "gs"])
@pytest.mark.parametrize("ci", range(len(CASES)))
def test_first_sweep_of_the_correction(mgp_mod, gpu_ready, ci, rlx, inner, ns):
    m = mgp_mod
    dims, levels, bc = CASES[ci]
    h = 1.0 / (dims[0] - 1)
    it = 3
    rng = np.random.default_rng(31 + ci)
    rx = m.JACOBI if rlx == "jacobi" else m.GAUSSSEIDEL
    e = m.Solver(dims, levels, h, bc, m.FULLWEIGHTING, rx, m.F64, it, 1, 0.0, strict_bc=True,
                 flags=m.FLAG_REFINE_F32 if inner == "f32" else m.FLAG_REFINE_F64)
    b = m.Batch(m.FULLWEIGHTING, rx, m.F32 if inner == "f32" else m.F64, "Vcycle", ns, max_problems=1)
    p = b.problem(b.add(dims, levels, h, bc, strict_bc=True))
    f = rng.uniform(-1, 1, size=e.level[0].pad)
    faces = [rng.uniform(-1, 1, size=e.level[0].face_shape[fc]) for fc in range(6)]
    for s in (e, p):
        s.upload("f", f)
        for fc in range(6):
            s.upload_face(fc, faces[fc])
        s.write_bc(0)
    for _ in range(2):  # a second solve starts from the first one's u
        e.solve("Vcycle", ns)
    b.solve(0.0, it)
    b.solve(0.0, it)
    for name in ("u", "r"):
        assert np.array_equal(e.download(name), p.download(name)), name
    e.close()
    b.close()
