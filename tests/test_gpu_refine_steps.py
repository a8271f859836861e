"""GPU: refinement steps against the same steps composed from plain solvers.  The refinement
residual writes the correction's first sweep along (also in a batch); here the correction cycle
is run by a plain solver from u = 0, so every sweep of it is launched: r from an FP64 residual of
u, e from one cycle with zero boundary data on f = (Ti) r, u += e at the relaxed points in numpy.
u and r must be bit-identical for two steps in a row, for 1, 2 and 3 sweeps (with one, the only
Jacobi sweep is the one the residual writes), V- and F-cycles, both smoothers, both inner types
and every kind of face."""
import numpy as np
import pytest

from _util import make_engine

pytestmark = pytest.mark.gpu

CASES = [
    # dims, levels, bc (strict), restriction, relaxation
    ((33, 17, 17), 3, (0, 0, 1, 0, 1, 0), "inj", "jacobi"),
    ((65, 33, 17), 4, (1, 1, 1, 1, 0, 1), "fw", "jacobi"),
    ((65, 65, 33), 4, (0, 0, 0, 0, 0, 0), "fw", "gs"),
    ((33, 17, 33), 3, (1, 1, 1, 0, 1, 1), "inj", "gs"),
]


@pytest.mark.parametrize("ns", [1, 2, 3])
@pytest.mark.parametrize("inner", ["f32", "f64"])
@pytest.mark.parametrize("cycle", ["Vcycle", "Fcycle"])
@pytest.mark.parametrize("ci", range(len(CASES)))
def test_steps_match_composed_steps(mgp_mod, gpu_ready, ci, cycle, inner, ns):
    m = mgp_mod
    dims, levels, bc, rst, rlx = CASES[ci]
    cfg = {"dims": dims, "levels": levels, "bc": bc, "restriction": rst, "relaxation": rlx, "h": 1.0 / (dims[0] - 1),
           "strict_bc": True}
    npdt = np.float32 if inner == "f32" else np.float64
    R = make_engine(m, cfg, maxiter=1, tol=0.0, flags=m.FLAG_REFINE_F32 if inner == "f32" else m.FLAG_REFINE_F64)
    P = make_engine(m, cfg)
    Q = make_engine(m, cfg, dtype=m.F32 if inner == "f32" else m.F64)
    B = m.Batch(m.FULLWEIGHTING if rst == "fw" else m.INJECTION, m.JACOBI if rlx == "jacobi" else m.GAUSSSEIDEL,
                m.F32 if inner == "f32" else m.F64, cycle, ns, max_problems=1)
    pid = B.add(dims, levels, cfg["h"], bc, strict_bc=True)
    lv = R.level[0]
    rng = np.random.default_rng(700 + ci)
    u0, f = rng.uniform(-1, 1, size=lv.pad), rng.uniform(-1, 1, size=lv.pad)
    faces = [rng.uniform(-1, 1, size=lv.face_shape[fc]) for fc in range(6)]
    for e in (R, P, B.problem(pid)):
        e.upload("u", u0)
        e.upload("f", f)
        for fc in range(6):
            e.upload_face(fc, faces[fc])
        e.write_bc(0)
    # the relaxed points of level 0 (all but the Dirichlet planes) in the host layout
    kind = dict(zip(("north", "south", "east", "west", "top", "bottom"), lv.face_kind))
    rb = tuple(slice(h + (kind[lo] == 0), h + n - (kind[hi] == 0))
               for h, n, lo, hi in zip((lv.halo["west"], lv.halo["south"], lv.halo["bottom"]), lv.shape,
                                       ("west", "south", "bottom"), ("east", "north", "top")))
    u = P.download("u")
    P.residual(0)
    for step in range(2):
        fi = np.zeros(lv.pad, dtype=npdt)
        fi[rb] = P.download("r")[rb].astype(npdt)
        for l in range(levels):
            for name in ("u", "uprev", "f", "r") if rlx == "jacobi" else ("u", "f", "r"):
                Q.upload(name, np.zeros(Q.level[l].pad, dtype=npdt), l)
        Q.upload("f", fi)
        getattr(Q, cycle.lower())(0, -1.0, ns)
        u[rb] = u[rb] + Q.download("u")[rb].astype(np.float64)
        P.upload("u", u)
        P.residual(0)
        R.solve(cycle, ns)
        B.solve(0.0, 1)
        for e in (R, B.problem(pid)):
            assert np.array_equal(e.download("u")[lv.interior], u[lv.interior]), step
            assert np.array_equal(e.download("r")[rb], P.download("r")[rb]), step
    for e in (R, P, Q, B):
        e.close()
