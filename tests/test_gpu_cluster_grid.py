"""GPU: the coarse levels in a cluster against the same levels by the per-level kernels.  A launch
shape set on the coarsest level keeps every level out of the cluster, so small levels take the
grid kernels (and the one-kernel set-up, or the separate kernels on request); the one-CTA form is
the third.  The three leave the same bits in every field and face, in FP64 and FP32."""
import numpy as np
import pytest

from _util import make_oracle, randomize

pytestmark = pytest.mark.gpu

CASES = [
    # dims, levels, bc (strict), relaxation, restriction
    ((33, 17, 17), 3, (1, 1, 1, 1, 1, 0), "jacobi", "fw"),
    ((17, 33, 9), 2, (0, 1, 0, 1, 1, 0), "jacobi", "inj"),
    ((33, 33, 33), 4, (0, 0, 0, 0, 0, 0), "gs", "inj"),
    ((65, 33, 33), 4, (1, 1, 1, 0, 0, 0), "gs", "fw"),
    ((65, 65, 33), 3, (0, 0, 1, 1, 0, 1), "jacobi", "fw"),
]


@pytest.mark.parametrize("ns", [1, 2])
@pytest.mark.parametrize("cycle", ["vcycle", "fcycle"])
@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("ci", range(len(CASES)))
def test_cluster_matches_grid_kernels(mgp_mod, gpu_ready, ci, dtype, cycle, ns):
    m = mgp_mod
    dims, levels, bc, rlx, rst = CASES[ci]
    h = 1.0 / (dims[0] - 1)
    o = make_oracle({"dims": dims, "levels": levels, "bc": bc, "restriction": rst, "relaxation": rlx, "h": h,
                     "strict_bc": True})
    randomize(o, 330 + ci)
    jac = rlx == "jacobi"
    npdt = np.float64 if dtype == "f64" else np.float32
    names = ("u", "uprev", "f") if jac else ("u", "f")
    engines = []
    for form in ("cluster", "grid", "separate", "tail"):
        e = m.Solver(dims, levels, h, bc, m.FULLWEIGHTING if rst == "fw" else m.INJECTION,
                     m.JACOBI if jac else m.GAUSSSEIDEL, m.F64 if dtype == "f64" else m.F32, 2, 1, 0.0, strict_bc=True)
        if form == "tail":
            e.set_tuning(0, m.TUNE_TAIL, 1)
        elif form != "cluster":
            e.set_tuning(levels - 1, m.TUNE_RELAX_PLANES, 1)
            for l in range(levels - 1):
                e.set_tuning(l, m.TUNE_SETUP_FORM, 1 if form == "separate" else 2)
        for l in range(levels):
            for name in names + ("r",):
                e.upload(name, o.field(name, l).astype(npdt), l)
            for fc in range(6):
                e.upload_face(fc, o.face(fc, l).astype(npdt), l)
        getattr(e, cycle)(0, -1.0, ns)
        # solve iterations: the residual and its norm too
        st = e.solve(cycle.capitalize(), ns)
        engines.append((e, st))
    a, sa = engines[0]
    launches = [st.kernel_launches for _, st in engines]
    assert launches[0] < min(launches[1:3])
    for b, sb in engines[1:]:
        assert (sa.rel_res, sa.first_rel_res) == (sb.rel_res, sb.first_rel_res)
        for l in range(levels):
            for name in names + (("r",) if l == 0 else ()):
                assert np.array_equal(a.download(name, l), b.download(name, l)), (name, l)
            for fc in range(6):
                assert np.array_equal(a.download_face(fc, l), b.download_face(fc, l)), (fc, l)
    for e, _ in engines:
        e.close()
