"""GPU: the residual of a set-up and the Neumann face restriction in one launch (levels of more than
30000 and fewer than 2^22 points that take the built-in shapes).  Cycles against the oracle in
FP64, and against an explicit residual shape (which keeps the separate launches) in FP32: one plane
per block and two, an odd number of planes, planes of one block and of many, faces of several
blocks, every kind of face; and no launch more than with Dirichlet faces only."""
import numpy as np
import pytest

from _util import assert_face_equal, assert_field_equal, make_engine, make_oracle, push, randomize

pytestmark = pytest.mark.gpu

CASES = [
    # dims, levels, bc (strict), relaxation, restriction
    ((65, 33, 33), 2, (1, 1, 1, 1, 1, 1), "jacobi", "fw"),
    ((33, 37, 65), 2, (1, 0, 0, 1, 0, 1), "jacobi", "inj"),
    ((129, 65, 65), 3, (0, 0, 1, 0, 1, 1), "gs", "fw"),
    ((1025, 9, 9), 2, (1, 1, 0, 1, 0, 0), "jacobi", "fw"),
    ((9, 129, 257), 2, (0, 1, 1, 0, 1, 0), "jacobi", "fw"),
    ((129, 161, 97), 3, (1, 1, 1, 1, 0, 0), "gs", "inj"),
    ((257, 129, 113), 3, (0, 0, 0, 0, 1, 0), "jacobi", "fw"),
]


def config(ci):
    dims, levels, bc, rlx, rst = CASES[ci]
    return {"dims": dims, "levels": levels, "bc": bc, "restriction": rst, "relaxation": rlx, "h": 1.0 / (max(dims) - 1),
            "strict_bc": True}


@pytest.mark.parametrize("cycle", ["vcycle", "fcycle"])
@pytest.mark.parametrize("ci", range(len(CASES)))
def test_cycles_match_oracle(mgp_mod, gpu_ready, ci, cycle):
    cfg = config(ci)
    o = make_oracle(cfg)
    randomize(o, 820 + ci)
    e = make_engine(mgp_mod, cfg)
    push(o, e)
    om = o.default_omega()
    for ns in (1, 2):
        getattr(o, cycle)(0, om, ns)
        getattr(e, cycle)(0, om, ns)
    for l in range(o.levels):
        for name in ("u", "f"):
            assert_field_equal(o, e, name, l)
        for fc in range(6):
            if cfg["bc"][fc] == 1:
                assert_face_equal(o, e, fc, l)
    e.close()


@pytest.mark.parametrize("ci", range(len(CASES)))
def test_fp32_matches_separate_launches(mgp_mod, gpu_ready, ci):
    cfg = config(ci)
    o = make_oracle(cfg)
    randomize(o, 840 + ci)
    jac = cfg["relaxation"] == "jacobi"
    engines = []
    for planes in (0, 5):
        e = make_engine(mgp_mod, cfg, dtype=mgp_mod.F32)
        e.set_tuning(0, mgp_mod.TUNE_RESID_PLANES, planes)
        for l in range(o.levels):
            for name in ("u", "uprev", "f", "r") if jac else ("u", "f", "r"):
                e.upload(name, o.field(name, l).astype(np.float32), l)
            for fc in range(6):
                e.upload_face(fc, o.face(fc, l).astype(np.float32), l)
        e.vcycle(0, -1.0, 2)
        engines.append(e)
    for l in range(o.levels):
        for name in ("u", "f"):
            assert np.array_equal(engines[0].download(name, l), engines[1].download(name, l)), (name, l)
        for fc in range(6):
            assert np.array_equal(engines[0].download_face(fc, l), engines[1].download_face(fc, l)), (fc, l)
    assert np.array_equal(engines[0].download("r"), engines[1].download("r"))
    for e in engines:
        e.close()


@pytest.mark.parametrize("ci", range(len(CASES)))
def test_no_launch_of_its_own(mgp_mod, gpu_ready, ci):
    cfg = config(ci)
    n = []
    for bc in (cfg["bc"], (0, 0, 0, 0, 0, 0)):
        e = make_engine(mgp_mod, dict(cfg, bc=bc), maxiter=1, tol=0.0)
        n.append(e.solve("Vcycle", 2, -1.0).kernel_launches)
        e.close()
    assert n[0] == n[1]
