"""GPU: boxes with more planes than a grid has rows to give one to every two or three of them
(65535): the register form of the stencils takes them to the march, as every accepted size."""
import numpy as np
import pytest

from _util import assert_field_equal, make_engine, make_oracle, push, randomize

pytestmark = pytest.mark.gpu

CASES = [
    # dims, relaxation: two planes per block would take 65535 (the last that fits) and 65536 rows,
    # three 66668 of them
    ((131070, 3, 5), "jacobi"),
    ((131071, 3, 5), "jacobi"),
    ((131075, 3, 9), "gs"),
    ((200003, 5, 5), "jacobi"),
    ((300001, 3, 5), "gs"),
]


@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("ci", range(len(CASES)))
def test_operators(mgp_mod, gpu_ready, ci, dtype):
    """FP64 against the oracle, FP32 against an explicit launch shape."""
    dims, rlx = CASES[ci]
    m = mgp_mod
    cfg = {"dims": dims, "levels": 1, "bc": (0, 0, 1, 0, 0, 0), "restriction": "fw", "relaxation": rlx, "h": 1 / 64,
           "strict_bc": True}
    o = make_oracle(cfg)
    randomize(o, 950 + ci)
    if dtype == "f64":
        e = make_engine(m, cfg)
        push(o, e)
        om = o.default_omega()
        o.relax(0, om, 1)
        o.residual(0)
        assert e.relax_residual(0, om, 1, norm=True) == o.norm("r", 0)
        o.relax(0, om, 1)
        o.residual(0)
        e.relax(0, om, 1)
        e.residual(0)
        for name in ("u", "r"):
            assert_field_equal(o, e, name, 0)
        e.close()
        return
    got = []
    for planes in (0, 64):
        e = make_engine(m, cfg, dtype=m.F32)
        for p in (m.TUNE_RELAX_PLANES, m.TUNE_RESID_PLANES, m.TUNE_NORM_PLANES):
            e.set_tuning(0, p, planes)
        for name in ("u", "uprev", "f", "r") if rlx == "jacobi" else ("u", "f", "r"):
            e.upload(name, o.field(name, 0).astype(np.float32))
        for fc in range(6):
            e.upload_face(fc, o.face(fc, 0).astype(np.float32))
        n = e.relax_residual(0, -1.0, 1, norm=True)
        e.relax(0, -1.0, 1)
        e.residual(0)
        got.append((n, e.download("u"), e.download("r")))
        e.close()
    assert got[0][0] == got[1][0]
    assert np.array_equal(got[0][1], got[1][1]) and np.array_equal(got[0][2], got[1][2])
