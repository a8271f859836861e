"""GPU: long thin boxes, whose planes are one block of the stencils: with more planes than the chip
takes two per block, the sweeps (and the FP64 residual with its norm) take the march, below that
and with larger planes the register form.  Either side of both lines, against the oracle in FP64
and against an explicit launch shape in FP32."""
import numpy as np
import pytest

from _util import assert_field_equal, make_engine, make_oracle, push, randomize

pytestmark = pytest.mark.gpu

CASES = [
    # dims, bc (strict), relaxation; blocks of a plane: 256 threads of two (FP64) or four points
    ((1184, 9, 9), (0, 0, 1, 1, 0, 0), "jacobi"),   # 592 blocks of two planes: one wave of 148 x 4
    ((1185, 9, 9), (1, 0, 0, 1, 0, 1), "jacobi"),   # 593
    ((4097, 9, 9), (0, 0, 0, 0, 0, 0), "gs"),
    ((4098, 5, 5), (1, 1, 1, 0, 1, 1), "gs"),
    ((2049, 16, 31), (0, 1, 1, 0, 1, 0), "jacobi"),  # 256 threads
    ((2049, 17, 31), (0, 1, 1, 0, 1, 0), "jacobi"),  # 272: two blocks
    ((16385, 3, 4), (1, 1, 1, 1, 1, 1), "jacobi"),
]


@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("ci", range(len(CASES)))
def test_operators(mgp_mod, gpu_ready, ci, dtype):
    dims, bc, rlx = CASES[ci]
    m = mgp_mod
    cfg = {"dims": dims, "levels": 1, "bc": bc, "restriction": "fw", "relaxation": rlx, "h": 1 / 100, "strict_bc": True}
    o = make_oracle(cfg)
    randomize(o, 970 + ci)
    names = ("u", "r") + (("uprev",) if rlx == "jacobi" else ())
    if dtype == "f64":
        e = make_engine(m, cfg)
        push(o, e)
        om = o.default_omega()
        o.relax(0, om, 2)
        o.residual(0)
        assert e.relax_residual(0, om, 2, norm=True) == o.norm("r", 0)
        o.relax(0, om, 1)
        o.residual(0)
        e.relax(0, om, 1)
        e.residual(0)
        for name in names:
            assert_field_equal(o, e, name, 0)
        e.close()
        return
    engines, norms = [], []
    for planes in (0, 5):
        e = make_engine(m, cfg, dtype=m.F32)
        for p in (m.TUNE_RELAX_PLANES, m.TUNE_RESID_PLANES, m.TUNE_NORM_PLANES):
            e.set_tuning(0, p, planes)
        for name in ("u", "f", "r") + names[2:]:
            e.upload(name, o.field(name, 0).astype(np.float32))
        for fc in range(6):
            e.upload_face(fc, o.face(fc, 0).astype(np.float32))
        norms.append(e.relax_residual(0, -1.0, 2, norm=True))
        e.relax(0, -1.0, 1)
        e.residual(0)
        engines.append(e)
    assert norms[0] == norms[1]
    for name in names:
        assert np.array_equal(engines[0].download(name), engines[1].download(name)), name
    for e in engines:
        e.close()
