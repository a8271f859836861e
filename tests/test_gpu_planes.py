"""GPU: the stencil kernels that keep a block's planes in registers (k_stencil_planes: two planes per
block on middle levels, three on large ones).  Operators on one level against the oracle in FP64,
and against the staged march (an explicit launch shape keeps it) in FP32: numbers of planes that
the block's planes divide and do not, last vectors full and half-filled, rows of a few vectors,
every face kind, both colours."""
import numpy as np
import pytest

from _util import assert_field_equal, make_engine, make_oracle, push, randomize

pytestmark = pytest.mark.gpu

CASES = [
    # dims, bc (strict), relaxation; 2^22 points and more: three planes
    ((130, 127, 257), (0, 0, 0, 0, 0, 0), "jacobi"),
    ((129, 257, 129), (1, 1, 1, 1, 1, 1), "jacobi"),
    ((257, 129, 131), (1, 0, 0, 1, 0, 1), "jacobi"),
    ((129, 257, 129), (1, 1, 0, 1, 0, 0), "gs"),
    ((131, 129, 255), (0, 0, 0, 0, 1, 1), "gs"),
    # fewer: two planes
    ((129, 65, 65), (1, 1, 1, 1, 0, 0), "jacobi"),
    ((100, 129, 67), (0, 1, 0, 1, 1, 0), "jacobi"),
    ((129, 129, 33), (0, 0, 1, 0, 0, 0), "gs"),
    ((513, 257, 9), (1, 0, 1, 1, 0, 1), "jacobi"),
]


@pytest.mark.parametrize("ci", range(len(CASES)))
def test_operators_match_oracle(mgp_mod, gpu_ready, ci):
    dims, bc, rlx = CASES[ci]
    cfg = {"dims": dims, "levels": 1, "bc": bc, "restriction": "fw", "relaxation": rlx, "h": 1 / 100 if ci % 2 else 1 / 128,
           "strict_bc": True}
    o = make_oracle(cfg)
    randomize(o, 910 + ci)
    e = make_engine(mgp_mod, cfg)
    push(o, e)
    om = o.default_omega()
    o.relax(0, om, 2)
    o.residual(0)
    e.relax(0, om, 2)
    e.residual(0)
    for name in ("u", "r") + (("uprev",) if rlx == "jacobi" else ()):
        assert_field_equal(o, e, name, 0)
    o.relax(0, om, 1)
    o.residual(0)
    assert e.relax_residual(0, om, 1, norm=True) == o.norm("r", 0)
    for name in ("u", "r"):
        assert_field_equal(o, e, name, 0)
    e.close()


@pytest.mark.parametrize("ci", range(len(CASES)))
def test_fp32_matches_the_march(mgp_mod, gpu_ready, ci):
    dims, bc, rlx = CASES[ci]
    cfg = {"dims": dims, "levels": 1, "bc": bc, "restriction": "fw", "relaxation": rlx, "h": 1 / 100, "strict_bc": True}
    o = make_oracle(cfg)
    randomize(o, 930 + ci)
    engines, norms = [], []
    for shaped in (False, True):
        e = make_engine(mgp_mod, cfg, dtype=mgp_mod.F32)
        if shaped:
            for p in (mgp_mod.TUNE_RELAX_PLANES, mgp_mod.TUNE_RESID_PLANES, mgp_mod.TUNE_NORM_PLANES):
                e.set_tuning(0, p, 5)
        for name in ("u", "uprev", "f", "r") if rlx == "jacobi" else ("u", "f", "r"):
            e.upload(name, o.field(name, 0).astype(np.float32))
        for fc in range(6):
            e.upload_face(fc, o.face(fc, 0).astype(np.float32))
        e.relax(0, -1.0, 2)
        e.residual(0)
        norms.append(e.relax_residual(0, -1.0, 1, norm=True))
        engines.append(e)
    assert norms[0] == norms[1]
    for name in ("u", "r") + (("uprev",) if rlx == "jacobi" else ()):
        assert np.array_equal(engines[0].download(name), engines[1].download(name)), name
    for e in engines:
        e.close()
