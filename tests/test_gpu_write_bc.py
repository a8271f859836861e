"""GPU: Dirichlet data into u and u_prev in one launch.  Every combination of Dirichlet and Neumann
faces on a small box with different data on every face: the last Dirichlet face in the
reference's order (north, south, east, west, top, bottom) wins on shared edges and corners, and
nothing else is written."""
import numpy as np
import pytest

from _util import assert_field_equal, make_engine, make_oracle, push, randomize

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["f64", "f32"])
def test_write_bc_every_combination(mgp_mod, gpu_ready, dtype):
    for m in range(64):
        bc = tuple((m >> f) & 1 for f in range(6))
        cfg = {"dims": (6, 5, 7), "levels": 1, "bc": bc, "restriction": "fw", "relaxation": "jacobi", "h": 0.25,
               "strict_bc": True}
        o = make_oracle(cfg)
        randomize(o, 500 + m)
        for name in ("u", "uprev", "f", "r"):
            o.field(name, 0)[...] = o.field(name, 0).astype(np.float32)
        for fc in range(6):
            o.face(fc, 0)[...] = o.face(fc, 0).astype(np.float32)
        e = make_engine(mgp_mod, cfg, dtype=mgp_mod.F64 if dtype == "f64" else mgp_mod.F32)
        push(o, e)
        o.write_bc(0)
        e.write_bc(0)
        for name in ("u", "uprev"):
            assert_field_equal(o, e, name, 0)
        e.close()
