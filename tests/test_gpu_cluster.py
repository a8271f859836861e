"""GPU: the coarse levels of a cycle in one thread-block cluster (k_cluster).  Cycles whose every
level, or whose coarser levels, fit a cluster leave the oracle's bits in u, u_prev, f, the
Neumann faces and (with a solve) r and the residual history.  Shapes: slabs of two and more
planes, a short last slab, several passes of columns, one to five levels in the cluster, odd and
even extents on the coarsest level."""
import numpy as np
import pytest

from _util import assert_face_equal, assert_field_equal, make_engine, make_oracle, push, randomize

pytestmark = pytest.mark.gpu

CASES = [
    # dims, levels, bc (strict), relaxation, restriction
    ((17, 9, 9), 3, (1, 1, 1, 1, 0, 0), "jacobi", "fw"),
    ((33, 17, 17), 3, (1, 0, 1, 1, 0, 1), "jacobi", "inj"),
    ((65, 33, 17), 4, (1, 1, 1, 1, 1, 1), "jacobi", "fw"),
    ((13, 25, 37), 2, (0, 1, 0, 1, 1, 0), "jacobi", "fw"),
    ((33, 33, 33), 5, (0, 0, 0, 0, 0, 0), "gs", "inj"),
    ((33, 17, 33), 3, (1, 1, 1, 1, 1, 1), "gs", "fw"),
    ((65, 65, 65), 5, (0, 0, 1, 0, 0, 0), "gs", "fw"),
    ((129, 33, 65), 4, (1, 1, 0, 1, 0, 0), "jacobi", "fw"),
]


@pytest.mark.parametrize("ns", [1, 2, 3])
@pytest.mark.parametrize("cycle", ["vcycle", "fcycle"])
@pytest.mark.parametrize("ci", range(len(CASES)))
def test_cluster_cycles_match_oracle(mgp_mod, gpu_ready, ci, cycle, ns):
    dims, levels, bc, rlx, rst = CASES[ci]
    cfg = {"dims": dims, "levels": levels, "bc": bc, "restriction": rst, "relaxation": rlx,
           "h": 1.0 / (dims[0] - 1), "strict_bc": True}
    o = make_oracle(cfg)
    randomize(o, 210 + ci)
    e = make_engine(mgp_mod, cfg)
    push(o, e)
    om = o.default_omega()
    for _ in range(2):
        getattr(o, cycle)(0, om, ns)
        getattr(e, cycle)(0, om, ns)
    for l in range(levels):
        for name in ("u", "f") + (("uprev",) if rlx == "jacobi" else ()):
            assert_field_equal(o, e, name, l)
        for fc in range(6):
            if l == 0 or bc[fc] == 1:
                assert_face_equal(o, e, fc, l)
    # a visit that starts on a coarser level
    if levels > 2:
        o.vcycle(1, om, ns)
        e.vcycle(1, om, ns)
        for l in range(1, levels):
            assert_field_equal(o, e, "u", l)
    e.close()


@pytest.mark.parametrize("ci", range(len(CASES)))
def test_cluster_solve_matches_oracle(mgp_mod, gpu_ready, ci):
    """Solve iterations: where level 0 fits too, the whole iteration with its residual and
    max-norm (the stored r outside the relaxation bounds counts) is one launch."""
    dims, levels, bc, rlx, rst = CASES[ci]
    cfg = {"dims": dims, "levels": levels, "bc": bc, "restriction": rst, "relaxation": rlx,
           "h": 1.0 / (dims[0] - 1), "strict_bc": True}
    o = make_oracle(cfg)
    randomize(o, 240 + ci, lo=-3.0, hi=3.0)
    e = make_engine(mgp_mod, cfg, maxiter=3, tol=0.0)
    push(o, e)
    for cycle in ("Vcycle", "Fcycle"):
        st = e.solve(cycle, 2, -1.0)
        rr, it, _, _ = o.solve(cycle, 2, -1.0, 3, 1, 0.0)
        assert (st.rel_res, st.iterations) == (rr, it)
    for name in ("u", "r"):
        assert_field_equal(o, e, name, 0)
    assert np.isfinite(st.rel_res)
    e.close()
