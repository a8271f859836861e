"""GPU: failure detection of the coarse levels in a cluster.  With a bound of one poll the waits for
a neighbour's planes run out: the solve returns an error status that names the cluster, the
context stays usable, and the same solver then solves with the default bound, bit-identical to the
oracle."""
import numpy as np
import pytest

from _util import assert_field_equal, make_engine, make_oracle, push, randomize

pytestmark = pytest.mark.gpu

CASES = [
    # dims, levels, bc (strict), relaxation, restriction: the whole hierarchy in the cluster, or its coarser levels
    ((33, 17, 17), 3, (1, 0, 1, 1, 0, 1), "jacobi", "fw"),
    ((33, 17, 33), 3, (1, 1, 1, 1, 1, 1), "gs", "inj"),
    ((65, 65, 33), 4, (0, 0, 1, 0, 0, 0), "gs", "fw"),
    ((65, 33, 65), 4, (1, 1, 0, 1, 0, 0), "jacobi", "inj"),
]


@pytest.mark.parametrize("cycle", ["Vcycle", "Fcycle"])
@pytest.mark.parametrize("ci", range(len(CASES)))
def test_wait_that_runs_out(mgp_mod, gpu_ready, ci, cycle):
    dims, levels, bc, rlx, rst = CASES[ci]
    cfg = {"dims": dims, "levels": levels, "bc": bc, "restriction": rst, "relaxation": rlx,
           "h": 1.0 / (dims[0] - 1), "strict_bc": True}
    o = make_oracle(cfg)
    randomize(o, 270 + ci)
    e = make_engine(mgp_mod, cfg, maxiter=2, tol=0.0)
    for _ in range(2):
        e.set_wait_polls(1)
        push(o, e)
        with pytest.raises(mgp_mod.MgpError) as ei:
            e.solve(cycle, 3, -1.0)
        assert ei.value.status == mgp_mod.ERR_TIMEOUT and "cluster" in str(ei.value)
        e.set_wait_polls(0)
    push(o, e)
    st = e.solve(cycle, 3, -1.0)
    rr, it, _, _ = o.solve(cycle, 3, -1.0, 2, 1, 0.0)
    assert (st.rel_res, st.iterations) == (rr, it)
    for name in ("u", "r"):
        assert_field_equal(o, e, name, 0)
    e.close()


@pytest.mark.parametrize("bc", [(0, 0, 0, 0, 0, 0), (1, 1, 1, 0, 0, 0)])
def test_refinement_reports_it(mgp_mod, gpu_ready, bc):
    """Afterwards the solver gives the bits of one that never failed."""
    m = mgp_mod
    e, fresh = [m.Solver((33, 17, 17), 3, 1 / 32, bc, m.FULLWEIGHTING, m.JACOBI, m.F64, 4, 1, 0.0, strict_bc=True,
                         flags=m.FLAG_REFINE_F32) for _ in range(2)]
    f = np.random.default_rng(5).uniform(-1, 1, size=e.level[0].pad)
    for s in (e, fresh):
        s.upload("f", f)
    e.set_wait_polls(1)
    with pytest.raises(m.MgpError) as ei:
        e.solve("Vcycle", 2)
    assert ei.value.status == m.ERR_TIMEOUT and "cluster" in str(ei.value)
    e.set_wait_polls(0)
    e.zero_u(0)
    assert e.solve("Vcycle", 2).rel_res == fresh.solve("Vcycle", 2).rel_res
    for name in ("u", "r"):
        assert np.array_equal(e.download(name), fresh.download(name)), name
    e.close()
    fresh.close()
