"""GPU: batches whose step leaves the inner hierarchies in another buffer state than it found them
in (Jacobi F-cycles with an odd number of sweeps swap the finest level's buffers 3*ns times a
step).  Every step must use the buffers of its own state: the same bits as the same problems
solved one at a time, over enough steps that launched and captured ones take part, also when the
set of problems changes in between."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PROBLEMS = [
    # dims, levels, bc (strict)
    ((17, 17, 17), 3, (0, 0, 0, 0, 0, 0)),
    ((33, 17, 17), 3, (0, 0, 1, 1, 0, 0)),
    ((33, 33, 33), 4, (1, 1, 0, 1, 0, 1)),
    ((17, 9, 33), 2, (0, 0, 0, 0, 1, 1)),
]


def load(s, seed):
    rng = np.random.default_rng(seed)
    s.upload("f", rng.uniform(-1, 1, size=s.level[0].pad), 0)
    for fc in range(6):
        s.upload_face(fc, rng.uniform(-1, 1, size=s.level[0].face_shape[fc]), 0)
    s.write_bc(0)


def single(m, case, seed, rx, inner, cycle, ns, steps):
    dims, levels, bc = case
    e = m.Solver(dims, levels, 1.0 / (dims[0] - 1), bc, m.FULLWEIGHTING, rx, m.F64, steps, 1, 0.0, strict_bc=True,
                 flags=m.FLAG_REFINE_F32 if inner == "F32" else m.FLAG_REFINE_F64)
    load(e, seed)
    e.solve(cycle, ns)
    return e


@pytest.mark.parametrize("ns", [1, 2, 3])
@pytest.mark.parametrize("cycle", ["Fcycle", "Vcycle"])
@pytest.mark.parametrize("inner", ["F32", "F64"])
@pytest.mark.parametrize("rlx", ["JACOBI", "GAUSSSEIDEL"])
def test_steps_match_single_solves(mgp_mod, gpu_ready, rlx, inner, cycle, ns):
    m = mgp_mod
    rx = getattr(m, rlx)
    # red-black layouts want paired y and z kinds
    probs = [p for p in PROBLEMS if rlx == "JACOBI" or (p[2][0] == p[2][1] and p[2][4] == p[2][5])]
    for steps in (1, 2, 7):
        b = m.Batch(m.FULLWEIGHTING, rx, getattr(m, inner), cycle, ns)
        ids = []
        for i, (dims, levels, bc) in enumerate(probs):
            ids.append(b.add(dims, levels, 1.0 / (dims[0] - 1), bc, strict_bc=True))
            load(b.problem(ids[-1]), i)
        assert b.solve(0.0, steps) == steps
        for i, (case, pid) in enumerate(zip(probs, ids)):
            e = single(m, case, i, rx, inner, cycle, ns, steps)
            for name in ("u", "r"):
                assert np.array_equal(e.download(name), b.problem(pid).download(name)), (steps, case, name)
            e.close()
        b.close()


@pytest.mark.parametrize("ns", [1, 2])
def test_set_changes_between_steps(mgp_mod, gpu_ready, ns):
    """A problem that joins, pauses or leaves does not disturb the others' steps."""
    m = mgp_mod
    b = m.Batch(m.FULLWEIGHTING, m.JACOBI, m.F32, "Fcycle", ns, max_problems=3)

    def add(i):
        dims, levels, bc = PROBLEMS[i]
        pid = b.add(dims, levels, 1.0 / (dims[0] - 1), bc, strict_bc=True)
        load(b.problem(pid), i)
        return pid

    def check(i, pid, steps):
        e = single(m, PROBLEMS[i], i, m.JACOBI, "F32", "Fcycle", ns, steps)
        assert b.status(pid).iterations == steps
        assert np.array_equal(e.download("u"), b.problem(pid).download("u")), (i, steps)
        e.close()

    p0, p1 = add(0), add(1)
    for _ in range(3):
        b.step()
    p2 = add(2)
    for _ in range(6):
        b.step()
    b.set_active(p1, False)
    for _ in range(5):
        b.step()
    b.set_active(p1, True)
    for _ in range(6):
        b.step()
    b.remove(p0)
    b.step()
    check(1, p1, 16)
    check(2, p2, 18)
    b.close()
