"""The solves a program has this framework do, as cases that can be timed and compared.

A case is a solve (or a batch of solves) through the public binding: the hierarchy, the
right-hand side and the boundary data are on the GPU beforehand, and one pass resets the
iterate, runs a fixed number of cycles (tolerance 0, so that every pass does the same work) and
hands back u and r.  One kind keeps its data in host arrays and takes them through
PoissonSolver.to_device / solve / to_host, as a program written for the reference does.

Sizes are the repository's own (bench.py, tests, golden fixtures) or ragged ones of the same
form: a * 2^(levels-1) + 1 points per axis.
"""
from __future__ import annotations

import math
import sys
from pathlib import Path

import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "multigrid-poisson_b200"))
import mgp  # noqa: E402

DEV = "cuda"
KIND_LETTERS = {"D": 0, "N": 1}  # case["bc"]: kinds of north, south, east, west, top, bottom


def listed():
    def solve(name, dims, levels, **kw):
        c = {"name": name, "kind": "solve", "nx": dims[0], "ny": dims[1], "nz": dims[2], "levels": levels,
             "dtype": "f64", "relaxation": "jacobi", "restriction": "fw", "cycle": "Fcycle", "nsmooth": 2, "cycles": 4,
             "bc": "NNNNDD", "strict": False, "refine": ""}
        c.update(kw)
        return c

    return [
        # the smallest solve: the smoke check's hierarchy, all launches and read-backs
        solve("fcycle 33x17x17", (33, 17, 17), 3, bc="NNNNND"),
        # the reference's small cube (bench C1): Injection + red-black SOR, all Dirichlet
        solve("fcycle 65^3 sor", (65, 65, 65), 5, relaxation="gs", restriction="inj", bc="DDDDDD", cycles=10),
        # the default plug-ins and smoothing count of PoissonSolver.solve
        solve("vcycle 129^3 sor ns10", (129, 129, 129), 6, relaxation="gs", restriction="inj", cycle="Vcycle",
              nsmooth=10),
        # a ragged box, every requested kind honoured, h^2 not a power of two, odd smoothing
        solve("fcycle 161x97x193 ragged", (161, 97, 193), 5, nsmooth=3, bc="NDNDND", strict=True),
        # the headline F-cycle (bench metric) and the V-cycle on the same grid (bench C2)
        solve("fcycle 513x257x129", (513, 257, 129), 6, bc="NNNNND"),
        solve("vcycle 513x257x129", (513, 257, 129), 6, cycle="Vcycle"),
        # single precision throughout
        solve("fcycle 257^3 f32", (257, 257, 257), 7, dtype="f32", bc="DDNNDD"),
        # FullWeighting with red-black SOR, the combination of the batch and refinement workloads
        solve("fcycle 257x257x129 sor fw", (257, 257, 129), 6, relaxation="gs", bc="DDDDDD"),
        # mixed precision: FP32 corrections of an FP64 problem (bench C2 / C3)
        solve("refine f32 513x257x129", (513, 257, 129), 6, cycle="Vcycle", refine="f32"),
        solve("refine f32 1025x1025x513", (1025, 1025, 513), 8, relaxation="gs", bc="DDDDDD", refine="f32", cycles=2),
        # an ensemble: cubes of mixed sizes solved together (the batch engine; bench's 256-problem mix)
        {"name": "batch 24 cubes f32", "kind": "batch", "count": 24, "kmin": 5, "kmax": 7, "dtype": "f32", "steps": 6,
         "nsmooth": 2},
        # a program with host arrays: upload, solve, download
        solve("host 257x129x65", (257, 129, 65), 5, kind="host", cycles=3),
    ]


def draw(rng):
    """One more case: kind, operators, precision and boundary kinds at random, sizes spread over
    their logarithm from a few thousand points to the size of the headline grid."""
    kind = rng.choices(["solve", "refine", "batch", "host"], [12, 3, 2, 2])[0]
    if kind == "batch":
        return {"kind": "batch", "count": rng.randint(4, 30), "kmin": rng.randint(4, 5), "kmax": rng.randint(6, 7),
                "dtype": rng.choice(["f32", "f64"]), "steps": rng.randint(4, 6), "nsmooth": rng.randint(1, 3)}
    top = 1.7e7 if kind != "host" else 3e6
    target = math.exp(rng.uniform(math.log(4e3), math.log(top)))
    relaxation = rng.choice(["jacobi", "gs"])
    while True:
        levels = rng.randint(3, 7)
        # red-black colouring wants an odd extent on the coarsest level too
        unit = 1 << (levels - 1 if relaxation == "jacobi" else levels)
        side = target ** (1.0 / 3.0)
        least = 2 if relaxation == "jacobi" else 1
        n = [max(least, round(side * math.exp(rng.uniform(-0.7, 0.7)) / unit)) * unit + 1 for _ in range(3)]
        pts = n[0] * n[1] * n[2]
        if 0.5 * target < pts < 1.6 * target and pts < 1.6 * top:
            break
    strict = rng.random() < 0.5
    while True:
        bc = [rng.choice("DN") for _ in range(6)]
        if relaxation == "gs":  # red-black layouts: paired y and z kinds (the others are column-ordered or refused)
            bc[1], bc[5] = bc[0], bc[4]
        if "D" in bc:
            break
    return {"kind": "host" if kind == "host" else "solve", "nx": n[0], "ny": n[1], "nz": n[2], "levels": levels,
            "dtype": "f64" if kind == "refine" else rng.choice(["f64", "f64", "f32"]), "relaxation": relaxation,
            "restriction": rng.choice(["fw", "inj"]), "cycle": rng.choice(["Vcycle", "Fcycle"]),
            "nsmooth": rng.choice([1, 2, 2, 3, 4]), "cycles": rng.randint(2, 5), "bc": "".join(bc), "strict": strict,
            "refine": rng.choice(["f32", "f64"]) if kind == "refine" else ""}


# ---- inputs ---------------------------------------------------------------------------------
def _kinds(case):
    return [KIND_LETTERS[c] for c in case["bc"]]


def _h(case):
    return 1.0 / (max(case["nx"], case["ny"], case["nz"]) - 1)


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _smooth(shape, g, noise=0.05):
    """A few random sine modes plus a little noise, as an FP64 tensor."""
    out = torch.empty(shape, dtype=torch.float64, device=DEV)
    out.uniform_(-noise, noise, generator=g)
    for _ in range(3):
        p = torch.rand(7, dtype=torch.float64, device=DEV, generator=g).tolist()
        ax = [torch.sin(math.pi * (1 + int(3 * p[2 * a])) * torch.linspace(0, 1, n, dtype=torch.float64, device=DEV)
                        + p[2 * a + 1]) for a, n in enumerate(shape)]
        yz = (0.2 + p[6]) * ax[1][:, None] * ax[2][None, :]
        for i0 in range(0, shape[0], 64):  # in slabs: the product of a large grid is not formed at once
            out[i0:i0 + 64] += ax[0][i0:i0 + 64, None, None] * yz
    return out


def _face_shapes(shape):
    nx, ny, nz = shape
    return [(nx, 1, nz), (nx, 1, nz), (1, ny, nz), (1, ny, nz), (nx, ny, 1), (nx, ny, 1)]


def _data(case, seed):
    """Right-hand side and the six face arrays of a solve, FP64."""
    g = _gen(seed)
    shape = (case["nx"], case["ny"], case["nz"])
    f = _smooth(shape, g, 0.5)
    return f, [_smooth(fs, g) for fs in _face_shapes(shape)]


def _batch_problems(case, seed):
    g = _gen(seed)
    out = []
    for i in range(case["count"]):
        k = case["kmin"] + (i * 2654435761 >> 7) % (case["kmax"] - case["kmin"] + 1)
        n = 2 ** k + 1
        f = torch.empty((n, n, n), dtype=torch.float64, device=DEV)
        f.uniform_(-1.0, 1.0, generator=g)
        out.append((n, k - 1, f))
    return out


def _dt(name):
    return (mgp.F64, torch.float64) if name == "f64" else (mgp.F32, torch.float32)


class _Fields:
    """Device fields as tensors, wrapped once per buffer."""

    def __init__(self, solver):
        self.solver, self.seen = solver, {}

    def __call__(self, name):
        v = self.solver.device_field(name)
        t = self.seen.get(v.ptr)
        if t is None:
            t = self.seen[v.ptr] = torch.as_tensor(v, device=DEV)
        return t


def prepare(case, seed):
    if case["kind"] == "batch":
        dt, _ = _dt(case["dtype"])
        b = mgp.Batch(mgp.FULLWEIGHTING, mgp.GAUSSSEIDEL, dt, "Fcycle", case["nsmooth"], max_problems=case["count"])
        probs = []
        for n, levels, f in _batch_problems(case, seed):
            pid = b.add((n, n, n), levels, 1.0 / (n - 1))
            s = b.problem(pid)
            s.batch = b  # the problem's memory is the batch's: a tensor of it keeps the batch alive
            s.synchronize()
            fields = _Fields(s)
            fields("f").copy_(f)
            probs.append((pid, s, fields))
        torch.cuda.synchronize()
        return {"case": case, "batch": b, "probs": probs}
    shape, kinds = (case["nx"], case["ny"], case["nz"]), _kinds(case)
    dt, tdt = _dt(case["dtype"])
    f, faces = _data(case, seed)
    if case["kind"] == "host":
        st = mgp.Settings(levels=case["levels"], dims=list(shape), maxiter=case["cycles"], miniter=case["cycles"],
                          tolerance=0.0, h=_h(case), origin=[0.0, 0.0, 0.0])
        ps = mgp.PoissonSolver(st, mgp.BoundaryCondition(*kinds), restriction=case["restriction"],
                               relaxation=case["relaxation"], dtype=dt, strict_bc=case["strict"], pinned=True)
        ps.init_zero()
        ps.get_rhs().view[...] = f.to(tdt).cpu().numpy()
        for fc in range(6):
            ps.get_bc(fc).arr[...] = faces[fc].to(tdt).cpu().numpy()
        return {"case": case, "ps": ps}
    flags = {"": 0, "f32": mgp.FLAG_REFINE_F32, "f64": mgp.FLAG_REFINE_F64}[case["refine"]]
    s = mgp.Solver(shape, case["levels"], _h(case), kinds, case["restriction"], case["relaxation"], dt, case["cycles"],
                   case["cycles"], 0.0, strict_bc=case["strict"], flags=flags)
    fields = _Fields(s)
    fields("f").copy_(f)
    for fc in range(6):
        torch.as_tensor(s.device_face(fc), device=DEV).copy_(faces[fc])
    torch.cuda.synchronize()
    return {"case": case, "solver": s, "fields": fields}


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        b = state["batch"]
        for pid, s, _ in state["probs"]:
            s.zero_u(0)
            b.restart(pid)
        b.solve(0.0, case["steps"])
        return [t for _, _, fields in state["probs"] for t in (fields("u"), fields("r"))]
    if case["kind"] == "host":
        ps = state["ps"]
        ps.get_solution().arr[...] = 0  # the initial guess
        ps.to_device()
        ps.solve(case["cycle"], case["nsmooth"])
        ps.to_host()
        return {"u": ps.get_solution().view, "r": ps.get_residual().view, "rel_res": ps.relative_residual()}
    s, fields = state["solver"], state["fields"]
    s.zero_u(0)
    s.write_bc(0)
    st = s.solve(case["cycle"], case["nsmooth"])
    return {"u": fields("u"), "r": fields("r"), "rel_res": st.rel_res}


# ---- the work a pass cannot do without ---------------------------------------------------------
def _cycle_work(shape, levels, cycle, ns, es):
    """Bytes and operations of one cycle and the residual after it: each visit of a level reads u
    and f once and writes u once for all its sweeps, each set-up writes the coarse f and u, each
    prolongation reads the coarse u; the last residual is written."""
    n = [math.prod((d - 1 >> l) + 1 for d in shape) for l in range(levels)]
    tot = [0.0, 0.0]

    def visit(l, sweeps):
        tot[0] += 3 * es * n[l]
        tot[1] += 11.0 * n[l] * sweeps

    def down(l):
        tot[0] += 2 * es * n[l + 1]
        tot[1] += 9.0 * n[l] + 40.0 * n[l + 1]

    def up(l):
        tot[0] += es * n[l + 1]
        tot[1] += 4.0 * n[l]

    def v(l):
        visit(l, ns)
        if l < levels - 1:
            down(l)
            v(l + 1)
            up(l)
            visit(l, ns)

    def f(l):
        visit(l, ns)
        down(l)
        if l < levels - 2:
            f(l + 1)
        v(l + 1)
        up(l)
        if l == 0:
            v(0)

    (f if cycle == "Fcycle" else v)(0)
    tot[0] += es * n[0]
    tot[1] += 9.0 * n[0]
    return tot


def work(case):
    if case["kind"] == "batch":
        b = fl = 0.0
        es = 8 if case["dtype"] == "f64" else 4
        for i in range(case["count"]):
            k = case["kmin"] + (i * 2654435761 >> 7) % (case["kmax"] - case["kmin"] + 1)
            n = 2 ** k + 1
            w = _cycle_work((n, n, n), k - 1, "Fcycle", case["nsmooth"], es)
            b += case["steps"] * (w[0] + 24.0 * n ** 3)
            fl += case["steps"] * w[1]
        return {"bytes": b, "flops": fl}
    shape = (case["nx"], case["ny"], case["nz"])
    pts = math.prod(shape)
    es = 8 if case["dtype"] == "f64" else 4
    if case["refine"]:
        w = _cycle_work(shape, case["levels"], case["cycle"], case["nsmooth"], 4 if case["refine"] == "f32" else 8)
        # the correction cycle, then u += e and the FP64 residual: u and f read, u written
        return {"bytes": case["cycles"] * (w[0] + 24.0 * pts), "flops": case["cycles"] * (w[1] + 10.0 * pts)}
    w = _cycle_work(shape, case["levels"], case["cycle"], case["nsmooth"], es)
    extra = 7.0 * es * pts if case["kind"] == "host" else 0.0  # u, u_prev, f, r up; r, u, u_prev down
    return {"bytes": case["cycles"] * w[0] + extra, "flops": case["cycles"] * w[1]}


# ---- the same solves in plain torch, FP64 -----------------------------------------------------
class _Plain:
    """The multigrid cycles of a solve written with torch operations on whole arrays."""

    def __init__(self, shape, levels, h, requested, strict, restriction, relaxation):
        self.levels, self.fw, self.jacobi = levels, restriction == "fw", relaxation == "jacobi"
        kind = list(requested)
        if not strict:  # north, south and bottom are resolved to Dirichlet
            kind[0] = kind[1] = kind[5] = 0
        self.kind = kind
        self.shape = [tuple((d - 1 >> l) + 1 for d in shape) for l in range(levels)]
        self.h = [h * (1 << l) for l in range(levels)]
        self.poff = (requested[3] + requested[1] + requested[5]) & 1
        self.alternate = True
        self.omega = 6.0 / 7.0 if self.jacobi else 8.0 / 9.0
        self.u = [None] * levels
        self.f = [None] * levels
        self.g = [None] * levels
        self.mask = {}

    def box(self, l):
        n, k = self.shape[l], self.kind
        lo = (int(k[3] == 0), int(k[1] == 0), int(k[5] == 0))
        hi = (n[0] - int(k[2] == 0), n[1] - int(k[0] == 0), n[2] - int(k[4] == 0))
        return tuple(slice(a, b) for a, b in zip(lo, hi))

    def neighbours(self, l):
        """The sum of the six neighbours at the relaxed points, Neumann ghosts formed."""
        u, b, h2, g = self.u[l], self.box(l), 2.0 * self.h[l], self.g[l]
        s = None
        faces = ((3, 2), (1, 0), (5, 4))
        for ax in range(3):
            n = u.shape[ax]
            for side, sign in ((0, -1.0), (1, 1.0)):
                fc = faces[ax][side]
                lo, hi = b[ax].start, b[ax].stop
                if side == 0:
                    t = u.narrow(ax, max(lo - 1, 0), hi - 1 - max(lo - 1, 0))
                    if lo == 0:
                        t = torch.cat([sign * h2 * g[fc] + u.narrow(ax, 1, 1), t], dim=ax)
                else:
                    t = u.narrow(ax, lo + 1, min(hi + 1, n) - lo - 1)
                    if hi == n:
                        t = torch.cat([t, sign * h2 * g[fc] + u.narrow(ax, n - 2, 1)], dim=ax)
                t = t[tuple(slice(None) if a == ax else b[a] for a in range(3))]
                s = t.clone() if s is None else s.add_(t)
        return s

    def parity(self, l, colour):
        key = (l, colour)
        if key not in self.mask:
            b = self.box(l)
            i, j, k = (torch.arange(q.start, q.stop, device=DEV) for q in b)
            self.mask[key] = ((i[:, None, None] + j[None, :, None] + k[None, None, :] + self.poff) & 1) == colour
        return self.mask[key]

    def relax(self, l, ns):
        b, h, w = self.box(l), self.h[l], self.omega
        for _ in range(ns if self.jacobi else 2 * ns):
            new = self.neighbours(l).sub_(h * h * self.f[l][b]).mul_(w / 6.0).add_((1.0 - w) * self.u[l][b])
            if self.jacobi:
                u = self.u[l].clone()
                u[b] = new
                self.u[l] = u
            else:
                m = self.parity(l, 0 if self.alternate else 1)
                self.u[l][b] = torch.where(m, new, self.u[l][b])
                self.alternate = not self.alternate

    def residual(self, l):
        b, h = self.box(l), self.h[l]
        r = torch.zeros(self.shape[l], dtype=torch.float64, device=DEV)
        r[b] = self.f[l][b] - (self.neighbours(l) - 6.0 * self.u[l][b]) / (h * h)
        return r

    def restrict(self, a):
        if not self.fw:
            return a[tuple(slice(0, None, 2) for _ in range(3))].clone()
        for ax in range(3):
            n = a.shape[ax]
            if n == 1:
                a = 4.0 * a
                continue
            idx = torch.arange(0, n, 2, device=DEV)
            a = a.index_select(ax, (idx - 1).clamp(min=0)) + 2.0 * a.index_select(ax, idx) + \
                a.index_select(ax, (idx + 1).clamp(max=n - 1))
        return a / 64.0

    def setup(self, l):
        self.f[l + 1] = self.restrict(self.residual(l))
        self.u[l + 1] = torch.zeros(self.shape[l + 1], dtype=torch.float64, device=DEV)
        u, g = self.u[l], []
        for fc in range(6):
            gc = self.restrict(self.g[l][fc])
            if self.kind[fc] == 0:
                gc.zero_()
            else:
                ax = {0: 1, 1: 1, 2: 0, 3: 0, 4: 2, 5: 2}[fc]
                upper = fc in (0, 2, 4)
                at = [u.shape[ax] - 1 - q if upper else q for q in range(3)]
                even = tuple(slice(None) if a == ax else slice(0, None, 2) for a in range(3))
                v = [u.narrow(ax, p, 1)[even] for p in at]
                c = (1.5, -2.0, 0.5) if upper else (-1.5, 2.0, -0.5)
                gc -= (c[0] * v[0] + c[1] * v[1] + c[2] * v[2]) / self.h[l]
            g.append(gc)
        self.g[l + 1] = g

    def prolong_add(self, l):
        a = self.u[l + 1]
        for ax in range(3):
            n = 2 * a.shape[ax] - 1
            o = torch.empty([n if q == ax else a.shape[q] for q in range(3)], dtype=torch.float64, device=DEV)
            even = tuple(slice(0, None, 2) if q == ax else slice(None) for q in range(3))
            odd = tuple(slice(1, None, 2) if q == ax else slice(None) for q in range(3))
            o[even] = a
            o[odd] = 0.5 * (a.narrow(ax, 0, a.shape[ax] - 1) + a.narrow(ax, 1, a.shape[ax] - 1))
            a = o
        self.u[l] = self.u[l] + a

    def v(self, l, ns):
        self.relax(l, ns)
        if l < self.levels - 1:
            self.setup(l)
            self.v(l + 1, ns)
            self.prolong_add(l)
            self.relax(l, ns)

    def fc(self, l, ns):
        self.relax(l, ns)
        self.setup(l)
        if l < self.levels - 2:
            self.fc(l + 1, ns)
        self.v(l + 1, ns)
        self.prolong_add(l)
        if l == 0:
            self.v(0, ns)

    def cycle(self, name, ns):
        (self.fc if name == "Fcycle" else self.v)(0, ns)

    def write_bc(self):
        """Dirichlet face data into u: north, south, east, west, top, bottom, later faces win."""
        u = self.u[0]
        for fc, at in enumerate(((1, -1), (1, 0), (0, -1), (0, 0), (2, -1), (2, 0))):
            if self.kind[fc] == 0:
                u.narrow(at[0], u.shape[at[0]] - 1 if at[1] else 0, 1).copy_(self.g[0][fc])


def _refined(p, f, faces, cycle, ns, steps):
    """Iterative refinement: corrections with zero boundary data, u += e, the residual."""
    zero = torch.zeros_like(f)
    e = _Plain(p.shape[0], p.levels, p.h[0], [0] * 6, True, "fw" if p.fw else "inj", "jacobi" if p.jacobi else "gs")
    e.kind, e.poff = p.kind, p.poff
    p.f[0], p.g[0] = f, faces
    p.u[0] = zero
    p.write_bc()
    p.u[0] = p.u[0].clone()
    e.g[0] = [torch.zeros_like(g) for g in faces]
    r = p.residual(0)
    for _ in range(steps):
        e.f[0], e.u[0] = r, torch.zeros_like(f)
        e.cycle(cycle, ns)
        b = p.box(0)
        p.u[0][b] += e.u[0][b]
        r = p.residual(0)
    return p.u[0], r


def exact(case, seed):
    if case["kind"] == "batch":
        out = []
        for n, levels, f in _batch_problems(case, seed):
            p = _Plain((n, n, n), levels, 1.0 / (n - 1), [0] * 6, False, "fw", "gs")
            faces = [torch.zeros(fs, dtype=torch.float64, device=DEV) for fs in _face_shapes((n, n, n))]
            out += list(_refined(p, f, faces, "Fcycle", case["nsmooth"], case["steps"]))
        return out
    shape = (case["nx"], case["ny"], case["nz"])
    if math.prod(shape) > 1e8:
        return None  # minutes of whole-array passes
    f, faces = _data(case, seed)
    if case["dtype"] == "f32":  # the inputs the solver gets
        f, faces = f.float().double(), [g.float().double() for g in faces]
    p = _Plain(shape, case["levels"], _h(case), _kinds(case), case["strict"], case["restriction"], case["relaxation"])
    if case["refine"]:
        u, r = _refined(p, f, faces, case["cycle"], case["nsmooth"], case["cycles"])
        return {"u": u, "r": r, "rel_res": float(r.abs().max() / f.abs().max())}
    p.f[0], p.g[0] = f, faces
    p.u[0] = torch.zeros_like(f)
    p.write_bc()
    for _ in range(case["cycles"]):
        p.cycle(case["cycle"], case["nsmooth"])
    r = p.residual(0)
    out = {"u": p.u[0], "r": r, "rel_res": float(r.abs().max() / f.abs().max())}
    if case["kind"] == "host":
        out["u"], out["r"] = out["u"].cpu().numpy(), out["r"].cpu().numpy()
    return out
