"""Measured workloads of the insem B200 backend, through its public Python faces.

The shapes are the ones the package's own workloads have (``cases.config1`` ..
``cases.config4``, ``serving.request_stream``): Cartesian media of order 3 to
8 with 1k to 200k elements, the coupled ocean-bottom model, cased and open
boreholes of azimuthal order 0 and 1, batches of them, the set-up that every
request pays, and the two kernel seams.

A pass steps an existing solve on by a fixed number of steps (a solve is made
with far more steps than any number of passes takes) and reads what a program
reads then: the field, the streamed sample rows, the energy.  The initial
wavefield, the source signature and, for the set-up, the materials come from
the seed; the mesh is the case's own.
"""

from __future__ import annotations

import ctypes as C
import dataclasses
import functools
import importlib.util
import json
import math
import sys
from pathlib import Path

import numpy as np
import torch

_ROOT = Path(__file__).resolve().parent.parent


def _package():
    if "insem_b200" not in sys.modules:
        pkg = _ROOT / "in-house-sem_b200"
        spec = importlib.util.spec_from_file_location("insem_b200", pkg / "__init__.py",
                                                      submodule_search_locations=[str(pkg)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["insem_b200"] = mod
        spec.loader.exec_module(mod)
    import insem_b200.cases  # noqa: F401
    import insem_b200.kernels  # noqa: F401
    import insem_b200.serving  # noqa: F401
    return sys.modules["insem_b200"]


# --------------------------------------------------------------------- cases
def listed():
    return [
        # the smallest call: an interactive program steps the 32 x 32 acoustic
        # square on by a few steps and looks at the field
        dict(name="square_watch", use="advance", model="square", steps=4, energy=0),
        # the same model over the 287 steps of its 4 ms: launch latency
        dict(name="square_run", use="advance", model="square", steps=287, energy=0),
        # Cartesian elastic solve of high order with the energy monitor on
        dict(name="elastic_order8_energy", use="advance", model="elastic", order=8, nx=61, nz=67, steps=200, energy=10),
        # cased borehole, monopole, order 4, hanging nodes (one logging shot)
        dict(name="borehole_cased_m0", use="advance", model="cased", steps=500, energy=0),
        # dipole borehole of order 6 as one solve: streamed samples, the mud's pressure
        dict(name="borehole_m1", use="stream", model="borehole", index=3, steps=100),
        # coupled water / curved elastic layers with 512 seafloor receivers,
        # the largest single solve: a step moves more than L2 holds
        dict(name="ocean_bottom", use="stream", model="coupled", nx=384, receivers=512, steps=200),
        # the batched boreholes of the benchmark: m = 0 / 1, order 4 - 6
        dict(name="borehole_batch", use="batch", members="boreholes", first=0, count=12, steps=25),
        # a server's batch: Cartesian media of orders 3 - 8 beside boreholes, many small tile classes
        dict(name="serving_batch", use="batch", members="requests", first=0, count=10, steps=50),
        # the set-up of one request: upload, stable time step, tiling
        dict(name="setup_borehole", use="setup", model="borehole", index=0),
        dict(name="setup_elastic", use="setup", model="elastic", order=4, nx=96, nz=96),
        # the per-block and DofMap seams: gather, element forces, assembly on device arrays
        dict(name="seam_curved", use="seam", model="coupled", nx=128, receivers=16),
        # internal forces on the caller's own arrays, axisymmetric with hanging nodes
        dict(name="forces_cased", use="forces", model="cased"),
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    use = rng.choice(["advance", "advance", "stream", "stream", "batch", "setup", "seam", "forces"])
    if use == "batch":
        return dict(use=use, members=rng.choice(["boreholes", "requests"]), first=rng.randrange(0, 24),
                    count=rng.randrange(2, 9), steps=_spread(rng, 5, 40))
    kinds = ["acoustic", "elastic", "elastic", "coupled", "borehole", "borehole"]
    model = rng.choice(kinds)
    if model in ("acoustic", "elastic"):
        order = rng.randrange(3, 9)
        n = _spread(rng, 1500, 60000 * 16 // (order * order) // 4)
        nx = _spread(rng, 24, max(32, int(math.sqrt(n) * 1.5)))
        case = dict(model=model, order=order, nx=nx, nz=max(9, n // nx))
    elif model == "coupled":
        case = dict(model=model, nx=_spread(rng, 33, 257), receivers=_spread(rng, 4, 256))
    else:
        case = dict(model=model, index=rng.choice([0, 1, 4, 5, 7, 8, 12, 14, 15, 16, 17, 20, 22]))
    if use == "advance":
        case.update(steps=_spread(rng, 1, 300), energy=rng.choice([0, 0, 7]))
    elif use == "stream":
        case.update(steps=_spread(rng, 1, 200))
    return dict(case, use=use)


# -------------------------------------------------------------------- models
def _model(case, n_steps, scale=1.0):
    """The model description of a case; `scale` multiplies the speeds of its elastic and acoustic media."""
    K = _package().cases
    kind = case["model"]
    if kind == "square":
        m = K.config1()
    elif kind == "cased":
        m = K.config2()
    elif kind == "coupled":
        m = K.config3(nx=case["nx"], n_steps=1, n_receivers=case["receivers"])
    elif kind == "borehole":
        p = K.config4_params(256, 4)[case["index"]]
        m = K.config4_model(p, *K.config4_geometry_table(256, 4)[case["index"]])
    else:  # a Cartesian request of the serving mix
        S = _package().serving
        spec = dict(elements=float(case["nx"] * case["nz"]), order=case["order"], duration=1e-3, vs_ratio=0.53,
                    vp=1500.0 if kind == "acoustic" else 3100.0, rho=2100.0)
        m = S.request_model(S.Request(0, 0.0, "cartesian-" + kind, spec))
        h = 0.05
        w, d = case["nx"] * h, case["nz"] * h
        m.mesh = K.rectangle((0.0, w), (-d, 0.0), nx=case["nx"], nz=case["nz"], material=int(kind == "elastic"))
        m.sources[0].x, m.sources[0].z = 0.5 * w, -0.5 * d
        for i, r in enumerate(m.receivers):
            r.x, r.z = (0.2 + 0.15 * i) * w, -0.2 * d
    m.materials = {r: dataclasses.replace(x, vp=x.vp * scale, vs=x.vs * scale) for r, x in m.materials.items()}
    m.duration, m.n_steps, m.energy_every = 0.0, n_steps, int(case.get("energy") or 0)
    return m


def _key(case):
    return json.dumps({k: v for k, v in case.items() if k not in ("name", "use", "steps")}, sort_keys=True)


@functools.lru_cache(maxsize=16)
def _built(key, n_steps):
    """(setup arrays, stable time step) of a case's model: the mesh work that a program does once."""
    pkg = _package()
    model = _model(json.loads(key), n_steps)
    arrays = pkg.cases.setup_arrays(model)
    probe = pkg.cases.build_from_arrays(model, arrays, stable_dt=1.0)
    return model, arrays, float("%.3g" % pkg.solver.estimate_stable_dt(probe))


def _budget(case):
    """Steps of a solve: more than all its passes take (a pass of more steps or points is repeated less often)."""
    return {"advance": 400_000, "stream": 200_000}.get(case["use"], 100_000)


def _problem(case):
    model, arrays, sdt = _built(_key(case), _budget(case))
    return _package().cases.build_from_arrays(model, arrays, stable_dt=sdt), arrays


def _requests():
    S = _package().serving
    out = [r for r in S.request_stream(50.0, 20.0, 5) if r.spec.get("elements", 0) < 40000]
    return [r for r in out if not r.kind.startswith("borehole") or r.spec["c4"] in (0, 1, 5, 7, 8, 12, 14, 15, 16, 17, 20, 22)
            or r.rid % 7 == 0]


@functools.lru_cache(maxsize=64)
def _member_built(members, index):
    pkg = _package()
    if members == "boreholes":
        model = _model(dict(model="borehole", index=index), 50_000)
    else:
        model = pkg.serving.request_model(_requests()[index])
        model.n_steps = 50_000
    arrays = pkg.cases.setup_arrays(model)
    probe = pkg.cases.build_from_arrays(model, arrays, stable_dt=1.0)
    return model, arrays, float("%.3g" % pkg.solver.estimate_stable_dt(probe))


def _member_problems(case):
    for k in range(case["first"], case["first"] + case["count"]):
        model, arrays, sdt = _member_built(case["members"], k)
        yield _package().cases.build_from_arrays(model, arrays, stable_dt=sdt), arrays


def _wavefield(prob, arrays, rng):
    """Smooth initial fields per domain: a few wave packets of random place, width and strength."""
    out = []
    for i, d in enumerate(prob.domains):
        xz = arrays[f"problem.domains.{i}.coords"].reshape(-1, 2)
        size = float(np.min(xz.max(0) - xz.min(0)))
        amp = 1e3 if d.medium == 0 else 1e-6
        u, v = np.zeros((d.ncomp, d.n_global)), np.zeros((d.ncomp, d.n_global))
        for _ in range(4):
            at, width = xz[rng.integers(0, len(xz))], size * rng.uniform(0.05, 0.2)
            q = (xz - at) / width
            bump = np.exp(-(q * q).sum(1))
            u += amp * rng.uniform(-1, 1, (d.ncomp, 1)) * bump
            v += amp * 1e3 * rng.uniform(-1, 1, (d.ncomp, 1)) * bump * q[:, 0]
        out.append((u, v))
    return out


def _signature(prob, steps, rng):
    """A measured source signature: band-limited noise per source, [steps][sources]."""
    t = np.arange(steps)[:, None]
    s = sum(rng.uniform(-1, 1, (1, len(prob.sources))) * np.sin(t * rng.uniform(0.01, 0.2) + rng.uniform(0, 6)) for _ in range(5))
    return np.ascontiguousarray(s, np.float32)


def _scale(seed):
    """Speed factor of the set-up cases' materials."""
    return 1.0 + 0.2 * float(np.random.default_rng(seed).uniform(-1, 1))


# ------------------------------------------------------------------- passes
def _start(prob, arrays, rng):
    s = _package().Solver(prob)
    for d, (u, v) in zip(prob.media, _wavefield(prob, arrays, rng)):
        s.set_state(d, u, v)
    return s


class _Handles:
    """What a program keeps between passes."""

    def __init__(self, case, **kw):
        self.case = case
        self.__dict__.update(kw)


def prepare(case, seed):
    pkg, rng, use = _package(), np.random.default_rng(seed), case["use"]
    if use == "setup":
        model = _model(case, 1000, _scale(seed))
        return _Handles(case, model=model, arrays=pkg.cases.setup_arrays(model))
    if use == "batch":
        batch = pkg.Batch()
        for prob, arrays in _member_problems(case):
            batch.adopt(_start(prob, arrays, rng))
        rows = torch.empty((case["steps"], batch.stream_layout()[1]), dtype=torch.float64, pin_memory=True)
        return _Handles(case, batch=batch, rows=rows)
    prob, arrays = _problem(case)
    if use == "advance":
        return _Handles(case, solver=_start(prob, arrays, rng))
    if use == "stream":
        s = _start(prob, arrays, rng)
        return _Handles(case, solver=s, amp=_signature(prob, case["steps"], rng), rows=np.empty((case["steps"], s.n_columns)))
    fields = _wavefield(prob, arrays, rng)
    u = [torch.from_numpy(f[0].astype(np.float32)).cuda() for f in fields]
    f = [torch.empty_like(x) for x in u]
    if use == "forces":
        return _Handles(case, solver=pkg.Solver(prob), u=u, f=f)
    ops = []
    for d, x in zip(prob.domains, u):
        local = [torch.zeros(d.ncomp * d.l2g.size, dtype=torch.float32, device="cuda") for _ in range(2)]
        ops.append((d.ncomp, d.n_elements, pkg.kernels.DofMapKernel(prob.ngll, d),
                    [pkg.kernels.BlockKernel(prob, b, d.medium) for b in d.blocks], local))
    return _Handles(case, ops=ops, u=u, f=f)


def run(st):
    use = st.case["use"]
    if use == "advance":
        s = st.solver
        s.advance(st.case["steps"])
        out = {m: s.state(m) for m in s.media}
        if st.case["energy"]:
            out["energy"] = s.energy[-1]
        return out
    if use == "stream":
        s = st.solver
        n = s.advance_streamed(st.case["steps"], st.amp, st.rows)
        out = {"rows": st.rows[:n]}
        if "acoustic" in s.media:
            out["acoustic"] = s.state("acoustic")
        return out
    if use == "batch":
        n = st.batch.advance_streamed(st.case["steps"], None, st.rows)
        return {"rows": st.rows[:n]}
    if use == "setup":
        prob, s = _package().cases.build_solver_from_arrays(st.model, st.arrays)
        out = {"stable_dt": s.stable_dt, "dt": s.dt, "n_steps": s.n_steps}
        s.close()
        return out
    stream = torch.cuda.current_stream().cuda_stream
    if use == "forces":
        native = _package().native
        for di, (u, f) in enumerate(zip(st.u, st.f)):
            native.check(native.lib().insem_cuda_solver_internal_forces_noalloc(
                st.solver._h, di, C.c_void_p(u.data_ptr()), C.c_void_p(f.data_ptr()), C.c_void_p(stream)))
        return st.f
    for (ncomp, n_el, dofs, blocks, (ul, fl)), u, f in zip(st.ops, st.u, st.f):
        dofs.gather_device(ncomp, u.data_ptr(), ul.data_ptr(), stream)
        for b in blocks:
            b.forces_device(n_el, ul.data_ptr(), fl.data_ptr(), stream)
        dofs.assemble_device(ncomp, fl.data_ptr(), f.data_ptr(), stream)
    return st.f


# --------------------------------------------------------------------- work
def _step_work(prob):
    """Bytes and operations of one time step.  Bytes: u and v read and written
    and the inverse mass read per point and component; per element the slot
    map, the metric (Rect 12 bytes, Affine 20, Curved 20 and axisymmetric 28
    per point) and one coefficient pair.  Operations: the derivative and
    divergence sums (8 ngll per point and component) and some 20 per point
    and component for stress, fluxes and the update."""
    npe, byts, ops = prob.ngll ** 2, 0, 0
    for d in prob.domains:
        byts += d.n_global * (16 * d.ncomp + 4)
        for b in d.blocks:
            byts += b.n_elements * (4 * npe + 8 + {0: 12, 1: 20, 2: 20 * npe, 3: 28 * npe}[b.kind])
            ops += b.n_elements * npe * d.ncomp * (8 * prob.ngll + 20)
    return byts, ops


def work(case):
    use = case["use"]
    if use == "batch":
        parts = [_step_work(p) for p, _ in _member_problems(case)]
        return {"bytes": case["steps"] * sum(p[0] for p in parts), "flops": case["steps"] * sum(p[1] for p in parts)}
    if use == "setup":
        model = _model(case, 1000)
        prob = _package().cases.build_from_arrays(model, _package().cases.setup_arrays(model), stable_dt=1.0)
        applied = 100 + (120 if len(prob.domains) > 1 else 0)  # applications of the operator in the power iteration
        byts, ops = _step_work(prob)
        return {"bytes": applied * byts, "flops": applied * ops}
    prob, _ = _problem(case)
    byts, ops = _step_work(prob)
    if use in ("advance", "stream"):
        return {"bytes": case["steps"] * byts, "flops": case["steps"] * ops}
    # one application: fields in and out once, the slot maps and the element data
    byts -= sum(d.n_global * (8 * d.ncomp + 4) for d in prob.domains)
    return {"bytes": byts, "flops": ops}


# ------------------------------------------------------------ 64-bit answers
class _Exact:
    """The same step in 64 bits, written with torch from the discrete equations."""

    def __init__(self, prob):
        self.p, self.ng, self.dev = prob, prob.ngll, "cuda" if torch.cuda.is_available() else "cpu"
        self.dt, self.step = float(prob.dt), 0
        self.D, self.Dj, self.w2 = (self._t(x).reshape(self.ng, self.ng) if len(x) else None for x in (prob.D, prob.Dj, prob.w2))
        self.dom = [self._domain(d) for d in prob.domains]
        self.solid = next((i for i, d in enumerate(prob.domains) if d.medium == 1), None)
        self.fluid = next((i for i, d in enumerate(prob.domains) if d.medium == 0), None)
        c = prob.coupling
        self.cpl = [self._t(c[k], torch.long if "points" in k else torch.float64) for k in ("fluid_points", "solid_points", "cx", "cz")]
        self.started = False

    def _t(self, x, dtype=torch.float64):
        return torch.as_tensor(np.asarray(x)).to(self.dev, dtype)

    def _domain(self, d):
        npe, q = self.ng ** 2, {}
        slots = self._t(d.l2g, torch.long)
        q["rows"] = torch.nonzero(slots < 0).flatten()
        q["l2g"] = slots.clamp(min=0)
        if d.n_rows:
            off = np.asarray(d.row_offsets)
            of = (-1 - np.asarray(d.l2g))[np.asarray(d.l2g) < 0]  # row of each constrained slot
            n = off[of + 1] - off[of]
            flat = np.concatenate([np.arange(a, b) for a, b in zip(off[of], off[of + 1])]) if len(of) else np.zeros(0, int)
            q["row_at"] = self._t(np.repeat(np.nonzero(np.asarray(d.l2g) < 0)[0], n), torch.long)
            q["row_dof"], q["row_w"] = self._t(np.asarray(d.row_dofs)[flat], torch.long), self._t(np.asarray(d.row_weights)[flat])
        q["mass"], q["zero"] = self._t(d.mass), torch.zeros((d.ncomp, d.n_global), dtype=torch.bool, device=self.dev)
        q["zero"][:, self._t(d.dirichlet_points, torch.long)] = True
        for c in d.axis_components:
            q["zero"][int(c), self._t(d.axis_points, torch.long)] = True
        q["abs"] = self._t(d.absorbing_points, torch.long)
        q["C"] = self._t(d.absorbing_coef).reshape(-1, d.ncomp, d.ncomp)
        q["blocks"] = []
        for b in d.blocks:
            shape = (b.n_elements, self.ng, self.ng)
            m = self._t(b.metric)
            if b.kind == 0:
                m = m.reshape(-1, 3, 1, 1)
                z = torch.zeros_like(m[:, 0])
                m = (m[:, 0], z, z, m[:, 1], m[:, 2])
            elif b.kind == 1:
                m = m.reshape(-1, 5, 1, 1).unbind(1)
            else:
                m = m.reshape(*shape, 5).unbind(-1)
            q["blocks"].append(dict(e=self._t(b.elements, torch.long), m=m, kind=b.kind, order=b.azimuthal_order,
                                    c0=self._t(b.coef0).reshape(shape), c1=self._t(b.coef1).reshape(shape) if b.coef1.size else None,
                                    wr=self._t(b.wr).reshape(shape) if b.wr.size else None, hoop=self._t(b.hoop).reshape(shape) if b.hoop.size else None,
                                    r=self._t(b.r).reshape(shape) if b.r.size else None, axial=torch.nonzero(self._t(b.axial, torch.long)).flatten()))
        q["u"], q["v"], q["a"] = (torch.zeros((d.ncomp, d.n_global), dtype=torch.float64, device=self.dev) for _ in range(3))
        return q

    def forces(self, di, u):
        d, q, ng = self.p.domains[di], self.dom[di], self.ng
        loc = u[:, q["l2g"]]
        if d.n_rows:
            loc[:, q["rows"]] = 0.0
            loc.index_add_(1, q["row_at"], u[:, q["row_dof"]] * q["row_w"])
        loc = loc.reshape(d.ncomp, -1, ng, ng)
        out = torch.zeros_like(loc)
        for b in q["blocks"]:
            out[:, b["e"]] = self._element(d, b, loc[:, b["e"]])
        out = out.reshape(d.ncomp, -1)
        f = torch.zeros_like(u)
        if d.n_rows:
            f.index_add_(1, q["row_dof"], out[:, q["row_at"]] * q["row_w"])
            out = out.clone()
            out[:, q["rows"]] = 0.0
        return f.index_add_(1, q["l2g"], out)

    def _element(self, d, b, u):
        D, ax = self.D, b["axial"]
        u_xi, u_eta = u @ D.T, D @ u
        if len(ax):
            u_xi[:, ax] = u[:, ax] @ self.Dj.T
        xx, xz, ex, ez, jac = b["m"]
        gx, gz = u_xi * xx + u_eta * ex, u_xi * xz + u_eta * ez
        axisym, lam, mu = b["kind"] == 3, b["c0"], b["c1"]
        w = b["wr"] if axisym else self.w2 * jac
        hoop, spread = {}, {}  # component -> direct term, and its value for the on-axis points
        if axisym:
            r = b["r"]
            on = r == 0.0
            rr = torch.where(on, torch.ones_like(r), r)
            over = lambda c: torch.where(on, gx[c], u[c] / rr)  # noqa: E731
        if d.medium == 0:
            qx, qz = [lam * gx[0]], [lam * gz[0]]
            if axisym and b["order"] == 1:
                hoop[0], spread[0] = lam * u[0] / rr, lam * gx[0]
        elif axisym and b["order"] == 1:
            h, s2 = math.sqrt(0.5), math.sqrt(2.0)
            rx, rz, tx, tz = (gx[0] + gx[1]) * h, (gz[0] + gz[1]) * h, (gx[0] - gx[1]) * h, (gz[0] - gz[1]) * h
            ett = s2 * over(0)
            ltr = lam * (rx + gz[2] + ett)
            srr, szz, stt = ltr + 2 * mu * rx, ltr + 2 * mu * gz[2], ltr + 2 * mu * ett
            srz, srt, stz = mu * (rz + gx[2]), mu * (tx - ett), mu * (tz - over(2))
            qx, qz = [(srr + srt) * h, (srr - srt) * h, srz], [(srz + stz) * h, (srz - stz) * h, szz]
            hoop = {0: s2 * (stt - srt), 2: -stz}
            spread = dict(hoop)
        else:
            ett = over(0) if axisym else torch.zeros_like(gx[0])
            ltr = lam * (gx[0] + gz[1] + ett)
            srz = mu * (gz[0] + gx[1])
            qx, qz = [ltr + 2 * mu * gx[0], srz], [srz, ltr + 2 * mu * gz[1]]
            if axisym:
                hoop[0] = ltr + 2 * mu * ett
                spread = dict(hoop)
        qx, qz = torch.stack(qx), torch.stack(qz)
        f_xi, f_eta = w * (qx * xx + qz * xz), w * (qx * ex + qz * ez)
        s = f_xi @ D + D.T @ f_eta
        if len(ax):
            s[:, ax] = f_xi[:, ax] @ self.Dj + D.T @ f_eta[:, ax]
        for c, t in hoop.items():
            direct = b["hoop"] * t
            if len(ax):
                direct[ax, :, 0] = 0.0
            s[c] += direct
            if len(ax):
                g = (w * spread[c])[ax, :, 0]
                s[c][ax] += (g * xx[ax, :, 0])[:, :, None] * self.Dj[0]
                s[c][ax, :, 0] += (g * ex[ax, :, 0]) @ D
        return -s

    def accelerate(self, di, amp, h, energy):
        p, q, d = self.p, self.dom[di], self.p.domains[di]
        f = self.forces(di, q["u"])
        pot = -0.5 * float((q["u"] * f).sum()) if energy else 0.0
        for k, s in enumerate(p.sources):
            if s.domain == di:
                f.index_add_(1, self._t(s.points, torch.long), self._t(s.coef).reshape(d.ncomp, -1) * float(amp[k]))
        fp, sp, cx, cz = self.cpl
        if len(fp):
            sd = self.dom[self.solid]
            pm = p.domains[self.solid].ncomp == 3
            if di == self.solid:
                pr, hs = self.dom[self.fluid]["u"][0, fp], math.sqrt(0.5)
                for c in (0, 1) if pm else (0,):
                    f[c].index_add_(0, sp, (hs if pm else 1.0) * cx * pr)
                f[-1].index_add_(0, sp, cz * pr)
            else:
                ar = math.sqrt(0.5) * (sd["a"][0, sp] + sd["a"][1, sp]) if pm else sd["a"][0, sp]
                f[0].index_add_(0, fp, -(cx * ar + cz * sd["a"][-1, sp]))
        a = f / q["mass"]
        if len(q["abs"]):
            at, damp = q["abs"], q["C"]
            rhs = f[:, at].T - (damp @ q["v"][:, at].T[:, :, None])[:, :, 0]
            lhs = h * damp + torch.diag_embed(q["mass"][at][:, None].expand(-1, d.ncomp))
            a[:, at] = torch.linalg.solve(lhs, rhs[:, :, None])[:, :, 0].T
        q["a"] = torch.where(q["zero"], torch.zeros_like(a), a)
        return pot

    def _solve(self, amp, h, energy):
        return sum(self.accelerate(di, amp, h, energy) for di in (self.solid, self.fluid) if di is not None)

    def start(self, fields, amp0, energy=False):
        for q, (u, v) in zip(self.dom, fields):
            for k, x in (("u", u), ("v", v)):
                q[k] = torch.where(q["zero"], torch.zeros_like(q["u"]), self._t(np.asarray(x, np.float32)))
        self._solve(amp0, 0.0, energy)

    def advance(self, amp, energy=False):
        dt = self.dt
        for q in self.dom:
            q["u"] = q["u"] + dt * q["v"] + 0.5 * dt * dt * q["a"]
            q["v"] = q["v"] + 0.5 * dt * q["a"]
        self.step += 1
        pot = self._solve(amp, 0.5 * dt, energy)
        for q in self.dom:
            q["v"] = q["v"] + 0.5 * dt * q["a"]
        if energy:
            kin = sum(float((q["mass"] * (0.5 * q["v"] ** 2 - dt * dt / 8 * q["a"] ** 2)).sum()) for q in self.dom)
            return [self.step * dt, kin, pot]

    def receivers(self):
        """(domain, field, points, weights) of every recorded quantity."""
        return [(r.domain, {"pressure": "u", "displacement": "u", "velocity": "v", "acceleration": "a"}[q],
                 self._t(r.points, torch.long), self._t(r.value)) for r in self.p.receivers for q in r.quantities]

    def row(self, recs):
        out = []
        for di, k, at, w in recs:
            x = (self.dom[di][k][:, at] * w).sum(1)
            out.append(torch.stack([(x[0] + x[1]), (x[0] - x[1]), x[2] * math.sqrt(2)]) * math.sqrt(0.5) if len(x) == 3 else x)
        return torch.cat(out)

    def state(self, di):
        return tuple(self.dom[di][k].cpu().numpy() for k in "uva")


def _own_amp(prob, step):
    """The sources' own time functions (Ricker wavelets) at a step."""
    out = []
    for s in prob.sources:
        x = (math.pi * s.f0 * (step * prob.dt - s.t0)) ** 2
        out.append(s.amplitude * (1.0 - 2.0 * x) * math.exp(-x))
    return out


def _power_iteration(prob):
    """2 / sqrt(lambda_max) by 100 power iterations per domain and 120 of the
    coupled operator, start vectors U(-1, 1) from mt19937(12345)."""
    gen = np.random.MT19937()
    gen._legacy_seeding(12345)

    def vector(d):
        raw = gen.random_raw(2 * d.ncomp * d.n_global).astype(np.float64)
        x = 2.0 * ((raw[0::2] + raw[1::2] * 4294967296.0) / 18446744073709551616.0) - 1.0
        return torch.from_numpy(x.astype(np.float32)).double().reshape(d.ncomp, -1).to(ex.dev)

    ex, lam = _Exact(prob), 0.0
    for di, d in enumerate(prob.domains):
        q, x = ex.dom[di], vector(d)
        for _ in range(100):
            x = torch.where(q["zero"], torch.zeros_like(x), x)
            f = ex.forces(di, x)
            lam = max(lam, float(-(x * f).sum() / (q["mass"] * x * x).sum()))
            y = -f / q["mass"]
            x = y / y.square().sum().sqrt()
    if len(ex.cpl[0]):
        order, none = (ex.solid, ex.fluid), [0.0] * len(prob.sources)
        norm = lambda k: sum(float((ex.dom[i]["mass"] * ex.dom[i][k] ** 2).sum()) for i in order)  # noqa: E731
        for i in order:
            ex.dom[i]["u"], ex.dom[i]["abs"] = vector(prob.domains[i]), ex.dom[i]["abs"][:0]
        for it in range(120):
            for i in order:
                ex.dom[i]["u"] = torch.where(ex.dom[i]["zero"], torch.zeros_like(ex.dom[i]["u"]), ex.dom[i]["u"])
            nx = norm("u")
            ex._solve(none, 0.0, False)
            ny = norm("a")
            if it >= 60:
                lam = max(lam, math.sqrt(ny / nx))
            for i in order:
                ex.dom[i]["u"] = -ex.dom[i]["a"] / math.sqrt(ny)
    return 2.0 / math.sqrt(lam)


def exact(case, seed):
    pkg, rng, use = _package(), np.random.default_rng(seed), case["use"]
    if use == "setup":
        model = _model(case, 1000, _scale(seed))
        prob = pkg.cases.build_from_arrays(model, pkg.cases.setup_arrays(model), stable_dt=1.0)
        sdt = _power_iteration(prob)
        return {"stable_dt": sdt, "dt": model.safety * sdt, "n_steps": 1000}
    if use == "batch":
        rows = []
        for prob, arrays in _member_problems(case):
            ex = _Exact(prob)
            ex.start(_wavefield(prob, arrays, rng), _own_amp(prob, 0))
            recs, own = ex.receivers(), []
            for k in range(case["steps"]):
                ex.advance(_own_amp(prob, k + 1))
                own.append(ex.row(recs))
            rows.append(torch.stack(own))
        return {"rows": torch.cat(rows, 1).cpu()}
    prob, arrays = _problem(case)
    ex, fields = _Exact(prob), _wavefield(prob, arrays, rng)
    if use in ("seam", "forces"):
        return [ex.forces(i, ex._t(f[0].astype(np.float32))).cpu() for i, f in enumerate(fields)]
    every = int(case.get("energy") or 0)
    ex.start(fields, _own_amp(prob, 0), every > 0)
    if use == "advance":
        energy = [0.0, None, None]
        for k in range(1, case["steps"] + 1):
            got = ex.advance(_own_amp(prob, k), every > 0 and k % every == 0)
            energy = got or energy
        out = {m: ex.state(i) for i, m in enumerate(prob.media)}
        if every:
            out["energy"] = np.array(energy) if case["steps"] >= every else None
        return out
    amp, recs, rows = _signature(prob, case["steps"], rng), ex.receivers(), []
    for k in range(case["steps"]):
        ex.advance(amp[k])
        rows.append(ex.row(recs))
    out = {"rows": torch.stack(rows).cpu().numpy()}
    if ex.fluid is not None:
        out["acoustic"] = ex.state(ex.fluid)
    return out
