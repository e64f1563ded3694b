"""Domains of several element blocks against the oracle: a block without
elements ahead of the others, in their middle or at the end, and one block
split in two.  The blocks of a domain follow one another in a chain of
launches of which only the first waits for what is ahead of it, so that first
one has to be a block that launches."""

from __future__ import annotations

import copy
import ctypes as C
from dataclasses import fields, replace

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FORMS = ["empty first", "empty middle", "empty last", "split"]


def _take(b, npe, lo, hi):
    """Elements [lo, hi) of a block."""
    n, out = b.n_elements, {}
    for f in fields(b):
        x = getattr(b, f.name)
        if isinstance(x, np.ndarray):
            out[f.name] = np.ascontiguousarray(x.reshape(n, -1)[lo:hi].ravel()) if x.size else x
    return replace(b, **out)


def _with_blocks(prob, form):
    """The problem with every domain's one block in the given form."""
    prob, npe = copy.deepcopy(prob), prob.ngll ** 2
    for d in prob.domains:
        (b,) = d.blocks
        n = b.n_elements
        first, second, none = _take(b, npe, 0, n // 2), _take(b, npe, n // 2, n), _take(b, npe, 0, 0)
        d.blocks = {"empty first": [none, first, second], "empty middle": [first, none, second],
                    "empty last": [first, second, none], "split": [first, second]}[form]
    return prob


def _problem(kind, n=24, n_steps=1, order=4):
    import insem_b200.cases as K

    if kind == "dipole":
        b = K.borehole((0.0, 0.1 * n), [("mud", 0.1)], formation_radius=0.08 * n, dz=0.1)
        mats = {b.regions["mud"]: K.MUD, b.regions["formation"]: K.FAST}
        m = K.Model(b.mesh, order=order, azimuthal_order=1, materials=mats, boundaries={b.boundaries["outer"]: "absorbing"},
                    sources=[K.Source("dipole", 0.0, 0.05 * n, (1.0, 0.0, 0.0), K.ricker(3000.0))], dt=1e-8,
                    receivers=[K.Receiver("p", 0.04, 0.043 * n, ["pressure"], "acoustic")])
    else:
        mesh = K.rectangle((0.0, float(n)), (0.0, float(n)), nx=n, nz=n, material=lambda x, z: int(z < 0.4 * n))
        m = K.Model(mesh, order=order, materials={0: K.Material.acoustic(1500.0, 1000.0), 1: K.FAST}, dt=1e-8,
                    boundaries={K.BOTTOM: "absorbing", K.LEFT: "rigid"}, energy_every=3,
                    sources=[K.Source("monopole", 0.41 * n, 0.83 * n, stf=K.ricker(300.0))],
                    receivers=[K.Receiver("p", 0.32 * n, 0.71 * n, ["pressure"], "acoustic")])
    m.n_steps = n_steps
    return K.build(m, stable_dt=1.0)


@pytest.mark.parametrize("form", FORMS + ["uncovered"])
@pytest.mark.parametrize("kind", ["plain", "dipole"])
def test_forces_without_allocation(pkg, oracle, kind, form):
    """Both domains one after the other, many times, over one scratch array and
    with the field rewritten ahead of each call."""
    import torch

    from insem_b200 import native as N

    prob = _problem(kind, n=48)
    if form == "uncovered":  # elements of no block contribute nothing (two-pass path only)
        prob = _with_blocks(prob, "empty first")
        for d in prob.domains:
            d.blocks.pop()
    else:
        prob = _with_blocks(prob, form)
    ref = oracle.OracleSolver(prob)
    rng = np.random.default_rng(5)
    with pkg.Solver(prob, path=1) as s:
        host = [rng.uniform(-1, 1, d.ncomp * d.n_global).astype(np.float32) for d in prob.domains]
        want = [ref.internal_forces(i, u) for i, u in enumerate(host)]
        src = [torch.from_numpy(u).cuda() for u in host]
        u = [torch.empty_like(x) for x in src]
        reps = 20
        f = [[torch.full_like(x, float("nan")) for x in src] for _ in range(reps)]
        side = torch.cuda.Stream()
        torch.cuda.synchronize()
        with torch.cuda.stream(side):
            for k in range(reps):
                for i in range(len(src)):
                    u[i].zero_()
                    torch.add(u[i], src[i], out=u[i])
                    N.check(N.lib().insem_cuda_solver_internal_forces_noalloc(
                        s._h, i, C.c_void_p(u[i].data_ptr()), C.c_void_p(f[k][i].data_ptr()), C.c_void_p(side.cuda_stream)))
        torch.cuda.synchronize()
        for k in range(reps):
            for i in range(len(src)):
                assert np.array_equal(f[k][i].cpu().numpy(), want[i]), (k, i)


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("kind", ["plain", "dipole"])
def test_stable_dt(pkg, kind, form):
    """The estimate of the problem as built, bit for bit: blocks only share out
    the elements."""
    from insem_b200.solver import estimate_stable_dt

    prob = _problem(kind)
    want, other = estimate_stable_dt(prob), _with_blocks(prob, form)
    for _ in range(3):
        assert estimate_stable_dt(other) == want


@pytest.mark.parametrize("kind", ["coupled", "dipole"])
@pytest.mark.parametrize("blocks", ["none", "empty"])
def test_stable_dt_with_a_solid_that_launches_nothing(pkg, oracle, kind, blocks):
    """The solid then has no stiffness; its mass still takes part in the coupled
    iteration, in which the fluid's forces come first."""
    from insem_b200.solver import estimate_stable_dt
    from test_gpu_stable_dt import _expected, _problem as small

    prob = small(4, kind)
    d = prob.domains[prob.domain_index("elastic")]
    d.blocks = [] if blocks == "none" else [_take(d.blocks[0], prob.ngll ** 2, 0, 0)]
    with np.errstate(invalid="ignore"):  # the solid alone: 0 / 0 after its first iteration, which no maximum takes
        want = _expected(prob, oracle)
    got = estimate_stable_dt(prob)
    assert abs(got - want) <= 2e-6 * want, (got, want)
    assert got == estimate_stable_dt(prob)


def _check(prob, s, ref):
    for name, quantity in prob.trace_list():
        assert np.array_equal(s.trace(name, quantity), ref.trace(name, quantity)), (name, quantity)
    for i, medium in enumerate(prob.media):
        for x, y in zip(s.state(medium), ref.state(i)):
            assert np.array_equal(x, y), medium


def _mixed(n, n_steps=1):
    """Rect, Affine and Curved elements: three blocks of one domain."""
    import insem_b200.cases as K

    a, b = 0.35 * n, 0.7 * n
    rise = lambda x: np.where(x < a, 0.0, np.where(x < b, 0.2 * (x - a), 0.2 * (b - a) + 0.3 * np.sin(x - b)))  # noqa: E731
    mesh = K.layered((0.0, float(n)), [rise, lambda x: n + rise(x)], [n], [1], nx=n, quadratic=True)
    m = K.Model(mesh, order=4, materials={1: K.FAST}, boundaries={K.LEFT: "absorbing", K.TOP: "free"}, dt=1e-6,
                sources=[K.Source("force", 0.36 * n, 0.49 * n, (0.0, 1.0, 0.0), K.ricker(300.0))],
                receivers=[K.Receiver("v", 0.68 * n, 0.46 * n, ["velocity"], "elastic")], energy_every=3)
    m.n_steps = n_steps
    prob = K.build(m, stable_dt=1.0)
    assert [x.kind for x in prob.domains[0].blocks] == [0, 1, 2]
    return prob


def _set(prob, *solvers):
    rng = np.random.default_rng(2)
    for d, medium in zip(prob.domains, prob.media):
        u, v = (1e3 if d.medium == 0 else 1e-6) * rng.standard_normal((2, d.ncomp, d.n_global))
        for s in solvers:
            s.set_state(medium, u, v)


def _steps_problem(kind, form, n_steps):
    return _mixed(20, n_steps) if kind == "mixed" else _with_blocks(_problem(kind, n_steps=n_steps), form)


CASES = [(kind, form) for kind in ("plain", "dipole") for form in FORMS] + [("mixed", "built")]


@pytest.mark.parametrize("kind,form", CASES)
@pytest.mark.parametrize("path", [0, 1])
def test_steps(pkg, oracle, kind, form, path):
    prob = _steps_problem(kind, form, 23)
    ref = oracle.OracleSolver(prob)
    with pkg.Solver(prob, path=path) as s:
        _set(prob, s, ref)
        for n in (1, 21, 1):
            s.advance(n)
        ref.run()
        _check(prob, s, ref)


def test_batched_steps(pkg, oracle):
    with pkg.Batch() as b:
        entries = []
        for kind, form in CASES:
            prob = _steps_problem(kind, form, 11)
            s, ref = b.add(prob), oracle.OracleSolver(prob)
            _set(prob, s, ref)
            entries.append((prob, s, ref))
        b.run()
        for prob, s, ref in entries:
            ref.run()
            _check(prob, s, ref)


def test_mixed_kinds_forces_and_stable_dt(pkg, oracle):
    import torch

    from insem_b200 import native as N
    from insem_b200.solver import estimate_stable_dt
    from test_gpu_stable_dt import _expected

    prob = _mixed(6)
    want, got = _expected(prob, oracle), estimate_stable_dt(prob)
    assert abs(got - want) <= 2e-6 * want, (got, want)
    assert got == estimate_stable_dt(prob)
    prob = _mixed(20)
    d = prob.domains[0]
    u = np.random.default_rng(4).uniform(-1, 1, d.ncomp * d.n_global).astype(np.float32)
    u_dev = torch.from_numpy(u).cuda()
    f = [torch.empty_like(u_dev) for _ in range(10)]
    torch.cuda.synchronize()
    with pkg.Solver(prob) as s:
        for x in f:
            N.check(N.lib().insem_cuda_solver_internal_forces_noalloc(s._h, 0, C.c_void_p(u_dev.data_ptr()),
                                                                      C.c_void_p(x.data_ptr()), None))
        torch.cuda.synchronize()
    want = oracle.OracleSolver(prob).internal_forces(0, u)
    assert all(np.array_equal(x.cpu().numpy(), want) for x in f)
