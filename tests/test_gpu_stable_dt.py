"""The device power iteration against the same iteration in 64 bits (numpy, on
the dense operator that the oracle's internal forces give), for every order,
one and two media, plain and weighted maps."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _start():
    gen = np.random.MT19937()
    gen._legacy_seeding(12345)

    def vector(n):
        raw = gen.random_raw(2 * n).astype(np.float64)
        x = 2.0 * ((raw[0::2] + raw[1::2] * 4294967296.0) / 18446744073709551616.0) - 1.0
        return x.astype(np.float32).astype(np.float64)

    return vector


def _expected(prob, oracle):
    ref = oracle.OracleSolver(prob)
    ops = []
    for i, d in enumerate(prob.domains):
        n = d.ncomp * d.n_global
        K = np.stack([ref.internal_forces(i, e).astype(np.float64) for e in np.eye(n, dtype=np.float32)], axis=1)
        zero = np.zeros((d.ncomp, d.n_global), bool)
        zero[:, d.dirichlet_points] = True
        for c in d.axis_components:
            zero[int(c), d.axis_points] = True
        ops.append((K, np.tile(d.mass.astype(np.float64), d.ncomp), zero.ravel()))
    vector, lam = _start(), 0.0
    for K, m, zero in ops:
        x = vector(m.size)
        for _ in range(100):
            x[zero] = 0.0
            f = K @ x
            lam = max(lam, -(x @ f) / (x @ (m * x)))
            x = -f / m
            x /= np.sqrt(x @ x)
    c = prob.coupling
    if c["fluid_points"].size:
        si = prob.domain_index("elastic")
        fi = 1 - si
        s, ng = prob.domains[si], prob.domains[si].n_global
        u = {i: vector(ops[i][1].size) for i in (si, fi)}
        h = np.sqrt(0.5)
        for it in range(120):
            for i in u:
                u[i][ops[i][2]] = 0.0
            nx = sum(ops[i][1] @ u[i] ** 2 for i in u)
            f = ops[si][0] @ u[si]
            p = u[fi][c["fluid_points"]]
            for comp in (0, 1) if s.ncomp == 3 else (0,):
                np.add.at(f, comp * ng + c["solid_points"], (h if s.ncomp == 3 else 1.0) * c["cx"] * p)
            np.add.at(f, (s.ncomp - 1) * ng + c["solid_points"], c["cz"] * p)
            a = {si: np.where(ops[si][2], 0.0, f / ops[si][1])}
            f = ops[fi][0] @ u[fi]
            ar = a[si][c["solid_points"]]
            if s.ncomp == 3:
                ar = h * (ar + a[si][ng + c["solid_points"]])
            np.add.at(f, c["fluid_points"], -(c["cx"] * ar + c["cz"] * a[si][(s.ncomp - 1) * ng + c["solid_points"]]))
            a[fi] = np.where(ops[fi][2], 0.0, f / ops[fi][1])
            ny = sum(ops[i][1] @ a[i] ** 2 for i in u)
            if it >= 60:
                lam = max(lam, np.sqrt(ny / nx))
            u = {i: -a[i] / np.sqrt(ny) for i in u}
    return 2.0 / np.sqrt(lam)


def _problem(order, kind):
    import insem_b200.cases as K

    if kind == "dipole":
        b = K.borehole((0.0, 0.3), [("mud", 0.1)], formation_radius=0.4, dz=0.15)
        mats = {b.regions["mud"]: K.MUD, b.regions["formation"]: K.FAST}
        m = K.Model(b.mesh, order=order, azimuthal_order=1, materials=mats, dt=1e-9,
                    boundaries={b.boundaries["top"]: "rigid"})
    else:
        mesh = K.rectangle((0.0, 3.0), (0.0, 2.0), nx=3, nz=2, material=lambda x, z: int(kind == "coupled" and z < 1.0))
        m = K.Model(mesh, order=order, materials={0: K.Material.acoustic(1500.0, 1000.0), 1: K.FAST}, dt=1e-9,
                    boundaries={K.LEFT: "rigid", K.TOP: "free"}, regions=[(0.0, 1.0, 1.0, 2.0, 1)] if kind == "hanging" else [])
    m.n_steps = 1
    return K.build(m, stable_dt=1.0)


@pytest.mark.parametrize("order", range(1, 9))
@pytest.mark.parametrize("kind", ["acoustic", "hanging", "coupled", "dipole"])
def test_estimate_matches_64_bits(pkg, oracle, order, kind):
    from insem_b200.solver import estimate_stable_dt

    prob = _problem(order, kind)
    got, want = estimate_stable_dt(prob), _expected(prob, oracle)
    # float fields renormalised each iteration: the quotients carry their rounding only
    assert abs(got - want) <= 2e-6 * want, (got, want)
    assert got == estimate_stable_dt(prob)
