"""Fluid-solid coupling in the halo kernel: points of one group share a CTA
(chunks of 256 per side); a group too large for a CTA takes two launches.
Interface entries are added to the layered model so that neighbouring points
join into groups of a given length."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(group, n_steps=9):
    import insem_b200.cases as K

    m = K.rectangle((0.0, 80.0), (0.0, 6.0), nx=80, nz=6, material=lambda x, z: int(z < 3.0))
    mats = {0: K.Material.acoustic(1500.0, 1000.0), 1: K.FAST}
    model = K.Model(m, order=4, materials=mats, boundaries={K.BOTTOM: "absorbing", K.LEFT: "absorbing"},
                    sources=[K.Source("monopole", 40.3, 4.6, stf=K.ricker(300.0))],
                    receivers=[K.Receiver("r", 30.2, 3.3, ["pressure"], "acoustic")], n_steps=n_steps, dt=1e-6,
                    energy_every=4)
    prob = K.build(model, stable_dt=1e-5)
    c = prob.coupling
    n = c["fluid_points"].size
    assert n == 321
    more = np.array([i for i in range(n - 1) if (i + 1) % group], dtype=int)  # entry i also joins point i + 1's solid
    solid = c["solid_points"]
    for k in ("fluid_points", "cx", "cz"):
        c[k] = np.ascontiguousarray(np.concatenate([c[k], c[k][more]]))
    c["solid_points"] = np.ascontiguousarray(np.concatenate([solid, solid[more + 1]]))
    return prob


def _check(prob, s, ref):
    for name, quantity in prob.trace_list():
        assert np.array_equal(s.trace(name, quantity), ref.trace(name, quantity))
    for i, medium in enumerate(prob.media):
        for x, y in zip(s.state(medium), ref.state(i)):
            assert np.array_equal(x, y), medium
    got, want = s.energy, ref.energy
    assert np.all(np.abs(got - want) <= 1e-9 * np.abs(want).max(0))


@pytest.mark.parametrize("group", [1, 3, 255, 256, 257, 321])
@pytest.mark.parametrize("batched", [False, True])
def test_coupled_groups(pkg, oracle, group, batched):
    prob = _problem(group)
    rng = np.random.default_rng(group)
    ref = oracle.OracleSolver(prob)
    b = pkg.Batch() if batched else None
    s = b.add(prob) if batched else pkg.Solver(prob)
    for d, medium in zip(prob.domains, prob.media):
        u, v = (1e3 if d.medium == 0 else 1e-6) * rng.standard_normal((2, d.ncomp, d.n_global))
        s.set_state(medium, u, v)
        ref.set_state(medium, u, v)
    (b or s).run()
    ref.run()
    _check(prob, s, ref)
    (b or s).close()
