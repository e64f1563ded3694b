"""Spans of steps against the oracle at the lengths where the captured
sequences (1, 4 and 16 steps) meet: receivers of one step run beside the next
step's tiles, constrained slots are gathered inside the tiles."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(n_steps, energy_every):
    import insem_b200.cases as K

    # borehole with a refined annulus: hanging nodes, two media, axis, Stacey
    b = K.borehole((0.0, 0.9), [("mud", 0.1), ("casing", 0.11)], formation_radius=0.8, dz=0.15)
    mats = {b.regions["mud"]: K.MUD, b.regions["casing"]: K.STEEL, b.regions["formation"]: K.FAST}
    recs = [K.Receiver("p", 0.05, 0.5, ["pressure", "particle_velocity"], "acoustic"),
            K.Receiver("s", 0.4, 0.45, ["velocity", "acceleration"], "elastic")]
    model = K.Model(b.mesh, order=4, regions=[(0.2, 0.2, 0.5, 0.5, 1)], materials=mats,
                    boundaries={b.boundaries["outer"]: "absorbing", b.boundaries["top"]: "absorbing"},
                    sources=[K.Source("monopole", 0.0, 0.45, stf=K.ricker(8000.0))], receivers=recs,
                    n_steps=n_steps, dt=1e-7, record_every=2, energy_every=energy_every)
    prob = K.build(model, stable_dt=1e-5)
    assert sum(d.n_rows for d in prob.domains) > 0
    return prob


def _fields(prob, seed):
    rng = np.random.default_rng(seed)
    return [(1e3 if d.medium == 0 else 1e-6) * rng.standard_normal((2, d.ncomp, d.n_global)) for d in prob.domains]


def _check(prob, s, ref):
    for name, quantity in prob.trace_list():
        assert np.array_equal(s.trace(name, quantity), ref.trace(name, quantity)), (name, quantity)
    if prob.energy_every:
        got, want = s.energy, ref.energy
        assert got.shape == want.shape and np.all(np.abs(got - want) <= 1e-9 * np.abs(want).max(0))
    for i, medium in enumerate(prob.media):
        for x, y in zip(s.state(medium), ref.state(i)):
            assert np.array_equal(x, y), medium


@pytest.mark.parametrize("graphs", [True, False])
@pytest.mark.parametrize("energy_every", [0, 3])
def test_spans_match_the_oracle(pkg, oracle, graphs, energy_every):
    spans = [1, 3, 4, 0, 5, 16, 64, 83, 2]
    prob = _problem(sum(spans), energy_every)
    ref = oracle.OracleSolver(prob)
    with pkg.Solver(prob, use_graphs=graphs) as s:
        for medium, (u, v) in zip(prob.media, _fields(prob, 1)):
            s.set_state(medium, u, v)
            ref.set_state(medium, u, v)
        for n in spans:
            s.advance(n)
            ref.advance(n)
            _check(prob, s, ref)


@pytest.mark.parametrize("graphs", [True, False])
def test_batch_spans_match_the_oracle(pkg, oracle, graphs):
    lengths = (1, 6, 21)  # members end in the middle of the batch's spans
    with pkg.Batch(use_graphs=graphs) as b:
        entries = []
        for k, n in enumerate(lengths):
            prob = _problem(n, 3 * (k % 2))
            ref, s = oracle.OracleSolver(prob), b.add(prob)
            for medium, (u, v) in zip(prob.media, _fields(prob, k)):
                s.set_state(medium, u, v)
                ref.set_state(medium, u, v)
            entries.append((prob, s, ref))
        for n in (2, 3, 16, 5):
            b.advance(n)
        assert b.active == 0
        for prob, s, ref in entries:
            ref.run()
            _check(prob, s, ref)
