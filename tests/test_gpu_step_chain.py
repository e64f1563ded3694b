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


def _samples(prob, ref):
    return np.concatenate([ref.trace(r, q) for r, q in prob.trace_list()], axis=1)


@pytest.mark.parametrize("path", [0, 1])
def test_streamed_spans_with_several_sources(pkg, oracle, path):
    import insem_b200.cases as K
    from insem_b200.stf import amplitudes

    spans = [1, 7, 64]
    prob = _problem(sum(spans), 0)
    extra = K.build(K.Model(**{**_source_model(), "n_steps": 1, "dt": 1e-7}), stable_dt=1e-5).sources
    prob.sources.extend(extra)
    ref = oracle.OracleSolver(prob)
    ref.run()
    want, step = _samples(prob, ref), 0
    with pkg.Solver(prob, path=path) as s:
        for n in spans:
            amp = np.ascontiguousarray(amplitudes(prob, step + 1, n))
            rows = np.full((n, s.n_columns), np.nan)
            got = s.advance_streamed(n, amp, rows)
            first = step // prob.record_every + 1
            assert np.array_equal(rows[:got], want[first:first + got]) and got == (step + n) // prob.record_every + 1 - first
            step += n


def _source_model():
    import insem_b200.cases as K

    b = K.borehole((0.0, 0.9), [("mud", 0.1), ("casing", 0.11)], formation_radius=0.8, dz=0.15)
    mats = {b.regions["mud"]: K.MUD, b.regions["casing"]: K.STEEL, b.regions["formation"]: K.FAST}
    return dict(mesh=b.mesh, order=4, regions=[(0.2, 0.2, 0.5, 0.5, 1)], materials=mats,
                sources=[K.Source("monopole", 0.0, 0.3, stf=K.gaussian(6000.0, 1e-5))])


def test_streamed_batch_spans(pkg, oracle):
    from insem_b200.stf import amplitudes

    lengths, n = (5, 12, 40), 21  # a whole sequence, then single steps; two members end inside
    probs = [_problem(k, 0) for k in lengths]
    refs = [oracle.OracleSolver(p) for p in probs]
    for r in refs:
        r.run()
    with pkg.Batch() as b:
        for p in probs:
            b.add(p)
        a_cols, r_cols = b.stream_layout()
        amp = np.ascontiguousarray(np.concatenate([amplitudes(p, 1, n) for p in probs], axis=1))
        assert amp.shape == (n, a_cols)
        rows = np.full((n, r_cols), np.nan)
        assert b.advance_streamed(n, amp, rows) == n
    at = 0
    for p, r in zip(probs, refs):
        want = _samples(p, r)
        for j in range(min(n, p.n_steps)):
            assert np.array_equal(rows[j, at:at + want.shape[1]], want[(j + 1) // p.record_every])
        at += want.shape[1]
