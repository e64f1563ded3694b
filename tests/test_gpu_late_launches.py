"""Launches of a sequence that read what earlier launches wrote without a wait
of their own: the halo points of a batch's second and third class, the
receivers and particle velocities beside the next step's tiles, and a coupled
model's fluid tiles.  Members of every halo class step together over whole
sequences; fields, traces and particle velocities equal the oracle's."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(kind, n_steps):
    import insem_b200.cases as K

    if kind == "dipole":
        b = K.borehole((0.0, 0.9), [("mud", 0.1)], formation_radius=0.8, dz=0.1)
        m = K.Model(b.mesh, order=5, azimuthal_order=1, regions=[(0.2, 0.2, 0.5, 0.5, 1)],
                    materials={b.regions["mud"]: K.MUD, b.regions["formation"]: K.FAST},
                    boundaries={b.boundaries["outer"]: "absorbing"},
                    sources=[K.Source("dipole", 0.0, 0.45, (1.0, 0.0, 0.0), K.ricker(3000.0))], dt=1e-7)
        where = [("acoustic", 0.05, 0.5), ("elastic", 0.4, 0.45)]
    else:
        fluid = kind == "fluid"
        mesh = K.rectangle((0.0, 9.0), (0.0, 9.0), nx=9, nz=9, material=0 if fluid else (lambda x, z: int(z < 4.0)))
        m = K.Model(mesh, order=4, materials={0: K.Material.acoustic(1500.0, 1000.0), 1: K.FAST},
                    regions=[(2.0, 5.0, 4.0, 7.0, 1)], boundaries={K.BOTTOM: "absorbing", K.LEFT: "absorbing"},
                    sources=[K.Source("monopole", 4.3, 6.2, stf=K.ricker(300.0))], dt=1e-6)
        where = [("acoustic", 6.3, 7.1)] + ([] if fluid else [("elastic", 3.7, 1.2)])
    for medium, x, z in where:
        q = ["pressure", "particle_velocity"] if medium == "acoustic" else ["velocity", "acceleration"]
        m.receivers.append(K.Receiver(medium, x, z, q, medium))
    m.n_steps = n_steps
    prob = K.build(m, stable_dt=1e-5)
    assert sum(d.n_rows for d in prob.domains) > 0
    return prob


@pytest.mark.parametrize("graphs", [True, False])
def test_halo_classes_side_by_side(pkg, oracle, graphs):
    spans = (8, 19, 64)
    with pkg.Batch(use_graphs=graphs) as b:
        entries = []
        for k, kind in enumerate(("fluid", "coupled", "dipole") * 2):
            prob = _problem(kind, sum(spans) - 5 * k)
            ref, s = oracle.OracleSolver(prob), b.add(prob)
            rng = np.random.default_rng(k)
            for d, medium in zip(prob.domains, prob.media):
                u, v = (1e3 if d.medium == 0 else 1e-6) * rng.standard_normal((2, d.ncomp, d.n_global))
                s.set_state(medium, u, v)
                ref.set_state(medium, u, v)
            entries.append((prob, s, ref))
        for n in spans:
            b.advance(n)
        assert b.active == 0
        for prob, s, ref in entries:
            ref.run()
            for name, quantity in prob.trace_list():
                assert np.array_equal(s.trace(name, quantity), ref.trace(name, quantity)), (name, quantity)
            for i, medium in enumerate(prob.media):
                for x, y in zip(s.state(medium), ref.state(i)):
                    assert np.array_equal(x, y), medium
