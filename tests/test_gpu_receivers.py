"""Receiver sums (one warp per recorded column) against the oracle, at point
counts below, across and above a warp's 32 lanes, with and without recorded
particle velocity."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [1, 2, 4, 5, 8])
@pytest.mark.parametrize("axisym", [False, True])
def test_receiver_columns_match_the_oracle(pkg, oracle, order, axisym):
    import insem_b200.cases as K

    if axisym:  # dipole borehole: three-component solid, U+- rotated columns
        b = K.borehole((0.0, 0.8), [("mud", 0.1)], formation_radius=0.6, dz=0.1)
        mats = {b.regions["mud"]: K.MUD, b.regions["formation"]: K.FAST}
        model = K.Model(b.mesh, order=order, azimuthal_order=1, materials=mats,
                        boundaries={b.boundaries["outer"]: "absorbing"},
                        sources=[K.Source("dipole", 0.0, 0.4, (1.0, 0.0, 0.0), K.ricker(3000.0))], n_steps=12, dt=1e-7)
        where = [("acoustic", 0.04, 0.33), ("elastic", 0.3, 0.41)]
    else:
        m = K.rectangle((0.0, 8.0), (0.0, 6.0), nx=8, nz=6, material=lambda x, z: int(z < 3.0))
        mats = {0: K.Material.acoustic(1500.0, 1000.0), 1: K.FAST}
        model = K.Model(m, order=order, materials=mats, boundaries={K.BOTTOM: "absorbing", K.TOP: "free"},
                        sources=[K.Source("monopole", 4.1, 4.6, stf=K.ricker(300.0))], n_steps=12, dt=1e-6)
        where = [("acoustic", 2.3, 4.4), ("elastic", 3.7, 1.2)]
    for medium, x, z in where:
        quantities = ["pressure", "particle_velocity"] if medium == "acoustic" else ["velocity", "acceleration", "displacement"]
        model.receivers.append(K.Receiver(medium, x, z, quantities, medium))
    model.receivers.append(K.Receiver("plain", where[0][1] * 1.1, where[0][2], ["pressure"], "acoustic"))
    prob = K.build(model, stable_dt=1e-5)
    rng = np.random.default_rng(order)
    start = [(1e3 if d.medium == 0 else 1e-6) * rng.standard_normal((2, d.ncomp, d.n_global)) for d in prob.domains]
    ref = oracle.OracleSolver(prob)
    with pkg.Solver(prob) as s:
        for medium, (u, v) in zip(prob.media, start):
            s.set_state(medium, u, v)
            ref.set_state(medium, u, v)
        s.run()
        ref.run()
        for name, quantity in prob.trace_list():
            assert np.array_equal(s.trace(name, quantity), ref.trace(name, quantity)), (name, quantity)
