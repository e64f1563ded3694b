"""The tile kernels of every order, element kind and medium against the oracle:
whole and partial tiles, elements whose inner points are finished in registers
beside elements that carry a source or receiver, and both register budgets
(launches that are resident at once, and larger ones)."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KINDS = ["rect", "affine", "curved", "monopole", "dipole", "bent monopole", "bent dipole", "flat monopole", "flat dipole"]


def _model(order, kind, nx, nz):
    import insem_b200.cases as K

    if kind in ("monopole", "dipole"):
        b = K.borehole((0.0, 0.1 * nz), [("mud", 0.1)], formation_radius=0.1 * nx, dz=0.1, growth=1.05, dr=0.2)
        mats = {b.regions["mud"]: K.MUD, b.regions["formation"]: K.FAST}
        m = K.Model(b.mesh, order=order, azimuthal_order=int(kind == "dipole"), materials=mats,
                    boundaries={b.boundaries["outer"]: "absorbing", b.boundaries["top"]: "rigid"},
                    sources=[K.Source(kind, 0.0, 0.05 * nz, (1.0, 0.0, 0.0), K.ricker(8000.0))], dt=1e-7)
        where = [("acoustic", 0.04, 0.043 * nz), ("elastic", 0.06 * nx + 0.05, 0.07 * nz)]
    elif kind.startswith(("bent", "flat")):  # axisymmetric, with a metric that varies inside the elements; a solid on the axis
        h = nz // 2
        top = lambda x: 0.1 * (h + 0.5 * np.sin(20.0 * x) * kind.startswith("bent"))  # noqa: E731
        mesh = K.layered((0.0, 0.1 * nx), [0.0, top, 0.1 * nz], [h, nz - h], [1, 0], nx=nx, quadratic=kind.startswith("bent"),
                         coords="axisymmetric")
        m = K.Model(mesh, order=order, azimuthal_order=int(kind.endswith("dipole")),
                    materials={0: K.MUD, 1: K.FAST}, boundaries={K.RIGHT: "absorbing", K.TOP: "rigid"},
                    sources=[K.Source(kind.split()[1], 0.0, 0.083 * nz, (1.0, 0.0, 0.0), K.ricker(8000.0))], dt=1e-7)
        where = [("acoustic", 0.04 * nx, 0.08 * nz), ("elastic", 0.06 * nx, 0.02 * nz)]
    else:
        slope = {"rect": lambda x: 0.0 * x, "affine": lambda x: 0.2 * x, "curved": lambda x: 0.3 * np.sin(x)}[kind]
        h = nz // 2
        mesh = K.layered((0.0, float(nx)), [lambda x: slope(x), lambda x: h + slope(x), lambda x: nz + slope(x)],
                         [h, nz - h], [1, 0], nx=nx, quadratic=kind == "curved")
        m = K.Model(mesh, order=order, materials={0: K.Material.acoustic(1500.0, 1000.0), 1: K.FAST},
                    boundaries={K.BOTTOM: "absorbing", K.LEFT: "rigid", K.TOP: "free"},
                    sources=[K.Source("monopole", 0.41 * nx, 0.8 * nz, stf=K.ricker(300.0))], dt=1e-6)
        where = [("acoustic", 0.3 * nx, 0.77 * nz), ("elastic", 0.6 * nx, 0.3 * nz)]
    for medium, x, z in where:
        m.receivers.append(K.Receiver(medium, x, z, ["pressure" if medium == "acoustic" else "velocity"], medium))
    m.n_steps, m.energy_every = 5, 2
    return K.build(m, stable_dt=1e-5)


def _check(pkg, oracle, prob, **kw):
    rng = np.random.default_rng(7)
    ref = oracle.OracleSolver(prob)
    with pkg.Solver(prob, **kw) as s:
        for d, medium in zip(prob.domains, prob.media):
            u, v = (1e3 if d.medium == 0 else 1e-6) * rng.standard_normal((2, d.ncomp, d.n_global))
            s.set_state(medium, u, v)
            ref.set_state(medium, u, v)
        s.advance(2)
        s.run()
        ref.run()
        for name, quantity in prob.trace_list():
            assert np.array_equal(s.trace(name, quantity), ref.trace(name, quantity)), (name, quantity)
        for i, medium in enumerate(prob.media):
            for x, y in zip(s.state(medium), ref.state(i)):
                assert np.array_equal(x, y), medium
        got, want = s.energy, ref.energy
        assert np.all(np.abs(got - want) <= 1e-9 * np.abs(want).max(0))


@pytest.mark.parametrize("order", range(1, 9))
@pytest.mark.parametrize("kind", KINDS)
def test_small_domains(pkg, oracle, order, kind):
    prob = _model(order, kind, 11, 8)
    assert {b.kind for d in prob.domains for b in d.blocks} == {{"rect": 0, "affine": 1, "curved": 2}.get(kind, 3)}
    _check(pkg, oracle, prob)
    _check(pkg, oracle, prob, tile_elements=7)


@pytest.mark.parametrize("order,kind,nx,nz", [(3, "rect", 300, 320), (5, "curved", 210, 220), (4, "monopole", 220, 230),
                                              (6, "dipole", 130, 140), (8, "affine", 120, 130), (5, "bent monopole", 200, 210)])
def test_domains_of_many_tiles(pkg, oracle, order, kind, nx, nz):
    _check(pkg, oracle, _model(order, kind, nx, nz))


@pytest.mark.parametrize("n,want", [(255, 8), (257, 32)])  # 4.16M and 4.23M points, about 2^22
def test_large_domains_take_full_tiles(pkg, n, want):
    import insem_b200.cases as K

    m = K.Model(K.layered((0.0, 1.0), [0.0, 1.0], [n], [0], nx=n), order=8,
                materials={0: K.Material.acoustic(1500.0, 1000.0)}, dt=1e-9)
    m.n_steps = 1
    prob = K.build(m, stable_dt=1e-6)
    with pkg.Solver(prob, tile_elements=8) as s:
        assert pkg.native.lib().insem_cuda_solver_tile_elements(s._h, 0) == want
