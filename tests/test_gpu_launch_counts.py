"""kernels_per_step says the same whatever length of steps a solve or batch was
first advanced by (and so whichever sequence of steps was captured first)."""

from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


def _problem():
    import insem_b200.cases as K

    mesh = K.rectangle((0.0, 9.0), (0.0, 9.0), nx=9, nz=9, material=lambda x, z: int(z < 4.0))
    m = K.Model(mesh, order=3, materials={0: K.Material.acoustic(1500.0, 1000.0), 1: K.FAST}, dt=1e-7, energy_every=5,
                receivers=[K.Receiver("p", 4.3, 6.2, ["pressure", "particle_velocity"], "acoustic")])
    m.n_steps = 100
    return K.build(m, stable_dt=1e-5)


def test_launches_of_a_step(pkg):
    # fluid and solid tiles, halo points, energy, particle velocity, record
    for first in (1, 3, 4, 64):
        with pkg.Solver(_problem()) as s:
            s.advance(first)
            assert s.kernels_per_step == 6, first
            s.advance(1)
            assert s.kernels_per_step == 6, first
    for first in (1, 8, 11):
        with pkg.Batch() as b:
            b.add(_problem())
            b.advance(first)
            assert b.kernels_per_step == 6, first
            b.advance(1)
            assert b.kernels_per_step == 6, first
