"""state(): renumbered on the device in one piece, field by field and by ranges
of points, on both paths, against what set_state was given."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# points: 81 (one copy), 160k (all at once), 400k (field by field, two
# components), 1.05M and 1.44M (ranges of 2^20 points, the last one short)
@pytest.mark.parametrize("path", [1, 2])
@pytest.mark.parametrize("medium,order,n", [("acoustic", 4, 2), ("acoustic", 4, 100), ("elastic", 4, 158),
                                            ("elastic", 4, 256), ("acoustic", 4, 300), ("elastic", 2, 512)])
def test_state_returns_what_was_set(pkg, medium, order, n, path):
    import insem_b200.cases as K

    mat = K.Material.acoustic(1500.0, 1000.0) if medium == "acoustic" else K.FAST
    mesh = K.layered((0.0, 1.0), [0.0, 1.0], [n], [0], nx=n)
    m = K.Model(mesh, order=order, materials={0: mat}, dt=1e-8)
    m.n_steps = 1
    prob = K.build(m, stable_dt=1e-6)
    d = prob.domains[0]
    rng = np.random.default_rng(3)
    u, v = rng.standard_normal((2, d.ncomp, d.n_global)).astype(np.float32).astype(np.float64)
    with pkg.Solver(prob, path=path) as s:
        s.set_state(medium, u, v)
        for _ in range(2):
            got = s.state(medium)
            assert np.array_equal(got[0], u) and np.array_equal(got[1], v) and not got[2].any()
