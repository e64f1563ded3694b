"""Gather, assembly and allocation-free internal forces against the oracle for
every order and component count, points of one to many contributions, plain
and weighted maps; and the same calls replayed from a captured graph."""

from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(order, kind):
    import insem_b200.cases as K

    if kind == "dipole":
        b = K.borehole((0.0, 0.6), [("mud", 0.1)], formation_radius=0.7, dz=0.15)
        mats = {b.regions["mud"]: K.MUD, b.regions["formation"]: K.FAST}
        m = K.Model(b.mesh, order=order, azimuthal_order=1, materials=mats, dt=1e-9)
    else:
        mesh = K.rectangle((0.0, 6.0), (0.0, 5.0), nx=6, nz=5, material=lambda x, z: int(z < 2.0))
        m = K.Model(mesh, order=order, materials={0: K.Material.acoustic(1500.0, 1000.0), 1: K.FAST}, dt=1e-9,
                    regions=[(0.0, 1.0, 3.0, 4.0, 1)] if kind == "hanging" else [])
    m.n_steps = 1
    return K.build(m, stable_dt=1.0)


@pytest.mark.parametrize("order", range(1, 9))
@pytest.mark.parametrize("kind", ["plain", "hanging", "dipole"])
def test_maps_and_forces(pkg, oracle, order, kind):
    import torch

    from insem_b200 import kernels, native as N

    prob = _problem(order, kind)
    rng = np.random.default_rng(order)
    side = torch.cuda.Stream()
    with pkg.Solver(prob) as s:
        for i, d in enumerate(prob.domains):
            u = rng.uniform(-1, 1, d.ncomp * d.n_global).astype(np.float32)
            loc = rng.uniform(-1, 1, d.ncomp * d.l2g.size).astype(np.float32)
            u_dev, l_in = torch.from_numpy(u).cuda(), torch.from_numpy(loc).cuda()
            l_out, g_out, f_out = torch.empty_like(l_in), torch.empty_like(u_dev), torch.empty_like(u_dev)
            dofs = kernels.DofMapKernel(prob.ngll, d)

            def calls(stream):
                dofs.gather_device(d.ncomp, u_dev.data_ptr(), l_out.data_ptr(), stream)
                dofs.assemble_device(d.ncomp, l_in.data_ptr(), g_out.data_ptr(), stream)
                N.check(N.lib().insem_cuda_solver_internal_forces_noalloc(
                    s._h, i, C.c_void_p(u_dev.data_ptr()), C.c_void_p(f_out.data_ptr()), C.c_void_p(stream)))

            def check(scale):
                torch.cuda.synchronize()
                us = (u * np.float32(scale)).astype(np.float32)
                assert np.array_equal(l_out.cpu().numpy(), oracle.gather(prob, i, us))
                assert np.array_equal(g_out.cpu().numpy(), oracle.assemble(prob, i, loc))
                assert np.array_equal(f_out.cpu().numpy(), oracle.OracleSolver(prob).internal_forces(i, us))

            torch.cuda.synchronize()
            calls(side.cuda_stream)
            check(1.0)
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=side):
                u_dev.mul_(2.0)  # a caller's kernel ahead of the seam's
                calls(side.cuda_stream)
            for k in (1, 2):
                graph.replay()
                check(2.0 ** k)
