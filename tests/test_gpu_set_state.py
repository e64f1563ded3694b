"""set_state() again and again on one solver, each time followed at once by a
read of the state or by the first step: the values just set are the ones read."""

from __future__ import annotations

import ctypes as C
from concurrent.futures import ThreadPoolExecutor
from threading import Barrier

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(n, order=4):
    import insem_b200.cases as K

    mesh = K.layered((0.0, 1.0), [0.0, 1.0], [n], [0], nx=n)
    m = K.Model(mesh, order=order, materials={0: K.Material.acoustic(1500.0, 1000.0)}, dt=1e-9)
    m.n_steps = 2
    return K.build(m, stable_dt=1e-6)


# points: 81 and 10k (copied through the driver's buffer at once), 160k, 1.05M
# (read by ranges, without a numbering uploaded on the first read)
@pytest.mark.parametrize("path", [1, 2])
@pytest.mark.parametrize("n", [2, 25, 100, 256])
def test_values_set_are_the_values_read(pkg, n, path):
    prob = _problem(n)
    d = prob.domains[0]
    rng = np.random.default_rng(n)
    with pkg.Solver(prob, path=path) as s:
        for _ in range(8):
            u, v = rng.standard_normal((2, d.ncomp, d.n_global)).astype(np.float32).astype(np.float64)
            s.set_state("acoustic", u, v)
            got = s.state("acoustic")
            assert np.array_equal(got[0], u) and np.array_equal(got[1], v) and not got[2].any()


@pytest.mark.parametrize("path", [1, 2])
@pytest.mark.parametrize("n", [2, 25, 100])
def test_the_first_step_starts_from_the_values_set(pkg, oracle, n, path):
    prob = _problem(n)
    d = prob.domains[0]
    rng = np.random.default_rng(n)
    ref = oracle.OracleSolver(prob)
    with pkg.Solver(prob, path=path) as s:
        for _ in range(3):
            u, v = rng.standard_normal((2, d.ncomp, d.n_global))
            s.set_state("acoustic", u, v)
        ref.set_state("acoustic", u, v)
        s.run()
        ref.run()
        for x, y in zip(s.state("acoustic"), ref.state(0)):
            assert np.array_equal(x, y)


@pytest.mark.parametrize("path", [1, 2])
def test_several_threads_read_one_solver(pkg, path):
    """The first reads of a solver's state come from several threads at once."""
    prob, threads = _problem(100), 6
    d = prob.domains[0]
    u, v = np.random.default_rng(1).standard_normal((2, d.ncomp, d.n_global)).astype(np.float32).astype(np.float64)
    with ThreadPoolExecutor(threads) as pool:
        for _ in range(10):
            with pkg.Solver(prob, path=path) as s:
                s.set_state("acoustic", u, v)
                start = Barrier(threads)

                def read():
                    start.wait(30)
                    return s.state("acoustic")

                for got in [f.result() for f in [pool.submit(read) for _ in range(threads)]]:
                    assert np.array_equal(got[0], u) and np.array_equal(got[1], v) and not got[2].any()


class _PoolProps(C.Structure):  # CUmemPoolProps: pinned memory of device 0
    _fields_ = [("alloc_type", C.c_int), ("handle_types", C.c_int), ("location_type", C.c_int), ("location_id", C.c_int),
                ("security", C.c_void_p), ("max_size", C.c_size_t), ("rest", C.c_ubyte * 56)]


class _NoDeviceMemory:
    """The process's allocations come from a small pool that is used up."""

    def __enter__(self):
        import torch

        self.cu = C.CDLL("libcuda.so.1")
        self.default, self.pool, self.taken = C.c_void_p(), C.c_void_p(), []
        props = _PoolProps(1, 0, 1, 0, None, 32 << 20)
        assert self.cu.cuDeviceGetMemPool(C.byref(self.default), 0) == 0
        assert self.cu.cuMemPoolCreate(C.byref(self.pool), C.byref(props)) == 0
        assert self.cu.cuDeviceSetMemPool(0, self.pool) == 0
        for size in [1 << k for k in range(25, 8, -1)]:  # at most a few times 32 MB
            while len(self.taken) < 4096:
                p = C.c_uint64()
                if self.cu.cuMemAllocFromPoolAsync(C.byref(p), C.c_size_t(size), self.pool, None) != 0:
                    break
                self.taken.append(p)
        torch.cuda.synchronize()
        assert len(self.taken) < 4096
        return self

    def __exit__(self, *exc):
        import torch

        assert self.cu.cuDeviceSetMemPool(0, self.default) == 0
        torch.cuda.synchronize()
        for p in self.taken:
            self.cu.cuMemFreeAsync(p, None)
        torch.cuda.synchronize()
        self.cu.cuMemPoolDestroy(self.pool)


# points: 10k, 160k (one numbering kept on the device), 1.05M (sent in ranges)
@pytest.mark.parametrize("path", [1, 2])
@pytest.mark.parametrize("n", [25, 100, 256])
def test_a_full_device_can_be_read(pkg, n, path):
    prob = _problem(n)
    d = prob.domains[0]
    u, v = np.random.default_rng(n).standard_normal((2, d.ncomp, d.n_global)).astype(np.float32).astype(np.float64)
    with pkg.Solver(prob, path=path) as s:
        s.set_state("acoustic", u, v)
        with _NoDeviceMemory():
            got = s.state("acoustic")
        for got in (got, s.state("acoustic")):
            assert np.array_equal(got[0], u) and np.array_equal(got[1], v) and not got[2].any()
