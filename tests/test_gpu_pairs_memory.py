"""Evaluations without a cutoff where the pair-tensor workspace is not to be had: the sweep gives the results, in
every call that takes the product otherwise, and the product is taken again for the next sizes that fit."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle as O
from threebodymdalgorithms_b200 import Context

pytestmark = pytest.mark.gpu

TOL = {"mixed": 1e-5, "fp64": 1e-12}


def set_most(ctx, size):
    f = ctx._lib.tbmd_probe_pair_workspace
    f.restype, f.argtypes = C.c_int, [C.c_void_p, C.c_int64]
    assert f(ctx.handle, size) == 0


def positions(n):
    m = int(np.ceil(n ** (1 / 3)))
    s = np.arange(n)
    return np.ascontiguousarray(np.stack([s % m, s // m % m, s // (m * m)]) +
                                np.random.default_rng(n).uniform(-0.2, 0.2, (3, n)))


def close(got, want, tol):
    return np.linalg.norm(np.stack(got) - np.stack(want)) <= tol * np.linalg.norm(np.stack(want))


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("algo", ["auta", "nata"])
def test_sweep_without_a_workspace(algo, precision):
    tol = TOL[precision]
    sizes = [400, 330]
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    x = [positions(n) for n in sizes]
    g = [np.random.default_rng(n).standard_normal((3, n)) for n in sizes]
    want = [O.forces(*p, 1.0, -1.0, nthreads=0)[:3] for p in x]
    ctx, full = Context(algo, precision, dt=1e-6), Context("auta", "fp64")
    for most in (0, 1 << 62, 0):
        set_most(ctx, most)
        for p, q, w in zip(x, g, want):
            ctx.set_particles(*p)
            full.set_particles(*p)
            assert close(ctx.forces()[:3], w, tol)
            assert close(ctx.adjoint(*q)[:3], full.adjoint(*q)[:3], tol)
            assert ctx.step(9).tolist() == [len(q[0]) * (len(q[0]) - 1) * (len(q[0]) - 2) // 6] * 9
        for p, q in ((np.concatenate(x, 1), np.concatenate(g, 1)),):
            for _ in range(2):
                b = ctx.batch_forces(off, *p)
                assert close(b[:3], [np.concatenate(c) for c in zip(*want)], tol)
                assert close(ctx.batch_adjoint(off, *p, *q, np.zeros(2))[:3],
                             full.batch_adjoint(off, *p, *q, np.zeros(2))[:3], tol)
    ctx.close()
    full.close()


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_kernels_that_ran(precision):
    """One sweep, or the product's several kernels."""
    x = positions(500)
    ctx = Context("auta", precision)
    used = []
    for n, most in ((500, 0), (500, 1 << 62), (499, 1 << 62), (500, 1000)):
        set_most(ctx, most)
        ctx.set_particles(*np.ascontiguousarray(x[:, :n]))
        before = ctx.kernel_launches()
        ctx.forces()
        used.append(ctx.kernel_launches() - before)
    ctx.close()
    assert used[0] == used[1] == used[3] < used[2]  # unchanged sizes are not tried again
