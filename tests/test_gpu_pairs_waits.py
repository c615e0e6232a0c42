"""A wait inside the pair-tensor kernels that runs out: every call with a status reports TBMD_TIMEOUT, the device
calls give NaN in all floating outputs, and the next evaluation is right again.  The limit of the waits is set to
zero, so that each block gives up at its first wait."""
import ctypes as C

import numpy as np
import pytest

from threebodymdalgorithms_b200 import Context
from threebodymdalgorithms_b200._lib import TbmdError

pytestmark = pytest.mark.gpu

TIMEOUT = 6


def set_limit(ctx, cycles):
    f = ctx._lib.tbmd_probe_pair_waits
    f.restype, f.argtypes = C.c_int, [C.c_void_p, C.c_int64]
    assert f(ctx.handle, cycles) == 0


def positions(n):
    m = int(np.ceil(n ** (1 / 3)))
    s = np.arange(n)
    return np.stack([s % m, s // m % m, s // (m * m)]) + np.random.default_rng(n).uniform(-0.2, 0.2, (3, n))


def status_of(call):
    with pytest.raises(TbmdError) as e:
        call()
    return e.value.status


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_host_calls_report_the_wait(precision):
    n = 333
    x = positions(n)
    g = np.random.default_rng(0).standard_normal((3, n))
    off = np.array([0, n], dtype=np.int64)
    ctx = Context("auta", precision, dt=1e-6)
    ctx.set_particles(*x)
    f = ctx.forces()
    batch = ctx.batch_forces(off, *x)
    calls = [ctx.forces, lambda: ctx.step(1), lambda: ctx.step(9), lambda: ctx.batch_forces(off, *x)]
    if precision == "mixed":  # the FP64 adjoint is a sweep, which waits for nothing
        h = ctx.adjoint(*g)
        calls += [lambda: ctx.adjoint(*g), lambda: ctx.batch_adjoint(off, *x, *g, np.zeros(1))]
    for call in calls:
        set_limit(ctx, 0)
        assert status_of(call) == TIMEOUT
        set_limit(ctx, 4_000_000_000)
        ctx.set_particles(*x)
        assert all(np.array_equal(a, b) for a, b in zip(ctx.forces(), f))
        assert all(np.array_equal(a, b) for a, b in zip(ctx.batch_forces(off, *x), batch))
    if precision == "mixed":
        assert all(np.array_equal(a, b) for a, b in zip(ctx.adjoint(*g), h))
    ctx.close()


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_device_calls_give_nan(precision):
    import torch

    n = 333
    x = torch.tensor(positions(n), device="cuda")
    g = torch.tensor(np.random.default_rng(0).standard_normal((3, n)), device="cuda")
    out, e = torch.zeros((6, n), dtype=torch.float64, device="cuda"), torch.zeros(1, dtype=torch.float64, device="cuda")
    ptr = lambda t: [C.c_void_p(r.data_ptr()) for r in t]
    stream = C.c_void_p(1)
    ctx = Context("auta", precision)

    def forces():
        ctx.forces_device(n, *ptr(x), *ptr(out[:3]), C.c_void_p(e.data_ptr()), None, stream=stream)
        torch.cuda.synchronize()
        return out[:3].clone(), e.clone()

    def adjoint():
        ctx.adjoint_device(n, [*ptr(x), *ptr(g), C.c_void_p(0), *ptr(out[:3]), C.c_void_p(e.data_ptr()), *ptr(out[3:])],
                           stream=stream)
        torch.cuda.synchronize()
        return out.clone(), e.clone()

    for call in [forces, adjoint] if precision == "mixed" else [forces]:
        want = call()
        assert all(bool(torch.isfinite(t).all()) for t in want)
        set_limit(ctx, 0)
        assert all(bool(torch.isnan(t).all()) for t in call())
        set_limit(ctx, 4_000_000_000)
        assert all(torch.equal(a, b) for a, b in zip(call(), want))
    ctx.close()
