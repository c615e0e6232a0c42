"""No-cutoff evaluations on streams that are destroyed with the work still in flight, so that a later stream can have
the same handle: each evaluation's results are those of its own positions."""
import ctypes as C

import numpy as np
import pytest

from threebodymdalgorithms_b200 import Context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,n", [("mixed", 1500), ("fp64", 900), ("fp64", 120)])
def test_streams_destroyed_in_flight(precision, n):
    import torch

    cuda = C.CDLL("libcuda.so.1")
    rng = np.random.default_rng(n)
    m = int(np.ceil(n ** (1 / 3)))
    s = np.arange(n)
    sites = np.stack([s % m, s // m % m, s // (m * m)])
    x = torch.tensor(np.stack([sites + rng.uniform(-0.2, 0.2, (3, n)) for _ in range(8)]), device="cuda")
    ctx = Context("auta", precision)

    def run(k, out, stream):
        p, f = x[k], out[k]
        ctx.forces_device(n, *[C.c_void_p(r.data_ptr()) for r in (*p, *f)], None, None, stream=stream)

    want, got = torch.zeros_like(x), torch.zeros_like(x)
    for k in range(len(x)):
        run(k, want, C.c_void_p(1))
        torch.cuda.synchronize()
    for _ in range(5):
        got.zero_()
        torch.cuda.synchronize()
        for k in range(len(x)):
            stream = C.c_void_p()
            assert cuda.cuStreamCreate(C.byref(stream), 1) == 0
            run(k, got, stream)
            assert cuda.cuStreamDestroy_v2(stream) == 0
        torch.cuda.synchronize()
        if precision == "mixed" or n >= 128:  # in a fixed order of summation
            assert torch.equal(got, want)
        else:
            assert float((got - want).norm() / want.norm()) <= 1e-12
    ctx.close()
