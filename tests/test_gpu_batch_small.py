"""Batches without a cutoff: many small systems are swept, larger ones go through the pair-tensor product, and an
uneven batch takes the side that costs less in all.  Launches tell the two apart: one sweep, or several kernels."""
import numpy as np
import pytest

from oracle import oracle as O
from threebodymdalgorithms_b200 import Context

pytestmark = pytest.mark.gpu

TOL = {"mixed": 1e-5, "fp64": 1e-12}


def batch(sizes):
    rng = np.random.default_rng(len(sizes))
    parts = []
    for n in sizes:
        m = max(1, int(np.ceil(n ** (1 / 3))))
        s = np.arange(n)
        parts.append(np.stack([s % m, s // m % m, s // (m * m)]) + rng.uniform(-0.2, 0.2, (3, n)))
    return np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64), np.ascontiguousarray(np.concatenate(parts, 1))


def launches(ctx, call):
    before = ctx.kernel_launches()
    out = call()
    return ctx.kernel_launches() - before, out


@pytest.mark.parametrize("precision,adjoint,sizes,product", [
    ("mixed", False, [8] * 60, False),
    ("mixed", False, [3, 0, 16, 1, 20] * 40, False),
    ("mixed", False, [40] * 20, True),
    ("mixed", False, [8] * 200 + [700], True),
    ("mixed", False, [3] * 400 + [60], False),
    ("fp64", False, [8] * 60, False),
    ("fp64", False, [30] * 20, True),
    ("mixed", True, [8] * 60, False),
    ("mixed", True, [32] * 12, False),
    ("mixed", True, [64] * 12, True),
])
def test_route_and_results(precision, adjoint, sizes, product):
    off, x = batch(sizes)
    g = np.random.default_rng(7).standard_normal(x.shape)
    ge = np.zeros(len(sizes))
    ctx, ref = Context("auta", precision), Context("auta", "fp64")
    if adjoint:
        count, out = launches(ctx, lambda: ctx.batch_adjoint(off, *x, *g, ge))
        want = ref.batch_adjoint(off, *x, *g, ge)  # the FP64 adjoint is always swept
    else:
        count, out = launches(ctx, lambda: ctx.batch_forces(off, *x))
    ctx.close()
    ref.close()
    assert (count > 2) == product
    for s, n in enumerate(sizes):
        a = slice(off[s], off[s + 1])
        got = np.stack([c[a] for c in out[:3]])
        if n < 3:
            assert not got.any()
            continue
        r = np.stack([c[a] for c in want[:3]]) if adjoint else \
            np.stack(O.forces(*np.ascontiguousarray(x[:, a]), 1.0, -1.0, nthreads=1)[:3])
        assert np.linalg.norm(got - r) <= TOL[precision] * np.linalg.norm(r)


@pytest.mark.parametrize("precision,n,product", [("mixed", 24, False), ("mixed", 31, True), ("fp64", 17, False), ("fp64", 24, True)])
def test_sizes_at_the_line(precision, n, product):
    """Planning a product on the host costs a system as much as the product gains at 24 particles."""
    off, x = batch([n] * 40)
    ctx = Context("auta", precision)
    count, out = launches(ctx, lambda: ctx.batch_forces(off, *x))
    ctx.close()
    assert (count > 2) == product
    want = np.concatenate([np.stack(O.forces(*np.ascontiguousarray(x[:, a:a + n]), 1.0, -1.0, nthreads=1)[:3])
                           for a in off[:-1]], 1)
    assert np.linalg.norm(np.stack(out[:3]) - want) <= TOL[precision] * np.linalg.norm(want)
