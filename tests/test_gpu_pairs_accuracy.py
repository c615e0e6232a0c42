"""How far the pair-tensor products are from sums in wider arithmetic."""
import numpy as np
import pytest

from threebodymdalgorithms_b200 import Context

pytestmark = pytest.mark.gpu


def lattice(n, seed):
    """n particles on a disordered cubic lattice of unit spacing."""
    rng = np.random.default_rng(seed)
    m = int(np.ceil(n ** (1 / 3)))
    s = np.sort(rng.permutation(m ** 3)[:n])
    return np.ascontiguousarray(np.stack([s % m, s // m % m, s // (m * m)]) + rng.uniform(-0.2, 0.2, (3, n)))


def tensors(r):
    """T = (3 r r^T - r^2) / r^5 of pair vectors r (.., 3); zero where r is."""
    r2 = (r * r).sum(-1)
    r2 = np.where(r2 > 0, r2, np.inf)
    i3 = 1 / (r2 * np.sqrt(r2))
    eye = np.eye(3, dtype=r.dtype)
    return 3 * (i3 / r2)[..., None, None] * r[..., :, None] * r[..., None, :] - i3[..., None, None] * eye


def forces_of(x, some):
    """Forces at strength 1 on the particles `some`, in 80-bit arithmetic: sum_j (T T)_ij : dT_ij / 3."""
    p = x.T.astype(np.longdouble)
    n, m = len(p), len(some)
    r = p[None] - p[some][:, None]
    a = tensors(r).transpose(0, 2, 1, 3).reshape(3 * m, 3 * n)
    b = tensors(p[None] - p[:, None]).transpose(0, 2, 1, 3).reshape(3 * n, 3 * n)
    g = (a @ b).reshape(m, 3, n, 3).transpose(0, 2, 1, 3)
    r2 = (r * r).sum(-1)
    r2 = np.where(r2 > 0, r2, np.inf)
    h = (g * r[..., None, :]).sum(-1) + (g * r[..., :, None]).sum(-2)  # 2 sym(G) r
    q, tr = (h * r).sum(-1) / 2, g[..., 0, 0] + g[..., 1, 1] + g[..., 2, 2]
    i5 = 1 / (r2 * r2 * np.sqrt(r2))
    return (i5[..., None] * (h + (tr - 5 * q / r2)[..., None] * r)).sum(1)


@pytest.mark.parametrize("n", [150, 300, 700, 1300])
def test_fp64_forces_are_as_accurate_as_sums_over_triplets(n):
    """5.5e-16 is the largest error that the FP64 sum over each particle's triplets has on thermal lattices."""
    x = lattice(n, n)
    some = np.random.default_rng(1).permutation(n)[:40]
    want = forces_of(x, some)
    ctx = Context("nata", "fp64")
    ctx.set_particles(*x)
    got = np.stack(ctx.forces()[:3], 1)[some].astype(np.longdouble)
    ctx.close()
    assert float(np.linalg.norm(got - want) / np.linalg.norm(want)) <= 5.5e-16


# The mixed form.  Relative errors of thermal lattices are 1.3e-7 .. 2.2e-7 in the forces and in H d; one of the
# small products left out would be 4e-6 off, a rounding instead of the compensation of the tensor core's truncation
# 6.4e-8 in the mean.
MIXED = 5e-7


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("n", [130, 420, 1000, 2500])
def test_mixed_forces(n):
    x = lattice(n, n)
    out = {}
    for precision in ("mixed", "fp64"):
        ctx = Context("auta", precision)
        ctx.set_particles(*x)
        out[precision] = np.stack(ctx.forces()[:3])
        ctx.close()
    assert rel(out["mixed"], out["fp64"]) <= MIXED


def test_mixed_adjoint_over_several_launches():
    """2,500 particles take two launches of 256 MB of tensors, whose H d are added up."""
    n = 2500
    x, g = lattice(n, n), np.random.default_rng(n).standard_normal((3, n))
    out = {}
    for precision in ("mixed", "fp64"):
        ctx = Context("auta", precision, nu=0.8)
        ctx.set_particles(*x)
        h = ctx.adjoint(*g, 0.3)
        out[precision] = np.stack(h[:3]), h[3]
        ctx.close()
    (hm, num), (h, nu) = out["mixed"], out["fp64"]
    assert rel(hm, h) <= MIXED
    assert abs(num - nu) <= MIXED * np.linalg.norm(g) * np.linalg.norm(h)


def test_mixed_batch_adjoint_over_several_launches():
    """Uneven systems, one of which begins in one launch and ends in the next."""
    sizes = [700, 43, 2500, 301, 0, 3, 1200]
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    x = np.ascontiguousarray(np.concatenate([lattice(n, 3 + n) for n in sizes if n], 1))
    g, ge = np.random.default_rng(0).standard_normal(x.shape), np.linspace(-0.4, 0.5, len(sizes))
    ctx = Context("auta", "mixed", nu=0.8)
    out = ctx.batch_adjoint(off, *x, *g, ge)
    fwd = ctx.batch_forces(off, *x)
    ctx.close()
    for s, n in enumerate(sizes):
        a = slice(off[s], off[s + 1])
        got = np.stack([c[a] for c in out[:3]])
        if n < 3:
            assert not got.any()
            continue
        one = Context("auta", "fp64", nu=0.8)
        one.set_particles(*np.ascontiguousarray(x[:, a]))
        h = one.adjoint(*np.ascontiguousarray(g[:, a]), ge[s])
        f = one.forces()
        one.close()
        tol = MIXED if n > 100 else 1e-5  # few triplets: the errors do not average
        assert rel(got, np.stack(h[:3])) <= tol, n
        assert rel(np.stack([c[a] for c in fwd[:3]]), np.stack(f[:3])) <= tol, n
        assert abs(out[3][s] - h[3]) <= tol * np.linalg.norm(g[:, a]) * np.linalg.norm(np.stack(h[:3])), n


def test_mixed_results_have_no_bias():
    """Mean of the signed errors over lattices, within half of the compensation (6.45e-8) of none: without it, or with
    its sign reversed, the means are 6.45e-8 or twice that off."""
    bias = {"f": [], "e": [], "h": []}
    for n in (300, 350, 512, 700, 1000, 1400):
        x, g = lattice(n, n + 1), np.random.default_rng(n).standard_normal((3, n))
        out = []
        for precision in ("mixed", "fp64"):
            ctx = Context("auta", precision)
            ctx.set_particles(*x)
            f = ctx.forces()
            out.append((np.stack(f[:3]), f[3], np.stack(ctx.adjoint(*g)[:3])))
            ctx.close()
        (fm, em, hm), (f, e, h) = out
        bias["f"].append(float((fm * f).sum() / (f * f).sum()) - 1)
        bias["e"].append(em / e - 1)
        bias["h"].append(float((hm * h).sum() / (h * h).sum()) - 1)
    for k, v in bias.items():
        assert abs(np.mean(v)) <= 3.2e-8, (k, v)
