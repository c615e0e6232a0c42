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
