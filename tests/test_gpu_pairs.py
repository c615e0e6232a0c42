"""The no-cutoff forces as a product of pair tensors, at the sizes where its tiling can go wrong: the edges of
the row blocks (42 particles mixed, 32 FP64), of the column blocks (84, 64) and of the ranges of k, against
the FP64 oracle.

Tolerance, FP64: 1e-12, as for every FP64 evaluation.  Mixed: an entry of G = T T is cut off twice and rounded at most 48 times (2 * 2^-23 + 48 * 2^-24 of its
partial sums, 3.1e-6), and its contraction with dT/dr rounds fewer than 18 times (1.1e-6)."""
import numpy as np
import pytest

from oracle import oracle as O
from threebodymdalgorithms_b200 import Context

pytestmark = pytest.mark.gpu

TOL = {"mixed": 4.2e-6, "fp64": 1e-12}
PRECISIONS = ["mixed", "fp64"]


def lattice(n, seed, scale=1.0):
    """n particles on a disordered cubic lattice of unit spacing, off the origin."""
    rng = np.random.default_rng(seed)
    m = int(np.ceil(n ** (1 / 3)))
    s = np.sort(rng.permutation(m ** 3)[:n])
    x = np.stack([s % m, s // m % m, s // (m * m)]) + rng.uniform(-0.2, 0.2, (3, n)) + 5.0
    return np.ascontiguousarray(x * scale)


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("algo", ["auta", "nata"])
@pytest.mark.parametrize("n", [128, 129, 167, 168, 169, 192, 193, 252, 253, 256, 383, 385, 420, 513, 769])
def test_pair_tensor_forces(algo, n, precision):
    x, y, z = lattice(n, n)
    ctx = Context(algo, precision, nu=1.3)
    ctx.set_particles(x, y, z)
    fx, fy, fz, e, c = ctx.forces()
    again = ctx.forces()
    ctx.close()
    rx, ry, rz, rc = O.forces(x, y, z, 1.3, -1.0, nthreads=0)
    assert c == rc
    assert rel(np.stack([fx, fy, fz]), np.stack([rx, ry, rz])) <= TOL[precision]
    assert abs(e - O.energy(x, y, z, 1.3, -1.0)) <= TOL[precision] * O.energy_abs(x, y, z, 1.3, -1.0)
    assert all(np.array_equal(a, b) for a, b in zip((fx, fy, fz, e), again))  # fixed order of summation


@pytest.mark.parametrize("n", [299, 300, 336, 337, 385, 504, 513, 640])
def test_pair_tensor_adjoint(n):
    """The mixed adjoint (H g and the strength's gradient) against the FP64 one, within the 1e-5 that every
    mixed adjoint is held to; the same in every run."""
    x, y, z = lattice(n, n)
    g = np.random.default_rng(n).standard_normal((3, n))
    out = {}
    for precision in ("fp64", "mixed", "mixed"):
        ctx = Context("auta", precision, nu=0.8)
        ctx.set_particles(x, y, z)
        h = ctx.adjoint(*g, 0.3)
        st = ctx.get_state()
        ctx.close()
        r = (np.stack(h[:3]), h[3], np.stack([st[k] for k in ("fx", "fy", "fz")]))
        if precision in out and n >= 300:
            assert all(np.array_equal(a, b) for a, b in zip(r, out[precision]))
        out[precision] = r
    (hm, num, fm), (h, nu, f) = out["mixed"], out["fp64"]
    assert rel(hm, h) <= 1e-5
    assert rel(fm, f) <= 1e-5
    assert abs(num - nu) <= 1e-5 * (np.abs(g * f).sum() + abs(nu))


@pytest.mark.parametrize("precision", PRECISIONS)
def test_pair_tensor_batch_of_uneven_systems(precision):
    sizes = [1, 84, 2, 0, 300, 43, 3, 42, 85, 126, 500]
    offsets = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    pos = np.concatenate([lattice(n, 7 + n) for n in sizes if n], 1)
    ctx = Context("auta", precision)
    fx, fy, fz, e, counts = ctx.batch_forces(offsets, *pos)
    ctx.close()
    for s, n in enumerate(sizes):
        sl = slice(offsets[s], offsets[s + 1])
        f = np.stack([fx[sl], fy[sl], fz[sl]])
        if n < 3:
            assert not f.any() and e[s] == 0.0 and counts[s] == 0
            continue
        x, y, z = (np.ascontiguousarray(p[sl]) for p in pos)
        rx, ry, rz, rc = O.forces(x, y, z, 1.0, -1.0, nthreads=0)
        assert counts[s] == rc
        assert rel(f, np.stack([rx, ry, rz])) <= TOL[precision], n
        assert abs(e[s] - O.energy(x, y, z, 1.0, -1.0)) <= TOL[precision] * O.energy_abs(x, y, z, 1.0, -1.0), n


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("scale", [0.05, 30.0])
def test_pair_tensor_range_of_lengths(scale, precision):
    """Pair tensors from 1 / 30^3 / 9^3 to 1 / 0.03^3: the same forces up to the scale's power."""
    x, y, z = lattice(300, 3, scale)
    ctx = Context("nata", precision)
    ctx.set_particles(x, y, z)
    f = np.stack(ctx.forces()[:3])
    ctx.close()
    assert rel(f, np.stack(O.forces(x, y, z, 1.0, -1.0, nthreads=0)[:3])) <= TOL[precision]


@pytest.mark.parametrize("algo,precision,tol", [("auta", "fp64", 1e-12), ("nata", "mixed", 1e-5)])
def test_fits_that_do_not_wait(algo, precision, tol):
    """Forward and backward of several sizes, issued without waiting on two streams: each call's work lists,
    tables and workspaces are those of its own size while earlier ones still run."""
    import torch

    from threebodymdalgorithms_b200.autograd import AxilrodTeller

    sizes = [100, 489, 100, 300, 127, 700]
    at = AxilrodTeller(algo, precision)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    got, want = [], []
    for q, n in enumerate(sizes):
        x = torch.tensor(lattice(n, n).T.copy(), device="cuda", requires_grad=True)
        nu = torch.tensor(1.1, dtype=torch.float64, device="cuda", requires_grad=True)
        torch.cuda.synchronize()
        with torch.cuda.stream(streams[q % 2]):
            f, e = at(x, nu)
            got.append((f, e, *torch.autograd.grad([f.square().sum() + e], [x, nu])))
    torch.cuda.synchronize()
    for n in sizes:
        x = torch.tensor(lattice(n, n).T.copy(), device="cuda", requires_grad=True)
        nu = torch.tensor(1.1, dtype=torch.float64, device="cuda", requires_grad=True)
        f, e = AxilrodTeller(algo, "fp64")(x, nu)
        want.append((f, e, *torch.autograd.grad([f.square().sum() + e], [x, nu])))
        torch.cuda.synchronize()
    for n, g, w in zip(sizes, got, want):
        for a, b in zip(g, w):
            assert float((a - b).detach().norm()) <= tol * max(float(b.detach().norm()), 1e-300), n


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("n", [451, 577, 600, 801, 1025])
def test_ranges_that_split_a_system_evenly(n, precision):
    """Sizes whose ranges of k are an even split (160 to 416 particles) with a shorter last one; the tolerance
    is that of the other ranges, as none is longer than 512."""
    x, y, z = lattice(n, n)
    ctx = Context("auta", precision, nu=1.3)
    ctx.set_particles(x, y, z)
    fx, fy, fz, e, c = ctx.forces()
    ctx.close()
    rx, ry, rz, rc = O.forces(x, y, z, 1.3, -1.0, nthreads=0)
    assert c == rc
    assert rel(np.stack([fx, fy, fz]), np.stack([rx, ry, rz])) <= TOL[precision]
    assert abs(e - O.energy(x, y, z, 1.3, -1.0)) <= TOL[precision] * O.energy_abs(x, y, z, 1.3, -1.0)
