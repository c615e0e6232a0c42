"""The mixed no-cutoff forces as a product of pair tensors, at the sizes where its tiling can go wrong: the
edges of the 42-particle row blocks, of the 84-particle column blocks and of the ranges of k, against the
FP64 oracle.

Tolerance: an entry of G = T T is cut off twice and rounded at most 48 times (2 * 2^-23 + 48 * 2^-24 of its
partial sums, 3.1e-6), and its contraction with dT/dr rounds fewer than 18 times (1.1e-6)."""
import numpy as np
import pytest

from oracle import oracle as O
from threebodymdalgorithms_b200 import Context

pytestmark = pytest.mark.gpu

TOL = 4.2e-6


def lattice(n, seed, scale=1.0):
    """n particles on a disordered cubic lattice of unit spacing, off the origin."""
    rng = np.random.default_rng(seed)
    m = int(np.ceil(n ** (1 / 3)))
    s = np.sort(rng.permutation(m ** 3)[:n])
    x = np.stack([s % m, s // m % m, s // (m * m)]) + rng.uniform(-0.2, 0.2, (3, n)) + 5.0
    return np.ascontiguousarray(x * scale)


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("algo", ["auta", "nata"])
@pytest.mark.parametrize("n", [128, 129, 167, 168, 169, 252, 253, 383, 385, 420, 513, 769])
def test_pair_tensor_forces(algo, n):
    x, y, z = lattice(n, n)
    ctx = Context(algo, "mixed", nu=1.3)
    ctx.set_particles(x, y, z)
    fx, fy, fz, e, c = ctx.forces()
    again = ctx.forces()
    ctx.close()
    rx, ry, rz, rc = O.forces(x, y, z, 1.3, -1.0, nthreads=0)
    assert c == rc
    assert rel(np.stack([fx, fy, fz]), np.stack([rx, ry, rz])) <= TOL
    assert abs(e - O.energy(x, y, z, 1.3, -1.0)) <= TOL * O.energy_abs(x, y, z, 1.3, -1.0)
    assert all(np.array_equal(a, b) for a, b in zip((fx, fy, fz, e), again))  # fixed order of summation


def test_pair_tensor_batch_of_uneven_systems():
    sizes = [1, 84, 2, 0, 300, 43, 3, 42, 85, 126, 500]
    offsets = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    pos = np.concatenate([lattice(n, 7 + n) for n in sizes if n], 1)
    ctx = Context("auta", "mixed")
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
        assert rel(f, np.stack([rx, ry, rz])) <= TOL, n
        assert abs(e[s] - O.energy(x, y, z, 1.0, -1.0)) <= TOL * O.energy_abs(x, y, z, 1.0, -1.0), n


@pytest.mark.parametrize("scale", [0.05, 30.0])
def test_pair_tensor_range_of_lengths(scale):
    """Pair tensors from 1 / 30^3 / 9^3 to 1 / 0.03^3: the same forces up to the scale's power."""
    x, y, z = lattice(300, 3, scale)
    ctx = Context("nata", "mixed")
    ctx.set_particles(x, y, z)
    f = np.stack(ctx.forces()[:3])
    ctx.close()
    assert rel(f, np.stack(O.forces(x, y, z, 1.0, -1.0, nthreads=0)[:3])) <= TOL
