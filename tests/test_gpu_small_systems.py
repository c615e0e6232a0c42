"""Contexts that step several particle sets of one size, each in its own periodic domain (the captured step
holds the domain and the cell grid it was captured with), and small systems, whose long lists are dealt out
over several work items."""
import numpy as np
import pytest

from oracle import oracle as O
from threebodymdalgorithms_b200 import Context, generators

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("iters", [1, 9])
def test_steps_after_a_particle_set_of_another_domain(iters):
    n, g = 700, (0.0, -9.81, 0.0)
    ctx = Context("p3bca", "fp64", 1.5, 0.0001, g)
    for side in (8.0, 8.0, 12.0, 6.5, 8.0):
        st = generators.uniform(n, (side,) * 3, mass=1e6)
        ref, counts = O.simulate("p3bca", iters, st, 0.0001, g, cutoff=1.5, nthreads=0)
        for _ in range(2):  # launched one by one, then as a graph
            ctx.set_state(st)
            assert np.array_equal(ctx.step(iters), counts), side
            got = ctx.get_state()
            f = np.stack([got[k] for k in ("fx", "fy", "fz")])
            r = np.stack([ref[k] for k in ("fx", "fy", "fz")])
            assert np.linalg.norm(f - r) <= 1e-10 * np.linalg.norm(r), side
    ctx.close()


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("mixed", 1e-5)])
@pytest.mark.parametrize("n,side,cutoff", [(3, 2.0, 1.5), (40, 2.5, 1.2), (150, 3.2, 1.6), (330, 4.0, 1.3),
                                           (900, 6.5, 1.5), (1180, 7.0, 1.2), (1185, 7.0, 1.2), (600, 6.0, 3.1)])
def test_small_systems(precision, tol, n, side, cutoff):
    """Lists dealt out in parts (up to 1,180 particles in FP64, 1,660 mixed) and cells shared by blocks: lists
    of 0 to 600 entries, one to several 64-entry chunks, wrapping and not."""
    st = generators.uniform(n, (side,) * 3, seed0=n)
    ctx = Context("p3bca", precision, cutoff, nu=0.7)
    ctx.set_state(st)
    fx, fy, fz, e, c = ctx.forces()
    ctx.close()
    x, y, z = st["x"], st["y"], st["z"]
    L, lo = O.domain(x, y, z)
    rx, ry, rz, rc = O.forces(x, y, z, 0.7, cutoff, L, lo, nthreads=0)
    assert c == rc
    f, r = np.stack([fx, fy, fz]), np.stack([rx, ry, rz])
    assert np.linalg.norm(f - r) <= tol * max(np.linalg.norm(r), 1e-300)
