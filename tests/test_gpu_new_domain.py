"""A context that steps several particle sets of one size: each in its own periodic domain (the step's
captured graph holds the domain and the cell grid it was captured with)."""
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
