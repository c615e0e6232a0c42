"""Nearly coincident particles in the mixed pair-tensor product, whose tensor's square passes the FP32 range."""
import numpy as np
import pytest

from threebodymdalgorithms_b200 import Context

pytestmark = pytest.mark.gpu


# particles of the first tile, of the two blocks of its pair of SMs, of two tiles, and the last two
@pytest.mark.parametrize("i, j", [(5, 17), (4, 5), (42, 83), (3, 200), (298, 299)])
@pytest.mark.parametrize("distance", [4e-6, 2e-7])
def test_close_pair(i, j, distance):
    """1e-5: the results are those of one pair, whose FP32 roundings do not average."""
    n = 300
    rng = np.random.default_rng(n)
    s = np.arange(n)
    x = np.stack([s % 7, s // 7 % 7, s // 49]) + rng.uniform(-0.2, 0.2, (3, n))
    x[:, j] = x[:, i] + distance * np.array([0.6, 0.0, -0.8])
    x, g = np.ascontiguousarray(x), rng.standard_normal((3, n))
    out = {}
    for precision in ("mixed", "fp64"):
        ctx = Context("auta", precision)
        ctx.set_particles(*x)
        f = ctx.forces()
        out[precision] = np.stack(f[:3]), np.array([f[3]]), np.stack(ctx.adjoint(*g)[:3])
        ctx.close()
    for got, want in zip(out["mixed"], out["fp64"]):
        assert np.isfinite(got).all()
        scale = np.abs(want).max()  # squares of H d leave FP64's comfortable range
        assert np.linalg.norm((got - want) / scale) <= 1e-5 * np.linalg.norm(want / scale)
