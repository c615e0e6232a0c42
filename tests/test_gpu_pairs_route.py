"""Which evaluations go through the pair-tensor product, as the library tells it (bench.py names the kernel by it)."""
import ctypes as C
import json
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

from threebodymdalgorithms_b200 import Context

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]


@pytest.mark.parametrize("algo,cutoff,n,product", [("auta", 0.0, 127, 0), ("auta", 0.0, 128, 1), ("nata", 0.0, 500, 1),
                                                   ("p3bca", 0.0, 500, 1), ("p3bca", 1.5, 500, 0)])
def test_route(algo, cutoff, n, product):
    ctx = Context(algo, "fp64", cutoff)
    ctx.set_particles(*np.random.default_rng(n).uniform(0.0, 8.0, (3, n)))
    ctx.forces()
    ctx._lib.tbmd_probe_pairs.argtypes = [C.c_void_p]
    assert ctx._lib.tbmd_probe_pairs(ctx.handle) == product
    ctx.close()


@pytest.mark.parametrize("workload,kernel", [("c1", "k_p64_gemm"), ("c3", "k_p3bca")])
def test_bench_names_the_kernel(workload, kernel):
    out = subprocess.run([sys.executable, str(ROOT / "bench.py"), "--workload", workload, "--precision", "fp64",
                          "--steps", "3", "--warmup", "3", "--no-e2e", "--no-cpu-baseline", "--no-autotune"],
                         capture_output=True, text=True, timeout=300, cwd=ROOT)
    assert out.returncode == 0, out.stderr[-2000:]
    assert json.loads(out.stdout.strip().splitlines()[-1])["roofline"]["kernel"] == kernel


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("mixed", 1e-5)])
def test_product_and_both_sweeps_agree(precision, tol):
    """8,192 uniform particles: AUTA and NATA both take the product, so the sweeps are asked for by leaving them no
    workspace."""
    from threebodymdalgorithms_b200 import generators

    st = generators.uniform(8192, (20.0,) * 3)
    out = {}
    for name, algo, most in (("product", "auta", 1 << 62), ("auta", "auta", 0), ("nata", "nata", 0)):
        ctx = Context(algo, precision)
        f = ctx._lib.tbmd_probe_pair_workspace
        f.restype, f.argtypes = C.c_int, [C.c_void_p, C.c_int64]
        assert f(ctx.handle, most) == 0
        ctx.set_state(st)
        r = ctx.forces()
        assert ctx._lib.tbmd_probe_pairs(ctx.handle) == (name == "product")
        ctx.close()
        out[name] = np.stack(r[:3])
    for name in ("auta", "nata"):
        assert np.linalg.norm(out["product"] - out[name]) <= tol * np.linalg.norm(out[name]), name
