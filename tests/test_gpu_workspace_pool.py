"""Workspaces that closed contexts leave for later ones: bounded, given back, and never shared by two contexts."""
import threading

import numpy as np
import pytest

from threebodymdalgorithms_b200 import Context
from threebodymdalgorithms_b200._lib import trim

pytestmark = pytest.mark.gpu

MB = 1 << 20


def positions(n, seed=0):
    m = int(np.ceil(n ** (1 / 3)))
    s = np.arange(n)
    rng = np.random.default_rng(n + 1000 * seed)
    return np.stack([s % m, s // m % m, s // (m * m)]) + rng.uniform(-0.2, 0.2, (3, n))


def forces(precision, x):
    ctx = Context("auta", precision)
    ctx.set_particles(*x)
    f = np.stack(ctx.forces()[:3])
    ctx.close()
    return f


def free_memory():
    import torch

    torch.cuda.synchronize()
    return torch.cuda.mem_get_info(0)[0]


def test_bounded_and_given_back():
    trim()
    first = forces("fp64", positions(512))  # kernels loaded
    trim()
    before = free_memory()
    assert np.array_equal(forces("fp64", positions(512)), first)
    kept = before - free_memory()
    assert 16 * MB <= kept <= 64 * MB  # 25 MB of tensors, and the results
    for n in (600, 300, 700, 512, 456, 800, 512, 1500, 150, 640):
        forces("fp64", positions(n))
        forces("mixed", positions(n))
        assert before - free_memory() <= 144 * MB  # 128, in the driver's granules
    assert np.array_equal(forces("fp64", positions(512)), first)
    trim()
    assert before - free_memory() <= 4 * MB
    trim()


def test_contexts_alive_at_once_share_nothing():
    """Four threads, each with contexts of its own that come and go."""
    sizes = [512, 500, 490, 480]
    want = {(p, n): forces(p, positions(n, 1)) for p in ("fp64", "mixed") for n in sizes}
    wrong = []

    def work(k):
        try:
            for q in range(6):
                p, n = ("fp64", "mixed")[(k + q) % 2], sizes[(k + q) % 4]
                a, b = Context("auta", p), Context("auta", p)
                for c in (a, b):
                    c.set_particles(*positions(n, 1))
                for _ in range(3):
                    for c in (a, b):
                        if not np.array_equal(np.stack(c.forces()[:3]), want[p, n]):
                            wrong.append((k, q))
                a.close()
                b.close()
        except Exception as e:  # reported by the assertion below
            wrong.append((k, repr(e)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
    trim()
