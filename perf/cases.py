"""The work that users of this package have it do, as cases that can be timed and compared.

Three kinds of program call the package:

  step    an MD program whose particles live in pinned host arrays: Context.step_host takes the state in,
          runs `iters` steps and gives the state back (positions, velocities, accelerations, forces, counts)
  field   a torch program that wants Axilrod-Teller forces and the energy of positions it has on the GPU,
          and, where it fits or optimises (`grad`), the gradients with respect to positions and strength.
          The FP64 form is used on float64 tensors; the mixed form, which works at FP32 accuracy, on
          float32 tensors, and its results go back into float32
  batch   force matching over many independent systems of uneven size (host arrays): one batched forward
          pass and one batched adjoint pass with the loss's cotangents; the mixed form's results feed a
          float32 model

`algorithm` is nata, auta (no cutoff) or p3bca (cutoff), `precision` fp64 or mixed.  Inputs are either
`uniform` (the generator's distribution), `liquid` (a cubic lattice with thermal disorder, which is what a
running simulation holds) or `clusters` (Gaussian clusters of unit width).  Densities are the 2.048 and 1
particles per unit volume of the repository's own workloads.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from threebodymdalgorithms_b200 import Context
from threebodymdalgorithms_b200.autograd import AxilrodTeller

DT, GRAVITY, NU = 0.001, (0.0, -9.81, 0.0), 1.0
IN = ("x", "y", "z", "vx", "vy", "vz", "ax", "ay", "az", "m")
OUT = ("x", "y", "z", "vx", "vy", "vz", "ax", "ay", "az", "m", "fx", "fy", "fz")


def listed():
    return [
        # the smallest whole run: 512 particles without a cutoff, one step, where latency counts
        dict(name="step_auta_fp64_512", kind="step", algorithm="auta", precision="fp64", n=512, cutoff=0.0,
             density=0.512, inputs="uniform", iters=1),
        # a small box with a cutoff (the size of the reference's own test fixture), a few steps per call
        dict(name="step_p3bca_fp64_1000", kind="step", algorithm="p3bca", precision="fp64", n=1000, cutoff=2.0,
             density=1.0, inputs="liquid", iters=5),
        # the main production run: 131,072 particles, cutoff 2, ten steps between two looks at the state
        dict(name="step_p3bca_mixed_131072", kind="step", algorithm="p3bca", precision="mixed", n=131072, cutoff=2.0,
             density=2.048, inputs="liquid", iters=10),
        # the same run in FP64 at the shorter cutoff of that workload
        dict(name="step_p3bca_fp64_131072", kind="step", algorithm="p3bca", precision="fp64", n=131072, cutoff=1.5,
             density=2.048, inputs="liquid", iters=10),
        # forces in a strongly clustered system: long neighbour lists, uneven work
        dict(name="field_p3bca_mixed_clusters_262144", kind="field", algorithm="p3bca", precision="mixed", n=262144,
             cutoff=2.0, density=1.0, inputs="clusters", grad=False),
        # forces of an odd-sized uniform system with a cutoff in FP64
        dict(name="field_p3bca_fp64_40013", kind="field", algorithm="p3bca", precision="fp64", n=40013, cutoff=2.0,
             density=2.048, inputs="uniform", grad=False),
        # a fit through the cutoff path: forward and backward
        dict(name="grad_p3bca_mixed_20011", kind="field", algorithm="p3bca", precision="mixed", n=20011, cutoff=2.0,
             density=2.048, inputs="uniform", grad=True),
        # all triplets of the largest no-cutoff workload, unique-triplet algorithm
        dict(name="field_auta_mixed_8192", kind="field", algorithm="auta", precision="mixed", n=8192, cutoff=0.0,
             density=1.024, inputs="uniform", grad=False),
        # all triplets seen from each particle, plain FP64, odd size
        dict(name="field_nata_fp64_4001", kind="field", algorithm="nata", precision="fp64", n=4001, cutoff=0.0,
             density=1.024, inputs="uniform", grad=False),
        # the same algorithm in mixed precision
        dict(name="field_nata_mixed_4096", kind="field", algorithm="nata", precision="mixed", n=4096, cutoff=0.0,
             density=1.024, inputs="uniform", grad=False),
        # force matching over 64 systems with a cutoff
        dict(name="batch_p3bca_mixed_64", kind="batch", algorithm="p3bca", precision="mixed", systems=64, nmin=512,
             nmax=4096, cutoff=2.0, density=2.048),
        # force matching over a few systems, all triplets
        dict(name="batch_auta_mixed_8", kind="batch", algorithm="auta", precision="mixed", systems=8, nmin=512,
             nmax=4096, cutoff=0.0, density=2.048),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "field", "field", "field", "batch"])
    algorithm = rng.choice(["p3bca", "p3bca", "auta", "nata"])
    cutoff = rng.choice([1.5, 2.0]) if algorithm == "p3bca" else 0.0
    if kind == "step":
        if algorithm == "p3bca":
            precision = rng.choice(["fp64", "mixed"])
            n = _log(rng, 1000 if precision == "fp64" else 20000, 131072)
            return dict(kind=kind, algorithm=algorithm, precision=precision, n=n, cutoff=cutoff, density=2.048,
                        inputs="liquid", iters=rng.randint(1, 10))
        return dict(kind=kind, algorithm=algorithm, precision="fp64", n=_log(rng, 100, 3000), cutoff=0.0,
                    density=1.024, inputs="liquid", iters=rng.randint(1, 3))
    if kind == "field":
        precision, grad = rng.choice(["fp64", "mixed"]), rng.random() < 0.4
        if algorithm == "p3bca":
            inputs = rng.choice(["uniform", "liquid", "clusters"])
            n = _log(rng, 1000, 65536 if inputs == "clusters" or grad else 131072)
            return dict(kind=kind, algorithm=algorithm, precision=precision, n=n, cutoff=cutoff,
                        density=1.0 if inputs == "clusters" else 2.048, inputs=inputs, grad=grad)
        return dict(kind=kind, algorithm=algorithm, precision=precision, n=_log(rng, 200, 2500 if grad else 4096),
                    cutoff=0.0, density=1.024, inputs=rng.choice(["uniform", "liquid"]), grad=grad)
    if algorithm == "p3bca":
        return dict(kind=kind, algorithm=algorithm, precision="mixed", systems=rng.randint(8, 64), nmin=512,
                    nmax=rng.randint(1024, 4096), cutoff=cutoff, density=2.048)
    return dict(kind=kind, algorithm="auta", precision="mixed", systems=rng.randint(2, 8), nmin=512,
                nmax=rng.randint(1024, 3000), cutoff=0.0, density=2.048)


# ---------------------------------------------------------------------------------------------
# inputs

def _side(n, density):
    return (n / density) ** (1.0 / 3.0)


def _positions(inputs, n, density, rng):
    """(n, 3) positions in a cube [0, side)."""
    side = _side(n, density)
    if inputs == "uniform":
        return rng.random((n, 3)) * side, side
    if inputs == "liquid":
        m = math.ceil(round(n ** (1.0 / 3.0), 9))
        a = side / m
        sites = np.sort(rng.permutation(m ** 3)[:n])
        lattice = np.stack([sites % m, (sites // m) % m, sites // (m * m)], 1).astype(np.float64)
        return (lattice + 0.5 + rng.uniform(-0.2, 0.2, (n, 3))) * a, side
    clusters = max(1, n // 1024)
    centres = 3.0 + rng.random((clusters, 3)) * (side - 6.0)
    x = centres[np.arange(n) % clusters] + rng.standard_normal((n, 3))
    return np.clip(x, 0.0, side * (1 - 1e-9)), side


def _step_state(case, seed):
    """The 10 input arrays of a step, as rows of one pinned host block."""
    rng = np.random.default_rng(seed)
    n = case["n"]
    x, _ = _positions(case["inputs"], n, case["density"], rng)
    block = torch.empty((10, n), dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy()
    block[0:3] = x.T
    block[3:6] = 0.1 * rng.standard_normal((3, n))
    block[6:9] = 0.0
    block[9] = 1.0
    return block


def _field_positions(case, seed):
    x, side = _positions(case["inputs"], case["n"], case["density"], np.random.default_rng(seed))
    dtype = torch.float64 if case["precision"] == "fp64" else torch.float32
    return torch.from_numpy(x).to(dtype), side


def _field_cotangents(case, seed):
    rng = np.random.default_rng(seed + 1000003)
    return torch.from_numpy(rng.standard_normal((case["n"], 3))), 0.5


def _batch_inputs(case, seed):
    """Packed systems (uneven sizes; the sizes themselves belong to the data set, not to the seed)."""
    sizes = np.random.default_rng(12345).integers(case["nmin"], case["nmax"] + 1, case["systems"])
    rng = np.random.default_rng(seed)
    offsets = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    sides = np.array([_side(int(n), case["density"]) for n in sizes])
    pos = np.concatenate([_positions("liquid", int(n), case["density"], rng)[0] for n in sizes])
    cot = rng.standard_normal((len(pos), 3))
    box = np.repeat(sides, 3)
    return offsets, np.ascontiguousarray(pos.T), np.ascontiguousarray(cot.T), box, np.zeros(3 * len(sizes))


# ---------------------------------------------------------------------------------------------
# one pass

def prepare(case, seed):
    if case["kind"] == "step":
        block, n = _step_state(case, seed), case["n"]
        out = torch.empty((13, n), dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy()
        ctx = Context(case["algorithm"], case["precision"], case["cutoff"], DT, GRAVITY, NU)
        return {"kind": "step", "ctx": ctx, "state": dict(zip(IN, block)), "iters": case["iters"],
                "out": dict(zip(OUT, out), id=np.zeros(n, dtype=np.int32))}
    if case["kind"] == "field":
        x, side = _field_positions(case, seed)
        at = AxilrodTeller(case["algorithm"], case["precision"], case["cutoff"], box=(side,) * 3, lo=(0.0,) * 3)
        x = x.cuda().requires_grad_(case["grad"])
        state = {"kind": "field", "at": at, "x": x, "grad": case["grad"],
                 "nu": torch.tensor(NU, dtype=torch.float64, device="cuda", requires_grad=case["grad"])}
        if case["grad"]:
            gf, ge = _field_cotangents(case, seed)
            state["cot"] = [gf.cuda(), torch.tensor(ge, dtype=torch.float64, device="cuda")]
        return state
    offsets, pos, cot, box, lo = _batch_inputs(case, seed)
    ctx = Context(case["algorithm"], case["precision"], case["cutoff"], nu=NU)
    return {"kind": "batch", "ctx": ctx, "offsets": offsets, "pos": pos, "cot": cot, "box": box, "lo": lo,
            "ge": np.zeros(len(offsets) - 1)}


def run(state):
    if state["kind"] == "step":
        res, counts = state["ctx"].step_host(state["state"], state["iters"], out=state["out"])
        return {"state": {k: res[k] for k in OUT}, "counts": counts.astype(np.int64)}
    if state["kind"] == "field":
        x = state["x"]
        f, e = state["at"](x, state["nu"])
        out = {"f": f.detach().to(x.dtype), "e": e.detach().to(x.dtype)}
        if state["grad"]:
            out["gx"], gnu = torch.autograd.grad([f, e], [x, state["nu"]], state["cot"])
            out["gnu"] = gnu.to(x.dtype)
        return out
    ctx, offsets, (x, y, z) = state["ctx"], state["offsets"], state["pos"]
    fx, fy, fz, e, counts = ctx.batch_forces(offsets, x, y, z, state["box"], state["lo"])
    gx, gy, gz, gnu = ctx.batch_adjoint(offsets, x, y, z, *state["cot"], state["ge"], state["box"], state["lo"])
    as32 = [a.astype(np.float32) for a in (fx, fy, fz, gx, gy, gz, e, gnu)]
    return {"f": as32[0:3], "g": as32[3:6], "e": as32[6], "gnu": as32[7], "counts": counts.astype(np.int64)}


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without

def _triplets(n, cutoff, density, inputs):
    """Expected triplets: all of them, or those of a uniform system with every side within the cutoff (the
    chance that two points of a ball of radius c are within c is 15/32), or dense clusters of 1024."""
    if cutoff <= 0:
        return n * (n - 1) * (n - 2) / 6
    if inputs == "clusters":
        return n / 1024 * 1024 ** 3 / 6 * 0.15
    near = density * 4.0 / 3.0 * math.pi * cutoff ** 3
    return n * near * near / 6 * 15 / 32


def work(case):
    """120 floating-point operations per triplet for energy and forces, three times that for the adjoint."""
    if case["kind"] == "batch":
        sizes = np.random.default_rng(12345).integers(case["nmin"], case["nmax"] + 1, case["systems"])
        t = sum(_triplets(int(n), case["cutoff"], case["density"], "liquid") for n in sizes)
        return {"bytes": float(sizes.sum()) * 8 * 15, "flops": t * 480}
    t = _triplets(case["n"], case["cutoff"], case["density"], case["inputs"])
    if case["kind"] == "step":
        return {"bytes": case["n"] * 8.0 * 23, "flops": t * 120 * case["iters"]}
    item = 8.0 if case["precision"] == "fp64" else 4.0
    return {"bytes": case["n"] * item * (12 if case["grad"] else 6), "flops": t * (480 if case["grad"] else 120)}


# ---------------------------------------------------------------------------------------------
# the same results in plain 64-bit torch

def _dense(x):
    """All triplets at strength 1, (forces, energy): with T_ij = (3 r r^T - r^2) / r^5 the energy of a triplet
    is -tr(T_ij T_jk T_ki) / 3, so the total is -tr(T^3) / 18 and the force on i sums (T T)_ij : dT_ij / 3."""
    n = len(x)
    r = x[None, :, :] - x[:, None, :]
    eye = torch.eye(n, dtype=x.dtype, device=x.device)
    r2 = (r * r).sum(-1) + eye
    i3 = (1.0 - eye) / (r2 * r2.sqrt())
    i5 = i3 / r2
    unit = torch.eye(3, dtype=x.dtype, device=x.device)
    t = 3.0 * i5[..., None, None] * r[..., :, None] * r[..., None, :] - i3[..., None, None] * unit
    m = t.permute(0, 2, 1, 3).reshape(3 * n, 3 * n)
    g = m @ m
    e = -(g * m).sum() / 18.0
    g = g.reshape(n, 3, n, 3).permute(0, 2, 1, 3)
    gr = (g * r[..., None, :]).sum(-1) + (g * r[..., :, None]).sum(-2)
    rgr = 0.5 * (gr * r).sum(-1)
    tr = g.diagonal(dim1=-2, dim2=-1).sum(-1)
    h = 3.0 * i5[..., None] * gr + (3.0 * i5 * tr - 15.0 * rgr * i5 / r2)[..., None] * r
    return h.sum(1) / 3.0, e


def _triple(xi, xj, xk):
    """(force on j, force on k, energy) of triplets at strength 1; the force on i is minus their sum."""
    u, v, w = xj - xi, xk - xi, xk - xj
    a, b, c = (u * u).sum(-1), (v * v).sum(-1), (w * w).sum(-1)
    p, q, s = (u * v).sum(-1), (u * w).sum(-1), (v * w).sum(-1)
    x = a * b * c
    t2 = 1.0 / x
    t3 = t2 / x.sqrt()
    d = p * q * s * t2
    m = -3.0 * t2 * t3
    b2 = m * (1.0 - 5.0 * d)
    alpha = b2 * b * c + m * (q * s - p * s - p * q)
    beta = b2 * a * c + m * (q * s + p * s + p * q)
    gamma = m * (q * s + p * s - p * q) - b2 * a * b
    fj = alpha[:, None] * u + gamma[:, None] * w
    fk = beta[:, None] * v - gamma[:, None] * w
    return fj, fk, (t3 * (1.0 - 3.0 * d)).sum()


def _near(xa, xb, box, cutoff):
    d = (xb - xa).abs()
    m = torch.minimum(d, box - d)
    m = m * m
    return (m[..., 0] + m[..., 1]) + m[..., 2] <= cutoff * cutoff


def _half_list(x, box, cutoff):
    """Pairs i < j within the cutoff, sorted by i."""
    n, rows, cols = len(x), [], []
    order = torch.argsort(x[:, 2])
    step = 512
    for s in range(0, n, step):
        own = order[s:s + step]
        lo, hi = x[own[0], 2], x[own[-1], 2]
        dz = (x[:, 2] - 0.5 * (lo + hi)).abs()
        cand = torch.nonzero(torch.minimum(dz, (box[2] - dz).abs()) <= cutoff * 1.01 + 0.5 * (hi - lo)).flatten()
        hit = _near(x[own][:, None, :], x[cand][None, :, :], box, cutoff) & (own[:, None] < cand[None, :])
        a, b = torch.nonzero(hit, as_tuple=True)
        rows.append(own[a])
        cols.append(cand[b])
    rows, cols = torch.cat(rows), torch.cat(cols)
    o = torch.argsort(rows, stable=True)
    return rows[o], cols[o]


def _cut_triplets(x, box, cutoff, chunk=6_000_000):
    """Chunks (i, j, k) of all triplets with every side within the cutoff; None if there are far too many."""
    rows, cols = _half_list(x, box, cutoff)
    n = len(x)
    length = torch.bincount(rows, minlength=n)
    start = torch.cumsum(length, 0) - length
    place = torch.arange(len(rows), device=x.device) - start[rows]
    later = length[rows] - place - 1  # partners after this entry in the same list
    total = torch.cumsum(later, 0)
    if len(total) == 0:
        return
    bounds, at, ends = [0], 0, total.cpu().numpy()
    while at < len(ends):
        base = 0 if at == 0 else int(ends[at - 1])
        at = max(at + 1, int(np.searchsorted(ends, base + chunk, side="right")))
        bounds.append(min(at, len(ends)))
    for a, b in zip(bounds[:-1], bounds[1:]):
        rep = later[a:b]
        e = torch.repeat_interleave(torch.arange(a, b, device=x.device), rep)
        off = torch.arange(len(e), device=x.device) - torch.repeat_interleave(torch.cumsum(rep, 0) - rep, rep)
        i, j, k = rows[e], cols[e], cols[e + 1 + off]
        keep = _near(x[j], x[k], box, cutoff)
        yield i[keep], j[keep], k[keep]


def _cut(x, box, cutoff, direction=None):
    """(forces, energy, count[, H direction]) at strength 1 with the cutoff."""
    f, h = torch.zeros_like(x), torch.zeros_like(x)
    e, count = x.new_zeros(()), 0
    for i, j, k in _cut_triplets(x, box, cutoff):
        count += len(i)
        if direction is None:
            fj, fk, de = _triple(x[i], x[j], x[k])
        else:
            (fj, fk, de), (hj, hk, _) = torch.func.jvp(_triple, (x[i], x[j], x[k]),
                                                        (direction[i], direction[j], direction[k]))
            h.index_add_(0, j, hj).index_add_(0, k, hk).index_add_(0, i, -(hj + hk))
        f.index_add_(0, j, fj).index_add_(0, k, fk).index_add_(0, i, -(fj + fk))
        e = e + de
    return (f, e, count) if direction is None else (f, e, count, h)


def _all(x, direction=None):
    count = len(x) * (len(x) - 1) * (len(x) - 2) // 6
    if direction is None:
        return (*_dense(x), count)
    (f, e), (h, _) = torch.func.jvp(_dense, (x,), (direction,))
    return f, e, count, h


def _evaluate(case, x, box, direction=None):
    return _cut(x, box, case["cutoff"], direction) if case["cutoff"] > 0 else _all(x, direction)


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if case["kind"] == "step":
        block = torch.from_numpy(np.array(_step_state(case, seed))).to(dev)
        x, v, a, m = block[0:3].T.contiguous(), block[3:6].T.contiguous(), block[6:9].T.contiguous(), block[9]
        box = (x.max(0).values + 0.0001) - (x.min(0).values - 0.0001)
        g = torch.tensor(GRAVITY, dtype=x.dtype, device=dev)
        counts = []
        for _ in range(case["iters"]):
            x = (x + v * DT) + a[:, 0:1] * (DT * DT * 0.5)  # the x acceleration on every axis, as the reference has it
            f, _, count = _evaluate(case, x, box)
            a = g - f / m[:, None]
            v = v + a * (DT * 0.5)
            counts.append(count)
        cols = [c.cpu().numpy() for c in (*x.T, *v.T, *a.T, m, *f.T)]
        return {"state": dict(zip(OUT, cols)), "counts": np.array(counts, dtype=np.int64)}
    if case["kind"] == "field":
        x, side = _field_positions(case, seed)
        x = x.to(dev).double()
        box = torch.full((3,), side, dtype=x.dtype, device=dev)
        if not case["grad"]:
            f, e, _ = _evaluate(case, x, box)
            return {"f": f * NU, "e": e * NU}
        gf, ge = _field_cotangents(case, seed)
        gf = gf.to(dev)
        f, e, _, h = _evaluate(case, x, box, gf)
        return {"f": f * NU, "e": e * NU, "gx": NU * (h + ge * f), "gnu": (gf * f).sum() + ge * e}
    offsets, pos, cot, sides, _ = _batch_inputs(case, seed)
    x, d = (torch.from_numpy(a.T.copy()).to(dev) for a in (pos, cot))
    fs, hs, es, gnu, counts = [], [], [], [], []
    for s in range(len(offsets) - 1):
        b, t = int(offsets[s]), int(offsets[s + 1])
        box = torch.full((3,), float(sides[3 * s]), dtype=x.dtype, device=dev)
        f, e, count, h = _evaluate(case, x[b:t].contiguous(), box, d[b:t].contiguous())
        fs.append(f)
        hs.append(h)
        es.append(float(e))
        gnu.append(float((d[b:t] * f).sum()))
        counts.append(count)
    f, h = torch.cat(fs).cpu().numpy(), torch.cat(hs).cpu().numpy()
    return {"f": [f[:, k] for k in range(3)], "g": [h[:, k] for k in range(3)], "e": np.array(es),
            "gnu": np.array(gnu), "counts": np.array(counts, dtype=np.int64)}
