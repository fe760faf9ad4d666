"""The work that users of this package have it do, as timed cases through its public entry
points: products with the truncated Gaussian operator, evaluation of an interpolant, solves
for the weights (plain FP64 and mixed precision, 2D and 3D, one and several right-hand
sides, batches of problems), the packed FP32 product and the training of the learned guess.

Widths are box widths in units of sigma, as in the package: 2D cells of 8 sigma with a one-
cell buffer and a cutoff 8 sigma past the cell's edge (batches: cells of 4 sigma), 3D cells
of 3 sigma with a 7 sigma buffer box and a cutoff 7 sigma past the edge. Points are lattices
over [-1, 1]^d with +-0.25 h of seeded jitter, sigma = h / overlap.
"""
import math

import numpy as np
import torch

from petrbf_gb300 import learned
from petrbf_gb300 import workloads as W
from petrbf_gb300.api import (Context, GaussianOperator, batch_interpolate, gpumatmult,
                              rbf_interpolation, vorticity_evaluation)

EPS = 1e-6  # the absolute slack of the cell grid and of the box tests

WIDTHS = {2: (8, 24, 24), 3: (3, 7, 17)}  # cell, Schwarz buffer box, truncation box
BATCH_WIDTHS = (4, 12, 20)


def listed():
    return [
        # one operator product of a small host program: 2500 points, host vectors
        {"name": "product_2d_small", "kind": "operator", "dim": 2, "m": 50, "overlap": 0.8},
        # the matvec inside a caller's own Krylov loop, at the headline size (4x10^6 points),
        # vectors on the device in the caller's order
        {"name": "product_2d_large", "kind": "product", "dim": 2, "m": 2000, "overlap": 0.8},
        # the same in 3D, 884736 points
        {"name": "product_3d", "kind": "product", "dim": 3, "m": 96, "overlap": 0.8},
        # the interpolant of 4.9x10^5 particles read at 3x10^5 scattered positions
        {"name": "evaluate_2d", "kind": "evaluate", "dim": 2, "m": 700, "nt": 300007, "overlap": 0.8},
        # the reference driver's own problem size in one call, context and all
        {"name": "solve_2d_1e4", "kind": "solve_once", "dim": 2, "m": 100, "overlap": 0.8},
        # a plain FP64 solve of a time step, 1.6x10^5 points, the context kept
        {"name": "solve_2d_fp64", "kind": "solve", "dim": 2, "m": 397, "nrhs": 1, "precision": "fp64",
         "pc": "rasm", "guess": "zero", "overlap": 0.8},
        # the largest solve: 4x10^6 points, mixed precision from the learned guess
        {"name": "solve_2d_mixed_large", "kind": "solve", "dim": 2, "m": 2000, "nrhs": 1, "precision": "mixed",
         "pc": "rasm", "guess": "learned", "overlap": 0.8},
        # a vortex ring's three components in lockstep, mixed precision, basic Schwarz
        {"name": "solve_3d_mixed", "kind": "solve", "dim": 3, "m": 56, "nrhs": 3, "precision": "mixed",
         "pc": "asm", "guess": "zero", "overlap": 0.8},
        # the same ring, coarser, in plain FP64
        {"name": "solve_3d_fp64", "kind": "solve", "dim": 3, "m": 26, "nrhs": 3, "precision": "fp64",
         "pc": "asm", "guess": "zero", "overlap": 0.8},
        # many independent problems of uneven size in one call
        {"name": "batch_2d", "kind": "batch", "nprob": 24, "nmin": 2000, "nmax": 120000, "precision": "fp64",
         "overlap": 0.8},
        # the reference's packed FP32 product, as its host code calls it
        {"name": "packed_fp32_2d", "kind": "packed", "m": 700},
        # two epochs of training of the guess network on the patches of one problem
        {"name": "train_guess", "kind": "train", "m": 300, "epochs": 2, "batch": 512},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["operator", "product", "product", "evaluate", "solve_once", "solve", "solve", "solve",
                       "batch", "packed", "train"])
    overlap = round(rng.uniform(0.8, 1.0), 3)
    dim = rng.choice([2, 3])
    if kind == "operator":
        return {"kind": kind, "dim": dim, "m": _log_int(rng, 30, 400) if dim == 2 else _log_int(rng, 10, 40),
                "overlap": overlap}
    if kind == "product":
        return {"kind": kind, "dim": dim, "m": _log_int(rng, 100, 2000) if dim == 2 else _log_int(rng, 16, 96),
                "overlap": overlap}
    if kind == "evaluate":
        return {"kind": kind, "dim": dim, "m": _log_int(rng, 60, 1000) if dim == 2 else _log_int(rng, 16, 64),
                "nt": _log_int(rng, 500, 500000 if dim == 2 else 100000), "overlap": overlap}
    if kind == "solve_once":
        return {"kind": kind, "dim": 2, "m": _log_int(rng, 40, 200), "overlap": overlap}
    if kind == "solve":
        precision = rng.choice(["fp64", "mixed"])
        if dim == 2:
            return {"kind": kind, "dim": 2, "m": _log_int(rng, 100, 450 if precision == "fp64" else 1400),
                    "nrhs": rng.choice([1, 1, 2, 3]), "precision": precision, "pc": "rasm",
                    "guess": rng.choice(["zero", "learned"]) if precision == "mixed" else "zero",
                    "overlap": overlap}
        return {"kind": kind, "dim": 3, "m": _log_int(rng, 12, 26 if precision == "fp64" else 48),
                "nrhs": rng.choice([1, 2, 3]), "precision": precision, "pc": "asm", "guess": "zero",
                "overlap": overlap}
    if kind == "batch":
        return {"kind": kind, "nprob": rng.randint(4, 24), "nmin": 2000, "nmax": _log_int(rng, 8000, 120000),
                "precision": rng.choice(["fp64", "mixed"]), "overlap": overlap}
    if kind == "packed":
        return {"kind": kind, "m": _log_int(rng, 40, 700)}
    return {"kind": "train", "m": _log_int(rng, 60, 300), "epochs": rng.randint(1, 2),
            "batch": rng.choice([256, 500, 512])}


# ---- inputs ---------------------------------------------------------------------------

def _points(dim, m, rng):
    """m^dim jittered lattice over [-1, 1]^dim: coordinates (z None in 2D) and h."""
    h = 2.0 / m
    k = -1.0 + h * np.arange(m)
    axes = np.meshgrid(*([k] * dim), indexing="ij")
    c = [a.ravel() + rng.uniform(-0.25 * h, 0.25 * h, a.size) for a in axes]
    return c[0], c[1], (c[2] if dim == 3 else None), h


def _field(x, y, z, nrhs, rng):
    """Right-hand sides: Lamb-Oseen vortices in 2D, the components of a vortex ring in 3D
    (the third is identically zero)."""
    if z is None:
        cols = []
        for _ in range(nrhs):
            gam, rc = rng.uniform(0.5, 2.0), rng.uniform(0.1, 0.3)
            xc, yc = rng.uniform(-0.5, 0.5, 2)
            cols.append(gam / (math.pi * rc * rc) * np.exp(-((x - xc) ** 2 + (y - yc) ** 2) / (rc * rc)))
        return cols[0] if nrhs == 1 else np.stack(cols, axis=1)
    w = W.vortex_ring(x, y, z, R=rng.uniform(0.4, 0.6), a=rng.uniform(0.1, 0.15))
    return w[0].copy() if nrhs == 1 else np.stack(w[:nrhs], axis=1)


def _problem(case, seed, nrhs=1):
    rng = np.random.default_rng(seed)
    x, y, z, h = _points(case["dim"], case["m"], rng)
    return rng, x, y, z, h / case["overlap"], _field(x, y, z, nrhs, rng), h


def _batch_problems(case, seed):
    # sizes from the case alone, so that every seed's batch is the same amount of work
    n = case["nprob"]
    sizes = np.exp(np.linspace(math.log(case["nmin"]), math.log(case["nmax"]), n))
    spread = np.random.default_rng(n).permutation(n) / max(n - 1, 1)
    rng = np.random.default_rng(seed)
    out = []
    for k in range(n):
        x, y, _, h = _points(2, max(8, int(round(math.sqrt(sizes[k])))), rng)
        ov = case["overlap"] + (1.0 - case["overlap"]) * spread[k]
        out.append({"x": x, "y": y, "f": _field(x, y, None, 1, rng), "sigma": h / ov, "nsigma_box": BATCH_WIDTHS[0],
                    "sigma_buffer": BATCH_WIDTHS[1], "sigma_trunc": BATCH_WIDTHS[2]})
    return out


def _evaluation(case, seed):
    rng, x, y, z, sigma, f, h = _problem(case, seed)
    g = f * h ** case["dim"]  # the size and shape of a solved field's weights
    t = [rng.uniform(-1.0, 1.0, case["nt"]) for _ in range(case["dim"])]
    return t, [x, y] + ([z] if z is not None else []), g, sigma


def _vector(case, seed):
    """A Krylov vector: the field with noise of its own size."""
    rng, x, y, z, sigma, f, _ = _problem(case, seed)
    return x, y, z, sigma, f / np.linalg.norm(f) + rng.standard_normal(f.size) / math.sqrt(f.size)


def _context(case, sigma, **opts):
    nb, nbuf, nt = WIDTHS[case["dim"]]
    return Context(dim=case["dim"], sigma=sigma, nsigma_box=nb, sigma_buffer=nbuf, sigma_trunc=nt, **opts)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "operator":
        x, y, z, sigma, v = _vector(case, seed)
        return {"kind": kind, "op": GaussianOperator(x, y, z, sigma, *WIDTHS[case["dim"]]), "v": v}
    if kind == "product":
        x, y, z, sigma, v = _vector(case, seed)
        ctx = _context(case, sigma)
        ctx.matvec_setup(x, y, z)
        v = torch.from_numpy(v).cuda()
        out = torch.empty_like(v)
        torch.cuda.synchronize()
        return {"kind": kind, "ctx": ctx, "v": v, "out": out}
    if kind == "evaluate":
        t, s, g, sigma = _evaluation(case, seed)
        return {"kind": kind, "args": (*t, *s, g, sigma, *WIDTHS[case["dim"]])}
    if kind == "solve_once":
        _, x, y, _, sigma, f, _ = _problem(case, seed)
        return {"kind": kind, "args": (x, y, f, sigma, *WIDTHS[2])}
    if kind == "solve":
        _, x, y, z, sigma, f, _ = _problem(case, seed, case["nrhs"])
        ctx = _context(case, sigma, precision=case["precision"], pc=case["pc"], guess=case["guess"])
        if case["guess"] == "learned":
            learned.install(ctx)
        return {"kind": kind, "ctx": ctx, "args": (x, y, z, f)}
    if kind == "batch":
        return {"kind": kind, "problems": _batch_problems(case, seed), "precision": case["precision"]}
    if kind == "packed":
        tx, ty, sx, sy, sg, off, sigma, _ = W.pack_gpumatmult_2d(case["m"], seed)
        return {"kind": kind, "args": (tx, ty, None, sx, sy, None, sg, off, float(sigma))}
    if kind == "train":
        rng = np.random.default_rng(seed)
        x, y, _, h = _points(2, case["m"], rng)
        f = _field(x, y, None, 1, rng)
        with Context(dim=2, sigma=h / 0.8, nsigma_box=8, sigma_buffer=24, sigma_trunc=24) as ctx:
            X, _, T, M = learned.patches(ctx, x, y, f, f * h * h)
        return {"kind": kind, "net": learned.Network(seed=seed), "data": (X, T, M), "epochs": case["epochs"],
                "batch": case["batch"], "seed": seed}
    raise ValueError("unknown kind %r" % (kind,))


def run(state):
    kind = state["kind"]
    if kind == "operator":
        return state["op"] @ state["v"]
    if kind == "product":
        state["ctx"].matvec_dev(state["v"].data_ptr(), state["out"].data_ptr())
        return state["out"]
    if kind == "evaluate":
        return vorticity_evaluation(*state["args"])
    if kind == "solve_once":
        return rbf_interpolation(*state["args"])[0]
    if kind == "solve":
        return state["ctx"].interpolate(*state["args"])[0]
    if kind == "batch":
        return batch_interpolate(state["problems"], precision=state["precision"])[0]
    if kind == "packed":
        return gpumatmult(*state["args"])
    net = state["net"]
    loss = net.train(*state["data"], epochs=state["epochs"], batch=state["batch"], seed=state["seed"])
    return {"loss": loss, "weights": net.weights}


# ---- work -----------------------------------------------------------------------------

def _counts(dim, n, overlap, widths, m=None):
    """Ordered pairs of a product, and multiply-adds (x 2) of the blocks' Cholesky."""
    m = m or n ** (1.0 / dim)
    h, sigma = 2.0 / m, 2.0 / m / overlap
    cells = max(1.0, 2.0 / (widths[0] * sigma)) ** dim
    inside = lambda width: min(n, (width * sigma / h) ** dim)  # noqa: E731
    return n * inside(widths[2]), cells * inside(widths[1]) ** 3 / 3.0


def work(case):
    """Inputs read once and outputs written once, and the arithmetic of one pass: 15
    operations a pair of a product (the reference's count), one product and one block
    factorisation for a solve, whose number of iterations is the method's own."""
    kind = case["kind"]
    if kind in ("operator", "product"):
        dim, n = case["dim"], case["m"] ** case["dim"]
        pairs, _ = _counts(dim, n, case["overlap"], WIDTHS[dim])
        return {"bytes": 8 * (dim + 2) * n, "flops": 15 * pairs}
    if kind == "evaluate":
        dim, n = case["dim"], case["m"] ** case["dim"]
        pairs, _ = _counts(dim, n, case["overlap"], WIDTHS[dim])
        return {"bytes": 8 * (dim + 1) * (n + case["nt"]), "flops": 15 * pairs / n * case["nt"]}
    if kind in ("solve", "solve_once"):
        dim, n, nrhs = case["dim"], case["m"] ** case["dim"], case.get("nrhs", 1)
        pairs, chol = _counts(dim, n, case["overlap"], WIDTHS[dim])
        return {"bytes": 8 * (dim + 2 * nrhs) * n, "flops": 15 * pairs + chol}
    if kind == "batch":
        flops = by = 0
        for n in np.exp(np.linspace(math.log(case["nmin"]), math.log(case["nmax"]), case["nprob"])):
            pairs, chol = _counts(2, n, case["overlap"], BATCH_WIDTHS)
            flops, by = flops + 15 * pairs + chol, by + 32 * n
        return {"bytes": int(by), "flops": flops}
    if kind == "packed":
        cells = max(1, (case["m"] * 0.8 / 8)) ** 2
        return {"bytes": int(cells * (128 * 12 + 900 * 12)), "flops": 12 * cells * 128 * 900}
    patches = case["m"] ** 2 / 6.25
    params = learned.param_count()
    return {"bytes": int(4 * patches * (learned.IN + 2 * learned.OUT) + 8 * params),
            "flops": 6 * params * patches * case["epochs"]}


# ---- 64-bit values --------------------------------------------------------------------

def _grid(coords, sigma, nb):
    """Cell edge, lower corner and cell counts of the grid over all given points."""
    box = nb * sigma + EPS
    lo = [float(min(c[k].min() for c in coords)) - EPS for k in range(len(coords[0]))]
    hi = [float(max(c[k].max() for c in coords)) + EPS for k in range(len(coords[0]))]
    return box, lo, [int(math.ceil((b - a) / box)) for a, b in zip(lo, hi)]


def _cells(pts, box, lo, dims):
    return [torch.floor((p - a) / box).long().clamp_(0, d - 1) for p, a, d in zip(pts, lo, dims)]


def _table(idx, dims):
    """Points of each cell as rows of indices, padded with the point count."""
    flat = idx[0]
    for i, d in zip(idx[1:], dims[1:]):
        flat = flat * d + i
    ncell = int(np.prod(dims))
    order = torch.argsort(flat, stable=True)
    count = torch.bincount(flat, minlength=ncell)
    start = torch.cumsum(count, 0) - count
    tab = torch.full((ncell, int(count.max())), len(flat), dtype=torch.long, device=flat.device)
    tab[flat[order], torch.arange(len(flat), device=flat.device) - start[flat[order]]] = order
    return tab


def _gauss_sum(tgt, src, g, sigma, nb, nt):
    """The truncated Gaussian sum at tgt of the sources src with weights g: a source counts
    when it lies within the truncation box of the target's cell, or in that cell."""
    dev = torch.device("cuda")
    box, lo, dims = _grid([tgt, src], sigma, nb)
    T = [torch.as_tensor(np.asarray(t, np.float64), device=dev) for t in tgt]
    S = [torch.as_tensor(np.asarray(s, np.float64), device=dev) for s in src]
    G = torch.cat([torch.as_tensor(np.asarray(g, np.float64), device=dev), torch.zeros(1, device=dev).double()])
    length, reach = nt * sigma / 2 + EPS, int(math.ceil((nt - nb + EPS) / 2 / nb))
    ti, si = _cells(T, box, lo, dims), _cells(S, box, lo, dims)
    ttab, stab = _table(ti, dims), _table(si, dims)
    far = torch.full((1,), 1e30, device=dev, dtype=torch.float64)
    T = [torch.cat([t, far * 0]) for t in T]
    S = [torch.cat([s, far]) for s in S]
    ncell = ttab.shape[0]
    ids = torch.arange(ncell, device=dev)
    at, rest = [], ids
    for d in reversed(dims):
        at.insert(0, rest % d)
        rest = rest // d
    acc = torch.zeros(ncell, ttab.shape[1], device=dev, dtype=torch.float64)
    chunk = max(1, int(4e7 // (ttab.shape[1] * stab.shape[1])))
    offsets = [()]
    for _ in dims:
        offsets = [o + (k,) for o in offsets for k in range(-reach, reach + 1)]
    for off in offsets:
        there = [a + k for a, k in zip(at, off)]
        ok = torch.ones(ncell, dtype=torch.bool, device=dev)
        for p, d in zip(there, dims):
            ok &= (p >= 0) & (p < d)
        rows = ids[ok]
        other = torch.zeros_like(rows)
        for p, d in zip(there, dims):
            other = other * d + p[ok]
        for a in range(0, len(rows), chunk):
            r, s = rows[a:a + chunk], stab[other[a:a + chunk]]
            w = G[s]
            if any(off):  # (all of the target's own cell counts)
                for k in range(len(dims)):
                    centre = lo[k] + (at[k][r].double() + 0.5) * box
                    w = torch.where((S[k][s] - centre[:, None]).abs() < length, w, 0.0)
            d2 = 0.0
            for k in range(len(dims)):
                diff = T[k][ttab[r]][:, :, None] - S[k][s][:, None, :]
                d2 = d2 + diff * diff
            acc[r] += torch.bmm(torch.exp(d2 * (-1.0 / (2.0 * sigma * sigma))), w[:, :, None])[:, :, 0]
    out = torch.empty(len(tgt[0]) + 1, device=dev, dtype=torch.float64)
    out[ttab.reshape(-1)] = acc.reshape(-1)
    return out[:-1] / (2.0 * math.pi * sigma * sigma)


def _dense_solve(pts, f, sigma, nb, nt):
    """Weights of the truncated Gaussian system, assembled densely and solved by LU with
    one step of refinement."""
    dev = torch.device("cuda")
    box, lo, dims = _grid([pts], sigma, nb)
    P = [torch.as_tensor(p, device=dev) for p in pts]
    idx = _cells(P, box, lo, dims)
    length = nt * sigma / 2 + EPS
    d2 = sum((p[:, None] - p[None, :]) ** 2 for p in P)
    A = torch.exp_(d2.mul_(-1.0 / (2.0 * sigma * sigma))).div_(2.0 * math.pi * sigma * sigma)
    same = torch.ones_like(A, dtype=torch.bool)
    for i in idx:
        same &= i[:, None] == i[None, :]
    keep = torch.ones_like(same)
    for p, i, a in zip(P, idx, lo):
        keep &= (p[None, :] - (a + (i.double() + 0.5) * box)[:, None]).abs() < length
    A.mul_((keep | same).double())
    del same, keep
    b = torch.as_tensor(f, device=dev)
    b = b[:, None] if b.ndim == 1 else b
    lu, piv = torch.linalg.lu_factor(A)
    x = torch.linalg.lu_solve(lu, piv, b)
    x = x + torch.linalg.lu_solve(lu, piv, b - A @ x)
    return x[:, 0] if np.ndim(f) == 1 else x


def exact(case, seed):
    kind = case["kind"]
    if kind in ("operator", "product"):
        x, y, z, sigma, v = _vector(case, seed)
        pts = [x, y] + ([z] if z is not None else [])
        nb, _, nt = WIDTHS[case["dim"]]
        return _gauss_sum(pts, pts, v, sigma, nb, nt)
    if kind == "evaluate":
        t, s, g, sigma = _evaluation(case, seed)
        nb, _, nt = WIDTHS[case["dim"]]
        return _gauss_sum(t, s, g, sigma, nb, nt)
    if kind in ("solve", "solve_once"):
        n = case["m"] ** case["dim"]
        if n > 20000:
            return None  # a dense solve takes too long
        _, x, y, z, sigma, f, _ = _problem(case, seed, case.get("nrhs", 1))
        nb, _, nt = WIDTHS[case["dim"]]
        return _dense_solve([x, y] + ([z] if z is not None else []), f, sigma, nb, nt)
    if kind == "batch":
        out = []
        for q in _batch_problems(case, seed):
            small = q["x"].size <= 8000
            out.append(_dense_solve([q["x"], q["y"]], q["f"], q["sigma"], q["nsigma_box"], q["sigma_trunc"])
                       if small else None)
        return out
    if kind == "packed":
        tx, ty, sx, sy, sg, off, sigma, _ = W.pack_gpumatmult_2d(case["m"], seed)
        dev = torch.device("cuda")
        t = [torch.as_tensor(a, device=dev).double().view(-1, 128) for a in (tx, ty)]
        s = [torch.cat([torch.as_tensor(a, device=dev).double(), torch.zeros(1, device=dev).double()])
             for a in (sx, sy, sg)]
        off = torch.as_tensor(off.astype(np.int64), device=dev)
        count = off[1:] - off[:-1]
        k = torch.arange(int(count.max()), device=dev)
        out = []
        for a in range(0, len(count), 256):
            at = off[a:a + 256, None][:len(count[a:a + 256])] + k
            at = torch.where(k[None, :] < count[a:a + 256, None], at, len(sx))
            d2 = sum((t[q][a:a + 256][:, :, None] - s[q][at][:, None, :]) ** 2 for q in (0, 1))
            e = torch.exp(d2 * (-1.0 / (2.0 * float(sigma) ** 2)))
            out.append(torch.bmm(e, s[2][at][:, :, None])[:, :, 0])
        return torch.cat(out).reshape(-1) / (2.0 * math.pi * float(sigma) ** 2)
    return None  # training: 16-bit operands in every layer
