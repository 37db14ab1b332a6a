"""The calls whose speed matters here, one case each, with their inputs and
their results in 64 bits.

A case goes through the public entry points (``svd``, ``UnevenBatch``,
``jacobi_eigh``) with the sizes, precisions and options that the workloads
of this repository and its tests use.  Singular vectors are only determined
up to a sign or phase each (and, between equal singular values, up to a
rotation), so a pass goes on to what a program makes of them, which is
unique: the polar factor U V^H (orthogonal Procrustes, rotation extraction),
the low-rank approximation U diag(s) V^H or the whitening matrix H^(-1/2).
"""
from __future__ import annotations

import importlib
import math
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

_pkg = importlib.import_module("pavel-s_svd_b200")
_eigh = importlib.import_module("pavel-s_svd_b200.eigh")
_batch = importlib.import_module("pavel-s_svd_b200.batch")

DEV = "cuda"
DTYPES = {"float32": torch.float32, "float64": torch.float64, "complex64": torch.complex64,
          "complex128": torch.complex128}
OPTIONS = ("precision", "tol", "block_size", "rank", "values_only")
SKETCH_SEED, OVERSAMPLE, POWER = 20261011, 8, 2          # the defaults of the projected solvers


def listed():
    def svd(name, algorithm, dtype, batch, m, n, spectrum, decades=0.0, result="polar", **options):
        return dict(name=name, kind="svd", algorithm=algorithm, dtype=dtype, batch=batch, m=m, n=n,
                    spectrum=spectrum, decades=decades, result=result, **options)

    return [
        # one small matrix in the middle of a host program: latency, launches, the status read-back
        svd("one_32x16", "jacobi", "float32", 1, 32, 16, "gaussian"),
        # the single matrix of the plain workload, s_i = 10^(-4 i / 127): one matrix, one SM
        svd("one_256x128", "jacobi", "float32", 1, 256, 128, "log", 4.0, tol=1e-6),
        # the headline: thousands of matrices of different shapes in one call
        dict(name="uneven_8192", kind="uneven", count=8192, n_lo=8, n_hi=64, precision="mixed"),
        # a large batch of one shape with spectra over three decades (the 128 x 64 family), default precision
        svd("family_128x64", "jacobi", "float32", 4096, 128, 64, "loguniform", 3.0),
        # plain FP32 arithmetic, odd wide matrices
        svd("fp32_45x61", "jacobi", "float32", 2048, 45, 61, "gaussian", precision="fp32"),
        # double precision batch
        svd("f64_64x32", "jacobi", "float64", 1024, 64, 32, "gaussian"),
        # complex batch (channel matrices and the like)
        svd("c64_48x32", "jacobi", "complex64", 1024, 48, 32, "gaussian"),
        # one tall and skinny matrix, least-squares shaped
        svd("tall_2048x32", "jacobi", "float32", 1, 2048, 32, "gaussian"),
        # truncated factors of a decaying spectrum from a random sketch
        svd("randomized_256x96", "randomized", "float32", 256, 256, 96, "geometric", result="approximation", rank=8),
        # covariance matrices to whiten
        dict(name="eigh_32", kind="eigh", dtype="float64", batch=1024, n=32),
        # block Jacobi in double precision: the rounds engine
        svd("rounds_f64_96x64", "block_jacobi", "float64", 256, 96, 64, "gaussian", block_size=8),
        # block Jacobi of one large low-rank matrix with noise: the tensor-core engine
        svd("block_8192x2048", "block_jacobi", "float32", 1, 8192, 2048, "lowrank", result="approximation",
            block_size=64),
    ]


def _log(rng, lo, hi):
    """An integer in [lo, hi], spread over its logarithm."""
    return max(lo, min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def _many(rng, most, cost, budget):
    """A batch size up to `most` whose cost (per matrix) stays within the budget."""
    return _log(rng, 1, max(1, min(most, int(budget / cost))))


def draw(rng):
    kind = rng.choice(["batch", "batch", "uneven", "double", "complex", "large", "tall", "projected", "eigh", "rounds",
                       "tensor"])
    if kind == "uneven":
        return dict(kind="uneven", count=_log(rng, 64, 8192), n_lo=rng.randint(2, 8), n_hi=rng.randint(12, 64),
                    precision="mixed")
    if kind == "eigh":
        n = _log(rng, 6, 96)
        return dict(kind="eigh", dtype=rng.choice(["float64", "float32"]), batch=_many(rng, 1024, n ** 3, 1e8), n=n)
    case = dict(kind="svd", algorithm="jacobi", spectrum="gaussian", decades=0.0, result="polar")
    if kind == "batch":
        n = _log(rng, 4, 64)
        m = rng.randint(n, 2 * n)
        style = rng.random()
        if style < 0.3:                  # FP32 arithmetic and steep spectra: not the nearly singular square ones
            m = max(m, n + -(-n // 4))
            case.update(precision="fp32")
        elif style < 0.5:
            m = max(m, n + -(-n // 4))
            case.update(spectrum="loguniform", decades=3.0)
        case.update(dtype="float32", batch=_many(rng, 4096, m * n * n, 2e9), m=m, n=n)
        if rng.random() < 0.2:
            case.update(values_only=True, result="values")
    elif kind in ("double", "complex"):
        n = _log(rng, 4, 64)
        m = rng.randint(n + -(-n // 4), 2 * n)
        dtype = "float64" if kind == "double" else rng.choice(["complex64", "complex128"])
        if kind == "double" and rng.random() < 0.3:
            m = 2 * n                    # the Gram squares the condition number
            case.update(algorithm=rng.choice(["gram_jacobi", "qr"]))
        case.update(dtype=dtype, batch=_many(rng, 1024, m * n * n, 1e8), m=m, n=n)
    elif kind == "large":
        n = rng.randint(65, 128)
        case.update(dtype="float32", batch=_log(rng, 1, 64), m=rng.randint(n, 256), n=n, spectrum="log", decades=3.0)
    elif kind == "tall":
        n = _log(rng, 4, 64)
        m = _log(rng, 300, 4096)
        case.update(dtype=rng.choice(["float32", "float32", "float64"]), batch=_many(rng, 64, m * n * n, 1e8), m=m, n=n,
                    algorithm=rng.choice(["jacobi", "jacobi", "qr", "tsqr"]))
    elif kind == "projected":
        m, n = _log(rng, 64, 512), rng.randint(32, 128)
        case.update(algorithm=rng.choice(["randomized", "subspace"]), dtype=rng.choice(["float32", "float64"]),
                    batch=_many(rng, 256, m * n, 8e6), m=m, n=n, spectrum="geometric", result="approximation",
                    rank=rng.randint(4, 16))
    elif kind == "rounds":
        n = rng.randint(24, 64)
        case.update(algorithm="block_jacobi", dtype="float64", batch=_log(rng, 16, 256), m=rng.randint(n, 2 * n), n=n,
                    block_size=8)
    else:
        n = _log(rng, 128, 2048)
        m = _log(rng, max(n, 512), 8192)
        case.update(algorithm="block_jacobi", dtype="float32", batch=1, m=m, n=n, block_size=rng.choice([32, 64]))
        if n > 512 or m > 2048 or rng.random() < 0.5:
            case.update(spectrum="lowrank", result="approximation")
    if kind not in ("tensor", "projected", "large") and rng.random() < 0.3:
        case.update(m=case["n"], n=case["m"])
    return case


def _matrices(case, seed):
    """The batch of input matrices, made on the device from the seed."""
    gen = torch.Generator(device=DEV).manual_seed(seed)
    dtype = DTYPES[case["dtype"]]
    b, m, n = case["batch"], max(case["m"], case["n"]), min(case["m"], case["n"])

    def normal(*shape, dtype=dtype):
        return torch.randn(*shape, dtype=dtype, device=DEV, generator=gen)

    spectrum = case["spectrum"]
    if spectrum == "gaussian":
        a = normal(b, m, n)
    elif spectrum == "lowrank":          # rank 64 of spectral norm about 1, plus noise of 1e-6
        r = min(64, n)
        a = (normal(b, m, r) @ normal(b, r, n)) / ((math.sqrt(m) + math.sqrt(r)) * (math.sqrt(n) + math.sqrt(r)))
        a += 1e-6 * normal(b, m, n)
    else:                                # U diag(s) V^T, V = exp of a skew matrix
        u = normal(b, m, n) / math.sqrt(m)   # near-orthogonal columns
        if spectrum == "log":
            u = torch.linalg.qr(u.double())[0].to(dtype)
        if spectrum == "log":            # evenly spaced decades
            s = 10.0 ** (-case["decades"] * torch.arange(n, device=DEV, dtype=dtype) / max(1, n - 1)).expand(b, n)
        elif spectrum == "geometric":    # the projected solvers' decaying spectrum
            s = (0.8 ** torch.arange(n, device=DEV, dtype=dtype)).expand(b, n)
        else:                            # "loguniform": unsorted, random decades
            s = 10.0 ** (-case["decades"] * torch.rand(b, n, device=DEV, dtype=dtype, generator=gen))
        k = normal(b, n, n)
        v = torch.linalg.matrix_exp((k - k.mT) * (1.2 / math.sqrt(2.0 * n)))
        a = u * s[:, None, :] @ v.mT
    return (a if case["m"] >= case["n"] else a.mH.resolve_conj()).contiguous()


def _uneven_shapes(case):
    """Shapes n ~ U{n_lo..n_hi}, m ~ U{n..2n}: part of the case, not of the seed."""
    rng = np.random.default_rng(case["count"] * 1000 + case["n_lo"] * 100 + case["n_hi"])
    n = rng.integers(case["n_lo"], case["n_hi"] + 1, size=case["count"])
    return rng.integers(n, 2 * n + 1).astype(np.int64), n.astype(np.int64)


def _classes(plan):
    """The matrices by width, 16 columns to a class: their indices and the
    height and width that hold a class."""
    for c in np.unique((plan.n - 1) // 16):
        at = np.flatnonzero((plan.n - 1) // 16 == c)
        yield at, int(plan.m[at].max()), int(plan.n[at].max())


def _padded(plan):
    """Per class, where the entries of U (height x width) and Vh (width x
    width) stand in the flat results, their end for the padding."""
    def places(off, rows, cols, end, height, width):
        i, j = torch.arange(height, device=DEV), torch.arange(width, device=DEV)
        at = [torch.from_numpy(x).to(DEV)[:, None, None] for x in (off, rows, cols)]
        inside = (i[:, None] < at[1]) & (j < at[2])
        return torch.where(inside, at[0] + i[:, None] * at[2] + j, end).to(torch.int32)

    return [(places(plan.u_off[at], plan.m[at], plan.n[at], plan.U.numel(), height, width),
             places(plan.v_off[at], plan.n[at], plan.n[at], plan.Vh.numel(), width, width))
            for at, height, width in _classes(plan)]


def prepare(case, seed):
    state = dict(case)
    if case["kind"] == "uneven":
        m, n = _uneven_shapes(case)
        plan = _batch.UnevenBatch(m, n, DEV, precision=case["precision"])
        size = int(plan.a_off[-1]) + -(-int(m[-1] * n[-1]) // 4) * 4
        gen = torch.Generator(device=DEV).manual_seed(seed)
        state.update(plan=plan, a=torch.randn(size, device=DEV, generator=gen), places=_padded(plan),
                     end=torch.zeros(1, device=DEV))
    elif case["kind"] == "eigh":
        gen = torch.Generator(device=DEV).manual_seed(seed)
        x = torch.randn(case["batch"], 2 * case["n"], case["n"], dtype=DTYPES[case["dtype"]], device=DEV, generator=gen)
        state.update(a=x.mT @ x / (2 * case["n"]))
    else:
        state.update(a=_matrices(case, seed), options={k: case[k] for k in OPTIONS if k in case})
    return state


def run(state):
    if state["kind"] == "uneven":
        plan = state["plan"]
        plan.launch(state["a"])
        plan.check()
        u, vh = (torch.cat([x, state["end"]]) for x in (plan.U, plan.Vh))
        return {"s": plan.S, "polar": [u[at_u] @ vh[at_v] for at_u, at_v in state["places"]]}
    if state["kind"] == "eigh":
        w, v, _ = _eigh.jacobi_eigh(state["a"])
        return {"w": w, "whiten": (v * w.rsqrt()[:, None, :]) @ v.mT}
    u, s, vh = _pkg.svd(state["a"], state["algorithm"], **state["options"])
    if state["result"] == "values":
        return {"s": s}
    if state["result"] == "approximation":
        return {"s": s, "approximation": (u * s[:, None, :]) @ vh}
    return {"s": s, "polar": u @ vh}


def work(case):
    """Each input read once, each result written once; the flops of a dense
    SVD with vectors, 6 m n^2 + 20 n^3 (Golub and Van Loan's R-SVD), of a
    symmetric eigen-decomposition, 9 n^3, or of the products of a sketch."""
    if case["kind"] == "uneven":
        m, n = _uneven_shapes(case)
        return {"bytes": float(4 * (m * n + m * n + n + n * n).sum()), "flops": float((6 * m * n * n + 20 * n ** 3).sum())}
    if case["kind"] == "eigh":
        b, n, e = case["batch"], case["n"], 8 if case["dtype"] == "float64" else 4
        return {"bytes": float(e * b * (2 * n * n + n)), "flops": float(b * 9 * n ** 3)}
    b, m, n = case["batch"], max(case["m"], case["n"]), min(case["m"], case["n"])
    e = {"float32": 4, "float64": 8, "complex64": 8, "complex128": 16}[case["dtype"]]
    k = case.get("rank", n)
    vectors = 0 if case.get("values_only") else m * k + k * n
    flops = 6 * m * n * n + 20 * n ** 3
    if case["spectrum"] == "lowrank":
        flops = 6 * m * n * min(64, n)
    elif "rank" in case:
        ell = min(k + OVERSAMPLE, n)
        flops = 2 * m * n * ell * (2 * POWER + 2)
    return {"bytes": float(b * e * (m * n + vectors) + 4 * b * k), "flops": float(b * flops * (4 if e > 8 or "complex" in case["dtype"] else 1))}


def _each(f, items):
    with ThreadPoolExecutor(16) as pool:      # LAPACK runs outside the interpreter lock
        return list(pool.map(f, items))


def _lapack(a):
    return np.linalg.svd(a, full_matrices=False)


def exact(case, seed):
    state = prepare(case, seed)
    if case["kind"] == "uneven":
        plan, flat = state["plan"], state["a"].cpu().numpy().astype(np.float64)
        s, q = np.zeros(plan.S.numel()), [None] * plan.count

        def one(i):
            m, n, o = int(plan.m[i]), int(plan.n[i]), int(plan.a_off[i])
            ui, si, vi = _lapack(flat[o:o + m * n].reshape(m, n))
            s[plan.s_off[i]:plan.s_off[i] + n] = si
            q[i] = ui @ vi

        _each(one, range(plan.count))
        polar = []
        for at, height, width in _classes(plan):
            polar.append(np.zeros((len(at), height, width)))
            for z, i in enumerate(at):
                polar[-1][z, :q[i].shape[0], :q[i].shape[1]] = q[i]
        return {"s": s, "polar": polar}
    a = state["a"].to(torch.complex128 if state["a"].is_complex() else torch.float64)
    if case["kind"] == "eigh":
        w, v = torch.linalg.eigh(a.cpu())
        return {"w": w, "whiten": (v * w.rsqrt()[:, None, :]) @ v.mT}
    if case["spectrum"] == "lowrank":
        # the values above the cut eps32 max(m, n) s_1 and what they carry; below it there is nothing
        tall = a[0] if case["m"] >= case["n"] else a[0].mT
        w, v = (t.flip(-1) for t in torch.linalg.eigh(tall.mT @ tall))
        s = w.clamp_min(0).sqrt()
        keep = s > torch.finfo(torch.float32).eps * max(case["m"], case["n"]) * s[0]
        v = v[:, keep]
        low = (tall @ v) @ v.mT
        return {"s": torch.where(keep, s, torch.zeros_like(s))[None].cpu(),
                "approximation": (low if case["m"] >= case["n"] else low.mT)[None].cpu()}
    if case["algorithm"] in ("randomized", "subspace"):
        return _projected(case, a.cpu())
    if case["batch"] * case["m"] * case["n"] * min(case["m"], case["n"]) > 2.5e10:
        return None
    u, s, vh = (np.stack(x) for x in zip(*_each(_lapack, a.cpu().numpy())))
    return {"s": s} if case["result"] == "values" else {"s": s, "polar": u @ vh}


def _projected(case, a):
    """The randomized range finder with two power iterations, from the same sketch."""
    gen = torch.Generator(device=DEV).manual_seed(SKETCH_SEED)
    ell = min(case["rank"] + OVERSAMPLE, min(case["m"], case["n"]))
    omega = torch.randn(case["batch"], case["n"], ell, dtype=DTYPES[case["dtype"]], device=DEV, generator=gen)
    q = torch.linalg.qr(a @ omega.to(a.dtype).cpu())[0]
    for _ in range(POWER):
        z = torch.linalg.qr(a.mH @ q)[0]
        q = torch.linalg.qr(a @ z)[0]
    u, s, vh = torch.linalg.svd(q.mH @ a, full_matrices=False)
    k = case["rank"]
    s = s[:, :k]
    return {"s": s, "approximation": (q @ u[:, :, :k] * s[:, None, :]) @ vh[:, :k]}
