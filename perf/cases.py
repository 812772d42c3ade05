"""What is timed: QR factorizations through the library's public entry points.

The cases are the calls a user makes, by how they make them:

* ``host``: the reference's own C signature (``orth.h``) on host arrays, the way
  the reference's test driver and a code ported from it call it. X is refilled
  before each call because Q overwrites it.
* ``dev``: X and R already on the GPU (``run_dev``), enqueued on the caller's
  stream, in the FP64 mode or in one of the two split modes. The copy that refills
  X before each call is the caller's own (it keeps X for its residual).
* ``batch``: many independent matrices of uneven shapes behind one plan that the
  program keeps (``Batch``).

X = G diag(sigma) W^T with Gaussian G (m >> n, so G is well conditioned), sigma
log-spaced from 1 to 1/kappa and W a product of reflectors: the graded matrices of
the library's benchmark and tests, in a form that is quick to build. ``uniform``
entries in [0, 1) are those of the reference's test driver. kappa stays where every
variant completes: after a Cholesky breakdown (beyond about 1e8, or 1e5 in the
48-bit mode) Q is not a result that could be compared.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.abspath("one-synchronization-bcgs_gb300"))

from bcgs_gb300 import orth  # noqa: E402

PRECISION = {"fp64": orth.FP64, "split": orth.SPLIT_BF16, "split_fast": orth.SPLIT_BF16_FAST}


def _dev(name, variant, precision, m, n, s, kappa, pad=0):
    """pad: rows between the end of one column of X and the next (ld = m + pad)."""
    return {"name": name, "kind": "dev", "variant": variant, "precision": precision, "m": m, "n": n, "s": s,
            "kappa": kappa, "pad": pad}


def _host(name, variant, m, n, s, data, kappa=0.0):
    return {"name": name, "kind": "host", "variant": variant, "precision": "fp64", "m": m, "n": n, "s": s,
            "data": data, "kappa": kappa}


def _batch(name, precision, count, m_max, shapes):
    """shapes: the seed the matrices' sizes are drawn from."""
    return {"name": name, "kind": "batch", "variant": "bcgsi2P1s", "precision": precision, "count": count,
            "m_max": m_max, "shapes": shapes}


def listed():
    return [
        # The reference's own test call: a drop-in user's smallest problem.
        _host("host_test_driver", "bcgsi2P1s", 550, 39, 5, "uniform"),
        # One s-step cycle of a small solver on the device: latency and launches.
        _dev("dev_small_pipi", "bcgspipi2", "fp64", 3001, 64, 4, 1e4),
        # The reference's CPU-runnable configuration through orth.h, malloc'd arrays.
        _host("host_config0", "bcgsi2P1s", 100000, 200, 10, "graded", 1e6),
        # The same configuration on device buffers: the split mode, and BCGSI+ (the
        # robust two-synchronization variant with a TSQR per pass) in FP64.
        _dev("dev_config0_split", "bcgsi2P1s", "split", 100000, 200, 10, 1e6),
        _dev("dev_config0_bcgsi2", "bcgsi2", "fp64", 100000, 200, 10, 1e6),
        # FP64 (the default mode) on a mid-sized basis, rows not a multiple of anything.
        _dev("dev_fp64_odd", "bcgsi2P1s", "fp64", 300007, 256, 16, 1e6),
        # One-synchronization BCGSI+A with a ragged last block and a padded ld.
        _dev("dev_21s_ragged", "bcgsi21s", "split", 700001, 250, 16, 1e6, 3),
        # Robust one-synchronization variant, wider blocks: a TSQR per block step.
        _dev("dev_p2s_wide", "bcgsi2P2s", "split", 400000, 256, 32, 1e6),
        # The widest blocks the library takes.
        _dev("dev_s64", "bcgsi2P1s", "split", 524288, 512, 64, 1e6),
        # The flagship shape, a quarter of its rows.
        _dev("dev_large", "bcgsi2P1s", "split", 2097152, 512, 16, 1e6),
        # Ensembles: uneven matrices, one plan, both precisions.
        _batch("batch_split", "split", 96, 50000, 11),
        _batch("batch_fp64", "fp64", 48, 20000, 12),
    ]


def _log(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    kind = rng.choice(["host", "dev", "dev", "dev", "dev", "batch"])
    if kind == "batch":
        precision = rng.choice(["fp64", "split"])
        top = 64 if precision == "fp64" else 128
        c = _batch("", precision, _log(rng, 4, top), _log(rng, 4000, 20000 if precision == "fp64" else 60000),
                   rng.randrange(1 << 20))
    else:
        s = rng.choice([4, 5, 8, 10, 16]) if kind == "host" else rng.choice([4, 5, 8, 10, 16, 20, 32, 64])
        n = s * rng.randint(2, max(2, min(20, 320 // s))) + rng.choice([0, 0, rng.randrange(s)])
        variant = rng.choice(list(orth.VARIANTS))
        precision = "fp64" if kind == "host" else rng.choice(["fp64", "split", "split", "split_fast"])
        # Bounded by the work of the largest listed case: the FP64 products run at the
        # FP64 pipe's rate, and so does the TSQR of each step of the two TSQR variants.
        if precision == "fp64":
            top = min(4e10 / (4.0 * n * n), 1.5e8 / n)
        else:
            top = 2.5e8 / n
        if variant in ("bcgsi2", "bcgsi2P2s"):
            top = min(top, 2e9 / (n * s))
        m = max(_log(rng, 500 if kind == "host" else 2000, 30000 if kind == "host" else max(4000.0, top)), n + 1)
        kappa = rng.choice([1e2, 1e4] if precision == "split_fast" else [1e2, 1e4, 1e6])
        if kind == "host":
            c = _host("", variant, m, n, s, rng.choice(["uniform", "graded"]), kappa)
        else:
            c = _dev("", variant, precision, m, n, s, kappa, rng.choice([0, 0, 1, 6]))
    del c["name"]
    return c


def _shapes(case):
    """Sizes of a batch: m log-uniform from 2000, s in {4, 8, 16}, 2 to 16 blocks."""
    rng = np.random.default_rng(case["shapes"])
    k = case["count"]
    ms = np.exp(rng.uniform(np.log(2000), np.log(case["m_max"]), k)).astype(np.int64)
    ss = rng.choice([4, 8, 16], k)
    ps = rng.integers(2, 17, k)
    ks = np.exp(rng.uniform(np.log(1e2), np.log(1e6), k))
    return [int(m) for m in ms], [int(s * p) for s, p in zip(ss, ps)], [int(s) for s in ss], [float(x) for x in ks]


def _graded(m, n, kappa, g, out):
    """Fills out (n x m, a row per column of X, rows may be padded) with a graded X."""
    out.normal_(generator=g)
    sigma = torch.logspace(0.0, -math.log10(kappa), n, device="cuda", dtype=torch.float64)
    out.mul_(sigma[:, None])
    for _ in range(3):
        v = torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
        v /= v.norm()
        out.addr_(v, v @ out, alpha=-2.0)


def prepare(case, seed):
    orth.load()
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    if case["kind"] == "batch":
        ms, ns, ss, ks = _shapes(case)
        offs = np.concatenate([[0], np.cumsum([m * n for m, n in zip(ms, ns)])])
        roffs = np.concatenate([[0], np.cumsum([n * n for n in ns])])
        X0 = torch.empty(int(offs[-1]), device="cuda", dtype=torch.float64)
        for b in range(case["count"]):
            _graded(ms[b], ns[b], ks[b], g, X0[int(offs[b]):int(offs[b + 1])].view(ns[b], ms[b]))
        X = X0.clone()
        R = torch.zeros(int(roffs[-1]), device="cuda", dtype=torch.float64)
        plan = orth.Batch(ms, ns, ss, [X.data_ptr() + 8 * int(o) for o in offs[:-1]],
                          [R.data_ptr() + 8 * int(o) for o in roffs[:-1]], precision=PRECISION[case["precision"]],
                          stream=torch.cuda.current_stream().cuda_stream)
        if plan.rc != 0:
            raise RuntimeError(f"batch plan: {plan.rc}")
        return {"case": case, "X0": X0, "X": X, "R": R, "plan": plan}
    m, n = case["m"], case["n"]
    if case["kind"] == "host":
        if case["data"] == "uniform":
            X0 = torch.rand((n, m), generator=g, device="cuda", dtype=torch.float64)
        else:
            X0 = torch.empty((n, m), device="cuda", dtype=torch.float64)
            _graded(m, n, case["kappa"], g, X0)
        return {"case": case, "X0": X0.cpu().numpy().T, "X": np.zeros((m, n), order="F"),
                "R": np.zeros((n, n), order="F"), "work": np.zeros(1)}
    X0 = torch.empty((n, m + case["pad"]), device="cuda", dtype=torch.float64)
    X0[:, m:] = 0.0
    _graded(m, n, case["kappa"], g, X0[:, :m])
    return {"case": case, "X0": X0, "X": torch.empty_like(X0),
            "R": torch.zeros((n, n), device="cuda", dtype=torch.float64)}


def run(state):
    """One QR (or one batch of them): {"Q": columns of Q as rows, "R": columns of R as rows}."""
    case, X0, X, R = state["case"], state["X0"], state["X"], state["R"]
    if case["kind"] == "batch":
        X.copy_(X0)
        rc = state["plan"].run(torch.cuda.current_stream().cuda_stream)
        out = {"Q": X, "R": R}
    elif case["kind"] == "host":
        np.copyto(X, X0)
        rc = orth.call(case["variant"], case["m"], case["n"], case["s"], X, case["m"], R, case["n"], state["work"])
        out = {"Q": X.T, "R": R.T}
    else:
        X.copy_(X0)
        rc, _ = orth.run_dev(case["variant"], case["m"], case["n"], case["s"], X.data_ptr(), X.stride(0),
                             R.data_ptr(), case["n"], PRECISION[case["precision"]],
                             torch.cuda.current_stream().cuda_stream, want_status=False)
        out = {"Q": X[:, :case["m"]], "R": R}
    if rc != 0:
        raise RuntimeError(f"{case['variant']}: {rc}")
    return out


def work(case):
    """Read X and write Q and R once; a reorthogonalized QR by block Gram-Schmidt is
    two projections of every column against those before it (4 m n^2)."""
    if case["kind"] == "batch":
        ms, ns, _, _ = _shapes(case)
        sizes = list(zip(ms, ns))
    else:
        sizes = [(case["m"], case["n"])]
    return {"bytes": float(sum(16 * m * n + 8 * n * n for m, n in sizes)),
            "flops": float(sum(4 * m * n * n for m, n in sizes))}


def _qr64(Xt):
    """Q^T and R^T of the QR factorization with a positive diagonal of R, from X^T
    (n x m): three rounds of Cholesky QR in 64 bits."""
    n = Xt.shape[0]
    Rt = np.eye(n)
    for _ in range(3):
        G = (Xt @ Xt.t()).cpu().numpy()
        L = np.linalg.cholesky(0.5 * (G + G.T))
        Rt = Rt @ L
        Xt = torch.linalg.solve_triangular(torch.from_numpy(L), torch.eye(n, dtype=torch.float64),
                                           upper=False).to(Xt.device) @ Xt
    return Xt, torch.from_numpy(np.tril(Rt)).to(Xt.device)


def exact(case, seed):
    if case["kind"] == "batch":
        ms, ns, _, ks = _shapes(case)
        g = torch.Generator(device="cuda")
        g.manual_seed(seed)
        offs = np.concatenate([[0], np.cumsum([m * n for m, n in zip(ms, ns)])])
        X0 = torch.empty(int(offs[-1]), device="cuda", dtype=torch.float64)
        Q, R = [], []
        for b in range(case["count"]):
            v = X0[int(offs[b]):int(offs[b + 1])].view(ns[b], ms[b])
            _graded(ms[b], ns[b], ks[b], g, v)
            q, r = _qr64(v)
            Q.append(q.reshape(-1))
            R.append(r.reshape(-1))
        return {"Q": torch.cat(Q), "R": torch.cat(R)}
    state = prepare(case, seed)
    if case["kind"] == "host":
        Q, R = np.linalg.qr(state["X0"])
        d = np.sign(np.diag(R))
        return {"Q": np.ascontiguousarray((Q * d).T), "R": np.ascontiguousarray((R * d[:, None]).T)}
    Q, R = _qr64(state["X0"][:, :case["m"]])
    return {"Q": Q, "R": R}
