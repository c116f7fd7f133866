"""What is timed: the calls a user of the kernel low-rank pipeline makes, at the sizes they are made at.

The three stages on Kuramoto-Sivashinsky states (bandwidth calibration, block
RPCholesky, bistochastic EVD), the hand-over of the stage-2 files to stage 3,
many uneven datasets in one call, and the out-of-sample queries behind the
serving loop; the mixed and the plain FP64 form.

Kinds of case and what stands behind them:

``calibrate``   the bandwidth sweep of one dataset (host sums back, as ``cuband`` needs them)
``sweep``       the sweeps of many uneven datasets in one launch
``median``      the exact median squared distance that centres a sweep
``rpchol``      the factorisation (``cuarpclm``); with b = 1 one pivot per round, latency-bound
``factorise``   the factorisations of many uneven datasets as one graph
``evd``         bistochastic normalisation and eigenpairs of a factor (``cukevd``)
``linv``        the factor from the stage-2 files ``/linv`` and ``/spiv``, which ``cukevd`` starts with
``nystrom``     eigenfunction values of new states against a resident model
``serve``       a burst of query batches through the serving loop, host buffers in and out

States come from the GPU KS generator: many trajectories from seeded random
initial states, a warm-up onto the attractor, then consecutive snapshots.
"""
import math
import random

import numpy as np
import torch

from kernel_evd_gb300 import api, datagen

DT = 0.25
WARM_STEPS = 800          # 200 time units: past the growth of the initial noise
EPS_OVER_MEDIAN = 0.17    # what the calibration selects for these states: 0.125 .. 0.18 of their median squared distance


def listed():
    return [
        # the sweep of a small dataset: 41 bandwidths over 20,000 states
        {"name": "calibrate_20k", "kind": "calibrate", "N": 20000, "d": 64, "L": 22.0, "n_eps": 41},
        # the sweep of a large one: 64 bandwidths over 2e10 pairs, the heaviest single pass of stage 1
        {"name": "calibrate_200k", "kind": "calibrate", "N": 200000, "d": 64, "L": 22.0, "n_eps": 64},
        # ten uneven datasets (d = 32, 64 or 128), 41 bandwidths each, in one call
        {"name": "sweep_batch", "kind": "sweep", "sets": 10, "N_lo": 10000, "N_hi": 60000, "mix": 5},
        # the exact median over all pairs of the small dataset
        {"name": "median_20k", "kind": "median", "N": 20000, "d": 64, "L": 22.0},
        # plain FP64, one pivot a round: 500 rounds of small launches
        {"name": "rpchol_fp64_b1", "kind": "rpchol", "precision": "fp64", "N": 20000, "d": 64, "L": 22.0, "k": 500,
         "b": 1},
        # the headline factorisation: 2,000,000 states to rank 2000
        {"name": "rpchol_2m", "kind": "rpchol", "precision": "mixed", "N": 2000000, "d": 64, "L": 22.0, "k": 2000,
         "b": 64},
        # eight uneven datasets (ranks not rounded to anything) as one graph of factorisations
        {"name": "factorise_batch", "kind": "factorise", "sets": 8, "N_lo": 10000, "N_hi": 100000, "mix": 3, "b": 32},
        # the headline decomposition: rank 2000 over 2,000,000 states, top 32
        {"name": "evd_2m", "kind": "evd", "precision": "mixed", "N": 2000000, "d": 64, "L": 22.0, "k": 2000,
         "k_out": 32},
        # the plain FP64 decomposition that mixed results are held against
        {"name": "evd_fp64_200k", "kind": "evd", "precision": "fp64", "N": 200000, "d": 64, "L": 22.0, "k": 1000,
         "k_out": 32},
        # stage 3 fed from stage 2's files: the FP64 factor from pivots and inverse Cholesky factor
        {"name": "linv_fp64", "kind": "linv", "precision": "fp64", "N": 100000, "d": 64, "L": 22.0, "k": 1024},
        # a query of the usual size: 64 new states (the middle of 1 .. 4096 in the logarithm)
        {"name": "nystrom_64", "kind": "nystrom", "n": 64, "N": 100000, "d": 64, "L": 22.0, "k": 2000, "k_out": 32},
        # 24 query batches of 1 .. 4096 states arriving at once at the serving loop
        {"name": "serve_burst", "kind": "serve", "queries": 24, "n_hi": 4096, "mix": 11, "N": 100000, "d": 64,
         "L": 22.0, "k": 2000, "k_out": 32},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["calibrate", "sweep", "median", "rpchol", "rpchol", "factorise", "evd", "evd", "linv", "nystrom",
                       "nystrom", "serve"])
    d, L = rng.choice([32, 64, 64, 128]), rng.choice([16.0, 22.0, 22.0, 36.0])
    if kind == "calibrate":
        return {"kind": kind, "N": _log_int(rng, 500, 150000), "d": d, "L": L, "n_eps": rng.randint(8, 64)}
    if kind == "sweep":
        return {"kind": kind, "sets": rng.randint(2, 12), "N_lo": 1000, "N_hi": _log_int(rng, 8000, 60000),
                "mix": rng.randrange(1 << 20)}
    if kind == "median":
        return {"kind": kind, "N": _log_int(rng, 500, 40000), "d": d, "L": L}
    if kind == "rpchol":
        if rng.random() < 0.5:
            N = _log_int(rng, 2000, 40000)
            return {"kind": kind, "precision": "fp64", "N": N, "d": d, "L": max(L, 22.0),
                    "k": min(N // 8, rng.randint(50, 500)), "b": rng.choice([1, 1, 8, 32, 64])}
        N = _log_int(rng, 10000, 1000000)
        return {"kind": kind, "precision": "mixed", "N": N, "d": 64, "L": 22.0,
                "k": min(N // 8, rng.randint(200, 1600)), "b": rng.choice([16, 32, 64, 64, 128])}
    if kind == "factorise":
        return {"kind": kind, "sets": rng.randint(2, 8), "N_lo": 10000, "N_hi": _log_int(rng, 12000, 100000),
                "mix": rng.randrange(1 << 20), "b": rng.choice([16, 32, 64])}
    if kind == "evd":
        if rng.random() < 0.5:
            N = _log_int(rng, 10000, 150000)
            return {"kind": kind, "precision": "fp64", "N": N, "d": d, "L": 22.0, "k": rng.randint(100, 1000),
                    "k_out": rng.choice([16, 32, 64])}
        N, k = _log_int(rng, 20000, 1000000), rng.randint(200, 1600)
        return {"kind": kind, "precision": "mixed", "N": N, "d": 64, "L": 22.0, "k": k,
                "k_out": rng.choice([16, 32, 32, 64, 256 if k >= 512 and N < 300000 else 32])}
    if kind == "linv":
        N = _log_int(rng, 10000, 100000)
        return {"kind": kind, "precision": rng.choice(["fp64", "mixed"]), "N": N, "d": d, "L": 22.0,
                "k": rng.randint(200, 1024)}
    model = {"N": 100000, "d": 64, "L": 22.0, "k": rng.randint(300, 2000), "k_out": rng.choice([8, 16, 32, 32, 64])}
    if kind == "nystrom":
        return {"kind": kind, "n": _log_int(rng, 1, 4096), **model}
    return {"kind": kind, "queries": rng.randint(2, 32), "n_hi": _log_int(rng, 16, 4096),
            "mix": rng.randrange(1 << 20), **model}


# ---- inputs ------------------------------------------------------------------
def _states(ctx, n, d, L, seed):
    """n KS states of d grid points: up to 1024 trajectories, consecutive snapshots of each."""
    t = max(1, min(1024, n // 128))
    rng = np.random.default_rng(seed)
    v0 = np.fft.rfft(0.1 * rng.standard_normal((t, d)), axis=1)
    per = [n // t + (1 if q < n % t else 0) for q in range(t)]
    parts = datagen.run_gpu([(L, v0[q], per[q]) for q in range(t)], d, DT, WARM_STEPS, ctx=ctx, precision="fp32")
    return torch.cat(parts).contiguous()


def _median(X, seed=0):
    """Median squared distance of 100,000 random pairs."""
    g = torch.Generator(device="cpu").manual_seed(seed)
    i = torch.randint(0, X.shape[0], (2, 100000), generator=g).to(X.device)
    return float(((X[i[0]].double() - X[i[1]].double()) ** 2).sum(1).median())


def _scale(X):
    return 1.0 / (EPS_OVER_MEDIAN * _median(X))


def _uneven(case):
    """(L, d, N, k) of each dataset of a batch; a function of the case alone.  The small domain L = 16 only in sweeps:
    there a factorisation may stop at its rounding floor before rank k, at a rank that depends on the states."""
    rng = random.Random(case["mix"])
    sets = []
    for _ in range(case["sets"]):
        n = _log_int(rng, case["N_lo"], case["N_hi"])
        sets.append((rng.choice([16.0, 22.0, 36.0] if case["kind"] == "sweep" else [22.0, 36.0]), rng.choice([32, 64, 128]), n, min(rng.randint(100, 1000), n // 8)))
    return sets


def _query_sizes(case):
    rng = random.Random(case["mix"])
    return [_log_int(rng, 1, case["n_hi"]) for _ in range(case["queries"])]


def _kernel(X, S, scale):
    """K(X, S) in FP64."""
    D = torch.cdist(X.double(), S.double(), compute_mode="donot_use_mm_for_euclid_dist")
    return torch.exp(-scale * D * D)


def prepare(case, seed):
    ctx = api.Context(0)
    st = {"case": case, "ctx": ctx, "seed": seed % (1 << 31)}
    kind = case["kind"]
    if kind in ("sweep", "factorise"):
        sets = _uneven(case)
        st["Xs"] = [_states(ctx, n, d, L, seed * 1000 + q) for q, (L, d, n, _) in enumerate(sets)]
        med = [_median(X) for X in st["Xs"]]
        if kind == "sweep":
            st["scales"] = [1.0 / api.log_sweep(m, 41) for m in med]
        else:
            st["scales"] = [1.0 / (EPS_OVER_MEDIAN * m) for m in med]
            st["k"] = [k for _, _, _, k in sets]
        return st
    N, d = case["N"], case["d"]
    X = _states(ctx, N + case.get("n", 0), d, case["L"], seed)
    if kind == "calibrate":
        st["X"], st["scales"] = X, 1.0 / api.log_sweep(_median(X), case["n_eps"])
        return st
    if kind == "median":
        st["X"] = X
        return st
    st["scale"] = _scale(X)
    if kind == "rpchol":
        st["X"] = X
        return st
    if kind == "serve":
        sizes = _query_sizes(case)
        Y = _states(ctx, sum(sizes), d, case["L"], seed + 7).cpu().numpy()
        at = np.cumsum([0] + sizes)
        st["Y"] = [np.ascontiguousarray(Y[at[q]:at[q + 1]]) for q in range(len(sizes))]
        srv = api.Server(factor_workers=1, max_query_batch=16384)
        rid = srv.submit_factorization(X.cpu().numpy(), st["scale"], case["k"], 64, case["k_out"], seed=st["seed"])
        st["model_id"], st["server"] = srv.wait(rid).model_id, srv
        return st
    if kind == "nystrom":
        Xl = X[:N].contiguous()
        fac = api.rpcholesky(ctx, Xl, st["scale"], case["k"], 64, seed=st["seed"])
        st["model"] = api.NystromModel(ctx, Xl, fac, k_out=min(case["k_out"], fac.rank))
        st["Y"] = X[N:].contiguous()
        return st
    # a factor: the pivots of the mixed factorisation
    fac = api.rpcholesky(ctx, X, st["scale"], case["k"], 64, seed=st["seed"])
    if kind == "evd" and case["precision"] == "mixed":
        st["F"] = fac.factor
        return st
    S = X[torch.from_numpy(fac.piv).cuda()]
    Linv = torch.linalg.solve_triangular(torch.linalg.cholesky(_kernel(S, S, st["scale"])),
                                         torch.eye(fac.rank, dtype=torch.float64, device="cuda"), upper=False)
    del fac
    if kind == "linv":
        st["X"], st["S"], st["Linv"] = X, S, Linv
        st["piv"] = _rows_of(X, S)
        st["Linv_host"] = np.asfortranarray(Linv.cpu().numpy())
        return st
    st["F"] = torch.cat([_kernel(x, S, st["scale"]) @ Linv.T for x in X.split(50000)]).contiguous()
    return st


def _rows_of(X, S):
    """Row numbers of the rows S of X."""
    where = {r.tobytes(): i for i, r in enumerate(X.cpu().numpy())}
    return np.array([where[r.tobytes()] for r in S.cpu().numpy()], dtype=np.int64)


# ---- one pass ------------------------------------------------------------------
def _by_round(a, case):
    """A per-round array at the length of the round limit (the number of rounds depends on the draws)."""
    out = np.zeros(4 * -(-case["k"] // case["b"]) + 8, dtype=a.dtype)
    out[:len(a)] = a
    return out


def _factorisation(f):
    return {"F": f.factor, "piv": f.piv, "trace_error": f.trace_error}


def run(state):
    case, ctx = state["case"], state["ctx"]
    kind = case["kind"]
    if kind == "calibrate":
        return api.calibrate(ctx, state["X"], state["scales"])
    if kind == "sweep":
        return api.calibrate_batched(ctx, state["Xs"], state["scales"])
    if kind == "median":
        return api.pair_median(ctx, state["X"])
    if kind == "rpchol":
        f = api.rpcholesky(ctx, state["X"], state["scale"], case["k"], case["b"], seed=state["seed"],
                           precision=case["precision"])
        return {**_factorisation(f), "err": _by_round(f.err, case), "accepted": _by_round(f.accepted, case)}
    if kind == "factorise":
        seeds = [state["seed"] + q for q in range(len(state["Xs"]))]
        facs = api.rpcholesky_batched(ctx, state["Xs"], state["scales"], state["k"], case["b"], seeds=seeds)
        return [_factorisation(f) for f in facs]
    if kind == "evd":
        e = api.bistochastic_evd(ctx, state["F"], k_out=case["k_out"])
        return {"lam": e.lam, "U": e.U}
    if kind == "linv":
        return api.factor_from_linv(ctx, state["X"], state["scale"], state["piv"], state["Linv_host"],
                                    precision=case["precision"])
    if kind == "nystrom":
        return state["model"](state["Y"])
    srv = state["server"]
    sent = [srv.submit_query(state["model_id"], y, case["k_out"]) for y in state["Y"]]
    for rid, _ in sent:
        srv.wait(rid)
    return [out for _, out in sent]


# ---- what a pass cannot do without ------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind in ("sweep", "factorise"):
        total = {"bytes": 0.0, "flops": 0.0}
        for L, d, n, k in _uneven(case):
            one = {"kind": "calibrate" if kind == "sweep" else "rpchol", "precision": "mixed", "N": n, "d": d, "k": k,
                   "n_eps": 41}
            for key, v in work(one).items():
                total[key] += v
        return total
    d, k = case["d"], case.get("k", 0)
    N = float(case["N"])
    pairs = N * (N - 1) / 2
    el = 8.0 if case.get("precision") == "fp64" else 4.0
    if kind == "calibrate":   # per pair a distance (3 d) and per bandwidth a scale, an exp and a sum
        return {"bytes": 4 * N * d + 16.0 * case["n_eps"], "flops": pairs * (3.0 * d + 3.0 * case["n_eps"])}
    if kind == "median":
        return {"bytes": 4 * N * d + 8.0, "flops": pairs * 3.0 * d}
    if kind == "rpchol":      # K(:, S), the products with the earlier columns, the solve with the pivot block
        return {"bytes": 4 * N * d + el * N * k, "flops": N * k * (3.0 * d + k)}
    if kind == "evd":         # four matrix-vector passes, two symmetric Grams, the dense solve, U
        return {"bytes": el * N * k + 4 * N * case["k_out"] + 8.0 * k,
                "flops": N * k * (8.0 + 2.0 * k + 2.0 * case["k_out"]) + 12.0 * k ** 3}
    if kind == "linv":        # K(:, S) and the product with the triangle
        return {"bytes": 4 * N * d + el * N * k + 8.0 * k * k, "flops": N * k * (3.0 * d + k)}
    n = float(case["n"] if kind == "nystrom" else sum(_query_sizes(case)))
    per = 4.0 * k * d + 8.0 * k * (case["k_out"] + 1)
    return {"bytes": 4 * n * (d + case["k_out"]) + per, "flops": n * k * (3.0 * d + 2.0 * (case["k_out"] + 1))}


# ---- the same in 64 bits ------------------------------------------------------------
def _pair_sums(X, scales):
    X = X.double()
    out = torch.zeros(len(scales), dtype=torch.float64, device=X.device)
    step = max(1, 32_000_000 // X.shape[0])
    for a in range(0, X.shape[0], step):
        D = torch.cdist(X[a:a + step], X[:a + step], compute_mode="donot_use_mm_for_euclid_dist").square()
        keep = torch.ones_like(D, dtype=torch.bool).tril(a - 1)
        D = torch.where(keep, D, torch.inf)
        for j, s in enumerate(scales):
            out[j] += torch.exp(-float(s) * D).sum()
    return out.cpu().numpy()


def _uniform(seed, rnd, stream, idx):
    """Draw (stream, idx) of round rnd: Philox4x32-10, 53 bits, in (0, 1]."""
    c, k = [idx, rnd, stream, 0], [seed & 0xFFFFFFFF, seed >> 32]
    for _ in range(10):
        p, q = 0xD2511F53 * c[0], 0xCD9E8D57 * c[2]
        c = [(q >> 32) ^ c[1] ^ k[0], q & 0xFFFFFFFF, (p >> 32) ^ c[3] ^ k[1], p & 0xFFFFFFFF]
        k = [(k[0] + 0x9E3779B9) & 0xFFFFFFFF, (k[1] + 0xBB67AE85) & 0xFFFFFFFF]
    return (((c[0] >> 5) << 26) + (c[1] >> 6) + 1) / 9007199254740992.0


def exact(case, seed):
    kind = case["kind"]
    pairs = float(case.get("N", 0)) ** 2 / 2
    # the eigenfunctions' signs are free, so U and what is built on it have no single exact value; the random
    # pivots of a factorisation are followed where a round is one proposal
    if kind in ("factorise", "nystrom", "serve"):
        return None
    if kind == "calibrate" and pairs * (case["n_eps"] + case["d"]) > 6e10:
        return None
    if kind == "sweep" and sum(n * n / 2.0 * (41 + d) for _, d, n, _ in _uneven(case)) > 6e10:
        return None
    if kind == "rpchol" and not (case["precision"] == "fp64" and case["b"] == 1):
        return None
    if kind == "evd" and float(case["N"]) * case["k"] ** 2 > 1e12:
        return None
    st = prepare(case, seed)
    if kind == "calibrate":
        return _pair_sums(st["X"], st["scales"])
    if kind == "sweep":
        return [_pair_sums(X, s) for X, s in zip(st["Xs"], st["scales"])]
    if kind == "median":
        return _exact_median(st["X"])
    if kind == "linv":
        return torch.cat([_kernel(x, st["S"], st["scale"]) @ st["Linv"].T for x in st["X"].split(50000)])
    if kind == "evd":
        return {"lam": _spectrum(st["F"].double()), "U": None}
    X, s, k = st["X"].double(), st["scale"], case["k"]
    N = X.shape[0]
    F = torch.zeros((N, k), dtype=torch.float64, device=X.device)
    dg = torch.ones(N, dtype=torch.float64, device=X.device)
    piv, err, acc = [], [], []
    for r in range(4 * k + 8):
        if len(piv) >= k:
            break
        c = torch.cumsum(dg, 0)
        i = min(int(torch.searchsorted(c, _uniform(st["seed"], r, 0, 0) * c[-1])), N - 1)
        h = 1.0 - float(F[i] @ F[i])
        ok = h > 1e-10 and h * _uniform(st["seed"], r, 1, 0) < h
        if ok:
            col = (torch.exp(-s * (X - X[i]).square().sum(1)) - F @ F[i]) / math.sqrt(h)
            F[:, len(piv)] = col
            dg = (dg - col * col).clamp_min(0.0)
            piv.append(i)
        acc.append(int(ok))
        err.append(float(dg.sum()) / N)
    return {"F": F[:, :len(piv)], "piv": np.array(piv), "trace_error": err[-1], "err": _by_round(np.array(err), case),
            "accepted": _by_round(np.array(acc, dtype=np.int32), case)}


def _exact_median(X):
    """Lower median of the pair distances, by bisection on its value."""
    X = X.double()
    N = X.shape[0]
    want = (N * (N - 1) // 2 - 1) // 2 + 1
    step = max(1, 64_000_000 // N)
    lo, hi = 0.9 * _median(X), 1.1 * _median(X)
    below, near = 0, []
    for a in range(0, N, step):
        D = torch.cdist(X[a:a + step], X[:a + step], compute_mode="donot_use_mm_for_euclid_dist").square()
        D = torch.where(torch.ones_like(D, dtype=torch.bool).tril(a - 1), D, torch.inf)
        below += int((D < lo).sum())
        near.append(D[(D >= lo) & (D <= hi)])
    near = torch.cat(near).sort().values
    return float(near[want - 1 - below])


def _spectrum(F):
    """Eigenvalues, ascending, of the bistochastic normalisation of F F^T."""
    dt = F @ F.sum(0)
    q = F @ (F / dt[:, None]).sum(0)
    A, B = (F / dt.square()[:, None]).T @ F, (F / q[:, None]).T @ F
    A += torch.finfo(torch.float64).eps * A.trace() * torch.eye(A.shape[0], dtype=A.dtype, device=A.device)
    C = torch.linalg.cholesky(A)
    W = C.T @ B @ C
    return torch.linalg.eigvalsh(0.5 * (W + W.T)).cpu().numpy()
