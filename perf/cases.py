"""What the engine's users run, as cases that can be timed: the reference drivers' block loop and
search, scan chunks of ordinary and frontier wheels, batched scans, counting probes, the
meet-in-the-middle search and the learned planner's network.

Each case goes through a public entry point of the package (``es_gb300.GpuSieve``,
``es_native.Context`` / ``Batch``, ``es_mitm.MitmEngine``, ``es_learned.MLP``).  Scan ranges are
laid around the recorded g(k) wherever the wheel's block holds it, so that the survivor list of a
range is not empty; the seed moves the range (or picks the blocks, the k, the bound, the rows).

Imported with the repository's root as the working folder.
"""
from __future__ import annotations

import functools
import json
import os
import random
import sys

import numpy as np

ROOT = os.getcwd()
PKG = os.path.join(ROOT, "erdos-selfridge_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import es_gb300  # noqa: E402
import es_learned  # noqa: E402
import es_mitm  # noqa: E402
import es_native as N  # noqa: E402

FEATURES = es_learned.FEATURE_DIM


def listed() -> list[dict]:
    return [
        # The resumable driver over a small k: one block is a few thousand positions, so a block is
        # host calls, one launch and one read-back.
        {"name": "blocks_k60", "kind": "blocks", "k": 60, "blocks": 8},
        # The engine's command line over eight consecutive k: block-ordered searches that end within
        # the first blocks.
        {"name": "search_k96", "kind": "search", "k": 96, "count": 8},
        # One drop-in launch chunk of the default size of the reference (2^30 positions), one-word
        # inner ring of 32 slots, ragged at both ends.
        {"name": "chunk_k300_2p30", "kind": "chunk", "k": 300, "positions": (1 << 30) + 12345},
        # The same wheel at the engine's own chunk size (2^34): the throughput benchmark's range.
        {"name": "chunk_k300_2p34", "kind": "chunk", "k": 300, "positions": 1 << 34},
        # A smaller chunk of a wheel whose inner ring fills a word only in part (18 of 32 slots).
        {"name": "chunk_k200_odd", "kind": "chunk", "k": 200, "positions": 123456789},
        # Frontier wheel with a three-word inner ring (72 slots), as whole-block replays scan it.
        {"name": "wheel_k379", "kind": "wheel", "k": 379, "role": "primary", "positions": 1 << 34},
        # Both recorded wheels of k = 390 (two-word inner rings) in one replayed graph: the
        # fixed-scope confirmation scan.
        {"name": "pair_k390", "kind": "pair", "k": 390, "positions": 1 << 35},
        # Sixteen uneven scans (k 150..400, 2^20..2^30 positions) in one persistent launch.
        {"name": "batch16", "kind": "batch", "items": 16, "k_lo": 150, "k_hi": 400, "log2_lo": 20.0,
         "log2_hi": 30.0},
        # The cost model's probe: a launch that counts the positions every filter stage passes.
        {"name": "counts_k260", "kind": "counts", "k": 260, "positions": 1 << 28},
        # One round of the meet-in-the-middle search.
        {"name": "mitm_k150", "kind": "mitm", "k": 150, "mem_gb": 8.0, "bound_mult": 3.0},
        # A stretch of the cost model's training: the campaign's 160 k give about 9,500 probed plans.
        {"name": "train_9467", "kind": "train", "rows": 9467, "dim": FEATURES, "hidden": 64, "batch": 256,
         "epochs": 8},
        # The model's predictions for the candidate plans of a few k.
        {"name": "predict_331", "kind": "predict", "rows": 331, "dim": FEATURES, "hidden": 64},
    ]


def _log_uniform(rng: random.Random, lo: float, hi: float) -> int:
    return int(2.0 ** rng.uniform(lo, hi))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["blocks", "search", "chunk", "chunk", "wheel", "wheel", "pair", "batch", "counts",
                       "mitm", "train", "predict"])
    if kind == "blocks":
        return {"kind": kind, "k": rng.randint(40, 150), "blocks": rng.randint(4, 16)}
    if kind == "search":
        return {"kind": kind, "k": rng.randint(40, 140), "count": rng.randint(4, 8)}
    if kind == "chunk":
        return {"kind": kind, "k": rng.randint(160, 400), "positions": _log_uniform(rng, 24, 34) | 1}
    if kind == "wheel":
        return {"kind": kind, "k": rng.randint(378, 400), "role": rng.choice(["primary", "confirmation"]),
                "positions": _log_uniform(rng, 26, 34) | 1}
    if kind == "pair":
        return {"kind": kind, "k": rng.randint(378, 400), "positions": _log_uniform(rng, 26, 34) | 1}
    if kind == "batch":
        lo = rng.uniform(18, 22)
        return {"kind": kind, "items": rng.randint(3, 16), "k_lo": 150, "k_hi": 400, "log2_lo": lo,
                "log2_hi": lo + rng.uniform(2, 8)}
    if kind == "counts":
        return {"kind": kind, "k": rng.randint(100, 400), "positions": _log_uniform(rng, 20, 28) | 1}
    if kind == "mitm":
        return {"kind": kind, "k": rng.randint(80, 152), "mem_gb": 8.0, "bound_mult": round(rng.uniform(1, 6), 3)}
    if kind == "train":
        return {"kind": kind, "rows": _log_uniform(rng, 9, 13), "dim": rng.choice([FEATURES, rng.randint(5, 64)]),
                "hidden": rng.choice([32, 64, 64]), "batch": rng.choice([64, 100, 128, 256, 300, 512]),
                "epochs": rng.randint(1, 8)}
    return {"kind": "predict", "rows": _log_uniform(rng, 2, 13), "dim": rng.choice([FEATURES, rng.randint(5, 64)]),
            "hidden": rng.choice([32, 64])}


# ------------------------------------------------------------------ plans (made once per process)
@functools.lru_cache(maxsize=None)
def _known() -> dict:
    with open(os.path.join(ROOT, "tests", "golden", "bfile.json")) as f:
        return {int(k): int(g) for k, g in json.load(f)["g"].items()}


@functools.lru_cache(maxsize=None)
def _recorded() -> dict:
    with open(os.path.join(ROOT, "tests", "golden", "replay_blocks.json")) as f:
        return {(c["k"], c["role"]): c["wheel"] for c in json.load(f)["cases"]}


@functools.lru_cache(maxsize=None)
def _plan(k: int, role: str | None = None):
    return es_gb300.Plan(k) if role is None else es_gb300.Plan(k, None, _recorded()[(k, role)])


@functools.lru_cache(maxsize=None)
def _mitm_plan(k: int, mem_gb: float):
    return es_mitm.MitmPlan(k, mem_gb)


def _range(plan, positions: int, rng: random.Random) -> tuple[int, int, int]:
    """(block, first outer index, outer indices): about `positions` positions that hold g(k)'s own,
    the seed choosing where in the range it lies; positions around the block's middle for a k
    beyond the recorded values."""
    r0 = plan.radix[0]
    outer = plan.R // r0
    count = max(1, min(outer, -(-positions // r0)))
    where = plan.n_to_idx(_known()[plan.k])
    t, o = (where[0], where[1] // r0) if where else (0, outer // 2)
    first = max(0, min(outer - count, o - rng.randrange(count)))
    return t, first, count


# ------------------------------------------------------------------ prepare
def prepare(case: dict, seed: int) -> dict:
    rng = random.Random(seed)
    return dict(globals()["_prepare_" + case["kind"]](case, rng, seed), kind=case["kind"])


def _prepare_blocks(c, rng, seed):
    return {"sieve": es_gb300.GpuSieve(_plan(c["k"])), "t0": rng.randrange(1 << 20), "blocks": c["blocks"]}


def _prepare_search(c, rng, seed):
    k0 = c["k"] + rng.randrange(16)
    return {"sieves": [es_gb300.GpuSieve(_plan(k)) for k in range(k0, k0 + c["count"])]}


def _prepare_chunk(c, rng, seed):
    plan = _plan(c["k"])
    t, first, count = _range(plan, c["positions"], rng)
    sieve = es_gb300.GpuSieve(plan)
    return {"sieve": sieve, "t": t, "first": first, "count": count}


def _prepare_wheel(c, rng, seed):
    plan = _plan(c["k"], c["role"])
    t, first, count = _range(plan, c["positions"], rng)
    return {"sieve": es_gb300.GpuSieve(plan), "t": t, "first": first, "count": count}


def _prepare_pair(c, rng, seed):
    plans = [_plan(c["k"], role) for role in ("primary", "confirmation")]
    tune = N.make_tune(layout=N.layout_for_plan(plans[0], 4), mask_filters=4, count_stages=0)
    ctxs = [N.Context(p, tune) for p in plans]
    items = []
    for i, p in enumerate(plans):
        t, first, count = _range(p, c["positions"], rng)
        items.append((i, i, t, first, first + count))
    return {"batch": N.Batch(ctxs, items, tune), "items": items}


def _prepare_batch(c, rng, seed):
    tune = N.make_tune(layout=N.LAYOUT_AUTO, mask_filters=4, count_stages=0)
    ctxs, items = [], []
    shape = random.Random(c["items"])    # the k and the lengths belong to the case, the places to the seed
    for i in range(c["items"]):
        plan = _plan(shape.randint(c["k_lo"], c["k_hi"]))
        positions = int(2.0 ** shape.uniform(c["log2_lo"], c["log2_hi"]))
        t, first, count = _range(plan, positions, rng)
        ctxs.append(N.Context(plan, tune))
        items.append((i, i, t, first, first + count))
    return {"batch": N.Batch(ctxs, items, tune), "items": items}


def _prepare_counts(c, rng, seed):
    plan = _plan(c["k"])
    t, first, count = _range(plan, c["positions"], rng)
    ctx = N.Context(plan, N.make_tune(layout=N.layout_for_plan(plan, 4), mask_filters=4, count_stages=1))
    return {"ctx": ctx, "t": t, "first": first, "count": count}


def _prepare_mitm(c, rng, seed):
    plan = _mitm_plan(c["k"], c["mem_gb"])
    bound = min(plan.M, max(1, int(c["bound_mult"] * plan.E * rng.uniform(0.9, 1.1))))
    return {"engine": es_mitm.MitmEngine(plan), "bound": bound}


def _rows(c, seed):
    """Standardised features and the two standardised targets of the cost model: smooth in the
    features, with the probes' noise."""
    g = np.random.default_rng(seed)
    X = g.normal(size=(c["rows"], c["dim"])).astype(np.float32)
    w = g.normal(size=(c["dim"], 2)) / np.sqrt(c["dim"])
    T = (np.tanh(X @ w) + 0.05 * g.normal(size=(c["rows"], 2))).astype(np.float32)
    return X, T


def _params(c, seed):
    """He-uniform weights and zero biases, as a new model starts."""
    g = np.random.default_rng(seed + 1)
    D, H, O = c["dim"], c["hidden"], 2
    parts = []
    for rows, cols in ((H, D), (H, H), (O, H)):
        a = np.sqrt(6.0 / cols)
        parts += [g.uniform(-a, a, size=rows * cols), np.zeros(rows)]
    return np.concatenate(parts).astype(np.float32)


def _prepare_train(c, rng, seed):
    X, T = _rows(c, seed)
    return {"mlp": es_learned.MLP(c["dim"], 2, c["hidden"], seed=0), "X": X, "T": T, "p0": _params(c, seed),
            "epochs": c["epochs"], "batch": c["batch"], "seed": seed & 0xffff}


def _prepare_predict(c, rng, seed):
    mlp = es_learned.MLP(c["dim"], 2, c["hidden"], seed=0)
    mlp.set_params(_params(c, seed))
    return {"mlp": mlp, "X": _rows(c, seed)[0]}


# ------------------------------------------------------------------ run
def run(state: dict):
    return globals()["_run_" + state["kind"]](state)


def _sorted(idx, room: int = 256) -> np.ndarray:
    """A survivor list in ascending order, in a buffer of fixed size: its length, then the list, then -1."""
    idx = np.sort(np.asarray(idx, dtype=np.int64), axis=0)
    out = np.full((1 + room,) + idx.shape[1:], -1, dtype=np.int64)
    out[0] = len(idx)
    out[1:1 + min(room, len(idx))] = idx[:room]
    return out


def _run_blocks(s):
    out = {"t0": s["t0"]}
    for i in range(s["blocks"]):
        out[f"block{i:02d}"] = _sorted(s["sieve"].scan_block(s["t0"] + i))
    return out


def _run_search(s):
    found = [v.search(None) for v in s["sieves"]]
    return {"k": np.array([r["k"] for r in found]), "block": np.array([r["block"] for r in found]),
            "survivors": np.array([r["survivors_in_block"] for r in found]),
            "g": np.array([[r["g"] >> 62, r["g"] & ((1 << 62) - 1)] for r in found], dtype=np.int64)}


def _run_chunk(s):
    # the drivers' calls of one chunk: block constants in, launch, survivor count and survivors out
    v = s["sieve"]
    v.tconst_h[:] = N.tconst_for(v.plan, s["t"])[:v.tconst_h.size]
    v.tconst.set(v.tconst_h)
    v.out_n.fill(0)
    v._launch(s["first"], s["count"])
    n = int(v.out_n.get()[0])
    return {"t": s["t"], "first": s["first"], "survivors": _sorted(v.out[:n].get())}


_run_wheel = _run_chunk


def _run_batches(s):
    b = s["batch"]
    b.run(use_graph=True)
    b.sync()
    surv = b.survivors()
    by_item = [_sorted(surv["idx"][surv["item"] == i], 64) for i in range(len(s["items"]))]
    groups = [b.group_min(i) for i in range(len(s["items"]))]
    return {"first": np.array([it[3] for it in s["items"]]), "survivors": np.array(by_item),
            "good": int(surv["good"].sum()),
            "least": np.array([[-1, -1, -1] if g is None else [g[0], g[1] >> 62, g[1] & ((1 << 62) - 1)]
                               for g in groups], dtype=np.int64)}


_run_pair = _run_batch = _run_batches


def _run_counts(s):
    c = s["ctx"]
    c.set_block(s["t"])
    c.reset_counts()
    c.reset()
    c.launch(s["first"], s["count"])
    return {"first": s["first"], "counts": c.stage_counts().astype(np.int64), "survivors": _sorted(c.survivors())}


def _run_mitm(s):
    surv, tested = s["engine"].scan(s["bound"])
    n = np.full((256, 2), -1, dtype=np.int64)     # ascending, as (high, low 62 bits), then -1
    for i, x in enumerate(surv[:256]):
        n[i] = x >> 62, x & ((1 << 62) - 1)
    return {"n": n, "survivors": len(surv), "tested": tested}


def _run_train(s):
    m = s["mlp"]
    m.set_params(s["p0"])
    loss = m.train(s["X"], s["T"], s["epochs"], s["batch"], 2e-3, s["seed"])
    return {"params": m.params(), "loss": np.float32(loss)}


def _run_predict(s):
    return s["mlp"].forward(s["X"])


# ------------------------------------------------------------------ work
def work(case: dict) -> dict:
    """Scans read nothing per position: their work is one decision per position (or per residue of
    the two halves), counted as one operation.  The network's is its multiply-adds and its rows."""
    kind = case["kind"]
    if kind == "blocks":
        return {"bytes": 0, "flops": case["blocks"] * _plan(case["k"]).R}
    if kind == "search":
        ks = range(case["k"], case["k"] + 16)
        per = sum(_plan(k).R * (1 + _known()[k] // _plan(k).M) for k in ks) / 16
        return {"bytes": 0, "flops": case["count"] * per}
    if kind in ("chunk", "wheel", "counts"):
        return {"bytes": 0, "flops": min(case["positions"], _plan(case["k"], case.get("role")).R)}
    if kind == "pair":
        return {"bytes": 0, "flops": 2 * case["positions"]}
    if kind == "batch":
        shape, total = random.Random(case["items"]), 0
        for _ in range(case["items"]):
            plan = _plan(shape.randint(case["k_lo"], case["k_hi"]))
            total += min(plan.R, int(2.0 ** shape.uniform(case["log2_lo"], case["log2_hi"])))
        return {"bytes": 0, "flops": total}
    if kind == "mitm":
        P = _mitm_plan(case["k"], case["mem_gb"])
        hits = case["bound_mult"] * P.E * (P.n1 * P.n2 / P.M)
        return {"bytes": 16 * P.n2, "flops": P.n1 + hits}
    D, H, n = case["dim"], case["hidden"], case["rows"]
    macs = D * H + H * H + H * 2
    if kind == "train":
        return {"bytes": 4 * n * (D + 2), "flops": 6 * macs * n * case["epochs"]}
    return {"bytes": 4 * n * (D + 2), "flops": 2 * macs * n}


# ------------------------------------------------------------------ exact (64-bit) values
def _split(P, D, H, O):
    at, out = 0, []
    for shape in ((H, D), (H,), (H, H), (H,), (O, H), (O,)):
        n = int(np.prod(shape))
        out.append(P[at:at + n].reshape(shape))
        at += n
    return out


def _forward64(P, X, D, H):
    W1, b1, W2, b2, W3, b3 = _split(P, D, H, 2)
    a1 = np.maximum(X @ W1.T + b1, 0.0)
    a2 = np.maximum(a1 @ W2.T + b2, 0.0)
    return a1, a2, a2 @ W3.T + b3


def _permutations(n: int, epochs: int, seed: int):
    """The trainer's seeded order of rows, one permutation per epoch (Fisher-Yates over splitmix64)."""
    mask, s, perm = (1 << 64) - 1, seed, list(range(n))
    for _ in range(epochs):
        for i in range(n - 1, 0, -1):
            s = (s + 0x9e3779b97f4a7c15) & mask
            z = ((s ^ (s >> 30)) * 0xbf58476d1ce4e5b9) & mask
            z = ((z ^ (z >> 27)) * 0x94d049bb133111eb) & mask
            j = (z ^ (z >> 31)) % (i + 1)
            perm[i], perm[j] = perm[j], perm[i]
        yield np.array(perm)


def exact(case: dict, seed: int):
    """The network's outputs in 64 bits; the scans' outputs are whole numbers."""
    if case["kind"] not in ("train", "predict"):
        return None
    D, H = case["dim"], case["hidden"]
    X, T = (a.astype(np.float64) for a in _rows(case, seed))
    P = _params(case, seed).astype(np.float64)
    if case["kind"] == "predict":
        return _forward64(P, X, D, H)[2]
    lr, b1, b2, eps = 2e-3, 0.9, 0.999, 1e-8
    m, v, step = np.zeros_like(P), np.zeros_like(P), 0
    for perm in _permutations(case["rows"], case["epochs"], seed & 0xffff):
        for at in range(0, case["rows"], case["batch"]):
            rows = perm[at:at + case["batch"]]
            x, t = X[rows], T[rows]
            a1, a2, y = _forward64(P, x, D, H)
            W1, _, W2, _, W3, _ = _split(P, D, H, 2)
            go = 2.0 * (y - t) / y.size
            g2 = (go @ W3) * (a2 > 0)
            g1 = (g2 @ W2) * (a1 > 0)
            g = np.concatenate([(g1.T @ x).ravel(), g1.sum(0), (g2.T @ a1).ravel(), g2.sum(0),
                                (go.T @ a2).ravel(), go.sum(0)])
            step += 1
            m = b1 * m + (1 - b1) * g
            v = b2 * v + (1 - b2) * g * g
            P = P - lr * (m / (1 - b1 ** step)) / (np.sqrt(v / (1 - b2 ** step)) + eps)
    y = _forward64(P, X, D, H)[2]
    return {"params": P, "loss": np.float64(np.mean((y - T) ** 2))}
