"""The measured workloads of the clustering library: what its users have it do,
through the public Python entry points (the C ABI of include/ngia.h).

Kinds of case:
  pairs   Context.pair_scores: one representative against a handful of records.
  scores  rep_scores_noalloc: one representative against records that are
          already in device memory owned by the caller.
  open    the `cluster` tool's path: open a database, cluster it, close it.
  whole   Context.cluster to the end with the tool's driver (speculative rounds).
  greedy  the first greedy iterations of a large database with the graph
          driver: begin, step, end (a large job runs for minutes, step by step).
  batch   Batch.run: independent jobs side by side.
  serve   Server: query batches against a resident representative set.

Databases come from the library's seeded generator (families of mutated
ancestors).  All outputs are whole numbers (assignments, scores, counts).
"""
from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parents[1]
if str(ROOT / "ngia-metax_gb300") not in sys.path:
    sys.path.insert(0, str(ROOT / "ngia-metax_gb300"))

import ngia  # noqa: E402

MODES = {"graph": ngia.MODE_GRAPH, "spec": ngia.MODE_SPEC, "plain": ngia.MODE_PLAIN, "pool": ngia.MODE_POOL}


def listed():
    return [
        # checking one sequence against a few others: the smallest call
        dict(name="pairs_dna_32", kind="pairs", type=0, n=256, length=1450, spread=80, s=0.85, w=5, precise=0, pairs=32),
        # scoring inside another application's loop, its buffers on the device
        dict(name="scores_dna_4k", kind="scores", type=0, n=4096, length=1450, spread=80, s=0.85),
        dict(name="scores_protein_1k", kind="scores", type=1, n=1000, length=380, spread=0, s=0.7),
        # the cluster tool on a small set of reads
        dict(name="open_dna_500", kind="open", type=0, n=500, length=600, spread=60, s=0.85, w=5, precise=0),
        # the 20,000-sequence 16S-like job, clustered to the end
        dict(name="whole_dna_20k", kind="whole", type=0, n=20000, length=1450, spread=80, s=0.85, w=5, precise=0),
        # the million-sequence job: representatives far longer than the candidates
        dict(name="greedy_dna_1m", kind="greedy", type=0, n=1000000, length=1450, spread=120, s=0.85, w=5, precise=0,
             iters=12),
        # the same families at a species-level cut-off
        dict(name="greedy_dna_s95", kind="greedy", type=0, n=250000, length=1450, spread=120, s=0.95, w=5, precise=0,
             iters=24),
        # peptides at high similarity: long tail of lengths, few members
        dict(name="greedy_protein_s90", kind="greedy", type=1, n=100000, length=380, spread=0, s=0.9, w=3, precise=0,
             iters=48),
        # peptides at low similarity, clustered to the end
        dict(name="whole_protein_s50", kind="whole", type=1, n=30000, length=380, spread=0, s=0.5, w=2, precise=0),
        # mixed jobs side by side: some samples of DNA, some of protein
        dict(name="batch_mixed_12", kind="batch", jobs=12, n_max=4000, iters=32, mode="graph"),
        # one small request to the service
        dict(name="serve_one", kind="serve", reps=6000, batches=1, n_max=24, s=0.9, w=5),
        # requests of many sizes at once
        dict(name="serve_burst", kind="serve", reps=6000, batches=16, n_max=2048, s=0.9, w=5),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cells(n, iters, length):
    """Rough cost of a greedy run, to keep drawn cases below the largest listed one."""
    return float(n) * iters * length * length


def draw(rng):
    kind = rng.choice(["pairs", "scores", "open", "whole", "whole", "greedy", "greedy", "batch", "serve", "serve"])
    t = rng.choice([0, 0, 1])
    c = dict(kind=kind, type=t)
    if kind in ("batch", "serve"):
        del c["type"]
    else:
        c["length"] = _log(rng, 150, 2600) if t == 0 else _log(rng, 120, 600)
        c["spread"] = max(1, int(c["length"] * rng.uniform(0.02, 0.12))) if t == 0 else 0
        c["s"] = rng.choice([0.8, 0.85, 0.9, 0.95, 0.99]) if t == 0 else rng.choice([0.5, 0.6, 0.7, 0.8, 0.9])
    if kind in ("pairs", "open", "whole", "greedy"):
        c["w"] = rng.choice([4, 5, 6, 8]) if t == 0 else rng.choice([2, 3])
        c["precise"] = 1 if rng.random() < 0.15 else 0
    if kind == "pairs":
        c["n"] = _log(rng, 40, 4000)
        c["pairs"] = rng.randint(1, c["n"])
    elif kind == "scores":
        c["n"] = _log(rng, 1, 20000)
    elif kind == "open":
        c["n"] = _log(rng, 2, 3000)
    elif kind == "whole":
        n = _log(rng, 300, 20000)
        while _cells(n, n, c["length"]) > _cells(16000, 16000, 1450):
            n = n * 3 // 4
        c["n"] = n
    elif kind == "greedy":
        n, c["iters"] = _log(rng, 20000, 400000), _log(rng, 4, 64)
        while _cells(n, c["iters"], c["length"]) > _cells(400000, 24, 1450):
            n = n * 3 // 4
        c["n"] = n
    elif kind == "batch":
        c["jobs"], c["n_max"] = rng.randint(2, 16), _log(rng, 1200, 4000)
        c["iters"], c["mode"] = _log(rng, 4, 32), rng.choice(["graph", "graph", "pool", "spec"])
    else:
        c["reps"], c["batches"] = _log(rng, 200, 6000), rng.randint(1, 12)
        c["n_max"], c["s"], c["w"] = _log(rng, 2, 2048), rng.choice([0.85, 0.9, 0.95]), rng.choice([4, 5, 7])
    return c


# ---- inputs --------------------------------------------------------------------


def _unknown(seqs, seed):
    """A few unread positions (N, or X-like characters the alphabet skips), as sequencers leave them."""
    rng = np.random.default_rng(seed)
    size = len(seqs.seq)
    if size:
        seqs.seq[rng.integers(0, size, size // 4000)] = ord("N")


def _database(case, seed, n=None):
    """One database of the case's type, size and lengths."""
    n = case["n"] if n is None else n
    length, spread = case["length"], case["spread"]
    if case["type"] == 0:
        seqs = ngia.synth(type=0, n_seqs=n, n_ancestors=max(1, n // 50), len_dist=0, len_a=float(length),
                          len_b=float(spread), len_min=max(1, length - 5 * spread), len_max=length + 5 * spread,
                          subst_max=0.2, indel_frac=0.05, indel_max=3, seed=seed)
        _unknown(seqs, seed)
    else:
        seqs = ngia.synth(type=1, n_seqs=n, n_ancestors=max(1, n // 25), len_dist=1, len_a=float(length), len_b=0.7,
                          len_min=20, len_max=35000, subst_max=0.5, indel_frac=0.05, indel_max=5, seed=seed)
    db = ngia.DB.pack(case["type"], seqs, seqs.off)
    seqs.close()
    return db


def _params(case):
    return ngia.params_clamp(case["type"], case["s"], case["w"], case["precise"])


def _spread(j):
    """0 <= x < 1, spread evenly for j = 0, 1, 2, ... (the golden ratio's multiples)."""
    return (j * 0.6180339887498949) % 1.0


def _batch_jobs(case, seed):
    """Jobs of sizes spread over the logarithm: DNA of log-uniform length 100-10,000 or proteins."""
    dbs, params = [], []
    for j in range(case["jobs"]):
        t = j % 2
        n = int(round(1000 * (case["n_max"] / 1000) ** _spread(j)))
        if t == 0:
            seqs = ngia.synth(type=0, n_seqs=n, n_ancestors=max(1, n // 50), len_dist=2, len_a=100.0, len_b=10000.0,
                              len_min=100, len_max=10000, subst_max=0.2, indel_frac=0.05, indel_max=3,
                              seed=seed * 1009 + j)
        else:
            seqs = ngia.synth(type=1, n_seqs=n, n_ancestors=max(1, n // 25), len_dist=1, len_a=380.0, len_b=0.7,
                              len_min=20, len_max=35000, subst_max=0.5, indel_frac=0.05, indel_max=5,
                              seed=seed * 1009 + j)
        dbs.append(ngia.DB.pack(t, seqs, seqs.off))
        seqs.close()
        params.append(ngia.params_clamp(t, (0.9, 0.8, 0.95)[j // 2 % 3], 5, 0))
    return dbs, params


def _serving(case, seed):
    """A resident set and query batches: windows of log-uniform length 200-3,000 over
    descendants of the same ancestors, one in ten from novel ones."""
    rng = np.random.default_rng(seed)
    family = dict(type=0, n_ancestors=400, len_dist=0, len_a=1450.0, len_b=80.0, len_min=1200, len_max=1700,
                  subst_max=0.2, indel_frac=0.05, indel_max=3)
    sizes = [case["n_max"]] + [int(round(case["n_max"] ** _spread(j))) for j in range(1, case["batches"])]
    seqs = ngia.synth(n_seqs=case["reps"], seed=seed, **family)
    reps = ngia.DB.pack(0, seqs, seqs.off)
    seqs.close()
    pool = ngia.synth(n_seqs=case["reps"] + sum(sizes) + 2, seed=seed, novel_frac=0.1, **family)
    batches, k = [], case["reps"]
    for m in sizes:
        parts, off = [], np.zeros(m + 1, dtype=np.int64)
        for q in range(m):
            want = int(round(math.exp(rng.uniform(math.log(200), math.log(3000)))))
            start = int(pool.off[k])
            start += int(rng.integers(0, max(1, int(pool.off[k + 1]) - start - want + 1)))
            part = pool.seq[start:start + want]
            parts.append(part)
            off[q + 1] = off[q] + len(part)
            k += 1
        batches.append(ngia.DB.pack(0, np.concatenate(parts), off))
    pool.close()
    return reps, batches


def prepare(case, seed):
    kind = case["kind"]
    state = dict(case=case)
    if kind == "batch":
        state["dbs"], state["params"] = _batch_jobs(case, seed)
        state["batch"] = ngia.Batch(state["dbs"])
    elif kind == "serve":
        state["reps"], state["batches"] = _serving(case, seed)
        slots = max(1, min(16, case["batches"]))
        state["server"] = ngia.Server(state["reps"], ngia.params_clamp(0, case["s"], case["w"], 0), slots=slots,
                                      max_batch=4096, max_record_blocks=96)
    elif kind == "scores":
        db = _database(case, seed, case["n"] + 1)
        state["rep"] = int(db.rec_off[db.n // 4])  # a representative of ordinary length
        state["words"] = torch.from_numpy(np.ascontiguousarray(db.words).view(np.int32)).cuda()
        order = np.random.default_rng(seed).permutation(db.n)[:case["n"]]
        state["queries"] = torch.from_numpy(db.rec_off[order].astype(np.int64)).cuda()
        state["out"] = torch.empty(case["n"], dtype=torch.int32, device="cuda")
    else:
        state["db"] = _database(case, seed)
        state["params"] = _params(case)
        if kind != "open":
            state["ctx"] = ngia.Context(state["db"])
        if kind == "pairs":
            state["rep"] = state["db"].n // 4
            rng = np.random.default_rng(seed)
            state["cands"] = rng.permutation(state["db"].n)[:case["pairs"]].astype(np.int32)
    return state


# ---- one pass -------------------------------------------------------------------


def _counts(st):
    return np.array([st[k] for k in ("iterations", "members")], dtype=np.int64)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "pairs":
        return state["ctx"].pair_scores(state["params"], state["rep"], state["cands"])
    if kind == "scores":
        ngia.rep_scores_noalloc(state["words"].data_ptr(), state["rep"], state["queries"].data_ptr(), case["n"],
                                case["type"], case["s"], state["out"].data_ptr(),
                                torch.cuda.current_stream().cuda_stream)
        return state["out"]
    if kind == "open":
        with ngia.Context(state["db"]) as ctx:
            cl, ident, st = ctx.cluster(state["params"], ngia.MODE_SPEC)
        return cl, ident, _counts(st)
    if kind == "whole":
        cl, ident, st = state["ctx"].cluster(state["params"], ngia.MODE_SPEC)
        return cl, ident, _counts(st)
    if kind == "greedy":
        ctx = state["ctx"]
        ctx.begin(state["params"], ngia.MODE_GRAPH)
        ctx.step(case["iters"])
        cl, ident, st = ctx.end()
        return cl, ident, _counts(st)
    if kind == "batch":
        cls, ids, st = state["batch"].run(state["params"], MODES[case["mode"]], case["iters"])
        return cls, ids, _counts(st)
    server = state["server"]
    tickets = [server.submit(b) for b in state["batches"]]
    got = [server.wait(t) for t in tickets]
    return np.concatenate([g[0] for g in got]), np.concatenate([g[1] for g in got])


# ---- the work a pass cannot do without --------------------------------------------


def _record_bytes(t, length):
    return 4 * ((6 if t == 0 else 30) + math.ceil(length / 32) * (2 if t == 0 else 5))


def _pair_ops(t, l1, l2, s):
    """Integer operations of one banded comparison: per 32 cells a match, an add and a
    merge (protein: five planes make the match), over the diagonals a result can reach."""
    band = min(l1, (l1 - s * l2) + (1 - s) * l2 + 32)
    return (3 if t == 0 else 7) * l2 * band / 32


def work(case):
    kind = case["kind"]
    if kind == "batch":
        # geometric mean sizes of the jobs; about half of a job's pairs are compared to the end
        n = math.sqrt(1000 * case["n_max"])
        dna, pro = (case["jobs"] + 1) // 2, case["jobs"] // 2
        per = n * case["iters"]
        flops = dna * per * _pair_ops(0, 8000, 2000, 0.9) / 4 + pro * per * 40
        size = dna * n * (_record_bytes(0, 2150) + 8) + pro * n * (_record_bytes(1, 486) + 8)
        return {"bytes": size, "flops": flops}
    if kind == "serve":
        q = case["n_max"] + (case["batches"] - 1) * case["n_max"] / max(1.0, math.log(max(2, case["n_max"])))
        size = case["reps"] * _record_bytes(0, 1450) + q * (_record_bytes(0, 800) + 8)
        # a query that no representative takes is compared with most of the resident set
        return {"bytes": size, "flops": q * case["reps"] / 2 * _pair_ops(0, 1450, 800, case["s"]) / 2}
    t, n, s = case["type"], case["n"], case["s"]
    mean = case["length"] * (1.0 if t == 0 else 1.28)
    size = n * _record_bytes(t, mean)
    if kind == "pairs":
        return {"bytes": (case["pairs"] + 1) * _record_bytes(t, mean) + 16 * case["pairs"],
                "flops": case["pairs"] * _pair_ops(t, mean, mean, s)}
    if kind == "scores":
        return {"bytes": size + 12 * n, "flops": n * _pair_ops(t, mean, mean, s)}
    if kind == "greedy":
        longest = case["length"] + 4.5 * case["spread"]
        # most DNA candidates are compared (about half of a comparison decides it); few protein pairs are
        flops = n * case["iters"] * (_pair_ops(0, longest, mean, s) / 2 if t == 0 and s < 0.93 else 10 if t == 0 else 40)
        return {"bytes": size + 8 * n, "flops": flops}
    # to the end: about half of the sequences become representatives, each against the sequences left
    share = 0.5 if t == 0 else 0.3
    pairs = n * n * share / 2
    flops = pairs * (_pair_ops(t, mean, mean, s) / 2 if t == 0 and s < 0.93 else 40)
    return {"bytes": size + 8 * n, "flops": flops}


def exact(case, seed):
    """Every output is a whole number; there is nothing to compute in 64 bits."""
    return None
