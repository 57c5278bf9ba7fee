"""Performance cases of the alignment library: what its users have it do, through
the C ABI (by way of the Python binding's declarations), from one short pair to
the 1 Mbp pair and the 100,000-pair batch.

Sizes are the named workloads (2,000 bp pair, 1 Mbp pair, batch, serving mix),
the sizes of the FASTA fixtures (organelle- and virus-sized genomes) and ragged
ones between them.  Sequences are seeded synthetic DNA: a random sequence and a
mutated copy of a window of it between random flanks.
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.abspath("projekt-2012_b200"))
import swb200  # noqa: E402
from swb200 import chain, synth  # noqa: E402

DNA = (1, -3, -5, -2)       # the pair workloads' scoring
DNA_BATCH = (2, -3, -5, -2)  # the batch workload's scoring
OPS_PER_CELL = 7            # int32 max/add operations of one cell of the recurrence


def listed():
    return [
        # the smallest call: two short reads or primers, full alignment from host memory
        {"name": "pair_600", "kind": "pair", "rows": 611, "cols": 437, "sub": 0.08, "where": "host"},
        # the plain small pair of the named workloads: latency of one call
        {"name": "pair_2k", "kind": "pair", "rows": 2000, "cols": 1993, "sub": 0.10, "where": "host"},
        # organelle-sized genomes (mitochondria), ragged
        {"name": "pair_17k", "kind": "pair", "rows": 17353, "cols": 12803, "sub": 0.07, "where": "host"},
        # herpesvirus-sized genomes (the 162 kbp x 172 kbp fixture pair's lengths), resident on the GPU
        {"name": "pair_172k", "kind": "pair", "rows": 172764, "cols": 162114, "sub": 0.05, "where": "device"},
        # the headline: the 1 Mbp pair, full path
        {"name": "pair_1m", "kind": "pair", "rows": 1000000, "cols": 999983, "sub": 0.05, "where": "device"},
        # screening: score and end cell only, resident sequences
        {"name": "score_61k", "kind": "score", "rows": 61003, "cols": 47111, "sub": 0.12, "where": "device"},
        # assembled contigs with N runs and IUPAC ambiguity codes (more than four letters)
        {"name": "iupac_41k", "kind": "iupac", "rows": 41234, "cols": 33333, "sub": 0.05, "where": "host"},
        # a pair whose special rows and columns exceed the caller's HBM budget (coarse grid and recompute)
        {"name": "budget_260k", "kind": "budget", "rows": 261111, "cols": 237007, "sub": 0.03, "where": "device"},
        # one block of a long pair split over GPUs by columns: borders in, borders out
        {"name": "block_131k", "kind": "block", "rows": 131072, "cols": 100003, "sub": 0.05, "where": "device"},
        # a small batch, every pair aligned: one iteration of a service
        {"name": "batch_24", "kind": "batch", "pairs": 24, "median": 2200, "traced": 1.0},
        # the batch workload: 100,000 uneven pairs, the best 1% aligned
        {"name": "batch_100k", "kind": "batch", "pairs": 100000, "median": 1000, "traced": 0.01},
        # a burst of short requests through the serving loop
        {"name": "serve_48", "kind": "serve", "pairs": 48},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pair", "pair", "pair", "score", "iupac", "budget", "block", "batch", "batch", "serve"])
    if kind == "batch":
        pairs = _log_uniform(rng, 1, 50000)
        return {"kind": "batch", "pairs": pairs, "median": rng.randint(400, 2500) if pairs < 3000 else rng.randint(400, 1100),
                "traced": 1.0 if pairs <= 512 else rng.choice([0.0, 0.01, 0.05])}
    if kind == "serve":
        return {"kind": "serve", "pairs": rng.randint(1, 200)}
    lo, hi = {"pair": (150, 700000), "score": (150, 700000), "iupac": (500, 200000), "budget": (190000, 400000),
              "block": (5000, 300000)}[kind]
    cols = _log_uniform(rng, lo, hi)
    rows = int(round(cols * rng.uniform(1.0, 2.0)))
    if kind == "block":
        rows = max(512, rows // 512 * 512)
        cols = min(cols, rows - 1)
    return {"kind": kind, "rows": rows, "cols": cols, "sub": round(rng.uniform(0.02, 0.14), 3),
            "where": rng.choice(["host", "device"]) if kind in ("pair", "score", "iupac") else "device"}


# ------------------------------------------------------------------ inputs

KINDS = {"pair": 1, "score": 2, "iupac": 3, "budget": 4, "block": 5, "batch": 6, "serve": 7}


def _rng(case, seed):
    return np.random.Generator(np.random.PCG64([seed, KINDS[case["kind"]], case.get("rows", 0), case.get("cols", 0),
                                                case.get("pairs", 0)]))


def _fit(rng, seq, n):
    """seq cut or filled with random bases to n."""
    return seq[:n] if len(seq) >= n else np.concatenate([seq, synth.random_dna(rng, n - len(seq))])


def _pair(case, seed):
    """rows and cols: cols holds a mutated copy of a window of rows between random flanks."""
    rng = _rng(case, seed)
    m, n = case["rows"], case["cols"]
    a = synth.random_dna(rng, m)
    flank = n // 10
    core = n - 2 * flank
    at = int(rng.integers(0, m - core + 1))
    b = np.concatenate([synth.random_dna(rng, flank), synth.mutate(rng, a[at:at + core], case["sub"], 0.01, 4.0)])
    b = _fit(rng, b, n)
    if case["kind"] == "iupac":
        a, b = _ambiguous(rng, a), _ambiguous(rng, b)
    return a, b


def _ambiguous(rng, s):
    s = s.copy()
    codes = np.frombuffer(b"RYKMSWN", dtype=np.uint8)
    at = rng.integers(0, len(s), size=max(1, len(s) // 500))
    s[at] = codes[rng.integers(0, len(codes), size=len(at))]
    for start in rng.integers(0, len(s), size=max(1, len(s) // 8000)).tolist():
        s[start:start + int(rng.integers(10, 200))] = ord("N")
    return s


def _requests(case, seed):
    """The serving mix's short requests: (query, target) with target 1.5 times the query."""
    rng = _rng(case, seed)
    out = []
    for n in _query_lengths(case).tolist():
        q = synth.random_dna(rng, n)
        left = int(rng.integers(0, n // 2 + 1))
        t = np.concatenate([synth.random_dna(rng, left), synth.mutate(rng, q, 0.07, 0.01, 3.0)])
        out.append((q, _fit(rng, t, int(round(1.5 * n)))))
    return out


def _query_lengths(case):
    """Query lengths are part of the case, not of the seed: outputs keep their shapes."""
    rng = _rng(case, 0)
    if case["kind"] == "serve":
        return rng.integers(200, 5001, size=case["pairs"])
    return np.clip(np.round(rng.lognormal(math.log(case["median"]), 0.75, size=case["pairs"])), 100,
                   10000).astype(np.int64)


def _batch(case, seed):
    """One buffer of queries and targets (target 1.5 times its query: a mutated copy
    of it at a random offset inside random padding) and the pairs' byte ranges."""
    q = _query_lengths(case)
    t = np.round(1.5 * q).astype(np.int64)
    ends = np.cumsum(q + t)
    offs = ends - q - t
    refs = np.stack([offs, q, offs + q, t], axis=1)
    g = torch.Generator(device="cuda").manual_seed(1000003 * seed + case["pairs"])
    dev, total = "cuda", int(ends[-1])
    bases = torch.tensor(list(b"ACGT"), dtype=torch.uint8, device=dev)
    buf = bases[torch.randint(0, 4, (total,), generator=g, device=dev)]
    nt = int(t.sum())
    td, qd, od = (torch.from_numpy(x).to(dev) for x in (t, q, offs))
    pair = torch.repeat_interleave(torch.arange(len(q), device=dev), td)
    pos = torch.arange(nt, device=dev) - (torch.cumsum(td, 0) - td)[pair]        # position in the target
    left = (torch.rand(len(q), generator=g, device=dev) * (td - qd + 1)).long()
    event = torch.rand(nt, generator=g, device=dev)
    size = 1 + (torch.empty(nt, device=dev).exponential_(0.4, generator=g)).long()  # indel lengths
    step = torch.where(event < 0.005, 1 + size, torch.where(event < 0.01, 1 - size, torch.ones_like(size)))
    walk = torch.cumsum(step, 0)
    first = (torch.cumsum(td, 0) - td) + left                                    # the copy's first target position
    src = walk - walk[first][pair]
    live = (pos >= left[pair]) & (src >= 0) & (src < qd[pair])
    live &= torch.rand(nt, generator=g, device=dev) >= 0.08                       # substitutions
    where = (od + qd)[pair] + pos
    buf[where[live]] = buf[(od[pair] + src)[live]]
    host = buf.cpu().numpy()
    del buf, pair, pos, event, size, step, walk, src, live, where
    torch.cuda.empty_cache()
    return host, refs


# ------------------------------------------------------------------ calls

def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        host, refs = _batch(case, seed)
        return {"case": case, "ctx": swb200.Context(device=0), "seq": host, "refs": swb200.pair_refs(refs),
                "sc": swb200.scoring(*DNA_BATCH)}
    if kind == "serve":
        return {"case": case, "server": swb200.Server(swb200.scoring(*DNA), hbm_budget_bytes=8 << 30),
                "reqs": [(q.tobytes(), t.tobytes()) for q, t in _requests(case, seed)]}
    a, b = _pair(case, seed)
    st = {"case": case, "sc": swb200.scoring(*DNA),
          "ctx": swb200.Context(device=0, hbm_budget_bytes=(1 << 30) if kind == "budget" else 0)}
    if kind == "block":
        _prepare_block(st, a, b)
    elif case["where"] == "host":
        st["a"], st["b"] = a.tobytes(), b.tobytes()
    else:
        st["a"], st["b"] = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
        torch.cuda.synchronize()
    return st


def _prepare_block(st, a, b):
    """The block's place in a larger matrix: 512 rows above it and 1,024 columns left
    of it, whose borders are what the block gets from its neighbours."""
    rng = np.random.Generator(np.random.PCG64(len(a)))
    rows = np.concatenate([synth.random_dna(rng, 1536), a])
    cols = np.concatenate([synth.random_dna(rng, 1024), b])
    dr, dc = torch.from_numpy(rows).cuda(), torch.from_numpy(cols).cuda()
    torch.cuda.synchronize()
    blk = chain.GpuBlocks(st["ctx"], dr, dc, st["sc"])
    r0, c0, m, n = 512, 1024, st["case"]["rows"], len(cols)
    top, _, _ = blk(0, r0, 0, n, None, None, 0, True, False)
    _, right, _ = blk(r0, r0 + m, 0, c0, top[:c0].contiguous(), None, 0, False, True)
    st["blk"] = blk
    st["args"] = (r0, r0 + m, c0, n, top[c0:].contiguous(), right, int(top[c0 - 1][0]), True, True)


def _whole(ptr, count, record, capacity):
    """`count` records of `record` bytes at ptr, whole, zero-filled to `capacity` records."""
    out = np.zeros(capacity * record, dtype=np.uint8)
    if count:
        C.memmove(out.ctypes.data, C.cast(ptr, C.c_void_p), count * record)
    return out


def _result(r):
    """The outputs of a swb_result: score, cells, operations and crosspoints, whole."""
    return {"score": int(r.score), "end": np.array([r.end_row, r.end_col], dtype=np.int64),
            "start": np.array([r.start_row, r.start_col], dtype=np.int64),
            "ops": _whole(r.ops, r.n_ops, 1, r.rows + r.cols),
            "xpoints": _whole(r.xpoints, r.n_xpoints, C.sizeof(swb200.XPoint), r.rows // 20 + 4).view(np.int32)}


def run(state):
    kind = state["case"]["kind"]
    if kind == "batch":
        return _run_batch(state)
    if kind == "serve":
        return _run_serve(state)
    if kind == "block":
        bottom, right, best = state["blk"](*state["args"])
        return {"bottom": bottom, "right": right, "best": np.array(best, dtype=np.uint64).view(np.int64)}
    L, ctx, a, b = swb200.lib(), state["ctx"], state["a"], state["b"]
    flags = swb200.FLAG_SCORE_ONLY if kind == "score" else 0
    r = swb200.Result()
    if state["case"]["where"] == "host":
        rc = L.swb_align_pair(ctx._h, a, len(a), b, len(b), C.byref(state["sc"]), flags, C.byref(r))
    else:
        rc = L.swb_align_pair_device(ctx._h, a.data_ptr(), a.numel(), b.data_ptr(), b.numel(), C.byref(state["sc"]),
                                     flags, C.byref(r))
    if rc != swb200.SWB_OK:
        raise swb200.SwbError(rc, L.swb_last_error(ctx._h).decode())
    out = _result(r)
    L.swb_result_free(C.byref(r))
    return out


def _run_batch(state):
    L, ctx, seq, refs = swb200.lib(), state["ctx"], state["seq"], state["refs"]
    r = swb200.BatchResult()
    rc = L.swb_batch_align(ctx._h, seq.ctypes.data, seq.nbytes, refs, len(refs), C.byref(state["sc"]), 0,
                           state["case"]["traced"], C.byref(r))
    if rc != swb200.SWB_OK:
        raise swb200.SwbError(rc, L.swb_last_error(ctx._h).decode())
    item = np.dtype({"names": [f for f, _ in swb200.BatchItem._fields_],
                     "formats": [np.dtype(t) for _, t in swb200.BatchItem._fields_],
                     "offsets": [getattr(swb200.BatchItem, f).offset for f, _ in swb200.BatchItem._fields_],
                     "itemsize": C.sizeof(swb200.BatchItem)})
    items = np.frombuffer(C.string_at(r.items, r.npairs * C.sizeof(swb200.BatchItem)), dtype=item)
    out = {f: items[f].copy() for f in item.names}
    most = np.sort(_shapes(state["case"]).sum(axis=1))[len(refs) - r.n_traced:].sum()
    out["ops"] = _whole(r.ops, r.ops_bytes, 1, most)
    out["xpoints"] = _whole(r.xpoints, r.n_xpoints, C.sizeof(swb200.XPoint), most // 20 + 4 * r.n_traced).view(np.int32)
    L.swb_batch_result_free(C.byref(r))
    return out


def _run_serve(state):
    L, srv = swb200.lib(), state["server"]
    ids = [srv.submit(q, t) for q, t in state["reqs"]]
    outs = []
    for rid in ids:
        r, info = swb200.Result(), swb200.RequestInfo()
        rc = L.swb_server_wait(srv._h, rid, -1, C.byref(r), C.byref(info))
        if rc != swb200.SWB_OK:
            raise swb200.SwbError(rc, (L.swb_server_last_error(srv._h) or b"").decode())
        outs.append(_result(r))
        L.swb_result_free(C.byref(r))
    out = {k: np.concatenate([o[k] for o in outs]) for k in ("end", "start", "ops", "xpoints")}
    out["score"] = np.array([o["score"] for o in outs], dtype=np.int64)
    return out


# ------------------------------------------------------------------ what a pass needs

def _shapes(case):
    """(rows, cols) of every pair of the case."""
    if case["kind"] in ("batch", "serve"):
        q = _query_lengths(case)
        return np.stack([np.round(1.5 * q).astype(np.int64), q], axis=1)
    return np.array([[case["rows"], case["cols"]]])


def work(case):
    """Sequences in, results out, and the recurrence's operations.  An aligned pair
    returns about one operation byte per column and a 24-byte crosspoint per 20 rows."""
    s = _shapes(case).astype(np.float64)
    cells = float((s[:, 0] * s[:, 1]).sum())
    nbytes = float(s.sum()) + 64.0 * len(s)
    traced = {"batch": case.get("traced", 0.0), "score": 0.0, "block": 0.0}.get(case["kind"], 1.0)
    nbytes += traced * float(s[:, 1].sum()) * (1 + 24 / 20)
    if case["kind"] == "block":
        nbytes += 16.0 * float(s.sum())  # borders in and out
    return {"bytes": nbytes, "flops": OPS_PER_CELL * cells}


def _score64(rows, cols, sc):
    """Best local score with affine gaps, row by row in 64 bits.  Within a row the
    horizontal gaps are a running maximum (opening costs at least extending)."""
    match, mismatch, gap_open, gap_ext = sc
    n = len(cols)
    ramp = np.arange(n, dtype=np.int64) * gap_ext
    h = np.zeros(n + 1, dtype=np.int64)
    f = np.full(n, -(1 << 40), dtype=np.int64)
    best = 0
    for ch in rows:
        f = np.maximum(f + gap_ext, h[1:] + gap_open)
        t = np.maximum(np.maximum(h[:-1] + np.where(cols == ch, match, mismatch), f), 0)
        run_max = np.maximum.accumulate(t - ramp)
        h[1:] = t
        h[2:] = np.maximum(t[1:], run_max[:-1] + ramp[:-1] + gap_open)
        best = max(best, int(h.max()))
    return best


def exact(case, seed):
    kind = case["kind"]
    cells = work(case)["flops"] / OPS_PER_CELL
    if kind in ("block", "batch") or cells > 6e8:
        return None
    if kind == "serve":
        scores = [_score64(t, q, DNA) for q, t in _requests(case, seed)]
        return {"score": np.array(scores, dtype=np.int64), "end": None, "start": None, "ops": None, "xpoints": None}
    a, b = _pair(case, seed)
    return {"score": _score64(a, b, DNA), "end": None, "start": None, "ops": None, "xpoints": None}
