"""Benchmark of the SW/Gotoh long-pair path on B200 (one JSON line on rank 0).

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]
                    [--workload long|small|chromosome]

A step is one full alignment of the workload pair through the library's C ABI.
`value` is GCUPS (rows * cols / seconds) with the sequences resident in HBM,
timed with CUDA events on the stream the library runs on; `e2e` is the same
metric through swb_align_pair() from pinned host buffers (host->device copy of
both sequences and the device->host read of the result inside the timed
region).  With N > 1 every rank aligns its own replica of the pair (weak
scaling, no collective on the data path) and the time is the max over ranks.
"""
from __future__ import annotations

import argparse
import json
import os
import subprocess
import sys
import tempfile
import threading
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(ROOT, "projekt-2012_b200"))

METRIC = "GCUPS (long pair, bit-exact); mixed-size pairs/s + p50/p99 latency vs plain"


def parse_args():
    p = argparse.ArgumentParser()
    p.add_argument("--gpus", type=int, default=1)
    p.add_argument("--steps", type=int, default=5)
    p.add_argument("--warmup", type=int, default=3)
    p.add_argument("--impl", choices=["ours", "reference"], default="ours")
    p.add_argument("--workload", choices=["long", "long200k", "long1mx250k", "long1mx64k", "tall10mx100k", "small",
                                          "chromosome"],
                   default="long")
    p.add_argument("--score-only", action="store_true", help="stage 1 only (diagnostics)")
    p.add_argument("--no-cpu-baseline", action="store_true")
    p.add_argument("--no-mixed", action="store_true", help="skip the batched and serving measurements")
    p.add_argument("--batch-pairs", type=int, default=100_000, help="pairs of the batched workload")
    p.add_argument("--serve-seconds", type=float, default=60.0, help="length of the Poisson serving run")
    p.add_argument("--no-serving", action="store_true", help="skip the serving measurement")
    p.add_argument("--no-chromosome", action="store_true", help="skip the 10 Mbp chromosome-pair sub-record")
    return p.parse_args()


def workload(name):
    from swb200 import synth
    if name == "long":
        a, b, sc = synth.long_pair()
        desc = ("long pair: 1 Mbp iid ACGT vs its central 800 kbp (5% sub, 1% indel, geometric "
                "mean 4) with 100 kbp random flanks; scoring 1/-3/-5/-2")
    elif name == "long200k":
        a, b, sc = synth.long_pair(length=200_000)
        desc = ("long pair scaled to 200 kbp (same construction and rates as the 1 Mbp pair), "
                "for profiling")
    elif name == "long1mx250k":
        a, b, sc = synth.long_pair()
        b = b[:250_000]
        desc = ("the 1 Mbp long pair's rows against the first 250 kbp of its columns (same strip "
                "count and occupancy as the full pair, a quarter of the steps), for profiling")
    elif name == "long1mx64k":
        a, b, sc = synth.long_pair()
        b = b[:65_536]
        desc = ("the 1 Mbp long pair's rows against the first 65,536 of its columns (same strips and grid as the "
                "full pair, about 3 GB of special rows and columns), for multi-pass profiles")
    elif name == "tall10mx100k":
        a, b, sc = synth.tall_pair()
        desc = ("10 Mbp iid rows against a mutated 100 kbp window of them (same strip count and occupancy "
                "as the chromosome-scale pair, 1% of its cells), for profiling")
    elif name == "small":
        a, b, sc = synth.plain_small()
        desc = "plain pair: 2,000 bp vs 400 + mutated 1,200 bp window + 400; scoring 1/-3/-5/-2"
    else:
        a, b, sc = synth.chromosome_pair()
        desc = ("chromosome pair: two ~10 Mbp from an 8 Mbp ancestor (3% sub, 0.5% indel, mean 4) + 1 Mbp "
                "random flanks on both ends; scoring 1/-3/-5/-2; special rows/columns within a 40 GB budget")
    return a, b, sc, desc


class ClockSampler:
    """nvidia-smi clocks and throttle reasons sampled every 200 ms."""

    def __init__(self, index: int):
        self.index = index
        self.proc = None
        self.lines = []

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--id={self.index}",
                 "--query-gpu=clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
                 "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
                 "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap",
                 "--format=csv,noheader,nounits", "-lms", "200"],
                stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            threading.Thread(target=self._read, daemon=True).start()
        except Exception:
            self.proc = None
        return self

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def __exit__(self, *exc):
        if self.proc:
            time.sleep(0.25)
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except Exception:
                self.proc.kill()

    def summary(self):
        sm, mx, reasons = [], 0, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in self.lines:
            f = [x.strip() for x in ln.split(",")]
            if len(f) < 8:
                continue
            try:
                sm.append(float(f[0]))
                mx = max(mx, float(f[1]))
            except ValueError:
                continue
            for nm, v in zip(names, f[4:8]):
                if v.lower().startswith("active"):
                    reasons.add(nm)
        if not sm:
            return None
        sm.sort()
        return {"sm_mhz": sm[len(sm) // 2], "sm_max_mhz": mx, "reasons": sorted(reasons),
                "samples": len(sm)}


def profile_traffic(workload_name):
    """DRAM bytes per stage-1 launch from the committed ncu summary, if any."""
    path = os.path.join(ROOT, "profiles", f"stage1_{workload_name}_pair.md")
    if not os.path.exists(path):
        return None
    for line in open(path):
        if line.startswith("dram_bytes_per_launch:"):
            try:
                return float(line.split(":", 1)[1].split()[0])
            except ValueError:
                return None
    return None


def cpu_model() -> str:
    """The host CPU's model name (from /proc/cpuinfo) and logical CPU count."""
    name = "unknown"
    try:
        for line in open("/proc/cpuinfo"):
            if line.startswith("model name"):
                name = line.split(":", 1)[1].strip()
                break
    except OSError:
        pass
    return f"{name}, {os.cpu_count()} logical CPUs"


def cpu_baseline(a: bytes, b: bytes, sc):
    """The oracle's fastest multithreaded CPU wavefront on this host (the AVX-512
    one where the CPU has it, else the scalar one; same int32 recurrence and tie
    rule) on a bounded sample of the same pair: a band of rows against all
    columns, sized for about 12 s on the host cores."""
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import oracle_ctypes as O
    rows, cols, _ = O.orient(a, b)
    threads = os.cpu_count() or 1
    lo = len(rows) // 10
    probe_rows = max(1, min(len(rows) - lo, int(2e9 // len(cols))))
    _, t, kind = O.stage1_fast(rows[lo:lo + probe_rows], cols, O.scoring(*sc), threads=threads)
    rate = probe_rows * len(cols) / max(t, 1e-6)
    nrows = max(1, min(len(rows) - lo, int(rate * 12.0 // len(cols))))
    _, t, kind = O.stage1_fast(rows[lo:lo + nrows], cols, O.scoring(*sc), threads=threads)
    cells = nrows * len(cols)
    impl = ("orc_stage1_simd: AVX-512 anti-diagonal strips of 16 rows" if kind == "avx512"
            else "orc_stage1_mt: scalar blocked wavefront")
    return {"value": cells / t / 1e9, "unit": "GCUPS", "cores": threads, "kind": "port", "cpu": cpu_model(),
            "sample": f"rows {lo}..{lo + nrows} of the rows sequence x all {len(cols)} columns "
                      f"({cells:.3e} cells, {t:.1f} s), score + end cell; {impl}"}


def reference_arm(args):
    """The reference's own kernels, compiled for the CPU (oracle/_ref, host threads
    standing in for its 2 x 5 CUDA threads), stage 1 on a bounded sample."""
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    a, b, sc, desc = workload(args.workload)
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import oracle_ctypes as O
    if not os.path.exists(O.REFEMU_PATH):
        print(json.dumps({"impl": "reference", "unavailable": "oracle/_ref/swalign_emu was not built"}))
        return
    rows, cols, _ = O.orient(a, b)
    lo = len(rows) // 10
    na = min(len(rows) - lo, 6000)
    nb = min(len(cols) - lo if len(cols) > lo + 100 else len(cols), 6000)
    sa = rows[lo:lo + na]
    sb = cols[lo:lo + nb] if len(cols) > lo + nb else cols[:nb]
    td = tempfile.mkdtemp()
    fa, fb = os.path.join(td, "a.fa"), os.path.join(td, "b.fa")
    open(fa, "wb").write(b">sample a\n" + sa + b"\n")
    open(fb, "wb").write(b">sample b\n" + sb + b"\n")
    for _ in range(args.warmup):
        O.run_reference(fa, fb, *sc, stage1_only=True)
    t0 = time.perf_counter()
    for _ in range(args.steps):
        O.run_reference(fa, fb, *sc, stage1_only=True)
    dt = time.perf_counter() - t0
    cells = len(sa) * len(sb) * args.steps
    v = cells / dt / 1e9
    cores = 5  # one block of the reference's forced 2 x 5 runs at a time, one host thread per CUDA thread
    line = {"metric": METRIC, "value": v, "unit": "GCUPS", "n_gpus": args.gpus, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": dt * 1e3 / args.steps, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "int32", "data": "synthetic",
            "impl": "reference",
            "config": {"workload": desc, "sample_rows": len(sa), "sample_cols": len(sb),
                       "stages": "stage 1 (score + end cell)"},
            "cpu_baseline": {"value": v, "unit": "GCUPS", "cores": cores, "kind": "reference", "cpu": cpu_model(),
                             "sample": f"{len(sa)} x {len(sb)} sub-pair of the workload, stage 1, "
                                       f"reference kernels on host threads"},
            "e2e": {"value": v, "unit": "GCUPS", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)


def percentile(xs, q):
    xs = sorted(xs)
    if not xs:
        return None
    k = min(len(xs) - 1, max(0, int(round(q / 100.0 * (len(xs) - 1)))))
    return xs[k]


def chromosome_metrics(args, device, peak_cells_per_s):
    """The chromosome-scale pair (two ~10 Mbp sequences, about 10^14 cells, special
    rows and columns within a 40 GB budget): one warm-up and one timed full
    alignment with the sequences resident in HBM, CUDA events on the library's
    stream, clocks sampled during the timed step; checked against the oracle's
    committed full-matrix golden when it exists."""
    import torch
    import swb200
    a, b, sc_t, desc = workload("chromosome")
    rows_b, cols_b = (a, b) if len(a) >= len(b) else (b, a)
    m, n = len(rows_b), len(cols_b)
    stream = torch.cuda.current_stream()
    ctx = swb200.Context(device=device, cuda_stream=stream.cuda_stream, hbm_budget_bytes=40_000_000_000)
    d_rows = torch.frombuffer(bytearray(rows_b), dtype=torch.uint8).cuda()
    d_cols = torch.frombuffer(bytearray(cols_b), dtype=torch.uint8).cuda()
    sc = swb200.scoring(*sc_t)
    ctx.align_device(d_rows.data_ptr(), m, d_cols.data_ptr(), n, sc, 0)  # warm-up
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    with ClockSampler(device) as clk:
        e0.record(stream)
        r = ctx.align_device(d_rows.data_ptr(), m, d_cols.data_ptr(), n, sc, 0)
        e1.record(stream)
        torch.cuda.synchronize()
    ms = e0.elapsed_time(e1)
    ctx.close()
    del d_rows, d_cols
    torch.cuda.empty_cache()
    golden = None
    gpath = os.path.join(ROOT, "tests", "golden", "chromosome_golden.json")
    if os.path.exists(gpath):
        g = json.load(open(gpath))["reference"]
        golden = (r.score, r.end_row, r.end_col) == (g["score"], g["end_row"], g["end_col"])
    achieved = m * n / (r.stage1_ms * 1e-3) / 1e9
    return {"workload": desc, "rows": m, "cols": n, "score": r.score, "end": [r.end_row + 1, r.end_col + 1],
            "oracle_golden_match": golden, "gcups": m * n / (ms * 1e-3) / 1e9, "ms": ms,
            "stage1_ms": r.stage1_ms, "stage2_ms": r.stage2_ms, "special_interval": r.special_interval,
            "special_bytes": r.special_bytes, "alignment_ops": len(r.ops),
            "roofline": {"achieved": achieved, "peak": peak_cells_per_s / 1e9, "unit": "GCUPS",
                         "frac": achieved * 1e9 / peak_cells_per_s, "kernel": "stage1_packed_kernel (scoring wavefront)"},
            "timing": "1 warm-up + 1 timed full alignment (stage 1 + special rows + GPU traceback)",
            "clocks": clk.summary()}


def batched_metrics(args, device):
    """The batched workload (100,000 pairs, log-normal query lengths, 1% traced)
    through swb_batch_align from a host buffer (copies inside the timed region),
    against the plain pair path (swb_align_pair, score only) on a sample of the
    same pairs."""
    import numpy as np
    import swb200
    from swb200 import synth
    buf, refs, sc_t = synth.batched(args.batch_pairs)
    sc = swb200.scoring(*sc_t)
    ctx = swb200.Context(device=device)
    for _ in range(2):
        ctx.batch_align(buf, refs, sc, trace_frac=0.01)
    runs = []
    for _ in range(3):
        t0 = time.perf_counter()
        r = ctx.batch_align(buf, refs, sc, trace_frac=0.01)
        runs.append((time.perf_counter() - t0, r.stage1_ms, r.stage2_ms, r.kernel_launches))
    wall = min(x[0] for x in runs)
    rng = np.random.default_rng(0)
    sample = rng.choice(len(refs), size=min(400, len(refs)), replace=False)
    t0 = time.perf_counter()
    for i in sample:
        ao, al, bo, bl = (int(v) for v in refs[i])
        p = ctx.align(buf[ao:ao + al].tobytes(), buf[bo:bo + bl].tobytes(), sc, swb200.FLAG_SCORE_ONLY)
        assert (p.score, p.end_row, p.end_col) == (r.score[i], r.end_row[i], r.end_col[i])
    plain = len(sample) / (time.perf_counter() - t0)
    # per-call cost of a serving-sized batch (32 pairs of 300-700 bp, every pair
    # traced): one replayed CUDA graph against the same kernels launched directly
    srng = np.random.default_rng(5)
    parts, srefs, off = [], [], 0
    for _ in range(32):
        la, lb = int(srng.integers(300, 700)), int(srng.integers(300, 700))
        a = srng.choice(np.frombuffer(b"ACGT", np.uint8), la)
        b = np.concatenate([a[: lb // 2], srng.choice(np.frombuffer(b"ACGT", np.uint8), lb - lb // 2)])
        parts += [a, b]
        srefs.append((off, la, off + la, lb))
        off += la + lb
    sbuf = np.concatenate(parts)
    srefs = np.array(srefs, dtype=np.int64)
    small = {}
    for mode in ("1", "0"):
        os.environ["SWB_BATCH_GRAPH"] = mode
        for _ in range(5):
            ctx.batch_align(sbuf, srefs, sc, trace_frac=1.0)
        ts = []
        for _ in range(60):
            t0 = time.perf_counter()
            rs = ctx.batch_align(sbuf, srefs, sc, trace_frac=1.0)
            ts.append((time.perf_counter() - t0) * 1e3)
        ts.sort()
        small[mode] = (ts[len(ts) // 2], rs.kernel_launches)
    os.environ.pop("SWB_BATCH_GRAPH", None)
    ctx.close()
    n = len(refs)
    return {"workload": f"{n} pairs, query clip(round(lognormal(ln 1000, 0.75)), 100, 10000), target 1.5x "
                        "(8% sub, 1% indel); scoring 2/-3/-5/-2; score + end cell of every pair, alignment of "
                        "the best 1%",
            "pairs_per_s": n / wall, "gcups": r.cells / wall / 1e9, "ms_per_batch": wall * 1e3,
            "stage1_ms": min(x[1] for x in runs), "stage2_ms": min(x[2] for x in runs),
            "kernel_launches": runs[-1][3], "plain_pairs_per_s": plain, "vs_plain": n / wall / plain,
            "plain_sample": f"{len(sample)} pairs of the same batch through swb_align_pair, score only, equal results",
            "timing": "wall clock of swb_batch_align from host memory (host->device copy, results back)",
            "small_batch": {"workload": "32 pairs of 300-700 bp, every pair traced (a serving iteration's size)",
                            "graph_ms_p50": small["1"][0], "graph_kernels": small["1"][1],
                            "direct_ms_p50": small["0"][0], "direct_kernels": small["0"][1],
                            "timing": "wall clock per swb_batch_align call, median of 60"}}


def serving_metrics(args, device):
    """Poisson stream of the serving mix at 80% of the measured capacity through
    the serving loop (swb_server_*), with latency per request; then the same
    arrivals through the plain path (swb_align_pair, one pair at a time in
    arrival order), measured the same way."""
    import numpy as np
    import swb200
    from swb200 import synth
    sc_t = (1, -3, -5, -2)
    sc = swb200.scoring(*sc_t)
    budget = 100 << 30
    # capacity: a burst from an independent draw of the same mix
    cap_rng = synth.rng_for(4, 99)
    burst = [synth.serving_request(cap_rng) for _ in range(160)]
    with swb200.Server(sc, device=device, hbm_budget_bytes=budget) as srv:
        t0 = time.perf_counter()
        ids = [srv.submit(q, t) for q, t, _ in burst]
        for i in ids:
            srv.wait(i)
        cap_t = time.perf_counter() - t0
    capacity = len(burst) / cap_t
    rate = 0.8 * capacity
    stream = synth.serving_stream(args.serve_seconds, rate)
    lat, lanes, cells = [], [], 0
    with swb200.Server(sc, device=device, hbm_budget_bytes=budget) as srv:
        ids = []
        start = time.perf_counter()
        for t_arr, q, tg, _ in stream:
            now = time.perf_counter() - start
            if t_arr > now:
                time.sleep(t_arr - now)
            ids.append(srv.submit(q, tg))
        for (t_arr, q, tg, lg), i in zip(stream, ids):
            res, info = srv.wait(i)
            lat.append(info["total_ms"])
            lanes.append(info["lane"])
            cells += len(q) * len(tg)
        span = time.perf_counter() - start
        st = srv.stats()
    # plain path, measured: the same arrivals served one pair at a time, in arrival
    # order, through swb_align_pair (full path) on one context; latency = finish -
    # arrival on the same clock
    ctx = swb200.Context(device=device, hbm_budget_bytes=budget // 2)
    ctx.align(stream[0][1], stream[0][2], sc)  # warm-up outside the stream
    plain_lat, plain_short, plain_long = [], [], []
    start = time.perf_counter()
    for t_arr, q, tg, lg in stream:
        now = time.perf_counter() - start
        if t_arr > now:
            time.sleep(t_arr - now)
        ctx.align(q, tg, sc)
        done = (time.perf_counter() - start - t_arr) * 1e3
        plain_lat.append(done)
        (plain_long if lg else plain_short).append(done)
    plain_span = time.perf_counter() - start
    ctx.close()
    short_lat = [x for x, l in zip(lat, lanes) if l == 0]
    long_lat = [x for x, l in zip(lat, lanes) if l == 1]
    return {"workload": f"Poisson arrivals for {args.serve_seconds:g} s at 80% of measured capacity; 95% short "
                        "(query U[200, 5000], target 1.5x, 7% sub + 1% indel), 5% long (query U[100k, 2M], target "
                        "1.5x, 2.5% sub + 0.5% indel); scoring 1/-3/-5/-2; full traceback; HBM budget 100 GiB",
            "capacity_pairs_per_s": capacity, "arrival_rate": rate, "requests": len(stream),
            "long_requests": int(sum(lanes)), "pairs_per_s": len(stream) / span, "gcups": cells / span / 1e9,
            "p50_ms": percentile(lat, 50), "p99_ms": percentile(lat, 99),
            "short_p50_ms": percentile(short_lat, 50), "short_p99_ms": percentile(short_lat, 99),
            "long_p50_ms": percentile(long_lat, 50), "long_p99_ms": percentile(long_lat, 99),
            "iterations": st["iterations"], "max_batch": st["max_batch_seen"],
            "plain_p50_ms": percentile(plain_lat, 50), "plain_p99_ms": percentile(plain_lat, 99),
            "plain_short_p99_ms": percentile(plain_short, 99), "plain_long_p99_ms": percentile(plain_long, 99),
            "plain_pairs_per_s": len(stream) / plain_span,
            "plain": "measured: the same arrivals through swb_align_pair one pair at a time in arrival order "
                     "(full path, one context), latency from arrival to result"}


def main():
    args = parse_args()
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if args.impl == "reference":
        reference_arm(args)
        return

    import torch
    import torch.distributed as dist
    import swb200
    from swb200.ranks import max_over_ranks, replica_throughput

    torch.cuda.set_device(local)
    if world > 1:
        dist.init_process_group("nccl", timeout=__import__("datetime").timedelta(seconds=120))

    a, b, sc_t, desc = workload(args.workload)
    sc = swb200.scoring(*sc_t)
    m, n = max(len(a), len(b)), min(len(a), len(b))
    rows_b, cols_b = (a, b) if len(a) >= len(b) else (b, a)
    cells = m * n
    stream = torch.cuda.current_stream()
    # the chromosome-scale pair keeps its special rows / columns within 40 GB
    budget = 40_000_000_000 if args.workload == "chromosome" else 0
    ctx = swb200.Context(device=local, cuda_stream=stream.cuda_stream, hbm_budget_bytes=budget)
    flags = swb200.FLAG_SCORE_ONLY if args.score_only else 0

    d_rows = torch.frombuffer(bytearray(rows_b), dtype=torch.uint8).cuda()
    d_cols = torch.frombuffer(bytearray(cols_b), dtype=torch.uint8).cuda()
    h_a = torch.frombuffer(bytearray(a), dtype=torch.uint8).pin_memory()
    h_b = torch.frombuffer(bytearray(b), dtype=torch.uint8).pin_memory()
    flush = torch.empty(256 << 20, dtype=torch.uint8, device="cuda")

    def step_device():
        flush.zero_()
        return ctx.align_device(d_rows.data_ptr(), m, d_cols.data_ptr(), n, sc, flags)

    def step_host():
        flush.zero_()
        return ctx.align_ptr(h_a.data_ptr(), len(a), h_b.data_ptr(), len(b), sc, flags)

    first = None
    for _ in range(args.warmup):
        first = step_device()
    torch.cuda.synchronize()

    def timed(fn):
        if world > 1:
            dist.barrier()
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        res = []
        e0.record(stream)
        for _ in range(args.steps):
            res.append(fn())
        e1.record(stream)
        torch.cuda.synchronize()
        ms = e0.elapsed_time(e1)
        if world > 1:
            ms = max_over_ranks(ms, "cuda")
            dist.barrier()
        return ms, res

    with ClockSampler(local) as clk:
        ms_dev, res_dev = timed(step_device)
    ms_e2e, res_e2e = timed(step_host)

    for r in res_dev + res_e2e:
        assert (r.score, r.end_row, r.end_col) == (first.score, first.end_row, first.end_col)

    value = replica_throughput(world, cells, args.steps, ms_dev) / 1e9
    e2e = replica_throughput(world, cells, args.steps, ms_e2e) / 1e9
    k_ms = sum(r.stage1_ms for r in res_dev) / len(res_dev)
    achieved = cells / (k_ms * 1e-3) / 1e9
    peak_cells = swb200.probe_packed_peak(local)
    wide_cells = swb200.probe_cell_peak(local)
    peak = peak_cells["cells_per_s"] / 1e9
    traffic = profile_traffic(args.workload)
    launches = sum(r.kernel_launches for r in res_dev)
    if rank != 0:
        if world > 1:
            dist.destroy_process_group()
        return
    # the CPU baseline and the single-GPU sub-records (batched, serving, 10 Mbp
    # pair) belong to the N = 1 line; at N > 1 they would hold every GPU for
    # minutes while rank 0 alone works
    single = world == 1
    cpu = None if (args.no_cpu_baseline or not single) else cpu_baseline(a, b, sc_t)
    mixed_batched = mixed_serving = chrom = None
    ctx.close()
    del d_rows, d_cols, flush
    torch.cuda.empty_cache()
    if not args.no_mixed and single:
        mixed_batched = batched_metrics(args, local)
        mixed_serving = None if args.no_serving else serving_metrics(args, local)
    if not args.no_chromosome and args.workload == "long" and single:
        chrom = chromosome_metrics(args, local, peak_cells["cells_per_s"])
    d2h = 64 + first.n_ops + 24 * len(first.xpoints)
    line = {
        "metric": METRIC, "value": value, "unit": "GCUPS", "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": ms_dev / args.steps, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "int32", "data": "synthetic",
        "config": {"workload": desc, "rows": m, "cols": n, "score": first.score,
                   "arithmetic": "exact int32 values, held in packed strips as a 32-bit base and 16-bit offsets; "
                                 "a pass whose offsets do not fit runs again in 32 bits",
                   "end": [first.end_row + 1, first.end_col + 1],
                   "stages": "stage 1 only" if args.score_only else
                             "stage 1 + special rows + GPU traceback (alignment, crosspoints)",
                   "special_interval": first.special_interval,
                   "parallelism": f"replicas x{world}" if world > 1 else "single GPU",
                   "l2": "256 MiB buffer written before every step (inside the timed region)"},
        "roofline": {"bound": "int16x2_dpx", "achieved": achieved, "peak": peak, "unit": "GCUPS",
                     "frac": achieved / peak, "traffic": traffic,
                     "kernel": "stage1_packed_kernel (scoring wavefront)",
                     "peak_source": "measured: swb_probe_packed_peak (the packed step's op mix, two cells per op, "
                                    "full occupancy)",
                     "peak_int32_mix": wide_cells["cells_per_s"] / 1e9,
                     "stage1_ms": k_ms, "stage2_ms": sum(r.stage2_ms for r in res_dev) / len(res_dev)},
        "cpu_baseline": cpu,
        "e2e": {"value": e2e, "unit": "GCUPS", "h2d_bytes_per_step": len(a) + len(b),
                "d2h_bytes_per_step": d2h},
        "gpu_launches": launches,
        "batched": mixed_batched,
        "serving": mixed_serving,
        "chromosome": chrom,
        "clocks": clk.summary(),
    }
    print(json.dumps(line), flush=True)
    if world > 1:
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
