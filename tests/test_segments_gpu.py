"""Stage 2 in segments walked at the same time (csrc/traceback.cu): paths whose
crossing of the special rows is not where the guess looks, for pairs and batches,
against the oracle's alignment."""
import random

import pytest

import oracle_ctypes as O
import swb200

pytestmark = pytest.mark.gpu


def _seq(rng, n):
    return bytes(rng.choice(b"ACGT") for _ in range(n))


def _mut(rng, s, p):
    out = bytearray()
    for ch in s:
        x = rng.random()
        if x < 0.6 * p:
            out.append(rng.choice(b"ACGT"))
        elif x < 0.8 * p:
            pass
        elif x < p:
            out += bytes([ch]) + _seq(rng, rng.randint(1, 5))
        else:
            out.append(ch)
    return bytes(out)


def _case(kind, rng):
    a = _seq(rng, 9000)
    if kind == "along the diagonal":
        return a, _mut(rng, a, 0.08)
    if kind == "a stronger alignment in the same rows":  # its H is higher than the path's there
        return a, _mut(rng, a[:3500], 0.01) + _seq(rng, 1500) + _mut(rng, a, 0.12)
    if kind == "long gaps":
        return a, _mut(rng, a[:4000], 0.04) + _seq(rng, 2300) + _mut(rng, a[4600:], 0.04)
    return a, _seq(rng, 8500)  # unrelated: linear-gap-like paths of random matches


@pytest.mark.parametrize("kind", ["along the diagonal", "a stronger alignment in the same rows", "long gaps", "unrelated"])
@pytest.mark.parametrize("sc", [(1, -3, -5, -2), (5, -4, -4, -4), (30, -20, -40, -10)])
def test_segments_give_the_serial_path(gpu_ctx, monkeypatch, kind, sc):
    rng = random.Random(len(kind) + sc[0])
    a, b = _case(kind, rng)
    rows, cols, _ = O.orient(a, b)
    e = O.stage1_fast(rows, cols, O.scoring(*sc), O.TIE_REFERENCE)[0]
    r = gpu_ctx.align(a, b, swb200.scoring(*sc))
    ops, sr, scol, xps = O.traceback_xp(rows, cols, O.scoring(*sc), e.row, e.col, r.xpoint_interval)
    want = (e.score, e.row, e.col, ops, sr, scol)
    assert (r.score, r.end_row, r.end_col, r.ops, r.start_row, r.start_col) == want
    assert [tuple(x) for x in r.xpoints[1:-1]] == [tuple(x) for x in xps]
    pairs = [(a[:1300], b[:900]), (a, b), (a[:40], b[:40]), (a[:2600], a[:2600])]
    buf, refs, off = b"".join(x + y for x, y in pairs), [], 0
    for x, y in pairs:
        refs.append((off, len(x), off + len(x), len(y)))
        off += len(x) + len(y)
    for graph in ("1", "0"):
        monkeypatch.setenv("SWB_BATCH_GRAPH", graph)
        t = gpu_ctx.batch_align(buf, refs, swb200.scoring(*sc), trace_frac=1.0)
        assert (t.score[1], t.end_row[1], t.end_col[1], t.ops[1], t.start_row[1], t.start_col[1]) == want
        assert [tuple(x) for x in t.xpoints[1][1:-1]] == [tuple(x) for x in xps]
        for i in (0, 2, 3):
            one = gpu_ctx.align(*pairs[i], swb200.scoring(*sc))
            assert (t.ops[i], t.start_row[i], t.start_col[i]) == (one.ops, one.start_row, one.start_col)
