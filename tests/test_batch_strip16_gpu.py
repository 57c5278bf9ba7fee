"""Batched passes in packed 16-bit strips (batch.cu over strip16.cuh): pairs at the
edges of strips and runs, both strip heights, all modes, against the oracle."""
import random

import pytest

import oracle_ctypes as O
import swb200

pytestmark = pytest.mark.gpu


def _pairs(rng, count, sizes, alph):
    out = []
    for _ in range(count):
        m = rng.choice(sizes)
        n = rng.choice([x for x in sizes if x <= m])
        a = bytes(rng.choice(alph) for _ in range(m))
        at = rng.randint(0, m - n)
        out.append((a, bytes(c if rng.random() > 0.07 else rng.choice(alph) for c in a[at:at + n])))
    return out


@pytest.mark.parametrize("sc", [(2, -3, -5, -2), (5, -5, -5, -5), (60, -40, -40, -30)])
@pytest.mark.parametrize("count", [3, 400])
def test_pairs_at_the_edges_of_strips_and_runs(gpu_ctx, monkeypatch, sc, count):
    """3 pairs take 256-row strips, 400 pairs 512-row ones; (60, ...) is too wide for
    the 16-bit window and takes 32-bit strips."""
    rng = random.Random(count + sc[0])
    sizes = [1, 31, 32, 33, 64, 95, 96, 97, 255, 256, 257, 288, 319, 321, 511, 512, 513, 767, 769, 1023, 1025]
    pairs = _pairs(rng, count, sizes, rng.choice([b"ACGT", b"ACGTN"]))
    buf, refs, off = b"".join(x + y for x, y in pairs), [], 0
    for x, y in pairs:
        refs.append((off, len(x), off + len(x), len(y)))
        off += len(x) + len(y)
    want = []
    for x, y in pairs:
        rows, cols, _ = O.orient(x, y)
        e = O.stage1(rows, cols, O.scoring(*sc), O.TEXTBOOK, O.TIE_REFERENCE)
        want.append((e, rows, cols))
    for graph, frac in (("1", 1.0), ("0", 1.0), ("1", 0.3), ("0", 0.0)):
        monkeypatch.setenv("SWB_BATCH_GRAPH", graph)
        r = gpu_ctx.batch_align(buf, refs, swb200.scoring(*sc), trace_frac=frac)
        for i, (e, rows, cols) in enumerate(want):
            assert (r.score[i], r.end_row[i], r.end_col[i]) == (e.score, e.row, e.col), (graph, frac, i)
            if r.traced[i] and e.score > 0:
                ops, sr, scol, xps = O.traceback_xp(rows, cols, O.scoring(*sc), e.row, e.col, int(r.xpoint_interval[i]))
                assert (r.ops[i], r.start_row[i], r.start_col[i]) == (ops, sr, scol), (graph, frac, i)
                assert [tuple(x) for x in r.xpoints[i][1:-1]] == [tuple(x) for x in xps]
