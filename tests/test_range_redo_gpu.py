"""A pass in packed 16-bit strips that reports that its offsets did not fit is done
again in 32-bit strips: every form of a batch, with results that do not change and a
context that stays usable.  After such a report nothing walks on the stores that the
aborted scoring kernel left unwritten."""
import random

import pytest

import swb200

pytestmark = pytest.mark.gpu


def _batch(rng, count):
    pairs = []
    for _ in range(count):
        a = bytes(rng.choices(b"ACGT", k=rng.randint(1, 2600)))
        b = bytes(c if rng.random() > 0.08 else rng.choice(b"ACGT") for c in a[:rng.randint(1, len(a))])
        pairs.append((a, b))
    refs, off = [], 0
    for a, b in pairs:
        refs.append((off, len(a), off + len(a), len(b)))
        off += len(a) + len(b)
    return b"".join(a + b for a, b in pairs), refs


@pytest.mark.parametrize("count,graph,frac", [(1, "1", 1.0), (40, "1", 1.0), (40, "1", 0.3), (40, "1", 0.0), (40, "0", 1.0),
                                              (40, "0", 0.3), (2100, "1", 0.01)])
def test_batch_redone_in_32_bits(gpu_ctx, monkeypatch, count, graph, frac):
    rng = random.Random(count)
    monkeypatch.setenv("SWB_BATCH_GRAPH", graph)
    buf, refs = _batch(rng, count)
    sc = swb200.scoring(2, -3, -5, -2)
    for _ in range(3):
        plain = gpu_ctx.batch_align(buf, refs, sc, trace_frac=frac)
        redone = gpu_ctx.batch_align(buf, refs, sc, swb200.FLAG_TEST_PACK_ANY, trace_frac=frac)
        for f in ("score", "end_row", "end_col", "start_row", "start_col", "swapped", "traced"):
            assert (getattr(plain, f) == getattr(redone, f)).all(), f
        assert plain.ops == redone.ops and plain.xpoints == redone.xpoints
        monkeypatch.setenv("SWB_BATCH_PACK", "0")
        wide = gpu_ctx.batch_align(buf, refs, sc, trace_frac=frac)
        monkeypatch.delenv("SWB_BATCH_PACK")
        assert redone.kernel_launches == wide.kernel_launches  # what ran last were 32-bit strips


def test_level1_recompute_redone_in_32_bits():
    """A small HBM budget keeps the coarse grid; the first round of recomputed cells is
    done again, which shows in the launches."""
    rng = random.Random(5)
    a = bytes(rng.choices(b"ACGT", k=6000))
    b = bytes(c if rng.random() > 0.08 else rng.choice(b"ACGT") for c in a[300:5600])
    sc = swb200.scoring(1, -3, -5, -2)
    with swb200.Context(device=0, hbm_budget_bytes=1 << 20) as ctx:
        plain = ctx.align(a, b, sc)
        redone = ctx.align(a, b, sc, swb200.FLAG_TEST_PACK_ANY)
    assert plain.score > 3000 and redone.kernel_launches == plain.kernel_launches + 2
    for f in ("score", "end_row", "end_col", "start_row", "start_col", "ops"):
        assert getattr(plain, f) == getattr(redone, f), f
    assert [tuple(x) for x in plain.xpoints] == [tuple(x) for x in redone.xpoints]
