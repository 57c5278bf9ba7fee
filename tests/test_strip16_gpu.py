"""Packed 16-bit strips of the pair path (csrc/strip16.cuh) where they can go
wrong: edges of strips, halves and 32-step runs, the moving base of the 16-bit
window, and boundaries that do not fit it (scored again in 32 bits)."""
import random

import numpy as np
import pytest

import oracle_ctypes as O
import swb200
from swb200 import chain

pytestmark = pytest.mark.gpu


def _related(rng, m, n, alph=b"ACGT", sub=0.08):
    a = bytes(rng.choice(alph) for _ in range(m))
    at = rng.randint(0, m - n)
    b = bytes(c if rng.random() > sub else rng.choice(alph) for c in a[at:at + n])
    return a, b


def _check(ctx, a, b, sc, flags):
    r = ctx.align(a, b, swb200.scoring(*sc), flags)
    rows, cols, _ = O.orient(a, b)
    e = O.stage1(rows, cols, O.scoring(*sc), O.TEXTBOOK,
                 O.TIE_ROWMAJOR if flags & swb200.FLAG_TIE_ROWMAJOR else O.TIE_REFERENCE)
    assert (r.score, r.end_row, r.end_col) == (e.score, e.row, e.col), (len(rows), len(cols), sc, flags)
    if not flags & swb200.FLAG_SCORE_ONLY and e.score > 0:
        ops, sr, scol, xps = O.traceback_xp(rows, cols, O.scoring(*sc), e.row, e.col, r.xpoint_interval)
        assert (r.ops, r.start_row, r.start_col) == (ops, sr, scol)
        assert [tuple(x) for x in r.xpoints[1:-1]] == [tuple(x) for x in xps]


@pytest.mark.parametrize("R", ["8", "14", "16", "32"])
def test_edges_of_strips_halves_and_runs(gpu_ctx, monkeypatch, R):
    monkeypatch.setenv("SWB_STAGE1_R", R)
    rng = random.Random(int(R))
    half = 16 * int(R)
    rows = [1, half - 1, half, half + 1, 2 * half - 1, 2 * half, 2 * half + 1, 3 * half + 5, 4 * half + 1]
    cols = [1, 2, 31, 32, 33, 63, 64, 65, 96, 97, 127, 128, 129, 255, 256, 257, 287, 288, 319, 320, 321, 511, 513]
    for m in rows:
        for n in rng.sample([c for c in cols if c <= m], min(6, sum(c <= m for c in cols))):
            a, b = _related(rng, m, n, rng.choice([b"ACGT", b"ACGTN", b"AC"]))
            sc = rng.choice([(1, -3, -5, -2), (5, -5, -5, -5), (3, -1, -1, -2)])
            _check(gpu_ctx, a, b, sc, rng.choice([0, swb200.FLAG_TIE_ROWMAJOR]))
            _check(gpu_ctx, a, b, sc, swb200.FLAG_SCORE_ONLY)


@pytest.mark.parametrize("alph", [b"ACGT", b"ACGTRN"])
def test_scores_beyond_sixteen_bits_move_the_base(gpu_ctx, monkeypatch, alph):
    """Scores up to 84,000 with the path leaving and entering strips: the base moves
    up along the path and down beside it; every strip height agrees with the oracle."""
    rng = random.Random(len(alph))
    a, b = _related(rng, 14_000, 12_000, alph, sub=0.02)
    b = b[:6000] + bytes(rng.choice(alph) for _ in range(700)) + b[6000:]
    sc = (7, -4, -9, -1)
    rows, cols, _ = O.orient(a, b)
    e = O.stage1_fast(rows, cols, O.scoring(*sc), O.TIE_REFERENCE)[0]
    assert e.score > 65_536
    for R in ("8", "14", "16", "32"):
        monkeypatch.setenv("SWB_STAGE1_R", R)
        r = gpu_ctx.align(a, b, swb200.scoring(*sc))
        assert (r.score, r.end_row, r.end_col) == (e.score, e.row, e.col), R
        assert O.score_ops(rows, cols, O.scoring(*sc), r.start_row, r.start_col, r.ops) == e.score


def test_scoring_too_wide_for_the_window(gpu_ctx):
    """Scores whose spread over a strip exceeds the window take 32-bit strips."""
    rng = random.Random(3)
    a, b = _related(rng, 3000, 2500)
    _check(gpu_ctx, a, b, (60, -40, -40, -30), 0)
    _check(gpu_ctx, a, b, (900, -700, -2000, -300), swb200.FLAG_SCORE_ONLY)


@pytest.mark.parametrize("jump", [0, 300, 40_000])
def test_block_with_borders_that_fit_no_matrix(gpu_ctx, jump):
    """A block's left and top borders may hold anything; where neighbouring values
    lie too far apart for the 16-bit window the block is scored in 32 bits."""
    import torch
    rng = random.Random(jump)
    rows, cols = _related(rng, 1024, 700)
    sc = (1, -3, -5, -2)
    left = np.zeros((1024, 2), dtype=np.int32)
    left[:, 0] = 20_000 + np.arange(1024) % 7
    left[500:, 0] += jump
    left[:, 1] = left[:, 0] - 3
    top = np.zeros((700, 2), dtype=np.int32)
    top[:, 0] = np.maximum(0, 20_000 - 2 * np.arange(700))
    top[:, 1] = top[:, 0] - 4
    s = O.scoring(*sc)
    exp_bottom, exp_right, e, _ = O.block(rows, cols, s, top, left, 20_001, 512, 256, 4096, 2048, O.TIE_REFERENCE)
    d_rows = torch.frombuffer(bytearray(512) + bytearray(rows) + bytearray(2560), dtype=torch.uint8).cuda()
    d_cols = torch.frombuffer(bytearray(256) + bytearray(cols) + bytearray(1092), dtype=torch.uint8).cuda()
    blk = chain.GpuBlocks(gpu_ctx, d_rows, d_cols, swb200.scoring(*sc))
    bottom, right, best = blk(512, 1536, 256, 956, torch.from_numpy(top).cuda(), torch.from_numpy(left).cuda(), 20_001,
                              True, True)
    assert np.array_equal(bottom.cpu().numpy(), exp_bottom)
    assert np.array_equal(right.cpu().numpy(), exp_right)
    assert best[:3] == (e.score, e.row, e.col)
