"""The best cell of one block (swb_score_block_device): only cells of the block
count, whatever its borders hold, for blocks with a top border, a left border, both,
any number of rows, and table and compare scores, against the oracle's block."""
import ctypes as C
import random

import numpy as np
import pytest

import oracle_ctypes as O
import swb200

pytestmark = pytest.mark.gpu


def _best(ctx, rows, cols, sc, top, left, corner, r0, c0, full_m, full_n, tie):
    """The block's best cell (score, row, col, key) on the GPU and from the oracle."""
    import torch
    dev = lambda x: None if x is None else torch.from_numpy(np.ascontiguousarray(x)).cuda()
    ptr = lambda t: None if t is None else C.c_void_p(t.data_ptr())
    d_rows, d_cols = dev(np.frombuffer(rows, np.uint8).copy()), dev(np.frombuffer(cols, np.uint8).copy())
    d_top, d_left, out, s = dev(top), dev(left), swb200.BlockBest(), swb200.scoring(*sc)
    rc = swb200.lib().swb_score_block_device(
        ctx._h, ptr(d_rows), len(rows), ptr(d_cols), len(cols), ptr(d_top), ptr(d_left), corner, r0, c0, full_m, full_n,
        C.byref(s), swb200.FLAG_TIE_ROWMAJOR if tie else 0, None, None, C.byref(out))
    assert rc == 0
    _, _, e, key = O.block(rows, cols, O.scoring(*sc), top, left, corner, r0, c0, full_m, full_n, tie)
    want = (e.score, e.row, e.col, key) if e.score > 0 else (0, -1, -1, (1 << 64) - 1)
    return (out.score, out.row, out.col, out.key), want


def _seq(rng, n, alph):
    return bytes(rng.choices(alph, k=n))


@pytest.mark.parametrize("n", [200, 700])
@pytest.mark.parametrize("m", [1, 40, 512, 700])
def test_cells_that_take_h_from_the_top_border_count(gpu_ctx, m, n):
    """A top border with one peak and no match below it, gaps cheaper than mismatches:
    the best cell is the one below the peak, whose H is its F (200 columns are scored in
    32-bit strips, 700 in packed ones)."""
    rng = random.Random(m + n)
    top = np.zeros((n, 2), dtype=np.int32)
    top[:, 0] = 300 - np.abs(np.arange(n) - n // 2)
    top[:, 1] = top[:, 0] - 2
    for alph in (b"CGT", b"CGTRYKM"):
        for tie in (O.TIE_REFERENCE, O.TIE_ROWMAJOR):
            got, want = _best(gpu_ctx, b"A" * m, _seq(rng, n, alph), (1, -3, -2, -2), top, None, 0, 512, 0, 4096, 1024, tie)
            assert want[:3] == (298, 512, n // 2) and got == want


@pytest.mark.parametrize("alph", [b"ACGT", b"ACGTRYKM"])
@pytest.mark.parametrize("last", [1, 24, 257, 512, 700])
def test_columns_right_of_the_block_do_not_count(gpu_ctx, alph, last):
    """The last rows of a matrix whose alignment ends in the row above the block, at
    the last column: the border is higher than every cell of the block, and a column
    past the last one would continue from it."""
    rng = random.Random(last + len(alph))
    n, above = 700, 1536
    cols = _seq(rng, n, alph)
    rows = _seq(rng, above - 500, alph) + cols[-500:] + _seq(rng, last, alph)
    m, sc = len(rows), (1, -3, -5, -2)
    for tie in (O.TIE_REFERENCE, O.TIE_ROWMAJOR):
        top = O.block(rows[:above], cols, O.scoring(*sc), None, None, 0, 0, 0, m, n, tie)[0]
        high = int(top[-1, 0])
        assert high >= 500
        got, want = _best(gpu_ctx, rows[above:], cols, sc, top, None, 0, above, 0, m, n, tie)
        assert want[0] == high - 5 and got == want


@pytest.mark.parametrize("alph", [b"ACGT", b"ACGTRYKM"])
@pytest.mark.parametrize("m", [3, 63, 255, 505, 520, 1000])
def test_rows_below_the_block_do_not_count(gpu_ctx, alph, m):
    """A left border that is highest at the block's last row, with mismatches cheaper
    than gaps: a row past the last one would continue from it along the diagonal."""
    rng = random.Random(m + len(alph))
    n = 600
    left = np.zeros((m, 2), dtype=np.int32)
    left[:, 0] = 40 + np.arange(m)
    left[:, 1] = left[:, 0] - 5
    for sc in ((1, -1, -5, -2), (2, -3, -9, -4)):
        got, want = _best(gpu_ctx, b"A" * m, _seq(rng, n, alph[1:]), sc, None, left, 0, 0, 256, 4096, 1024,
                          O.TIE_REFERENCE)
        assert got == want, sc


@pytest.mark.parametrize("alph", [b"ACGT", b"ACGTRYKM"])
@pytest.mark.parametrize("base", [0, 20_000])
@pytest.mark.parametrize("high", [5_000, 9_000, 20])
def test_a_top_border_that_jumps_up(gpu_ctx, alph, base, high):
    """A top border with one high value, and a slightly higher one far behind it
    followed by a match: no cell before it comes near the block's best."""
    rng = random.Random(high + base)
    m, n = 512, 700
    rows, cols = bytearray(_seq(rng, m, alph)), bytearray(_seq(rng, n, alph))
    cols[51] = ord("A") if rows[0] != ord("A") else ord("C")
    cols[401] = rows[0]
    top = np.zeros((n, 2), dtype=np.int32)
    top[:, 0] = base
    top[50, 0] = base + high
    top[400, 0] = base + high + 200
    top[:, 1] = np.maximum(top[:, 0] - 5, 0)
    got, want = _best(gpu_ctx, bytes(rows), bytes(cols), (1, -3, -5, -2), top, None, 0, 512, 0, 4096, 1024,
                      O.TIE_REFERENCE)
    assert want[:3] == (base + high + 201, 512, 401) and got == want
