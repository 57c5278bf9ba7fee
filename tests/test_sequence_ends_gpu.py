"""Sequences in device memory at any address and of any length: the pair walker reads
their bytes as aligned words, the first and the last of which may be partly outside."""
import random

import numpy as np
import pytest

import oracle_ctypes as O
import swb200

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("at", [0, 1, 2, 3])
@pytest.mark.parametrize("m,n", [(1, 1), (5, 3), (67, 66), (515, 511), (1030, 1027), (1302, 769)])
def test_any_alignment_and_length(gpu_ctx, at, m, n):
    import torch
    rng = random.Random(m * 4 + at)
    rows = bytes(rng.choices(b"ACGT", k=m))
    cols = bytes(c if rng.random() > 0.05 else rng.choice(b"ACGT") for c in rows[m - n:])
    if n > 2:
        cols = cols[:-1] + rows[-1:]  # the alignment reaches the last bytes
    buf = np.full(m + n + 64, ord("A"), dtype=np.uint8)
    c_at = (at + m + 8) // 4 * 4 + 4 + (3 - at)
    buf[at:at + m] = np.frombuffer(rows, np.uint8)
    buf[c_at:c_at + n] = np.frombuffer(cols, np.uint8)
    d = torch.from_numpy(buf).cuda()
    sc = (1, -3, -5, -2)
    r = gpu_ctx.align_device(d.data_ptr() + at, m, d.data_ptr() + c_at, n, swb200.scoring(*sc))
    e = O.stage1(rows, cols, O.scoring(*sc), O.TEXTBOOK, O.TIE_REFERENCE)
    assert (r.score, r.end_row, r.end_col) == (e.score, e.row, e.col)
    if e.score > 0:
        ops, sr, scol, _ = O.traceback_xp(rows, cols, O.scoring(*sc), e.row, e.col, r.xpoint_interval)
        assert (r.ops, r.start_row, r.start_col) == (ops, sr, scol)
