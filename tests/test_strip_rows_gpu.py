"""The pair path's rule for strip heights at its edges: 256 rows while every strip
has a scheduler to itself, then 448 or 512 by how many strips the fullest scheduler
gets."""
import random

import pytest

import oracle_ctypes as O
import swb200

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("over", [0, 1])
@pytest.mark.parametrize("rows", [256, 448, 512])
def test_heights_at_the_rules_edges(gpu_ctx, rows, over):
    rng = random.Random(rows + over)
    m, n = rows * 4 * 148 + over, 300
    a = bytes(rng.choices(b"ACGT", k=m))
    at = m - n - 5  # the best cell lies in the last strip
    b = bytes(c if rng.random() > 0.08 else rng.choice(b"ACGT") for c in a[at:at + n])
    sc = (1, -3, -5, -2)
    r = gpu_ctx.align(a, b, swb200.scoring(*sc))
    e = O.stage1_fast(a, b, O.scoring(*sc), O.TIE_REFERENCE)[0]
    assert (r.score, r.end_row, r.end_col) == (e.score, e.row, e.col)
    assert O.score_ops(a, b, O.scoring(*sc), r.start_row, r.start_col, r.ops) == e.score
    s = gpu_ctx.align(a, b, swb200.scoring(*sc), swb200.FLAG_SCORE_ONLY)
    assert (s.score, s.end_row, s.end_col) == (e.score, e.row, e.col)
