"""Device memory of stage 2's segments: it counts against the HBM budget, stays
bounded for tall pairs, and a call that has no room for it walks without."""
import random

import numpy as np
import pytest

import swb200

pytestmark = pytest.mark.gpu


def _pair(rng, n):
    a = bytes(rng.choices(b"ACGT", k=n))
    return a, bytes(c if rng.random() > 0.06 else rng.choice(b"ACGT") for c in a)


def _same(x, y):
    return (x.score, x.end_row, x.end_col, x.start_row, x.start_col, x.ops) == \
           (y.score, y.end_row, y.end_col, y.start_row, y.start_col, y.ops) and \
           [tuple(p) for p in x.xpoints] == [tuple(p) for p in y.xpoints]


def test_a_pair_without_room_for_segments():
    rng = random.Random(1)
    a, b = _pair(rng, 9000)
    sc = swb200.scoring(1, -3, -5, -2)
    with swb200.Context(device=0) as ctx:
        roomy = ctx.align(a, b, sc)
        kept = roomy.special_bytes
    # room for no segment, for a few of the pair's, for all
    for more, less_launches in ((4_000, True), (100_000, False), (400_000, False)):
        with swb200.Context(device=0, hbm_budget_bytes=kept + more) as ctx:
            r = ctx.align(a, b, sc)
        assert _same(r, roomy) and r.special_bytes == kept
        assert (r.kernel_launches < roomy.kernel_launches) == less_launches


@pytest.mark.parametrize("graph", ["0", "1"])
def test_a_batch_without_room_for_segments(monkeypatch, graph):
    monkeypatch.setenv("SWB_BATCH_GRAPH", graph)
    rng = random.Random(2)
    pairs = [_pair(rng, n) for n in (2600, 700, 5000)]
    refs, off = [], 0
    for a, b in pairs:
        refs.append((off, len(a), off + len(a), len(b)))
        off += len(a) + len(b)
    buf, sc = b"".join(a + b for a, b in pairs), swb200.scoring(1, -3, -5, -2)
    # special rows every 512 rows and columns every 256 of (H, F) and (H, E) pairs
    kept = sum(8 * (n // 512 * n + n // 256 * n) for n in (2600, 700, 5000))
    with swb200.Context(device=0) as ctx:
        roomy = ctx.batch_align(buf, refs, sc, trace_frac=1.0)
    with swb200.Context(device=0, hbm_budget_bytes=kept + 4_000) as ctx:
        tight = ctx.batch_align(buf, refs, sc, trace_frac=1.0)
    assert tight.ops == roomy.ops and tight.xpoints == roomy.xpoints
    assert tight.kernel_launches == roomy.kernel_launches - 2  # the two rounds of segments


def test_a_tall_pair_takes_no_scratch_for_rows_its_path_cannot_reach():
    import torch
    rng = np.random.Generator(np.random.PCG64(3))
    m, n = 60_000_000, 120
    rows = torch.from_numpy(rng.choice(np.frombuffer(b"ACGT", np.uint8), m)).cuda()
    cols = rows[m - 1000:m - 1000 + n].clone()
    with swb200.Context(device=0) as ctx:
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        r = ctx.align_device(rows.data_ptr(), m, cols.data_ptr(), n, swb200.scoring(1, -3, -5, -2))
        used = before - torch.cuda.mem_get_info()[0]
    assert (r.score, r.end_row, r.end_col) == (n, m - 1000 + n - 1, n - 1) and r.ops == "M" * n
    # codes (1), operations (1), crosspoints (1.6) and special rows (2.1) are about 6
    # bytes a row, the walker's blocks 97 MB; a segment for every 448 rows is 21 more
    assert used < 16 * m


def test_the_server_admits_requests_with_their_segments():
    """A request's reservation holds its segments, but a budget that only holds the
    request without them takes it all the same."""
    rng = random.Random(4)
    a, b = _pair(rng, 5000)
    m = n = 5000
    plain = 6 * (m + n) + 16 * n + 8 * (m // 512 * n + n // 256 * m) + (m + n + 8) + 32 * (m // 4 + 8) + 4096
    segments = 10 * (2 * 80 + 4096 + 8 * 4 * 160)
    sc = swb200.scoring(1, -3, -5, -2)
    results = []
    for budget, reserved in ((1 << 30, plain + segments), (plain + 1000, plain + 1000)):
        with swb200.Server(sc, hbm_budget_bytes=budget) as srv:
            results.append(srv.wait(srv.submit(a, b))[0])
            assert srv.stats()["peak_reserved_bytes"] == reserved
        with pytest.raises(swb200.SwbError) as ei:
            with swb200.Server(sc, hbm_budget_bytes=plain - 1) as srv:
                srv.submit(a, b)
        assert ei.value.code == swb200.SWB_ENOMEM_BUDGET
    assert _same(*results)
