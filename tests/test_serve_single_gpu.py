"""One client that sends a request and waits for it: the server starts it at once and
does not hold it for others."""
import random
import statistics

import pytest

import swb200

pytestmark = pytest.mark.gpu


def test_a_request_that_is_waited_for_is_not_held():
    rng = random.Random(31)
    queued = []
    with swb200.Server(swb200.scoring(1, -3, -5, -2)) as srv:
        for _ in range(60):
            a = bytes(rng.choices(b"ACGT", k=400))
            queued.append(srv.wait(srv.submit(a, a[50:350]))[1]["queued_ms"])
    # (a request that was held for others starts 0.1 ms after its submission or later)
    assert statistics.median(queued) < 0.09
