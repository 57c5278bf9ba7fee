"""Which strip height the pair path's rule takes, at its edges on this GPU: shown by the
spacing of the special rows, 512 rows for strips of 256 and 512, 448 for strips of 448."""
import random

import pytest

import swb200

pytestmark = pytest.mark.gpu


def test_heights_by_the_fullest_scheduler(gpu_ctx):
    import torch
    sched = 4 * torch.cuda.get_device_properties(0).multi_processor_count
    rng = random.Random(9)
    a = bytes(rng.choices(b"ACGT", k=2048 * sched + 1))
    b = a[100:180]
    for rows, spacing in ((256 * sched, 512),       # a 256-row strip for each scheduler
                          (256 * sched + 1, 448),   # one strip of 448 or of 512 rows at most
                          (448 * sched, 448),
                          (448 * sched + 1, 512),   # two of 448 rows, one of 512
                          (512 * sched, 512),
                          (512 * sched + 1, 448),   # two of either
                          (1344 * sched + 1, 512),  # four of 448 rows, three of 512
                          (1792 * sched + 1, 448),  # five of 448 rows: the next starts as soon as one ends
                          (2048 * sched + 1, 448)):
        r = gpu_ctx.align(a[:rows], b, swb200.scoring(1, -3, -5, -2))
        assert r.score == 80 and r.special_interval == spacing, rows
