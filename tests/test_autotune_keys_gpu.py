"""The autotuner's table keeps the choices of packed and 32-bit strips apart, in a
process and in a cache file, and does not take a batch choice of an older kernel."""
import os

import pytest

from test_autotune_gpu import _run, _run_batch

pytestmark = pytest.mark.gpu


def test_packed_and_wide_strips_have_entries_of_their_own(tmp_path):
    cache = str(tmp_path / "autotune.txt")
    env = {k: v for k, v in os.environ.items() if k not in ("SWB_STAGE1_R", "SWB_STAGE1_PACK")}
    env["SWB_AUTOTUNE_CACHE"] = cache
    wide = _run({**env, "SWB_STAGE1_PACK": "0"})
    lines = open(cache).read().splitlines()
    assert len(lines) == 1
    assert _run(env) == wide
    both = open(cache).read().splitlines()
    assert both[:1] == lines and len(both) == 2 and both[1].rsplit(" ", 1)[0] != lines[0].rsplit(" ", 1)[0]


def test_a_batch_entry_of_the_older_kernel_is_not_used(tmp_path):
    cache = str(tmp_path / "autotune.txt")
    env = {k: v for k, v in os.environ.items() if k not in ("SWB_BATCH16_R", "SWB_BATCH_PACK")}
    env["SWB_AUTOTUNE_CACHE"] = cache
    first, _, how = _run_batch(env)
    assert how == "probed"
    key, R = open(cache).read().split("\n")[0].rsplit(" ", 1)
    with open(cache, "w") as f:  # as the older kernel's entry was written
        f.write(f"{key.rstrip('p')} {R}\n")
    again, _, how = _run_batch(env)
    assert how == "probed" and again == first
