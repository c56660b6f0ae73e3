"""Kernels whose copies a lane issues (TMA): before a block ends it waits for those still under way, also where another warp's bounded wait runs out
after the issuing lane has looked at the abort flag.  So that wait depends on no flag, or stands behind a barrier of the whole block."""
import os
import re

import pytest

from arle_b200.ops import build

FILES = [f for f in build.sources() if "tma_load" in open(os.path.join(build.CSRC, f)).read()]


def _last_waits(text):
    """The text ahead of every last wait for copies, some lines of it."""
    for m in re.finditer(r"for \([^\n]*\)\s*(?:\{[^{}]*?)?mbar_wait_plain\(smem_addr\((?:&full|keys \? &k_full)", text):
        yield "\n".join(text[: m.start()].rstrip().splitlines()[-7:])


@pytest.mark.parametrize("name", FILES)
def test_copies_are_waited_for_whatever_the_flag_says(name):
    with open(os.path.join(build.CSRC, name)) as f:
        text = f.read()
    waits = list(_last_waits(text))
    assert waits, f"{name}: no last wait for copies found"
    for ahead in waits:
        look = re.search(r"if \([^;{}]*\*aborted", ahead)
        assert look is None or "__syncthreads();" in ahead[: look.start()], f"{name}: the last wait for copies goes by one look at the abort flag"
