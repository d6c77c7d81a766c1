"""A producer that gave up lets its copies land: what no run on a device reaches, checked in the sources."""
import glob
import os
import re

import vllm_b200

SOURCES = {os.path.basename(p): open(p).read() for p in glob.glob(os.path.join(os.path.dirname(vllm_b200.__file__), "csrc", "*.cu*"))}


class Barrier:
    """Phases of an mbarrier as a poll sees them: of the two parities, that of the phase before has always ended."""

    def __init__(self):
        self.phase = 0

    def poll(self, parity):
        return (self.phase & 1) != parity


def test_either_parity_says_nothing():
    b = Barrier()
    for b.phase in range(4):
        assert b.poll(0) or b.poll(1)                # a copy of this phase may still be on its way


def test_no_drain_ends_on_either_parity():
    either = re.compile(r"mbar_try_wait\(([^,]+), 0\)\s*\|\|\s*mbar_try_wait\(\1, 1\)|!mbar_try_wait\(([^,]+), 0\)\s*&&\s*!mbar_try_wait\(\2, 1\)")
    assert [f for f, text in SOURCES.items() if either.search(text)] == []


def test_producers_with_a_limit_drain():
    """A kernel that issues copies and has waits with a limit lets them land."""
    for f, text in SOURCES.items():
        if f.endswith(".cu") and "mbar_wait_lim(" in text and re.search(r"tma2?_load_\dd", text):
            assert "mbar_let_land(" in text or ".drain()" in text, f
