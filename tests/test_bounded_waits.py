"""What the kernels' sources promise about waits, checked in the sources: a wait that can run out never runs on a GPU here."""

import os
import re

import pytest

import qwen25vl_lite

CSRC = os.path.join(os.path.dirname(qwen25vl_lite.__file__), "csrc")
SOURCES = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")))


def _code(name):
    with open(os.path.join(CSRC, name)) as fh:
        return re.sub(r"//[^\n]*", "", fh.read())


@pytest.mark.parametrize("name", SOURCES)
def test_no_barrier_that_one_side_passes_without_waiting(name):
    """``bar.arrive`` lets its warp run ahead of the warp that waits at ``bar.sync``, which has no limit.  If the wait that keeps the
    two together runs out, two arrivals of the first warp complete a phase by themselves and the second waits for good.  Such a pair
    meets at an mbarrier, whose wait is bounded."""
    assert not re.search(r"\b(bar|barrier(\.cta)?)\.arrive\b", _code(name))


def test_every_wait_on_an_mbarrier_goes_through_the_bounded_one():
    for name in SOURCES:
        found = re.findall(r"mbarrier\.(?:try_wait|test_wait)", _code(name))
        assert len(found) == (1 if name == "common.cuh" else 0), name
