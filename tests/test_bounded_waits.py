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


def _kernels(name):
    """(kernel, body) of a source file."""
    code = _code(name)
    for m in re.finditer(r"__global__ void[^{;]*?(\w+_kernel)\(", code):
        at = code.index("{", code.index(")", m.end()))
        depth, end = 1, at + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(code[end], 0)
            end += 1
        yield m.group(1), code[at:end]


@pytest.mark.parametrize("name", ["gemm_f32x3.cu"])
def test_copies_have_landed_before_a_kernel_ends(name):
    """Where readers give up, copies may still be on their way: each ring's producer waits for its own last ones, and the thread that
    issues products for its own last commit, before shared and tensor memory go to another CTA."""
    rings = {"f3_rows_kernel": ["full"], "f3_tile_kernel": ["w_full", "x_full"]}
    found = dict(_kernels(name))
    assert set(rings) <= set(found)
    for kernel, body in found.items():
        assert re.findall(r"mbar_landed\((\w+),", body) == rings.get(kernel, [])
        if "tc5_mma" in body:
            last = body.index("mbar_wait(done + ((it - 1) & 1)")
            assert body.rindex("tc5_commit(") < last < body.index("tcgen05.dealloc")
