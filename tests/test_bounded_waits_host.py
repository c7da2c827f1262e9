"""CPU tests, by reading the kernel sources, that a bounded wait stays bounded.

A wait on an mbarrier gives up after a limit (test_failure_gpu.py); what its warp
does next must not leave other threads at a barrier that has no limit.  Such a
hang must not be brought about on a GPU, so these tests read the code.
"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sgemm.cu_b200",
                    "csrc")


def _code(name):
    """The file without comments."""
    with open(os.path.join(CSRC, name)) as f:
        text = re.sub(r"/\*.*?\*/", "", f.read(), flags=re.S)
    return re.sub(r"//[^\n]*", "", text)


def _body(code, head):
    """The braces of the first function (or block) whose head matches."""
    at = re.search(head, code)
    assert at, head
    i = code.index("{", at.end())
    depth = 0
    for j in range(i, len(code)):
        depth += {"{": 1, "}": -1}.get(code[j], 0)
        if depth == 0:
            return code[i:j + 1]
    raise AssertionError(head)


def _reaches(code, body, what, seen=()):
    """Whether `what` is in the body or in a function template it calls."""
    if what in body:
        return True
    for name in set(re.findall(r"\b(\w+)<C[^;(]*>\(", body)) - set(seen):
        head = r"void\s+" + name + r"\("
        if re.search(head, code) and _reaches(code, _body(code, head), what, (*seen, name)):
            return True
    return False


def test_plain_tile_warps_that_leave_alone_meet_no_hardware_barrier():
    """A compute warp of a TMA tile returns by itself when its wait expires, so none
    of the code its siblings go on to holds a bar.sync."""
    code = _code("ffma_kernel.cuh")
    kernel = _body(code, r"ffma_gemm_kernel\(")
    tma = _body(kernel, r"if constexpr \(C::TMA\)")
    after_loop = tma[tma.index("return;"):]  # the producer's end: compute warps from here
    assert "mbar_wait" in after_loop and "finish_tile" in after_loop
    assert not re.search(r"__syncthreads\s*\(|bar\.sync", after_loop)
    assert not _reaches(code, after_loop, "bar.sync")


@pytest.mark.parametrize("head", [r"bool multiply\(", r"bool convert\("])
def test_fused_split_roles_leave_as_whole_warps(head):
    """The fused split kernel's whole-warp roles go through collective instructions
    (votes, tensor-memory loads and stores), so no lane leaves on its own wait: a
    role returns false only where the warp has voted."""
    body = _body(_code("split_fused.cuh"), head)
    assert "__all_sync(" in body
    for leave in re.finditer(r"return false|\bbreak\b", body):
        before = body[:leave.start()].rsplit("\n", 1)[-1]
        if before.strip() == "if (u >= nt * 4)":  # the end of a loop without collectives
            continue
        assert re.search(r"if \(!(__all_sync\(0xffffffffu, \S+\)|drain_chunk\(\))\) $", before)


def test_fused_split_producer_arms_no_barrier_twice():
    """A split warp whose wait expired goes on to its chunk's vote and arrives on the
    way; the producer then issues no more copies, since the one that the warp gave up
    on may still be in flight on the same barrier."""
    code = _code("split_fused.cuh")
    produce = _body(code, r"bool produce\(")
    wait = produce.index("raw_empty")
    assert re.match(r"raw_empty[^;]*\|\| b\.gone\) return false;", produce[wait:])
    assert wait < produce.index("mbar_arrive_expect_tx")
    assert "b.gone = 1" in _body(code, r"bool wait_or_gone\(")


@pytest.mark.parametrize("kernel", ["split_gemm_kernel", "split_grouped_kernel"])
def test_planes_drain_warps_leave_as_whole_warps(kernel):
    """The drain warps of the kernels on planes read tensor memory with all their lanes:
    each wait, and the flag another role sets, goes into a vote before they leave."""
    body = _body(_code("split.cu"), kernel + r"\(")
    drain = body[body.index("float acc[128];"):body.index("tmem_dealloc")]
    loads = drain[:drain.rindex("tmem_ld_32x32b_x32")]
    waits = [w.start() for w in re.finditer(r"mbar_wait\(", loads)]
    assert len(waits) == 1
    after = loads[waits[0]:]
    assert re.match(r"mbar_wait\([^;]*\) && !abort_s;\s*ok = __all_sync\(0xffffffffu, ok\);", after)
    assert not re.search(r"if \([^;{]*abort_s", loads)
