"""Properties of the kernels that a run on the device does not show, checked on
the CPU: the order of reads that could race another grid, and what the compiler
made of the kernels."""
import os
import re

from avbd_b200 import build

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "avbd-metal_b200", "csrc")


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def body_of(text, pattern):
    """The braces that follow the first match of `pattern`."""
    at = text.index("{", re.search(pattern, text).end())
    depth = 0
    for i in range(at, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[at:i + 1]
    raise AssertionError(pattern)


def contact_words_written_by_the_dual():
    """16-byte words of a one-point manifold that dual_manifold stores to."""
    members = [m.strip() for m in re.search(r"struct ContactGPU\s*\{\s*f4([^;]*);", source("avbd_types.h")).group(1).split(",")]
    dual = body_of(source("solver.cu"), r"void dual_manifold\(")
    stored = {m for m in members if re.search(rf"\bc\.{m}(\.\w+)?\s*=[^=]", dual)}
    assert {"lambda", "penalty"} <= stored
    return {4 + members.index(m) for m in stored}          # header, pair, normal, tangent, then the contact


def test_staged_primal_reads_what_the_dual_writes_after_its_wait():
    """With `early` the dual of the iteration before may still be storing while
    the staged primal runs ahead of its wait."""
    kernel = body_of(source("solver.cu"), r"k_primal_staged\(const Params P")
    before, after = kernel.split("if (early) pdl_wait();")
    written = contact_words_written_by_the_dual()
    copied = lambda part: {int(w) for w in re.findall(r"copy16\([^,]*,\s*mw\s*\+\s*(\d+)\)", part)}
    assert written <= copied(after)
    assert not written & copied(before), written & copied(before)


def test_no_kernel_copies_its_arguments_to_local_memory():
    """A device function that is called instead of inlined takes the launch
    arguments by address: every thread of its callers then copies them (1.5 KB)
    to local memory, which cost the residual kernels of the learned warm start
    half their speed."""
    report = build.compile_report("solver.cu")
    functions = re.findall(r"Function properties for (\S+)\s+(\d+) bytes stack frame", report)
    called = [f for f, _ in functions if re.search(r"RKNS_(6Params|7DevPtrs)E", f)]
    assert not called, called
    residual = {f: int(frame) for f, frame in functions if re.search(r"k_primal_groupILi\d+ELb1ELb[01]ELb1E", f)}
    assert residual and not any(residual.values()), residual
