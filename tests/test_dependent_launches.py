"""Kernels launched as programmatic dependents are resident while the kernels before them still write.  What
those may write is read only after the wait, through plain pointers: `const __restrict__` parameters and __ldg
promise data that is read-only for the kernel's whole life and may be loaded before the wait.  Checked on the
sources, since a load moved above the wait is a race that no run shows reliably."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "microsim_b200", "csrc")

# written before the first launch of a chain and not by any kernel of it; flags_in of the FP32 full kernel is
# the previous step's, complete when the tile list (its only in-flight predecessor) starts
STATIC = {"insts", "models", "tile_inst", "tile_desc", "flags_in", "geo"}
WAIT = re.compile(r"gp_wait_for_earlier_kernels\(\)|griddepcontrol\.wait|begin_dependent\(\)")
READ_ONLY_LOADS = re.compile(r"__ldg\(|ld\.global\.nc|\bload_phi<|\bload_block<|\bload_mu<K1>")


def _closing(text, at, pair):
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return i
    raise AssertionError("unbalanced " + pair)


def _kernels():
    """(file, name, parameter list, body) of every kernel that waits for earlier ones."""
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        with open(os.path.join(CSRC, name)) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\()?", text):
            at = m.end()
            if text[at - 1] == "(":
                at = _closing(text, at - 1, "()") + 1
            sig = re.compile(r"\s*(\w+)\s*\(").match(text, at)
            end = _closing(text, sig.end() - 1, "()")
            if not re.compile(r"\s*\{").match(text, end + 1):
                continue
            start = text.index("{", end)
            body = text[start:_closing(text, start, "{}")]
            if WAIT.search(body):
                yield name, sig.group(1), text[sig.end():end], body


KERNELS = list(_kernels())


def test_the_dependent_kernels_are_found():
    assert {k[1] for k in KERNELS} >= {"k_lean64", "k_step64", "k_step32", "k_fwd", "k_rev_cell", "k_rev_jat", "k_rev_dphi"}


@pytest.mark.parametrize("kernel", KERNELS, ids=[k[1] for k in KERNELS])
def test_in_flight_buffers_are_not_declared_read_only(kernel):
    _, name, params, body = kernel
    for p in params.split(","):
        if "*" in p and "__restrict__" in p and "const" in p.split("*")[0]:
            assert p.split()[-1].strip("* ") in STATIC, (name, p.strip())
    assert not READ_ONLY_LOADS.search(body), name
