"""Source check of the device-side waits (no GPU): a bounded wait that gives up must not leave a warp
divided, which no run on a GPU may provoke."""
import os
import re

import pytest

OPS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "multi-device-model-compiler_b200", "csrc", "ops")


def _code(name):
    with open(os.path.join(OPS, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def _enclosing(code, position):
    """What opens each block that holds `position`, outermost first."""
    stack, start = [], 0
    for i, c in enumerate(code[:position]):
        if c == "{":
            stack.append(code[start:i].strip())
        elif c == "}":
            stack.pop()
        if c in "{};":
            start = i + 1
    return stack


@pytest.mark.parametrize("name", sorted(f for f in os.listdir(OPS) if f.endswith(".cu")))
def test_warps_wait_with_one_verdict(name):
    """mbar_wait is one thread's wait: its verdict mixes the barrier, the abort flag and the timer, and
    lanes that each ask for themselves can get different ones.  It may stand only where a single
    lane runs; whole warps use mbar_wait_all or mbar_wait_warp."""
    code = _code(name)
    for call in re.finditer(r"\bmbar_wait\(", code):
        assert any("lane == 0" in opener for opener in _enclosing(code, call.start())), code[call.start() - 80:call.end() + 60]


@pytest.mark.parametrize("name", sorted(f for f in os.listdir(OPS) if f.endswith(".cu")))
def test_elected_waits_stand_under_an_election(name):
    """mbar_wait_elected is mbar_wait where one elected thread runs the whole role.  Nothing warp-wide may stand there
    either: the other lanes never come to a second election, a vote or a shuffle."""
    code = _code(name)
    for call in re.finditer(r"\bmbar_wait_elected\(", code):
        assert "if (elect_one())" in " ".join(_enclosing(code, call.start())), code[call.start() - 80:call.end() + 60]
    for role in re.finditer(r"if \(elect_one\(\)\) \{", code):
        depth, end = 1, role.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(code[end], 0)
            end += 1
        assert not re.search(r"elect_one|_sync\(0x|_warp\(|_all\(|kblocks|umma_planes|mbar_wait_looked", code[role.end():end]), code[role.start():end][:300]


def test_the_warp_waits_are_uniform():
    code = _code("ptx_sm100.cuh")

    def body(function):
        return code[code.index("bool " + function):].split("\n}\n")[0]
    assert "__all_sync(0xffffffffu, mbar_wait(" in body("mbar_wait_all")
    assert "__shfl_sync(0xffffffffu, ok, 0)" in body("mbar_wait_warp")


@pytest.mark.parametrize("name", sorted(f for f in os.listdir(OPS) if f.endswith((".cu", ".h", ".cuh"))))
def test_a_tensor_map_is_judged_by_its_own_call(name):
    """A kernel launched with a map that was never written faults.  The status cannot tell: it may hold an earlier call's
    failure, or another thread's.  So the entry point that only sets the status is not for the operators."""
    code = _code(name)
    assert "mgpuTensorMapEncodeTiled" not in code and not re.search(r"before != 0 \|\| mgpuGetLastError", code)
    for call in re.finditer(r"\bencode_(tmap|tmap_2d|rows|operand)\(", code):
        before = code[max(0, call.start() - 120):call.start()]
        assert re.search(r"(if \([^;{}]*|ok = [^;{}]*|return |\|\|\s*!|inline bool |static bool )$", before), before[-80:]
