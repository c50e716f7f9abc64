"""Rules of the programming model that a GPU run cannot show to be broken, checked in the kernels' sources."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "t2fw_b200", "csrc")
SOURCES = sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))

# a condition on one of these differs between the threads of a block
PER_THREAD = re.compile(r"\b(threadIdx|tid|lane|warp|group|w)\b")


def _text(path):
    with open(path) as f:
        return re.sub(r"//[^\n]*|/\*.*?\*/", "", f.read(), flags=re.S)


def _block(text, start):
    """The text between the brace at `start` and its partner, and where that ends."""
    depth = 0
    for i in range(start, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[start:i + 1], i + 1
    raise AssertionError("unbalanced braces")


def _branches(text):
    """(condition, text of the branch) of every braced if, its else branches under the same condition."""
    for m in re.finditer(r"\bif (?:constexpr )?\(([^{};]*)\) \{", text):
        body, end = _block(text, m.end() - 1)
        yield m.group(1), body
        e = re.match(r"\s*else \{", text[end:])
        if e:
            yield m.group(1), _block(text, end + e.end() - 1)[0]


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_block_barriers_are_reached_by_the_whole_block(path):
    """__syncthreads() under a condition that differs within the block is undefined, also where every thread meets some
    __syncthreads(); groups of warps on different paths meet at named barriers."""
    for cond, body in _branches(_text(path)):
        if PER_THREAD.search(cond):
            assert not re.search(r"__syncthreads\(|\bsync_all\(", body), "if (%s)" % cond


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_dependent_launches_wait_first(path):
    """A kernel that may start before the one ahead of it has ended (launch_dependent) sees that one's writes, and those of
    every kernel before it, after its own griddepcontrol.wait only: it waits once and without a condition, in the outermost
    block."""
    text = _text(path)
    if "griddepcontrol.wait" in text:      # the definition
        return
    for m in re.finditer(r"__global__[^;{]*?\b(\w+_kernel)\([^;{]*\{", text):
        body, _ = _block(text, m.end() - 1)
        launched = re.search(r"launch_dependent\(\s*&?\s*%s\b|\*const \w+ = &%s\b" % (m.group(1), m.group(1)), text)
        if not launched:
            continue
        assert body.count("dependency_wait()") == 1, m.group(1)
        before = body[:body.index("dependency_wait()")]
        assert before.count("{") - before.count("}") == 1, m.group(1) + ": not in the outermost block"
        assert re.search(r"[;{}]\s*$", before), m.group(1) + ": under a condition"


def _kernels(text):
    """(name, body) of every kernel."""
    for m in re.finditer(r"__global__[^;{]*?\b(\w+_kernel)\([^;{]*\{", text):
        yield m.group(1), _block(text, m.end() - 1)[0]


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_copies_in_flight_are_waited_for_on_the_way_out(path):
    """Bulk copies that a kernel asked for may still be on their way when it gives up, into shared memory that the next block
    gets: behind the last place where it asks for more it waits once more for every barrier that they arrive on."""
    for name, body in _kernels(_text(path)):
        for m in re.finditer(r"auto (\w+) = \[&\]\([^)]*\) \{", body):
            fetch, _ = _block(body, m.end() - 1)
            if "mbar_expect_tx(" not in fetch:
                continue
            last = [c.end() for c in re.finditer(r"\b%s\(" % m.group(1), body)][-1]
            for bar in set(re.findall(r"&(bar\w+|full)\b", fetch)):
                assert re.search(r"\bmbar_wait\(&%s\b|\bdrain_ring<[^(]*\(%s\b" % (bar, bar), body[last:]), (name, m.group(1), bar)


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_copies_count_as_landed_only_after_a_wait_that_succeeded(path):
    """A wait that gave up says nothing about the copies it stood for: they are still due on the way out."""
    for m in re.finditer(r"[^;{}]*\b\w+_pending = false;", _text(path)):
        s = m.group(0).strip()
        assert s.startswith("bool ") or re.match(r"if \((acp::)?mbar_wait\(", s), s
