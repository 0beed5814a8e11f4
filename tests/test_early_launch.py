"""The kernels of a training step are launched before the kernel ahead of them has ended
(pacuda_b200/csrc/surrogate.cu, launch_early). What an earlier kernel wrote is only promised to be
seen behind griddepcontrol.wait, so no such kernel may touch the network's or the caller's arrays
before it, on any of its branches. (Read from the source: whether a load before the wait sees an old
value is a matter of timing that no run can show to be safe.)"""
import os
import re

import pytest

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pacuda_b200", "csrc", "surrogate.cu")


def code():
    text = open(SOURCE).read()
    return re.sub(r"//[^\n]*", "", text)


def body(text, name):
    at = re.search(r"__global__[^;{]*\b%s\([^;{]*\{" % name, text).end()
    depth, end = 1, at
    while depth:
        depth += {"{": 1, "}": -1}.get(text[end], 0)
        end += 1
    return text[at:end]


def early_kernels():
    text = code()
    return sorted(set(re.findall(r"launch_early\((?!void)(\w+)", text)))


def test_the_step_s_kernels_are_found():
    assert early_kernels() == ["chain_kernel", "dw_kernel", "update_kernel"]


@pytest.mark.parametrize("kernel", early_kernels())
def test_no_array_is_touched_before_the_wait(kernel):
    text = body(code(), kernel)
    arrays = r"\b[gu]\.(params|m1|m2|grad|loss|loss_sum|x|y|wimg|wtimg|x_img|h_img|dz_img|z|db|dw5|scalars|partial|dw)\b"
    waits = [m.start() for m in re.finditer(r"grid_wait\(\);", text)]
    assert waits
    for wait in waits:
        # the branch that this wait is on, from its start: what stands before it in the kernel's body at
        # the same or an outer level (other branches, behind their own waits, are left out)
        before, depth, k = [], 0, wait
        for ch in reversed(text[:wait]):
            k -= 1
            if ch == "}":
                depth += 1
            if depth == 0:
                before.append(ch)
            if ch == "{" and depth:
                depth -= 1
        prefix = "".join(reversed(before))
        # addresses may be formed (a select of pointers, an index added); no value may be loaded or stored
        for statement in prefix.split(";"):
            if not re.search(arrays, statement):
                continue
            assert "*reinterpret_cast" not in statement and not re.search(r"\[[^\]]*\]\s*[-+*/]?=[^=]", statement), statement
            assert not re.search(arrays + r"\s*\[[^\]]*(threadIdx|tile|\bt\b|\bk\b)", statement), statement
    # every load that is spelled as a vector load of the network's arrays comes behind a wait
    first = waits[0]
    assert not re.search(r"reinterpret_cast<const float4 \*>\(u\.(params|m1|m2)", text[:first])
