"""Rules for kernels that start before the kernel ahead of them has finished (dependent launches), read off their sources."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sc25-stof-ad_b200", "csrc")


def _braces(text, at):
    """The text from the `{` at or after `at` to its `}`."""
    start = text.index("{", at)
    depth, i = 0, start
    while True:
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        i += 1
        if depth == 0:
            return text[start:i]


def dependent_kernels():
    """(file:name, signature, body) of every kernel that waits for the one ahead of it."""
    found = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__[^;{]*?\b(\w+_kernel)\s*\(", text):
            body = _braces(text, m.end())
            if "grid_dependency_wait" in body:
                found.append(pytest.param(text[m.end():text.index("{", m.end())], body, id=f"{os.path.basename(path)}:{m.group(1)}"))
    return found


def test_every_launch_form_is_found():
    assert len(dependent_kernels()) >= 9


@pytest.mark.parametrize("signature,body", dependent_kernels())
def test_status_word_is_read_behind_the_dependency_wait(signature, body):
    """Ahead of it the kernel that reports a failure may still run, and the blocks of a cluster may see different words."""
    reads = [m.start() for m in re.finditer(r"\*\s*(?:p\.|report\.)?status\b|failure_reported\(", body)]
    assert all(at > body.index("grid_dependency_wait") for at in reads)


@pytest.mark.parametrize("signature,body", dependent_kernels())
def test_nothing_is_read_as_constant_by_kernels_that_start_early(signature, body):
    """__ldg, and plain loads through __restrict__ pointers to const, may be moved ahead of the wait: what the kernel ahead writes is not
    constant for the lifetime of a kernel that starts before it."""
    assert "__restrict__" not in signature and "__ldg" not in body


def test_nothing_is_read_as_constant_by_their_helpers():
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        assert "__ldg(" not in re.sub(r"//[^\n]*", "", open(path).read()), path
