"""How the libraries are built (pacuda_b200/build.py)."""
import os
import re

import pytest

from pacuda_b200 import build


def test_device_code_is_not_compressed():
    """A process's first call into a library waits for compressed device code to be unpacked, and nvcc
    compresses any file's past some megabytes unless told not to."""
    assert "--no-compress" in build.FLAGS and "--no-compress" in build.SG_FLAGS


def included(name, seen):
    """`name` and the files of csrc that it includes, at any depth."""
    if name in seen:
        return seen
    seen.add(name)
    for line in open(os.path.join(build.CSRC, name)):
        m = re.match(r'\s*#include "([^"/]+)"', line)
        if m and os.path.exists(os.path.join(build.CSRC, m.group(1))):
            included(m.group(1), seen)
    return seen


@pytest.mark.parametrize("sources,deps", [(build.SOURCES + ["tiled_fma.cu"], build.RUNNER_DEPS),
                                          (build.SG_SOURCES, build.SG_DEPS)])
def test_a_change_of_any_included_file_rebuilds(sources, deps):
    needed = set()
    for s in sources:
        included(s, needed)
    assert needed <= set(deps), sorted(needed - set(deps))
