"""The library is rebuilt when any of its sources or of the headers that they
include, directly or through another, is newer (CPU)."""
import os
import re

from feilab_b200 import build


def test_every_included_header_is_a_dependency():
    def includes(name, seen):
        if name not in seen and os.path.exists(os.path.join(build.CSRC, name)):
            seen.add(name)
            with open(os.path.join(build.CSRC, name)) as f:
                for inc in re.findall(r'#include "([^"]+)"', f.read()):
                    includes(inc, seen)
        return seen
    needed = set()
    for src, _, _ in build.LIB_UNITS:
        includes(src, needed)
    assert needed <= set(build.LIB_DEPS), needed - set(build.LIB_DEPS)
