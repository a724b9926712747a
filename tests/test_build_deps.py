"""A change to any of a library's sources makes it out of date: every file that
its translation units include is among the build's dependencies."""
import os
import re

import pytest

from nextgen_b200 import build


def includes(path, seen):
    if path in seen:
        return seen
    seen.add(path)
    for inc in re.findall(r'^\s*#include "([^"]+)"', open(path).read(), re.M):
        for d in (os.path.dirname(path), build.INC):
            p = os.path.normpath(os.path.join(d, inc))
            if os.path.exists(p):
                includes(p, seen)
                break
    return seen


@pytest.mark.parametrize("which", ["build_cgx", "build_meshgen"])
def test_every_included_file_is_a_dependency(which, monkeypatch):
    seen = []
    monkeypatch.setattr(build, "_stale", lambda out, deps: seen.append([os.path.normpath(d) for d in deps]))
    getattr(build, which)()
    units = [d for d in seen[0] if d.endswith((".cu", ".cpp"))]
    assert units
    need = set()
    for u in units:
        includes(u, need)
    assert need <= set(seen[0])
