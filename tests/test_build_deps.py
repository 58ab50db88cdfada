"""Every file that a source includes is among the build's dependencies, so that
a change of it alone rebuilds the objects."""
import os
import re

import build as build_mod


def test_included_files_are_dependencies():
    cu, cpp, hdr = build_mod._sources()
    deps = {os.path.realpath(h) for h in hdr}
    seen = set()
    todo = list(cu + cpp)
    while todo:
        f = os.path.realpath(todo.pop())
        if f in seen:
            continue
        seen.add(f)
        with open(f) as s:
            for name in re.findall(r'^\s*#\s*include\s*"([^"]+)"', s.read(), re.M):
                p = os.path.realpath(os.path.join(os.path.dirname(f), name))
                assert p in deps, (f, name)
                todo.append(p)
    assert any(f.endswith(".inc") for f in seen)
