"""What makes the library out of date: an edit of any source or of anything the sources include."""
import os
import re

from frovedis_gb300 import build


def test_every_included_file_triggers_a_rebuild():
    deps = {os.path.realpath(f) for f in build._deps()}
    seen, todo = set(), [os.path.join(build.CSRC, s) for s in build.SOURCES]
    while todo:
        path = os.path.realpath(todo.pop())
        if path in seen:
            continue
        seen.add(path)
        with open(path) as f:
            for name in re.findall(r'^\s*#include\s+"([^"]+)"', f.read(), re.M):
                found = [p for p in (os.path.join(d, name) for d in (os.path.dirname(path), build.INCLUDE))
                         if os.path.exists(p)]
                assert found, (path, name)
                todo.append(found[0])
    assert seen <= deps, sorted(seen - deps)
