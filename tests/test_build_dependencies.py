"""An edit of any header makes the objects that include it out of date."""
import os
import re

from exfemus_b200 import build


def test_every_included_header_is_a_dependency():
    seen = set()
    for src in build.sources():
        deps = {os.path.realpath(d) for d in build.dependencies(src)}
        todo = [src]
        while todo:
            f = todo.pop()
            for inc in re.findall(r'^\s*#include "([^"]+)"', open(f).read(), re.M):
                h = os.path.realpath(os.path.join(os.path.dirname(f), inc))
                assert h in deps, (src, inc)
                if h not in seen:
                    seen.add(h)
                    todo.append(h)
    assert any(h.endswith(".cuh") for h in seen)
