"""What an incremental build looks at: every file that a source includes is one whose change compiles it again (no GPU, no compiler)."""
import importlib
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "llm.metal_b200", "csrc")
SOURCES = sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))


def test_every_unit_is_built(pkg):
    build = importlib.import_module(pkg.__name__ + ".build")
    assert SOURCES == sorted(build.CU_SOURCES)


@pytest.mark.parametrize("source", SOURCES)
def test_includes_are_watched(pkg, source):
    build = importlib.import_module(pkg.__name__ + ".build")
    watched, todo, seen = {os.path.realpath(h) for h in build._headers()}, [os.path.join(CSRC, source)], set()
    while todo:
        path = todo.pop()
        with open(path) as f:
            for name in re.findall(r'^\s*#\s*include\s+"([^"]+)"', f.read(), re.M):
                at = os.path.realpath(os.path.join(os.path.dirname(path), name))
                assert at in watched, f"{os.path.basename(path)} includes {name}: a change there leaves {source}'s object as it is"
                if at not in seen:
                    seen.add(at)
                    todo.append(at)
