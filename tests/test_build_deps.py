"""The library's build knows every file that a translation unit includes (an
object that is not rebuilt after its table layout changed reads the new tables
by the old offsets)."""
import functools
import os
import re

import pytest

from vlxb import build


@functools.lru_cache(maxsize=None)
def quoted(path):
    with open(path) as fh:
        return re.findall(r'^[ \t]*#[ \t]*include[ \t]+"([^"]+)"', fh.read(), flags=re.M)


def includes(path, seen):
    """Quoted includes of a source file, followed through the files they name."""
    for name in quoted(path):
        for base in (os.path.dirname(path), build.CSRC):
            p = os.path.normpath(os.path.join(base, name))
            if os.path.exists(p):
                if p not in seen:
                    seen.add(p)
                    includes(p, seen)
                break
        else:
            pytest.fail(f"{path}: {name} is in neither place that the compiler looks")
    return seen


def test_every_include_is_a_dependency():
    srcs = build._sources()
    assert len(srcs) > 100
    for src in srcs:
        deps = {os.path.normpath(d) for d in build._deps(src)}
        missing = sorted(os.path.basename(p) for p in includes(src, set()) - deps)
        assert not missing, (os.path.basename(src), missing)
