"""The build compiles a translation unit again when a header that it includes has changed."""
import os
import re

from yune_gb300 import build


def _includes(path, seen):
    """Adds to `seen` the project headers that path includes, directly or not."""
    for name in re.findall(r'^\s*#\s*include\s+"([^"]+)"', open(path).read(), re.M):
        for base in (os.path.dirname(path), build.CSRC, os.path.join(build.ROOT, "include")):
            hdr = os.path.normpath(os.path.join(base, name))
            if os.path.exists(hdr):
                if hdr not in seen:
                    seen.add(hdr)
                    _includes(hdr, seen)
                break
        else:
            raise AssertionError("%s includes %s, which is nowhere" % (path, name))


def test_every_included_header_is_a_dependency():
    seen = set()
    for src in build.CU_SOURCES + build.CXX_SOURCES:
        _includes(os.path.join(build.CSRC, src), seen)
    assert seen and not seen - {os.path.normpath(p) for p in build._deps()}
