"""What decides that an object is stale covers every header its source names."""

import os
import re

from pymatting_b200 import build


def test_every_included_header_is_a_dependency():
    names = set()
    for f in os.listdir(build.CSRC):
        if f.endswith((".cu", ".cuh")):
            with open(os.path.join(build.CSRC, f)) as src:
                names |= set(re.findall(r'^\s*#\s*include\s+"([^"]+)"', src.read(), re.M))
    assert names
    deps = {os.path.basename(p) for p in build.headers()}
    assert names <= deps, sorted(names - deps)


def test_every_source_is_built():
    assert {f for f in os.listdir(build.CSRC) if f.endswith(".cu")} == set(build.SOURCES)


def test_a_newer_header_makes_an_object_stale(tmp_path):
    obj, dep = tmp_path / "a.o", tmp_path / "a.cuh"
    obj.write_text("")
    dep.write_text("")
    os.utime(obj, (1000, 1000))
    os.utime(dep, (2000, 2000))
    assert build._stale(str(obj), [str(dep)])
    os.utime(dep, (500, 500))
    assert not build._stale(str(obj), [str(dep)])
