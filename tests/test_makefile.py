"""The Makefile's dependencies: a change to any header under csrc/ or include/
recompiles every object whose source includes it, directly or through another
header (`make -n -W header`, nothing is built)."""
import os
import re
import shutil
import subprocess

import pytest

from conftest import ROOT

PKG = os.path.join(ROOT, "riken-braket_b200")
DIRS = [os.path.join(PKG, "csrc"), os.path.join(ROOT, "include")]


def includes(path, seen=None):
    seen = set() if seen is None else seen
    with open(path) as f:
        for name in re.findall(r'^\s*#include "([^"]+)"', f.read(), re.M):
            for d in DIRS:
                h = os.path.join(d, name)
                if os.path.exists(h) and h not in seen:
                    seen.add(h)
                    includes(h, seen)
    return seen


def test_every_included_header_is_a_dependency():
    if not shutil.which("make"):
        pytest.skip("no make")
    with open(os.path.join(PKG, "Makefile")) as f:
        makefile = f.read()
    objects = re.search(r"^OBJ :=(.*)$", makefile, re.M).group(1).split()
    missing, seen = [], set()
    for obj in objects:
        base = os.path.splitext(os.path.basename(obj))[0]
        source = next(p for e in (".cu", ".cpp") if os.path.exists(p := os.path.join(DIRS[0], base + e)))
        for header in sorted(includes(source)):
            seen.add(header)
            rel = os.path.relpath(header, PKG)
            r = subprocess.run(["make", "-C", PKG, "-n", "-W", rel, obj], capture_output=True, text=True, check=True)
            if f"-o {obj}" not in r.stdout:
                missing.append((obj, rel))
    assert len(seen) > 5
    assert not missing
