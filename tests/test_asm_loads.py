"""Loads from global memory by inline assembly are volatile: to the compiler
they read no memory, so nothing else keeps one behind a wait for the kernel that
wrote what it reads."""
import glob
import os
import re

import helpers


def test_inline_loads_are_volatile():
    found = 0
    for path in glob.glob(os.path.join(helpers.PKG, "csrc", "*")):
        if os.path.isfile(path):
            with open(path) as f:
                for m in re.finditer(r"\basm\b\s*(volatile)?\s*\(\s*\"(?:\{[^\"]*)?ld\.", f.read()):
                    assert m.group(1), (os.path.basename(path), m.group(0))
                    found += 1
    assert found >= 4
