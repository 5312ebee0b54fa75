"""Chained kernels read with ordinary loads (CPU: the sources are read).

A kernel that starts with chain_begin() is launched while its predecessor
still runs, and may read what that wrote only after the wait, through coherent
loads.  The read-only path (__ldg, ld.global.nc, and what the compiler makes of
pointers marked __restrict__ that the kernel only reads) needs data that stays
constant while the kernel runs, and such loads may be moved above the wait.
"""
from __future__ import annotations

import glob
import os
import re

from conftest import PKG_DIR

CSRC = os.path.join(PKG_DIR, "csrc")


def _strip(text):
    text = re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)
    return re.sub(r"__launch_bounds__\s*\([^()]*\)", "", text)


def _closing(text, at):
    """Index of the brace that closes the one at `at`."""
    depth = 0
    for i in range(at, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return i
    raise AssertionError("unbalanced braces")


def _functions(text):
    """(qualifier, name, parameters and body) of the kernels and device functions."""
    for m in re.finditer(r"__(global|device)__\s[^;{}=]*?(\w+)\s*\(([^;{}]*)\)\s*\{", text):
        yield m.group(1), m.group(2), text[m.start():_closing(text, m.end() - 1) + 1]


def test_chained_kernels_use_coherent_loads():
    functions = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        functions += list(_functions(_strip(open(path).read())))
    direct = re.compile(r"__ldg\s*\(|\.nc\b|__restrict__")
    readonly = {name for q, name, text in functions if q == "device" and direct.search(text)}
    chained = {name: text for q, name, text in functions if q == "global" and "chain_begin();" in text}
    assert len(chained) >= 20
    bad = {}
    for name, text in chained.items():
        hits = set(direct.findall(text)) | {f for f in readonly if re.search(rf"\b{f}\s*[<(]", text)}
        if hits:
            bad[name] = sorted(hits)
    assert not bad, bad
