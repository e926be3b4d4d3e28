"""Counters that blocks hand work over with are read with the width they are written with.

The PTX memory model orders nothing between a 64-bit load and 32-bit atomics
on its halves: an acquire of that kind may see a count without the exponent
(or the data) released before it.  Such a race does not show in a result on
demand, so the source is looked at: a hand-over word is written by 32-bit
atomics in every kernel of the library, and no acquire load is wider.
"""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pisces-1_gb300", "csrc")


def test_acquire_loads_are_as_wide_as_the_atomics():
    loads = 0
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, name)) as f:
                text = re.sub(r"//[^\n]*", "", f.read())
            found = re.findall(r"\bld\.acquire\.[\w.]*", text)
            loads += len(found)
            assert all(re.search(r"\.[ub]32$", f) for f in found), (name, found)
    assert loads > 0
