"""The lengths with mixed-radix kernels, as the translation units list them: a
length missing there would run the runtime-planned kernels without a word."""
from __future__ import annotations

import glob
import os
import re

from conftest import PKG_DIR

CSRC = os.path.join(PKG_DIR, "csrc")
TUNED = {128, 256, 512}  # every pass tuned; 64, 96, 192 and 384 have some mixed-radix passes


def _smooth(n):
    for q in (2, 3, 5, 7):
        while n % q == 0:
            n //= q
    return n == 1


def test_every_length_is_listed_once():
    lengths, parts = [], []
    for path in sorted(glob.glob(os.path.join(CSRC, "matvec_mx_*.cu"))):
        with open(path) as f:
            for m in re.finditer(r"GILA_MX_PART\(([^)]*)\)", f.read()):
                part, *ls = (int(v) for v in m.group(1).split(","))
                parts.append(part)
                lengths += ls
    assert sorted(lengths) == [n for n in range(4, 513, 2) if _smooth(n) and n not in TUNED]
    with open(os.path.join(CSRC, "matvec_mx.cuh")) as f:
        n = int(re.search(r"kMxParts = (\d+);", f.read()).group(1))
    assert sorted(parts) == list(range(n))
