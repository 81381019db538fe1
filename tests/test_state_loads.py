"""What the kernels read through the read-only path.

A read-only load (__ldg, or a const __restrict__ parameter) promises that the
data does not change while the kernel is resident, and a programmatic dependent
is resident before the kernel in front has ended: only tables that set-up
writes may be read so, never the solver's state, its gates or its fields.
"""

import glob
import os
import re

from aspher_b200 import build as B

TABLES = {"tw_2lr", "tw_m", "tb", "twm",          # twiddles
          "kh", "kxy", "own",                      # multiplier spectra
          "ctab"}                                  # the cosine table of a set-up kernel


def _sources():
    files = sorted(glob.glob(os.path.join(B.CSRC, "*.cu*")))
    assert files
    for f in files:
        yield os.path.basename(f), open(f).read()


def test_read_only_loads_read_tables():
    for name, text in _sources():
        for arg in re.findall(r"__ldg\(([^;]*?)\)", text):
            m = re.match(r"&(\w+)\[", arg)
            assert m and m.group(1) in TABLES, (name, arg)


def test_gates_and_state_are_not_restrict():
    for name, text in _sources():
        for arg in re.findall(r"const\s+(?:int|PkState)\s*\*\s*__restrict__\s+\w+", text):
            assert False, (name, arg)
