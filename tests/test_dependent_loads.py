"""Loads in the kernels' source that a dependent launch makes unsafe.

A kernel launched with programmatic stream serialization is resident before
the writes of the kernel ahead of it are visible.  The read-only data path
(__ldg, ld.global.nc) is defined only for memory that nothing writes while the
kernel is resident, so it may read the twiddle tables and nothing else:
residues, spectra and operands come from the launch before.  And a load in an
asm statement that is not volatile does not depend on memory for the compiler,
which may then move it above the wait.
"""

import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hypergeometrica_gb300", "csrc")
# (file, argument's pointer): the sub-transform, two-level and inter-pass twiddle tables
TABLES = {("hg_ntt_rounds.cuh", "src"), ("hg_ntt_rounds.cuh", "hi"), ("hg_ntt_rounds.cuh", "lo"),
          ("hg_ntt_rounds.cuh", "tws"), ("hg_ntt_bodies.cuh", "t")}


def _sources():
    for path in sorted(glob.glob(os.path.join(CSRC, "*"))):
        if path.endswith((".cu", ".cuh", ".h", ".inc")):
            text = "\n".join(line.split("//")[0] for line in open(path).read().splitlines())
            yield os.path.basename(path), text


def test_read_only_loads_are_of_tables():
    found = {(name, ptr) for name, text in _sources()
             for ptr in re.findall(r"__ldg\((?:reinterpret_cast<[^>]*>\()?\s*(\w+)", text)}
    assert found == TABLES


def test_loads_in_asm_stay_behind_the_wait():
    for name, text in _sources():
        assert "ld.global.nc" not in text, name
        for stmt in re.findall(r"\basm\b(?! volatile)[^;]*", text):
            assert not re.search(r"\bld\.", stmt), (name, stmt)
