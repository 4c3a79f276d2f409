"""Rules that count blocks per SM take the SM count from the device: no source
file spells out the 152 of one chip (comments may)."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "turbins_gb300", "csrc")


def test_no_sm_count_in_the_code():
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh")):
            src = open(os.path.join(CSRC, f)).read()
            src = re.sub(r'//[^\n]*|/\*.*?\*/|"[^"\n]*"', "", src, flags=re.S)
            assert not re.search(r"\b152\b", src), f
