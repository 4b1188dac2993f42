"""Loads from tensor memory fill their registers later: the instruction that waits for them has to carry these
registers, or the compiler may move what reads them above it."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "scwatter_gb300", "csrc")


def test_waits_carry_the_loaded_registers():
    loads, waits = set(), set()
    for path in glob.glob(os.path.join(CSRC, "*")):
        for asm in re.findall(r"asm\s+volatile\s*\((.*?)\);", open(path).read(), re.S):
            if "tcgen05.ld" in asm:
                loads.add(asm.count('"=r"'))
            if "tcgen05.wait::ld" in asm:
                assert '"memory"' in asm
                waits.add(asm.count('"+r"'))
    assert loads and waits == loads
