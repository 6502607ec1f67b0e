"""Inline PTX that a whole warp or block executes together (the .aligned forms and the block
barriers): volatile, so that the compiler keeps it where every lane reaches it."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "honei_b200", "csrc")


def test_collective_instructions_are_volatile():
    seen = 0
    for name in sorted(os.listdir(CSRC)):
        path = os.path.join(CSRC, name)
        if not os.path.isfile(path):
            continue
        for qualifier, text in re.findall(r'\basm\s*(volatile)?\s*\(\s*"([^"]*)"', open(path).read()):
            if ".aligned" in text or text.startswith(("bar.", "barrier.")):
                seen += 1
                assert qualifier, (name, text)
    assert seen >= 3
