"""Host code that only one kind of CPU or compiler takes stands behind a condition for it."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "evoc-rs_b200", "csrc")


def test_x86_attributes_are_conditional():
    seen = 0
    for path in glob.glob(os.path.join(CSRC, "*.c*")) + glob.glob(os.path.join(CSRC, "*.h")):
        conditions = []
        for line in open(path):
            word = re.match(r"\s*#\s*(ifdef|ifndef|if|elif|else|endif)\b(.*)", line)
            if word:
                if word[1].startswith("if"):
                    conditions.append(word[2])
                elif word[1] == "endif":
                    conditions.pop()
                else:
                    conditions[-1] = word[2]
            elif "target_clones" in line or "immintrin.h" in line:
                seen += 1
                assert any("__x86_64__" in c for c in conditions), (path, line)
    assert seen
