"""Exchange words of the on-chip marches: value and step number must arrive
together, which the PTX memory model promises for one 64-bit scalar and not
for the elements of a vector of 32-bit ones. No run can show a torn word, so
the sources are checked: every global access written as PTX is of 64-bit
scalars, with a scope."""
import os
import re

import conftest

CSRC = os.path.join(conftest.ROOT, "bristolfe-v2_gb300", "csrc")


def test_words_are_64_bit_scalars():
    found = []
    for name in ("bfe_onchip.cuh", "bfe_onchip.cu", "bfe_onchip_multi.cu"):
        with open(os.path.join(CSRC, name)) as f:
            found += re.findall(r'"((?:ld|st)\.[\w.:]*global[\w.:]*)', f.read())
    assert len(found) >= 4
    for op in found:
        assert re.fullmatch(r"(ld|st)\.relaxed\.gpu\.global(\.v2)?\.b64", op), op
