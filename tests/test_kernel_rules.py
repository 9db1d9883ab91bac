"""Rules that the CUDA sources keep and that no run on a GPU can show to be broken: read from the source."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gridbench_gb300", "csrc")


def sources():
    """File name -> its text without comments."""
    out = {}
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh", ".inl")):
            text = open(os.path.join(CSRC, name)).read()
            out[name] = re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)
    return out


def test_exchanges_name_their_lanes():
    """A shuffle's lanes are the ones that must take part, not the ones that happen to stand together."""
    assert [n for n, text in sources().items() if "__activemask" in text] == []
