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


def _block(text, at):
    """The text from the bracket at `at` to the one that closes it."""
    pair = {"(": ")", "{": "}"}[text[at]]
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == text[at]) - (text[i] == pair)
        if depth == 0:
            return text[at:i + 1]
    raise AssertionError("unbalanced")


def kernels(text):
    """Every __global__ function of a file: name -> (parameters, body)."""
    out = {}
    for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\s*)?", text):
        at = m.end()
        if text[at] == "(":  # the launch bounds
            at += len(_block(text, at))
        name = re.match(r"\s*(\w+)\s*", text[at:])
        at += name.end()
        params = _block(text, at)
        out[name.group(1)] = (params, _block(text, text.index("{", at + len(params))))
    return out


READ_ONLY = re.compile(r"__ldg\b|ld\.global\.nc|__restrict__")


def test_overlapped_kernels_wait_first_and_read_with_ordinary_loads():
    """A kernel that launch_after starts is resident while the launch before it writes: its first statement is
    the wait, and none of its loads, nor those of the device functions it may call, are read-only ones."""
    found, launched = {}, set()
    for name, text in sources().items():
        rest = text
        for k, (params, body) in kernels(text).items():
            found[k] = (params, body)
            rest = rest.replace(body, "").replace(params, "")
        assert not READ_ONLY.search(rest), name  # device functions
        launched |= set(re.findall(r"\bk_\w+", " ".join(re.findall(r"launch_after\(([^;]*)", text))))
    launched |= {"k_dhop_sweep", "k_dhop_tma", "k_dhop_tmaw"}  # through a variable
    assert len(launched) >= 15 and launched <= set(found), launched - set(found)
    for k in launched:
        params, body = found[k]
        assert re.match(r"\{\s*dep_wait\(\);", body), k
        assert not READ_ONLY.search(params + body), k
