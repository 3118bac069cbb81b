"""A kernel that may start before its predecessor has ended must not tell the compiler that what the
predecessor writes is read-only: no const __restrict__ argument and no __ldg in such a kernel or in the
device functions of its file. (The correlation kernels read the frames through __ldg; a placement or a
copy always lies between them and the preparation, so their frames are complete before they start.)"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "piv_b200", "csrc")


def _functions(text):
    """(head, body) of every __global__ and __device__ function definition."""
    for m in re.finditer(r"^(?:template[^\n]*\n)?[^\n;]*\b__(?:global|device)__\b", text, re.M):
        brace, semi = text.find("{", m.end()), text.find(";", m.end())
        if brace < 0 or 0 <= semi < brace:
            continue
        depth, i = 1, brace + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        yield text[m.start():brace], text[brace:i]


def _read_only(head, body):
    return "__ldg" in body or re.search(r"const\s+[\w:]+\s*\*\s*(const\s+)?__restrict__", head)


@pytest.mark.parametrize("unit", ["prep.cu", "field.cu"])
def test_no_read_only_loads_of_fresh_data(unit):
    with open(os.path.join(CSRC, unit)) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    found = list(_functions(text))
    assert any("dependent_wait()" in b for _, b in found)
    bad = [h.split("(")[0].split()[-1] for h, b in found
           if _read_only(h, b) and ("dependent_wait()" in b or "__global__" not in h)]
    assert not bad
