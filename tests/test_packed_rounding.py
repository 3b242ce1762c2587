"""The two forms of the guided taps (kernels_recon.cu, kernels_guided.cu) give
the same bits whatever the assembler makes of packed products: neither leaves a
packed product to a packed sum, which it may fuse or not, without writing the
fma out."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vapoursynth-lgcr_b200", "csrc")


def arguments(text, start):
    depth, at = 1, start
    while depth:
        depth += {"(": 1, ")": -1}.get(text[at], 0)
        at += 1
    return text[start:at - 1]


@pytest.mark.parametrize("name", ["kernels_recon.cu", "kernels_guided.cu", "guided.cuh"])
def test_packed_sums_take_no_packed_product(name):
    with open(os.path.join(CSRC, name)) as f:
        text = f.read()
    products = set(re.findall(r"f32x2 (\w+) = mul2\(", text))
    for m in re.finditer(r"\b(?:add2|sub2)\(", text):
        args = arguments(text, m.end())
        assert "mul2(" not in args, args
        assert not products & set(re.findall(r"\w+", args)), args
