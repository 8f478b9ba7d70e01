"""The product's device code does no FP64 arithmetic: doubles are bit patterns
there (softdouble.h), and sums are in integers or pairs of floats."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "simfast21_gb300", "csrc")


def _device_functions(text):
    """(head, body) of each __global__ or __device__ function, comments removed."""
    text = re.sub(r"/\*.*?\*/|//[^\n]*", "", text, flags=re.S)
    for m in re.finditer(r"__global__|__device__", text):
        if re.match(r"__host__\s+", text[m.start():]) or text[m.start() - 9:m.start()] == "__host__ ":
            continue  # host code too (tables, checks)
        brace, semi = text.find("{", m.end()), text.find(";", m.end())
        if brace < 0 or 0 <= semi < brace:
            continue
        depth, i = 1, brace + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        yield text[m.start():brace], text[brace:i]


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu*"))), ids=os.path.basename)
def test_no_double_in_device_code(path):
    with open(path) as f:
        for head, body in _device_functions(f.read()):
            name = re.findall(r"(\w+)\s*\(", head)
            assert not re.search(r"\bdouble[234]?\b|_as_double|\b__d(add|sub|mul|div)_", body), (path, name)
            # a floating literal without the suffix is a double
            assert not re.search(r"(?<![\w.])(\d+\.\d*|\.\d+)([eE][-+]?\d+)?(?![\w.])", body), (path, name)
