"""Kernels that may be set up while their predecessor drains wait for it first.

`launch_after` relaxes the order of consecutive launches; the order is given
back by `after_previous()` as the first statement of the kernel.  A kernel
without it would read buffers that its predecessor still writes.
"""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "aces-ii_b200", "csrc")
FILES = sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def _code(path):
    text = open(path).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return re.sub(r"//[^\n]*", "", text)


def _kernels(code):
    """name -> first statement of every __global__ function"""
    out = {}
    for m in re.finditer(r"__global__", code):
        sig = re.compile(r"\b(k_\w+)\s*\(").search(code, m.end())
        body = code.index("{", sig.end())
        out[sig.group(1)] = code[body + 1:code.index(";", body)].strip()
    return out


@pytest.mark.parametrize("path", FILES, ids=[os.path.basename(f) for f in FILES])
def test_overlapped_kernels_wait_first(path):
    code = _code(path)
    kernels = _kernels(code)
    for name in re.findall(r"launch_after\((k_\w+)", code):
        assert kernels[name] == "after_previous()", name
