"""Rules that the CUDA sources keep, checked on their text."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "sci-algorithms_gb300", "csrc")


def read(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def block(text, start):
    """text[start:] up to the brace that closes its first one."""
    depth = 0
    for i in range(start, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0 and text[i] == "}":
            return text[start:i + 1]
    raise AssertionError("no closing brace")


def waiting_kernels():
    """(file, definition) of the kernels that wait for their predecessor."""
    out = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = read(path)
        for m in re.finditer(r"__global__", text):
            k = block(text, m.start())
            if "grid_dep_wait()" in k:
                out.append((os.path.basename(path), k))
    return out


NC = re.compile(r"__ldg\s*\(|ldg4\s*\(|ld\.global\.nc")


def test_waiting_kernels_do_not_load_as_read_only():
    """A kernel launched programmatically may begin while its predecessor
    still writes: nothing it reads is read-only for its lifetime.  (T is the
    batch's table, uploaded before the first kernel.)"""
    kernels = waiting_kernels()
    assert len(kernels) >= 14
    for name, k in kernels:
        sig = k[:k.index("{")]
        assert not NC.search(k), (name, sig)
        for p in re.findall(r"const \w+ ?\*__restrict__ \w+", sig):
            assert p == "const Table *__restrict__ T", (name, p)


@pytest.mark.parametrize("name", ["sci_tv_tile.cuh", "sci_tv_adjoint.cuh", "sci_tv_slim.cuh",
                                  "sci_batch_lean.cu", "sci_sqerr.cuh"])
def test_what_waiting_kernels_call_does_not_load_as_read_only(name):
    assert not NC.search(read(name))


def test_masks_of_waiting_kernels_are_not_loaded_as_read_only():
    text = read("sci_ops.cu")
    for m in re.finditer(r"struct Mask<\d>\s*{", text):
        assert not NC.search(block(text, m.start()))


def test_memory_that_a_kernel_writes_is_not_loaded_as_read_only():
    """y1, which the accelerated projections update in place."""
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        assert not re.search(r"(__ldg|ldg4)\s*\(\s*(I\.)?y1\b", read(path)), path
