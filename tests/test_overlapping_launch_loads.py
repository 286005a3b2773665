"""Kernels that may be alive while the kernel before them still writes (those that call
stream_wait) must not read what it could write through the read-only path."""
import os
import re

import pytest

from conftest import PKG, ROOT

FILES = [os.path.join(d, f) for d in (os.path.join(PKG, "csrc"), os.path.join(ROOT, "include", "pbm"))
         for f in sorted(os.listdir(d)) if f.endswith((".cu", ".cuh"))]


def code_of(path):
    text = open(path).read()
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)


@pytest.mark.parametrize("path", FILES, ids=[os.path.basename(f) for f in FILES])
def test_no_read_only_loads(path):
    assert not re.search(r"\b__ldg\s*\(|__restrict__|\.nc\b", code_of(path))


def test_every_overlapping_kernel_waits_first():
    """Each kernel that is launched with launch_next calls stream_wait before it touches global memory."""
    code = "\n".join(code_of(f) for f in FILES)
    launched = set(re.findall(r"launch_next(?:_if)?\(\s*(?:!?\w+,\s*)?(?:\w+\s*\?\s*)?(k_\w+)", code))
    launched |= set(re.findall(r":\s*(k_\w+)\s*<", code)) | set(re.findall(r"go\((k_\w+)", code))
    launched |= set(re.findall(r"[?(]\s*(k_malloc\w+)<", code))
    assert {"k_round", "k_release", "k_gather_rows", "k_alloc_collab", "k_take_free", "k_malloc_plain",
            "k_malloc_persistent", "k_batch_persistent", "k_claim_write_free"} <= launched
    for k in sorted(launched):
        body = re.search(r"__global__[^;{]*\b" + k + r"\([^{;]*\)\s*\{(.{0,600})", code, flags=re.S)
        assert body and "stream_wait()" in body.group(1), k
