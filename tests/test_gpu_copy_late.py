"""Copying rounds whose waits for a piece of a page run out: the page's bytes are copied another
way before the page counts as resident, and nothing is reported as late."""
import os
import subprocess

import pytest

import test_gpu_bufmgr_forms as forms
from conftest import PKG, ROOT

pytestmark = pytest.mark.gpu
BUILD = os.path.join(ROOT, "tests", "caller", "_build")


@pytest.fixture(scope="module", params=[0, 1, 3])
def short_waits(request, pbm_mod):
    """The library with that many polls of each piece (with none, every wait runs out)."""
    os.makedirs(BUILD, exist_ok=True)
    obj, so = os.path.join(BUILD, f"bufmgr_polls{request.param}.o"), os.path.join(BUILD, f"libpbm_polls{request.param}.so")
    arch = ["-gencode", "arch=compute_103a,code=sm_103a", "-Xcompiler", "-fPIC"]
    src = os.path.join(PKG, "csrc", "bufmgr.cu")
    other = [os.path.join(PKG, "_build", f"{f}.o") for f in sorted(os.listdir(os.path.join(PKG, "csrc")))
             if f.endswith((".cu", ".cpp")) and f != "bufmgr.cu"]
    for cmd in (["nvcc", "-x", "cu", "-c", src, "-o", obj, "-O2", "-std=c++17", "--expt-relaxed-constexpr",
                 f"-DPBM_COPY_POLLS={request.param}", "-I", os.path.join(ROOT, "include"),
                 "-I", os.path.join(PKG, "csrc")] + arch,
                ["nvcc", "-shared", "-o", so, obj] + other + arch):
        r = subprocess.run(cmd, capture_output=True, text=True)
        assert r.returncode == 0, r.stdout + r.stderr
    return pbm_mod.load(so)


@pytest.mark.parametrize("frame_size", [16, 48, 4096, 4112, 12304])
@pytest.mark.parametrize("policy", [0, 1])
def test_late_pages_are_whole(cuda, pbm_mod, short_waits, monkeypatch, frame_size, policy):
    monkeypatch.setattr(pbm_mod, "_LIB", short_waits)
    forms.test_every_copied_frame_holds_its_page(cuda, pbm_mod, frame_size, policy, by_page=bool(policy))


def test_late_pages_of_a_large_round_are_whole(cuda, pbm_mod, short_waits, monkeypatch):
    monkeypatch.setattr(pbm_mod, "_LIB", short_waits)
    forms.test_large_copying_rounds_hold_their_pages(cuda, pbm_mod, 4112, 0, 5000)
