"""The build of the library and of the autograd extension beside it (a small
source tree; a stand-in compiler for the extension), and which library the
extension goes with."""
import os
import shutil
import stat
import subprocess
import sys

import pytest
import torch

from dmgs_gb300 import build as B


@pytest.fixture
def tree(tmp_path, monkeypatch):
    """build.py on a tree of one kernel source, the extension's compiler a
    script that writes its output and counts its calls."""
    csrc = tmp_path / "csrc"
    csrc.mkdir()
    (csrc / "one.cu").write_text('extern "C" int one() { return 1; }\n')
    (csrc / "autograd.cpp").write_text("// stands for the nodes\n")
    cxx = tmp_path / "cxx"
    cxx.write_text("#!/bin/sh\n"
                   f"echo x >> {tmp_path}/calls\n"
                   f"[ -e {tmp_path}/broken ] && exit 1\n"
                   "while [ $# -gt 0 ]; do [ \"$1\" = -o ] && echo x > \"$2\"; shift; done\n")
    cxx.chmod(cxx.stat().st_mode | stat.S_IXUSR)
    monkeypatch.setenv("CXX", str(cxx))
    for name, path in (("CSRC", csrc), ("BUILD", tmp_path / "_build"), ("LIB", tmp_path / "lib.so"), ("EXT", tmp_path / "ext.so"),
                       ("TAG", tmp_path / "_build" / "autograd.tag")):
        monkeypatch.setattr(B, name, str(path))
    monkeypatch.calls = lambda: len((tmp_path / "calls").read_text().split()) if (tmp_path / "calls").exists() else 0
    return tmp_path, monkeypatch


def test_the_library_does_not_wait_for_the_extension(tree):
    path, patch = tree
    (path / "broken").write_text("")
    with pytest.raises(RuntimeError):
        B.build()
    assert os.path.exists(B.LIB) and not os.path.exists(B.EXT)
    os.remove(path / "broken")
    B.build()
    assert os.path.exists(B.EXT)


@pytest.mark.parametrize("torch_is", ["missing", "without CUDA"])
def test_the_library_without_a_cuda_torch(tree, torch_is):
    path, patch = tree
    if torch_is == "missing":
        patch.setitem(sys.modules, "torch", None)
    else:
        patch.setattr(torch.version, "cuda", None)
    assert B.build() == B.LIB
    assert os.path.exists(B.LIB) and patch.calls() == 0


def test_the_extension_follows_the_torch_it_is_built_with(tree):
    path, patch = tree
    B.build()
    n = patch.calls()
    assert n == 2  # compiled and linked
    B.build()
    assert patch.calls() == n
    patch.setattr(torch, "__version__", "0.0.1")
    B.build()
    assert patch.calls() == 2 * n
    B.build()
    assert patch.calls() == 2 * n


def test_the_extension_goes_with_the_in_tree_library(tmp_path):
    """A program that loaded another library runs the general forms on it."""
    B.build()
    other = tmp_path / "libother.so"
    shutil.copy(B.LIB, other)
    code = ("import sys; sys.path.insert(0, sys.argv[2]); from dmgs_gb300 import _lib; _lib.load(sys.argv[1] or None); "
            "print(_lib.native() is not None, _lib.native_call('l1_ssim', None, None, 0.2))")
    for path, want in ((str(other), "False None"), (B.LIB, "True None"), ("", "True None")):
        r = subprocess.run([sys.executable, "-c", code, path, os.path.dirname(B.HERE)], capture_output=True, text=True)
        assert r.returncode == 0, r.stderr
        assert r.stdout.strip() == want
