"""Importing the package before its C++ host path is built, and with one that does not load."""
import os
import shutil
import subprocess
import sys

import pytest

PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ddfnet_b200")

PROGRAM = """
import os, shutil, sys, warnings
import torch
from ddfnet_b200 import DDFPack, ddf, op

def refused():
    x = torch.zeros(1, 2, 5, 5)
    try:
        ddf(x, torch.zeros(1, 2, 3, 3), torch.zeros(1, 9, 5, 5))
    except AssertionError as e:
        return "must be a CUDA tensor" in str(e)

with warnings.catch_warnings(record=True) as seen:
    warnings.simplefilter("always")
    assert refused() and refused() and op._native is None
mine = [str(w.message) for w in seen if "_native.so" in str(w.message)]
assert len(mine) == 1 and sys.argv[2] in mine[0], mine
there = os.path.join(os.path.dirname(op.__file__), "_native.so")
shutil.copy(sys.argv[1], there + ".tmp")
os.replace(there + ".tmp", there)
assert refused() and op._native is not None
"""


@pytest.mark.parametrize("content,says", [(None, "is not built"), (b"not a library", "failed to load")])
def test_the_host_path_may_come_after_the_import(tmp_path, content, says):
    built = os.path.join(PKG, "_native.so")
    if not os.path.exists(built):
        pytest.skip("_native.so is not built here")
    copy = tmp_path / "ddfnet_b200"
    shutil.copytree(PKG, copy, ignore=shutil.ignore_patterns("csrc", "*.so", "*.stamp", "__pycache__"))
    if content is not None:
        (copy / "_native.so").write_bytes(content)
    r = subprocess.run([sys.executable, "-c", PROGRAM, built, says], cwd=tmp_path, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
