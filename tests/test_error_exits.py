"""Kernels leave on a device error word by whole blocks.  Another block can
set the word between two threads' reads, and a warp or block collective that
some threads have left is undefined, so no thread returns on its own read of
it: grid_sync and block_error read it once per block."""
from __future__ import annotations

import glob
import os
import re

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
OWN_READ = re.compile(r"if\s*\(\s*!?\s*ld_volatile\([^;]*err[^;]*\)\s*return")


def test_no_thread_returns_on_its_own_read():
    files = glob.glob(os.path.join(REPO, "cuda-graph-traversal_b200", "csrc", "**", "*.cu*"), recursive=True)
    assert len(files) > 9
    found = [(os.path.basename(f), m.group(0)) for f in files for m in OWN_READ.finditer(open(f).read())]
    assert not found, found
