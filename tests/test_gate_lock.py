"""Threads that enqueue calls with a measured range wait for one another only where they share a workspace.  Needs no GPU, and
runs only without one: the calls get as far as their first CUDA call, which fails."""
import os
import subprocess
import sys

import pytest
import torch

CODE = """
import ctypes, threading
from deepshift_b200 import _ffi, kernels
lib = _ffi.lib()
A, B, BYTES = 1 << 40, 1 << 41, 65536   # addresses nobody reads
def call(ws):
    f = kernels._fuse(act_bits=-1)
    f.workspace, f.workspace_bytes = ws, BYTES
    assert lib.ds_linear_ex(4096, 4096, None, 4096, 100, 64, 64, 6, 0, f, None) not in (0, 1)
assert lib.ds_gate_debug_hold(A, BYTES, 1) == 0
ta, tb = (threading.Thread(target=call, args=(w,), daemon=True) for w in (A, B))
ta.start(); tb.start()
tb.join(60)
assert not tb.is_alive(), "waits for another workspace"
ta.join(1)
assert ta.is_alive(), "does not wait for its own"
assert lib.ds_gate_debug_hold(None, 0, 0) == 0
ta.join(60)
assert not ta.is_alive()
print("gate: ok")
"""


def test_only_calls_that_share_a_workspace_wait_for_one_another():
    from deepshift_b200 import _build
    if torch.cuda.is_available():
        pytest.skip("the calls would launch")
    if not os.path.exists(_build.CHECKED_LIB_PATH) and _build.nvcc_path() is None:
        pytest.skip("checked flavour not built and no nvcc here")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, DEEPSHIFT_B200_CHECKED="1", PYTHONPATH=root)
    res = subprocess.run([sys.executable, "-c", CODE], env=env, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=900)
    assert res.returncode == 0 and "gate: ok" in res.stdout, res.stdout[-3000:]
