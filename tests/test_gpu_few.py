"""Linear layers with few rows whose weights are expanded in the kernel, where a CTA walks several units: accumulator slots
used again, producers and loader crossing units in mid-group, K shared and not.  Whole calls through ``kernels.linear``,
and the bounds-checking flavour of the library."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

from helpers import weights

pytestmark = pytest.mark.gpu


def _few(dev, x, cw, bias, N, act_bits, workspace=None):
    """One direct call on poisoned buffers of exactly the asked size; (output, the scratch's first word)."""
    from deepshift_b200 import _ffi, kernels
    M, K = x.shape
    f = kernels._fuse(act_bits=act_bits, workspace=workspace)
    n = ctypes.c_longlong(0)
    assert _ffi.lib().ds_tc_few_bytes(M, K, N, cw.bits, 0, f, 1, ctypes.byref(n)) == 0 and n.value > 0
    xt = torch.from_numpy(x).to(dev)
    bt = torch.from_numpy(bias).to(dev) if bias is not None else None
    act = torch.full((n.value + 64,), 0xA5, dtype=torch.uint8, device=dev)
    out = torch.full((M * N + 16,), 0x5EADBEE, dtype=torch.int32, device=dev)
    rc = _ffi.lib().ds_tc_linear_few(xt.data_ptr(), cw.data.data_ptr(), bt.data_ptr() if bt is not None else None, out.data_ptr(), M, K, N,
                                     cw.bits, 0, f, act.data_ptr(), n.value, torch.cuda.current_stream(dev).cuda_stream)
    torch.cuda.synchronize(dev)
    assert rc == 0 and kernels.last_kernel_error() == 0
    assert bool((act[n.value:] == 0xA5).all()) and bool((out[-16:] == 0x5EADBEE).all())
    return out[:-16].reshape(M, N).cpu().numpy(), int(act[:4].view(torch.int32))


# (M, K, N): on 148 SMs 595 and 785 units of 80 columns, 600 and 440 of 144, K whole in the first of each, in fifths in the other
UNITS = [(20, 47, 76100), (79, 1500, 20000), (2860, 100, 3840), (1500, 1200, 1000)]


@pytest.mark.parametrize("M,K,N", UNITS)
@pytest.mark.parametrize("act_bits", [-1, 15])
def test_several_units_per_cta(oracle, cuda_device, M, K, N, act_bits):
    """``act_bits`` 15: nothing is measured, and the output is zeroed only where K is shared."""
    from deepshift_b200 import kernels, utils
    rng = np.random.default_rng(M + K)
    shift, sign = weights(rng, (N, K))
    bias = rng.integers(-2000, 2000, N).astype(np.int32)
    cw = utils.compress_bits(torch.from_numpy(shift).float(), torch.from_numpy(sign).float(), device=cuda_device)
    x = rng.integers(-16384, 16384, (M, K)).astype(np.int32)
    rows = sorted({0, 1, M // 3, M // 2, M - 2, M - 1} | set(range(M - M % 143, M, 29)))
    got, flag = _few(cuda_device, x, cw, bias, N, act_bits)
    assert np.array_equal(got[rows], oracle.linear(x[rows], shift, sign, bias))
    exact = kernels.linear(torch.from_numpy(x).to(cuda_device), torch.empty(N, 1), None, torch.from_numpy(bias).to(cuda_device), cw,
                           act_bits=0)
    assert np.array_equal(got, exact.cpu().numpy())
    assert flag == (0 if act_bits == -1 else int.from_bytes(b"\xa5" * 4, "little", signed=True))


@pytest.mark.parametrize("M", [64, 512])
@pytest.mark.parametrize("act_bits,wide", [(None, False), (None, True), (15, False)])
def test_whole_calls(oracle, cuda_device, monkeypatch, M, act_bits, wide):
    """4096 -> 4096, in range and with one code beyond it, which also ends in the workspace's last counter word."""
    from deepshift_b200 import kernels, utils
    rng = np.random.default_rng(M)
    K = N = 4096
    shift, sign = weights(rng, (N, K))
    bias = rng.integers(-2000, 2000, N).astype(np.int32)
    cw = utils.compress_bits(torch.from_numpy(shift).float(), torch.from_numpy(sign).float(), device=cuda_device)
    x = rng.integers(-16384, 16384, (M, K)).astype(np.int32)
    if wide:
        x[M - 1, K - 1] = 32768
    served, few = [], kernels._few_run
    monkeypatch.setattr(kernels, "_few_run", lambda *a: served.append(few(*a)) or served[-1])
    ws = kernels.workspace(cuda_device)
    ws[16383] = 77
    xt, bt = torch.from_numpy(x).to(cuda_device), torch.from_numpy(bias).to(cuda_device)
    got = kernels.linear(xt, torch.empty(N, 1), None, bt, cw, act_bits=act_bits)
    word = int(ws[16383])
    ws[16383] = 0
    assert served == [True] and kernels.last_kernel_error() == 0
    assert word == (int(wide) if act_bits is None and M > 64 else 77)
    rows = sorted({0, 1, 63, 77, 78, 79, 142, 143, 144, 285, 286, M - 2, M - 1} & set(range(M)))
    assert np.array_equal(got[rows].cpu().numpy(), oracle.linear(x[rows], shift, sign, bias))
    assert torch.equal(got, kernels.linear(xt, torch.empty(N, 1), None, bt, cw, act_bits=0))


def test_bounds_checking_flavour(cuda_device):
    """The checked flavour in a process of its own: exact with status 0, the checks fire when x is declared short, and waits
    that run out end the launch."""
    from deepshift_b200 import _build
    if not os.path.exists(_build.CHECKED_LIB_PATH) and _build.nvcc_path() is None:
        pytest.skip("checked flavour not built and no nvcc here")
    script = os.path.join(os.path.dirname(os.path.abspath(__file__)), "checked_build_few.py")
    res = subprocess.run([sys.executable, script], env=dict(os.environ, DEEPSHIFT_B200_CHECKED="1"), stdout=subprocess.PIPE,
                         stderr=subprocess.STDOUT, text=True, timeout=600)
    assert res.returncode == 0 and "checked build, few rows: ok" in res.stdout, res.stdout[-3000:]
