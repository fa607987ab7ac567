"""Run by test_gpu_memory_safety.py in a process of its own with DEEPSHIFT_B200_CHECKED=1: a spread of
linear and convolution shapes on the bounds-checking flavour of the library.  Every result must equal
the oracle's and the status word must stay 0; then the activations are declared 64 bytes shorter than
they are and the checks must report loads beyond that end (kind 1) -- while every access still lies
inside the real buffer."""
import ctypes
import os
import sys

import numpy as np
import torch

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.dirname(HERE))
sys.path.insert(0, HERE)

from helpers import acts_q16, acts_wide, weights  # noqa: E402


def status(lib):
    st, ck = ctypes.c_int(-1), ctypes.c_int(-1)
    assert lib.ds_bounds_status(ctypes.byref(st), ctypes.byref(ck)) == 0
    return st.value, ck.value


def waits_that_run_out(lib, dev, O, cw_of, rng):
    """Parts of the tensor-core kernel hold still, so that each kind of wait runs out: the launch ends by itself, says
    so, leaves the scratch header as it found it, and the next launch is exact again.  A linear layer with four units
    per CTA, a convolution with few tiles whose K is split."""
    from deepshift_b200 import kernels
    for (B, C, H, OC, k, p, holds) in [(60000, 64, 1, 33, 1, 0, (1, 2, 4, 7)), (2, 512, 7, 512, 3, 1, (1, 2))]:
        x = acts_q16(rng, (B, C, H, H))
        shift, sign = weights(rng, (OC, C, k, k))
        cw = cw_of(shift, sign)
        geo = (B, C, H, H, OC, k, k, 1, 1, p, p)
        f = kernels._fuse(act_bits=15)
        act, wt = kernels.tc_bytes(geo, cw, f, any_size=True)
        xt = torch.from_numpy(x).to(dev) // 2      # 15 bits
        wexp = kernels.tc_expand(geo, cw, f, wt, dev)
        want = O.conv2d(x // 2, shift, sign, None, (1, 1), (p, p))
        out = torch.empty(want.shape, dtype=torch.int32, device=dev)
        scratch = torch.zeros(act, dtype=torch.uint8, device=dev)

        def call():
            assert lib.ds_tc_conv2d(xt.data_ptr(), cw.data.data_ptr(), None, out.data_ptr(), *geo, cw.bits, cw.base, f,
                                    scratch.data_ptr(), act, wexp.data_ptr(), wt, torch.cuda.current_stream().cuda_stream) == 0
            torch.cuda.synchronize()
            return kernels.last_kernel_error()

        assert call() == 0 and np.array_equal(out.cpu().numpy(), want)
        for hold in holds:
            assert lib.ds_tc_debug_waits(5_000_000, hold) == 0
            assert call() == 1, hold
            assert lib.ds_tc_debug_waits(0, 0) == 0
            assert int(scratch[:2048].sum()) == 0, hold
            out.fill_(7)
            assert call() == 0 and np.array_equal(out.cpu().numpy(), want), hold
    assert lib.ds_tc_debug_waits(1 << 40, 0) != 0


def main():
    from deepshift_b200 import _ffi, kernels, utils
    from oracle import oracle as O
    O.build()
    lib = _ffi.lib()
    dev = torch.device("cuda:0")
    assert status(lib) == (0, 1), "not the checked flavour"
    rng = np.random.default_rng(77)

    def cw_of(shift, sign):
        return utils.compress_bits(torch.from_numpy(shift).float(), torch.from_numpy(sign).float(), device=dev)

    convs = [(3, 16, 28, 28, 40, 3, 1, 1), (3, 24, 14, 14, 70, 3, 1, 1), (2, 3, 32, 32, 64, 7, 2, 3), (4, 20, 7, 9, 70, 3, 1, 1),
             (3, 12, 10, 10, 33, 1, 2, 0), (2, 5, 9, 9, 12, 2, 1, 0), (5, 128, 7, 7, 130, 3, 1, 1), (49, 32, 28, 28, 100, 3, 1, 1)]
    for (B, C, H, W, OC, k, s, p) in convs:
        shift, sign = weights(rng, (OC, C, k, k))
        bias = rng.integers(-2000, 2000, OC).astype(np.int32)
        cw = cw_of(shift, sign)
        for x, ab in ((acts_q16(rng, (B, C, H, W)), 16), (acts_q16(rng, (B, C, H, W)), None), (acts_wide(rng, (B, C, H, W), 24), 0)):
            out = kernels.conv2d(torch.from_numpy(x).to(dev), torch.from_numpy(shift).to(dev), None,
                                 torch.from_numpy(bias).to(dev), cw, s, p, act_bits=ab)
            assert np.array_equal(out.cpu().numpy(), O.conv2d(x, shift, sign, bias, (s, s), (p, p))), (B, C, H, W, OC, k, ab)
    for (M, K, N) in [(1, 4096, 33), (5, 1031, 300), (16, 96, 4100), (40, 3000, 70), (300, 512, 200), (2304, 260, 130)]:
        shift, sign = weights(rng, (N, K))
        cw = cw_of(shift, sign)
        for ab in (16, 0):
            x = acts_q16(rng, (M, K))
            out = kernels.linear(torch.from_numpy(x).to(dev), torch.from_numpy(shift).to(dev), None, None, cw, act_bits=ab)
            assert np.array_equal(out.cpu().numpy(), O.linear(x, shift, sign, None)), (M, K, N, ab)
    # ... on the tensor cores: rows packed from measured int32 codes, 24-bit codes of fp32 input (kept tiles, used twice),
    # byte planes from layer to layer
    for (M, K, N) in [(66, 1031, 300), (300, 512, 200), (1000, 401, 129)]:
        shift, sign = weights(rng, (N, K))
        cw = cw_of(shift, sign)
        st, x = torch.from_numpy(shift).to(dev), acts_q16(rng, (M, K))
        assert kernels.tc_bytes((M, K, 1, 1, N, 1, 1, 1, 1, 0, 0), cw, kernels._fuse(act_bits=-1))[0] > 0
        out = kernels.linear(torch.from_numpy(x).to(dev), st, None, None, cw)
        assert np.array_equal(out.cpu().numpy(), O.linear(x, shift, sign, None)), (M, K, N)
        xf = rng.normal(0, 1, (M, K)).astype(np.float32)
        want = O.linear(np.trunc(xf.astype(np.float64) * 65536).astype(np.int32), shift, sign, None)
        for _ in range(2):
            out = kernels.linear_fused(torch.from_numpy(xf).to(dev), N, None, cw, in_kind=_ffi.IN_F32_LINEAR)
            assert np.array_equal(out.cpu().numpy(), want), (M, K, N)
    for (B, C, H, OC, halo) in [(3, 16, 9, 48, 1), (2, 64, 14, 144, 2), (2, 512, 7, 16, 1)]:
        shift, sign = weights(rng, (OC, C, 3, 3))
        s2, g2 = weights(rng, (20, OC, 1, 1))
        x = acts_q16(rng, (B, C, H, H))
        src, nxt = kernels.Planes(B, C, H, H, halo, dev), kernels.Planes(B, OC, H, H, 0, dev)
        cur = torch.cuda.current_stream().cuda_stream
        f, xt = kernels._fuse(_ffi.IN_I32_CLAMP, 0, 4, 12), torch.from_numpy(x).to(dev)
        assert lib.ds_planes_pack(xt.data_ptr(), _ffi.IN_I32_CLAMP, 4, 12, src.c, cur) == 0
        out = torch.empty((B, 20, H, H), dtype=torch.int32, device=dev)
        for cw, geo, a, b, o in ((cw_of(shift, sign), (B, C, H, H, OC, 3, 3, 1, 1, 1, 1), src.c, nxt.c, None),
                                 (cw_of(s2, g2), (B, OC, H, H, 20, 1, 1, 1, 1, 0, 0), nxt.c, None, out)):
            na, nw = kernels.tc_bytes(geo, cw, f, any_size=True)
            act = torch.zeros(na, dtype=torch.uint8, device=dev)
            tiles = kernels.tc_expand(geo, cw, f, nw, dev)
            assert lib.ds_tc_conv2d_ex(None, a, cw.data.data_ptr(), None, o.data_ptr() if o is not None else None, b, *geo,
                                       cw.bits, 0, f, act.data_ptr(), na, tiles.data_ptr(), nw, cur) == 0
            torch.cuda.synchronize()
        v = np.clip(O.conv2d(np.clip(x, -32768, 28672), shift, sign, None, (1, 1), (1, 1)), -32768, 28672)
        assert np.array_equal(out.cpu().numpy(), O.conv2d(v, s2, g2, None, (1, 1), (0, 0))), (B, C, H, OC)
    assert status(lib) == (0, 1), "an access left its extent"
    waits_that_run_out(lib, dev, O, cw_of, rng)
    assert status(lib) == (0, 1)
    # the checks fire: x declared 64 bytes short, nothing leaves the real buffer
    B, C, H, OC = 2, 8, 12, 20
    shift, sign = weights(rng, (OC, C, 3, 3))
    x = acts_q16(rng, (B, C, H, H))
    assert lib.ds_bounds_debug_shrink_x(64) == 0
    kernels.conv2d(torch.from_numpy(x).to(dev), torch.from_numpy(shift).to(dev), None, None, cw_of(shift, sign), 1, 1, act_bits=16)
    assert status(lib) == (1, 1), "loads beyond the declared end went unnoticed"
    assert lib.ds_bounds_debug_shrink_x(0) == 0
    out = kernels.conv2d(torch.from_numpy(x).to(dev), torch.from_numpy(shift).to(dev), None, None, cw_of(shift, sign), 1, 1, act_bits=16)
    assert np.array_equal(out.cpu().numpy(), O.conv2d(x, shift, sign, None, (1, 1), (1, 1)))
    assert status(lib) == (0, 1)
    print("checked build: ok")


if __name__ == "__main__":
    main()
