"""Run by test_gpu_few.py in a process of its own with DEEPSHIFT_B200_CHECKED=1: the few-row kernel on the bounds-checking
flavour of the library.  Every result must equal the oracle's and the status word must stay 0; with the activations declared
64 bytes shorter than they are the checks must report it while every access still lies inside the real buffers; and parts of
the kernel hold still, so that each kind of its waits runs out."""
import ctypes
import os
import sys

import numpy as np
import torch

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.dirname(HERE))
sys.path.insert(0, HERE)

from helpers import weights  # noqa: E402


def main():
    from deepshift_b200 import _ffi, kernels, utils
    from oracle import oracle as O
    O.build()
    lib = _ffi.lib()
    dev = torch.device("cuda:0")
    rng = np.random.default_rng(78)

    def status():
        st, ck = ctypes.c_int(-1), ctypes.c_int(-1)
        assert lib.ds_bounds_status(ctypes.byref(st), ctypes.byref(ck)) == 0
        return st.value, ck.value

    def case(M, K, N, act_bits, lo=-15, zeros=True):
        shift, sign = weights(rng, (N, K), lo, zeros)
        cw = utils.compress_bits(torch.from_numpy(shift).float(), torch.from_numpy(sign).float(), device=dev)
        x = rng.integers(-16384, 16384, (M, K)).astype(np.int32)
        xt, out = torch.from_numpy(x).to(dev), torch.empty((M, N), dtype=torch.int32, device=dev)
        f = kernels._fuse(act_bits=act_bits)
        n = ctypes.c_longlong(0)
        assert lib.ds_tc_few_bytes(M, K, N, cw.bits, 0, f, 1, ctypes.byref(n)) == 0 and n.value > 0
        act = torch.full((n.value,), 0xA5, dtype=torch.uint8, device=dev)

        def call():
            assert lib.ds_tc_linear_few(xt.data_ptr(), cw.data.data_ptr(), None, out.data_ptr(), M, K, N, cw.bits, 0, f,
                                        act.data_ptr(), n.value, torch.cuda.current_stream().cuda_stream) == 0
            torch.cuda.synchronize()
            return kernels.last_kernel_error()

        return call, out, O.linear(x, shift, sign, None)

    assert status() == (0, 1), "not the checked flavour"
    # both tile widths, rows and columns that fill no tile, K shared and whole, words and groups that K does not fill
    for (M, K, N, act_bits, lo, zeros) in [(17, 300, 127, -1, -15, True), (64, 2051, 300, -1, -15, True), (79, 1000, 129, 15, -7, False),
                                           (80, 1024, 129, -1, -3, False), (300, 515, 260, 15, -15, False), (20, 47, 76100, 15, -15, True)]:
        call, out, want = case(M, K, N, act_bits, lo, zeros)
        assert call() == 0 and np.array_equal(out.cpu().numpy(), want), (M, K, N)
    assert status() == (0, 1), "an access left its extent"
    # ... x declared 64 bytes short: noticed, skipped
    call, out, want = case(33, 300, 70, 15)
    assert lib.ds_bounds_debug_shrink_x(64) == 0
    assert call() == 0 and status() == (1, 1), "loads beyond the declared end went unnoticed"
    assert lib.ds_bounds_debug_shrink_x(0) == 0
    assert call() == 0 and np.array_equal(out.cpu().numpy(), want) and status() == (0, 1)
    # Waits run out: 595 units, four or five per CTA, so that accumulator slots come round again
    call, out, want = case(20, 47, 76100, 15)
    for hold in (1, 2, 4, 7):
        assert lib.ds_tc_debug_waits(5_000_000, hold) == 0
        assert call() == 1, hold
        assert lib.ds_tc_debug_waits(0, 0) == 0
        out.fill_(7)
        assert call() == 0 and np.array_equal(out.cpu().numpy(), want), hold
    assert status() == (0, 1)
    print("checked build, few rows: ok")


if __name__ == "__main__":
    main()
