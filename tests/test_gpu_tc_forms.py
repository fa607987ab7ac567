"""Both forms of the 128-column tile (two and three producer warpgroups) on either side of where they meet."""
import numpy as np
import pytest
import torch

from helpers import acts_q16, weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C", [17, 128, 144])       # two, eight and nine groups of K
@pytest.mark.parametrize("OC", [128, 162])          # one column tile, two
def test_long_runs_of_few_items(oracle, cuda_device, C, OC):
    from deepshift_b200 import _ffi, kernels, utils
    B, H = 48, 28
    rng = np.random.default_rng(C + OC)
    x = acts_q16(rng, (B, C, H, H))
    shift, sign = weights(rng, (OC, C, 1, 1))
    bias = rng.integers(-2000, 2000, OC).astype(np.int32)
    cw = utils.compress_bits(torch.from_numpy(shift).float(), torch.from_numpy(sign).float(), device=cuda_device)
    geo = (B, C, H, H, OC, 1, 1, 1, 1, 0, 0)
    f = kernels._fuse(_ffi.IN_I32_CLAMP, 0, 4, 12)
    act, wt = kernels.tc_bytes(geo, cw, f, any_size=True)
    if C > 17:
        assert _ffi.lib().ds_tc_columns(*geo, cw.bits, 0, f) == 128
    tiles = kernels.tc_expand(geo, cw, f, wt, cuda_device)
    scratch = torch.empty(act, dtype=torch.uint8, device=cuda_device)
    out = torch.full((B, OC, H, H), -7, dtype=torch.int32, device=cuda_device)
    xt, bt = torch.from_numpy(x).to(cuda_device), torch.from_numpy(bias).to(cuda_device)
    assert _ffi.lib().ds_tc_conv2d(xt.data_ptr(), cw.data.data_ptr(), bt.data_ptr(), out.data_ptr(), *geo, cw.bits, 0, f,
                                   scratch.data_ptr(), act, tiles.data_ptr(), wt,
                                   torch.cuda.current_stream(cuda_device).cuda_stream) == 0
    assert np.array_equal(out.cpu().numpy(), oracle.conv2d(x, shift, sign, bias, (1, 1), (0, 0)))
    assert kernels.last_kernel_error() == 0
