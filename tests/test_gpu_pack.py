"""compress_bits on fp32 parameters (two kernels) against the chain of torch passes it replaces."""
import numpy as np
import pytest
import torch

from helpers import weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1), (3, 7), (33, 64), (16, 3, 7, 7), (10, 45, 3, 3), (129, 20, 1, 1)])
@pytest.mark.parametrize("lo,hi,zeros", [(-15, 0, True), (-15, 0, False), (-7, 0, False), (-3, 0, False), (-1, 0, False),
                                         (0, 0, False), (-7, 3, True), (-2, 2, False), (-60, 0, True)])
def test_fp32_parameters_pack_as_integer_ones_do(oracle, cuda_device, shape, lo, hi, zeros):
    """float64 parameters take the general route; both give the oracle's words."""
    from deepshift_b200 import utils
    rng = np.random.default_rng(sum(shape) - 31 * lo + hi)
    shift = rng.integers(lo, hi + 1, shape).astype(np.int32)
    sign = weights(rng, shape, zeros=zeros)[1]
    s, g = torch.from_numpy(shift).to(cuda_device), torch.from_numpy(sign).to(cuda_device)
    fast = utils.compress_bits(s.float(), g.float())
    slow = utils.compress_bits(s.double(), g.double())
    assert (fast.base, fast.bits) == (slow.base, slow.bits)
    assert torch.equal(fast.data, slow.data)
    packed, base, bits = oracle.compress_bits(shift, sign)
    assert (base, bits) == (fast.base, fast.bits) and np.array_equal(packed.reshape(-1), fast.data.cpu().numpy())


def test_unrounded_parameters_and_views(cuda_device):
    """Halves round to even, signs below one count as negative, unaligned views pack like their copies."""
    from deepshift_b200 import utils
    g = torch.Generator(device=cuda_device).manual_seed(3)
    shift = torch.randint(-28, 1, (40, 61), generator=g, device=cuda_device).float() / 2
    sign = torch.rand((40, 61), generator=g, device=cuda_device) * 4 - 2
    sign[::3, ::5] = 0
    for s, q in ((shift, sign), (shift[1:, 1:], sign[1:, 1:]), (shift.reshape(-1)[1:2401].view(40, 60), sign.reshape(-1)[1:2401].view(40, 60)),
                 (shift.t(), sign.t())):
        fast, slow = utils.compress_bits(s, q), utils.compress_bits(s.double(), q.double())
        assert (fast.base, fast.bits) == (slow.base, slow.bits) and torch.equal(fast.data, slow.data)
