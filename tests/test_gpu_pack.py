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


@pytest.mark.parametrize("lo,hi,odd,far", [(-15, 0, None, False), (-15, 0, -16, True), (-15, 0, -31, True), (-15, 0, -32, False),
                                           (-60, -32, None, False), (-15, 2, -20, False)])
def test_shifts_of_16_to_31_are_noted(cuda_device, lo, hi, odd, far):
    """On both routes; zero weights (stored as 32) are none, and with left shifts (base < 0) nobody asks."""
    from deepshift_b200 import utils
    g = torch.Generator(device=cuda_device).manual_seed(5)
    shift = torch.randint(lo, hi + 1, (40, 61), generator=g, device=cuda_device).float()
    shift[0, 0] = hi
    sign = torch.where(torch.rand((40, 61), generator=g, device=cuda_device) < 0.5, -1.0, 1.0)
    sign[3, 3:9] = 0
    if odd is not None:
        shift[39, 60] = odd
    assert utils.compress_bits(shift, sign).far_shifts == far
    assert utils.compress_bits(shift.double(), sign.double()).far_shifts == far


@pytest.mark.parametrize("seen", [True, False])
def test_linear_layer_with_far_shifts_is_exact_on_either_path(oracle, cuda_device, seen):
    """The integer path when the packing saw them; found on the device when the packed words came otherwise."""
    from deepshift_b200 import _ffi, kernels, utils
    rng = np.random.default_rng(6)
    shift, sign = weights(rng, (70, 400), lo=-30)
    x = rng.normal(0, 1, (40, 400)).astype(np.float32)
    cw = utils.compress_bits(torch.from_numpy(shift).float(), torch.from_numpy(sign).float(), device=cuda_device)
    assert cw.far_shifts
    cw.far_shifts = seen
    want = oracle.linear(np.trunc(x.astype(np.float64) * 65536).astype(np.int32), shift, sign, None)
    for _ in range(2):
        got = kernels.linear_fused(torch.from_numpy(x).to(cuda_device), 70, None, cw, in_kind=_ffi.IN_F32_LINEAR)
        assert np.array_equal(got.cpu().numpy(), want)
    assert bool(cw.__dict__.get("_tc")) != seen
