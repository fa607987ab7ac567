"""compress_bits on fp32 parameters that are read once (a byte per weight, then the words): every field width, rows that are
no whole groups, unaligned and strided views, shifts of both signs up to where a byte ends."""
import numpy as np
import pytest
import torch

import test_gpu_pack as two_reads

pytestmark = pytest.mark.gpu


@pytest.fixture
def one_read(monkeypatch):
    """Layers of any size take the path of the large ones; counts the calls that made words from bytes."""
    from deepshift_b200 import kernels
    calls, pack = [], kernels.pack_codes
    monkeypatch.setattr(kernels, "_PACK_BYTES_FROM", 0)
    monkeypatch.setattr(kernels, "pack_codes", lambda *a: calls.append(a) or pack(*a))
    return calls


# (lo, hi, zeros): fields of 6, 4, 5, 3, 2, 1, 1, 4 (base < 0), 3 (base < 0), 6, 7 and 7 bits, the last to both ends of a byte
WIDTHS = [(-15, 0, True), (-15, 0, False), (-20, 0, False), (-7, 0, False), (-3, 0, False), (-1, 0, False), (0, 0, False),
          (-7, 3, False), (-2, 2, False), (-60, 0, True), (-60, 10, True), (-63, 64, False)]


@pytest.mark.parametrize("shape", [(1, 1), (3, 7), (33, 64), (16, 3, 7, 7), (10, 45, 3, 3), (129, 20, 1, 1), (5, 2048), (40, 62)])
@pytest.mark.parametrize("lo,hi,zeros", WIDTHS)
def test_every_width_and_row(oracle, cuda_device, one_read, shape, lo, hi, zeros):
    two_reads.test_fp32_parameters_pack_as_integer_ones_do(oracle, cuda_device, shape, lo, hi, zeros)
    assert len(one_read) == 1


def test_unrounded_parameters_and_views(cuda_device, one_read):
    two_reads.test_unrounded_parameters_and_views(cuda_device)
    assert len(one_read) == 4


@pytest.mark.parametrize("lo,hi,odd,far", [(-15, 0, None, False), (-15, 0, -16, True), (-15, 0, -31, True), (-15, 0, -32, False),
                                           (-60, -32, None, False), (-15, 2, -20, False)])
def test_shifts_of_16_to_31_are_noted(cuda_device, one_read, lo, hi, odd, far):
    two_reads.test_shifts_of_16_to_31_are_noted(cuda_device, lo, hi, odd, far)
    assert len(one_read) == 1


@pytest.mark.parametrize("shift,fits", [(-63, True), (-64, False), (64, True), (65, False)])
def test_shifts_beyond_a_byte_are_read_twice(cuda_device, one_read, shift, fits):
    """Right shifts of 64 and left shifts of 65 are outside the seven bits; the fields still hold them."""
    from deepshift_b200 import utils
    g = torch.Generator(device=cuda_device).manual_seed(9)
    s = torch.randint(-5, 1, (30, 43), generator=g, device=cuda_device).float()
    s[29, 42] = shift
    q = torch.where(torch.rand((30, 43), generator=g, device=cuda_device) < 0.5, -1.0, 1.0)
    fast, slow = utils.compress_bits(s, q), utils.compress_bits(s.double(), q.double())
    assert (fast.base, fast.bits) == (slow.base, slow.bits) and torch.equal(fast.data, slow.data)
    assert len(one_read) == int(fits)


@pytest.mark.parametrize("shape", [(1031, 1021), (1024, 1028), (512, 232, 3, 3)])
@pytest.mark.parametrize("lo,hi,zeros", WIDTHS[:5] + WIDTHS[7:8] + WIDTHS[10:])
def test_large_layers(cuda_device, shape, lo, hi, zeros):
    """Above the size where the path is taken: odd rows with a tail beyond the last 16 bytes, and rows of whole groups."""
    from deepshift_b200 import kernels, utils
    g = torch.Generator(device=cuda_device).manual_seed(-lo)
    s = torch.randint(lo, hi + 1, shape, generator=g, device=cuda_device).float()
    u = torch.rand(shape, generator=g, device=cuda_device)
    q = torch.where(u < 0.5, -1.0, 1.0)
    if zeros:
        q[(u > 0.45) & (u < 0.55)] = 0
    assert s.numel() >= kernels._PACK_BYTES_FROM
    for a, b in ((s, q), (s.reshape(-1)[1:-2].view(1, -1), q.reshape(-1)[1:-2].view(1, -1))):
        fast, slow = utils.compress_bits(a, b), utils.compress_bits(a.double(), b.double())
        assert (fast.base, fast.bits) == (slow.base, slow.bits) and torch.equal(fast.data, slow.data)
