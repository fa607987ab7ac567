"""The tensor-core path's size rule and the state it keeps, as far as they need no GPU."""
import copy
import pickle
import threading

import pytest
import torch


def _bytes(geo, in_kind, act_bits=0, I=4, F=12, base=0, bits=6, any_size=False):
    from deepshift_b200 import kernels, utils
    return kernels.tc_bytes(geo, utils.ConcWeight(None, base, bits), kernels._fuse(in_kind, 0, I, F, act_bits=act_bits), any_size)


def _linear(M, K, N):
    return (M, K, 1, 1, N, 1, 1, 1, 1, 0, 0)


@pytest.mark.parametrize("geo,in_kind,act_bits,served", [
    (_linear(8192, 4096, 4096), 0, -1, True), (_linear(65, 256, 10), 0, -1, True), (_linear(64, 4096, 4096), 0, -1, False),
    (_linear(8192, 255, 4096), 0, -1, False), (_linear(17, 320, 10), 2, 0, True), (_linear(17, 319, 10), 2, 0, False), (_linear(16, 4096, 4096), 2, 0, False),
    (_linear(8192, 4096, 4096), 0, 16, False), (_linear(8192, 4096, 4096), 0, 15, True), (_linear(8192, 4096, 4096), 0, 0, False),
    ((256, 64, 56, 56, 64, 3, 3, 1, 1, 1, 1), 3, 0, True), ((64, 64, 28, 28, 64, 1, 1, 1, 1, 0, 0), 0, -1, False),
    ((37, 45, 31, 29, 70, 3, 3, 2, 2, 1, 1), 0, -1, True), ((1, 64, 56, 56, 64, 3, 3, 1, 1, 1, 1), 0, -1, False), ((1, 64, 56, 56, 128, 1, 1, 2, 2, 0, 0), 3, 0, True),
    ((12, 16, 28, 28, 40, 3, 3, 1, 1, 1, 1), 3, 0, False), ((1024, 1, 28, 28, 20, 5, 5, 1, 1, 0, 0), 1, 0, False)])
def test_which_calls_are_served(geo, in_kind, act_bits, served):
    assert (_bytes(geo, in_kind, act_bits)[0] > 0) == served


def test_what_is_never_served():
    conv = (8, 64, 28, 28, 64, 3, 3, 1, 1, 1, 1)
    assert _bytes(conv, 3, any_size=True)[0] > 0
    assert _bytes(conv, 3, base=-1, any_size=True) == (0, 0)           # left shifts
    assert _bytes(conv, 3, I=5, F=12, any_size=True) == (0, 0)         # 17-bit codes
    assert _bytes(conv, 3, I=1, F=15, any_size=True) == (0, 0)         # one integer bit: codes down to -2^16
    assert _bytes(conv, 2, any_size=True) == (0, 0)                    # unclamped fp32 input of a convolution
    assert _bytes((1, 1 << 15, 128, 128, 8, 1, 1, 1, 1, 0, 0), 3, any_size=True) == (0, 0)  # an image of 2 GiB


def test_copies_of_packed_weights_leave_the_expanded_tiles_behind():
    from deepshift_b200 import utils
    cw = utils.ConcWeight(torch.arange(3, dtype=torch.int32), -2, 5)
    cw.__dict__["_tc"] = {"key": threading.Lock()}   # as unpicklable as a CUDA event
    for other in (copy.deepcopy(cw), pickle.loads(pickle.dumps(cw)), copy.copy(cw)):
        assert torch.equal(other.data, cw.data) and (other.base, other.bits) == (-2, 5) and "_tc" not in other.__dict__
    assert "_tc" in cw.__dict__


def test_layout_of_the_weights_does_not_depend_on_the_batch():
    """24-bit linear layers have one width of tile; convolutions at most three, whatever the batch."""
    from deepshift_b200 import _ffi, kernels
    columns = lambda geo, kind: kernels._tc_bytes(geo, 6, 0, kind, 0, 4, 12, True, 1)[1:]
    assert len({columns(_linear(m, 4096, 4096), _ffi.IN_F32_LINEAR) for m in (17, 64, 1000, 20000)}) == 1
    sizes = {columns((b, 64, 28, 28, 128, 3, 3, 1, 1, 1, 1), _ffi.IN_F32_CONV) for b in range(1, 400, 7)}
    assert {c for _, c in sizes} <= {32, 64, 128} and len(sizes) <= 3


@pytest.mark.parametrize("geo,plain,served", [
    ((65, 256, 10), True, False), ((128, 2048, 1000), True, False), ((256, 2048, 1000), True, True),
    ((512, 2048, 256), True, False), ((1024, 2048, 256), True, True), ((512, 4096, 256), True, False),
    ((512, 700, 1000), True, True), ((4096, 1024, 10), True, True), ((128, 4096, 1000), True, False),
    ((65, 320, 10), False, False), ((65, 400, 10), False, True), ((4096, 399, 4096), False, False)])
def test_promised_codes_move_only_where_it_is_faster(geo, plain, served):
    """Linear layers whose caller bounds the codes: the FP32-pipe path needs one launch, so small ones stay there."""
    from deepshift_b200 import kernels, utils
    f = kernels._fuse(0, 0 if plain else 1, 4, 8, act_bits=12)
    assert (kernels.tc_bytes(_linear(*geo), utils.ConcWeight(None, 0, 6), f)[0] > 0) == served
