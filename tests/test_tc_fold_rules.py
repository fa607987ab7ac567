"""Which 3-wide windows lie side by side in a tile (a "folded" window), as far as that needs no GPU."""
import pytest


def _columns(B, C, H, W, OC, pad, stride=1):
    from deepshift_b200 import _ffi, kernels
    f = kernels._fuse(_ffi.IN_F32_CONV, 0, 4, 12)
    return _ffi.lib().ds_tc_columns(B, C, H, W, OC, 3, 3, stride, stride, pad, pad, 6, 0, f)


@pytest.mark.parametrize("batch,channels,width,folded", [
    (64, 256, 10, False), (64, 256, 14, False), (64, 512, 7, False), (64, 512, 14, False), (64, 256, 28, False),
    (40000, 64, 3, False), (40000, 32, 3, False), (40000, 16, 3, False), (4096, 256, 3, False), (4096, 512, 10, False),
    (64, 64, 56, True), (4096, 32, 16, True), (4096, 16, 32, True),
    (1024, 64, 3, True), (64, 256, 7, True), (1, 512, 7, True), (1, 256, 14, True), (2, 32, 3, True)])
def test_windows_without_padding_count_the_pixels_that_own_no_output(batch, channels, width, folded):
    """The rows of a folded window are the pixels of the image, W of them for W - 2 outputs: what counts in more than one
    wave of tiles."""
    columns = _columns(batch, channels, width, width, channels, 0)
    assert (columns % 3 == 0) == folded and columns > 0


@pytest.mark.parametrize("channels,width", [(256, 14), (512, 7), (64, 56), (32, 16), (16, 32)])
def test_padded_windows_stay_folded(channels, width):
    assert _columns(64, channels, width, width, channels, 1) % 3 == 0


@pytest.mark.parametrize("C,OC,W", [(5, 17, 56), (5, 21, 56), (5, 33, 56), (5, 43, 56), (5, 20, 32), (5, 40, 32), (6, 18, 56),
                                    (6, 34, 56), (6, 17, 32), (6, 34, 32), (80, 4, 64), (114, 6, 12)])
def test_padding_of_one_form_never_makes_a_layer_unserved(C, OC, W):
    """Of one form's tiles less than a fifth of the product is live, of the other's more."""
    from deepshift_b200 import _ffi, kernels, utils
    f = kernels._fuse(_ffi.IN_F32_CONV, 0, 4, 12)
    assert kernels.tc_bytes((256, C, W, W, OC, 3, 3, 1, 1, 1, 1), utils.ConcWeight(None, 0, 6), f)[0] > 0


@pytest.mark.parametrize("C,OC,W,batch,folded", [
    (5, 17, 56, 64, False), (5, 64, 56, 64, False), (8, 32, 32, 256, False), (8, 48, 14, 256, False), (12, 144, 28, 64, False),
    (16, 192, 56, 64, False), (3, 64, 224, 64, False), (96, 256, 56, 64, False), (8, 16, 32, 256, True), (17, 33, 56, 64, True),
    (24, 32, 28, 64, True), (32, 160, 56, 64, True), (40, 144, 28, 64, True), (256, 256, 14, 64, True), (512, 512, 7, 256, True),
    (512, 160, 7, 256, True), (24, 144, 14, 8, True), (96, 256, 28, 1, True), (48, 256, 32, 4, True), (3, 64, 14, 1, False)])
def test_few_items_do_not_hide_the_epilogue_of_a_folded_tile(C, OC, W, batch, folded):
    """Three items of 96 or 192 columns take less time than their epilogue: that counts in long runs."""
    assert (_columns(batch, C, W, W, OC, 1) % 3 == 0) == folded
