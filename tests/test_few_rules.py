"""Which linear calls have their weights expanded in the kernel, as far as that needs no GPU."""
import pytest


@pytest.mark.parametrize("M,K,N,measured,promised", [
    (80, 1500, 400, True, False), (200, 1216, 256, True, False), (65, 1728, 10, True, False), (300, 2048, 128, True, False),
    (65, 2048, 1000, True, True), (128, 2048, 1000, True, True), (65, 4096, 512, True, True), (128, 4096, 1000, True, True),
    (256, 1024, 2048, True, True), (64, 4096, 4096, True, True), (64, 1024, 1024, False, False), (16, 4096, 4096, False, False)])
def test_promised_codes_move_only_where_it_is_faster(M, K, N, measured, promised):
    """A caller that bounds its codes has the FP32 pipe in one launch instead."""
    from deepshift_b200 import kernels
    assert (kernels._few_bytes(M, K, N, 6, -1) > 0) == measured
    assert (kernels._few_bytes(M, K, N, 6, 15) > 0) == promised
