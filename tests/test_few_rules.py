"""Which linear calls have their weights expanded in the kernel, as far as that needs no GPU."""
import random

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


@pytest.mark.parametrize("act_bits", [-1, 15])
def test_no_call_that_the_library_takes_goes_unasked(act_bits):
    """Up to 64 rows small layers are told apart before the question; that must be a true bound of its answer."""
    from deepshift_b200 import kernels
    rng = random.Random(1)
    taken = {False: 0, True: 0}
    for _ in range(20000):
        M = rng.choice([rng.randint(17, 64), rng.randint(65, 2000)])
        K, N = int(2 ** rng.uniform(4, 13.5)), int(2 ** rng.uniform(0, 13.5))
        if kernels._few_bytes.__wrapped__(M, K, N, rng.choice([1, 3, 4, 6, 7]), act_bits) > 0:
            assert kernels._few_asked(M, N * K), (M, K, N)
            taken[M > 64] += 1
    assert min(taken.values()) > 100


def test_what_is_not_asked():
    from deepshift_b200 import kernels
    assert not kernels._few_asked(16, 4096 * 4096) and not kernels._few_asked(64, 1024 * 1024)
    assert kernels._few_asked(65, 1728 * 10) and kernels._few_asked(200, 1216 * 256) and kernels._few_asked(17, 4096 * 4096)
