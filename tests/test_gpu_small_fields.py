"""The small-batch linear kernel over every field width: packed words of random bits, so that every field value occurs
(right shifts of 32 and more are zero weights), and activations over all of int32."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [1, 2, 3, 4, 5, 6, 7])
@pytest.mark.parametrize("M", [1, 2, 3, 5, 8, 16])
@pytest.mark.parametrize("base", [0, -3])
def test_every_field_value(oracle, cuda_device, bits, M, base):
    """Rows that are whole 16- and 8-byte groups of words and of activations, and rows that are neither."""
    from deepshift_b200 import kernels, utils
    rng = np.random.default_rng(100 * bits + M)
    for K, N in [(1, 3), (37, 70), (203, 33), (960, 129), (2051, 40), (3840, 66), (1024, 4100), (2048, 4100)]:
        if N * K > 1 << 22 and M not in (1, 8):
            continue   # sizes where one row, or eight, change the way fields are decoded
        row = (K + 32 // (bits + 1) - 1) // (32 // (bits + 1))
        packed = rng.integers(-2 ** 31, 2 ** 31, (N, row)).astype(np.int32)
        x = rng.integers(-2 ** 31, 2 ** 31, (M, K)).astype(np.int32)
        x.flat[0] = -2 ** 31
        bias = rng.integers(-2000, 2000, N).astype(np.int32)
        cw = utils.ConcWeight(torch.from_numpy(packed.reshape(-1)).to(cuda_device), base, bits)
        got = kernels.linear(torch.from_numpy(x).to(cuda_device), torch.empty(N, 1), None, torch.from_numpy(bias).to(cuda_device), cw)
        assert np.array_equal(got.cpu().numpy(), oracle.linear_packed(x, packed, bias, K, bits, base)), (K, N)
