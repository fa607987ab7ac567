"""compress_bits where there is no memory left for the bytes of its one-read path."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_without_room_for_the_bytes_the_parameters_are_read_twice(cuda_device, monkeypatch):
    from deepshift_b200 import kernels, utils
    g = torch.Generator(device=cuda_device).manual_seed(1)
    s = torch.randint(-15, 1, (1024, 1030), generator=g, device=cuda_device).float()
    q = torch.where(torch.rand((1024, 1030), generator=g, device=cuda_device) < 0.5, -1.0, 1.0)
    assert s.numel() >= kernels._PACK_BYTES_FROM
    want, empty = utils.compress_bits(s, q), torch.empty

    def full(*a, **k):
        if k.get("dtype") == torch.uint8:
            raise torch.OutOfMemoryError("planted")
        return empty(*a, **k)

    monkeypatch.setattr(torch, "empty", full)
    got = utils.compress_bits(s, q)
    assert (got.base, got.bits, got.far_shifts) == (want.base, want.bits, want.far_shifts) and torch.equal(got.data, want.data)
