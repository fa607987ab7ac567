"""What calls on the tensor cores keep of a layer's weights: always the packed words as they are, on every stream."""
import numpy as np
import pytest
import torch

from helpers import weights

pytestmark = pytest.mark.gpu


class Layer:
    """A linear layer on unclamped fp32 input (24-bit form, gated) or a 3x3 convolution (16-bit form)."""

    def __init__(self, oracle, dev, kind, batch=None, seed=1):
        from deepshift_b200 import utils
        self.oracle, self.dev, self.kind, self.utils = oracle, dev, kind, utils
        self.rng = np.random.default_rng(seed)
        self.shape = (70, 400) if kind == "linear" else (130, 64, 3, 3)
        x = (batch or 40, 400) if kind == "linear" else (batch or 3, 64, 14, 14)
        self.x_np = self.rng.normal(0, 1, x).astype(np.float32)
        self.x = torch.from_numpy(self.x_np).to(dev)
        self.cw, self.want = self.make()

    def make(self):
        """New packed weights and the result they give."""
        shift, sign = weights(self.rng, self.shape)
        sign.flat[0] = 0   # always the field width of layers with zero weights
        cw = self.utils.compress_bits(torch.from_numpy(shift).float(), torch.from_numpy(sign).float(), device=self.dev)
        if self.kind == "linear":
            codes = np.trunc(self.x_np.astype(np.float64) * 65536).astype(np.int32)
            return cw, self.oracle.linear(codes, shift, sign, None)
        codes = np.clip(np.floor(self.x_np * 4096.0), -32768, 28672).astype(np.int32)
        return cw, self.oracle.conv2d(codes, shift, sign, None, (1, 1), (1, 1))

    def run(self, out=None):
        from deepshift_b200 import _ffi, kernels
        if self.kind == "linear":
            return kernels.linear_fused(self.x, self.shape[0], None, self.cw, in_kind=_ffi.IN_F32_LINEAR, out=out)
        return kernels.conv2d_fused(self.x, self.shape, None, self.cw, 1, 1, in_kind=_ffi.IN_F32_CONV, act_integer_bits=4,
                                    act_fraction_bits=12, out=out)

    def check(self, got, want=None):
        assert np.array_equal(got.cpu().numpy(), self.want if want is None else want)


@pytest.mark.parametrize("kind", ["linear", "conv"])
def test_changed_packed_words_take_effect(oracle, cuda_device, kind):
    """In place, in place behind autograd's version counter (as collectives and raw pointers write), one word only,
    and by replacing the tensor twice, after which the allocator may hand the first address out again."""
    a = Layer(oracle, cuda_device, kind)
    for _ in range(2):
        a.check(a.run())
    for write in ("copy_", "data.copy_", "one word"):
        cw, want = a.make()
        if write == "copy_":
            a.cw.data.copy_(cw.data)
        elif write == "data.copy_":
            a.cw.data.data.copy_(cw.data)
        else:
            a.cw.data[1:] = cw.data[1:]
            a.run()
            a.cw.data.data[0] = cw.data[0]
        for _ in range(2):
            a.check(a.run(), want)
    for _ in range(3):
        cw, want = a.make()
        a.cw.data = cw.data.clone()
        del cw
        a.check(a.run(), want)


@pytest.mark.parametrize("kind", ["linear", "conv"])
def test_replays_of_a_graph_read_the_packed_words_of_the_moment(oracle, cuda_device, kind):
    a = Layer(oracle, cuda_device, kind)
    out = torch.empty(a.want.shape, dtype=torch.int32, device=cuda_device)
    a.run(out)   # kernel attributes, tiles kept by this stream
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        a.run(out)
    for _ in range(3):
        out.fill_(7)
        g.replay()
        a.check(out)
        cw, a.want = a.make()
        a.cw.data.copy_(cw.data)
        a.check(a.run())
    a.cw.__dict__.pop("_tc", None)   # a graph owns what it reads
    a.x.mul_(1.0)
    filler = [torch.full((1 << 20,), 0x5A, dtype=torch.uint8, device=cuda_device) for _ in range(8)]
    out.fill_(7)
    g.replay()
    a.check(out)
    del filler


@pytest.mark.parametrize("kind", ["linear", "conv"])
def test_streams_do_not_share_what_a_call_may_rewrite(oracle, cuda_device, kind):
    """First calls and changed weights on two streams at once."""
    a = Layer(oracle, cuda_device, kind)
    streams = [torch.cuda.Stream(cuda_device) for _ in range(2)]
    for _ in range(4):
        outs = []
        torch.cuda.synchronize()
        for s in streams:
            with torch.cuda.stream(s):
                outs += [a.run() for _ in range(3)]
        torch.cuda.synchronize()
        for o in outs:
            a.check(o)
        cw, a.want = a.make()
        a.cw.data.copy_(cw.data)


def test_batch_sizes_share_one_buffer(oracle, cuda_device):
    """A new number of rows, or of images, finds the tiles of the layout: no new buffer, at most one per tile width."""
    lin = Layer(oracle, cuda_device, "linear")
    for rows in (17, 40, 64, 200, 33):
        b = Layer(oracle, cuda_device, "linear", rows)
        lin.x, lin.cw.data = b.x, b.cw.data
        lin.check(lin.run(), b.want)
        assert len(lin.cw.__dict__["_tc"]) == 1
    conv = Layer(oracle, cuda_device, "conv", 1)
    for images in (1, 2, 3, 5, 9, 17, 33, 40):
        b = Layer(oracle, cuda_device, "conv", images)
        conv.x, conv.cw.data = b.x, b.cw.data
        conv.check(conv.run(), b.want)
        assert len(conv.cw.__dict__["_tc"]) <= 3
    before = torch.cuda.memory_allocated()
    conv.run()
    assert torch.cuda.memory_allocated() == before


def test_kept_tiles_are_bounded_and_given_back(oracle, cuda_device, monkeypatch):
    from deepshift_b200 import kernels
    a = Layer(oracle, cuda_device, "linear")
    a.check(a.run())
    size = next(iter(a.cw.__dict__["_tc"].values())).buf.numel()
    used = sum(t.buf.numel() for t in list(kernels._TC_KEPT))
    assert used >= size
    total = torch.cuda.get_device_properties(cuda_device).total_memory
    monkeypatch.setattr(kernels, "_TC_KEEP_SHARE", total // (used + size // 2))   # no room for one more of this size
    b = Layer(oracle, cuda_device, "linear", seed=2)
    for _ in range(2):
        b.check(b.run())
    assert not b.cw.__dict__["_tc"]
    a.check(a.run())                    # what is there stays in use
    del a.cw                            # ... and what is given up makes room
    b.check(b.run())
    assert len(b.cw.__dict__["_tc"]) == 1


@pytest.mark.parametrize("kind", ["linear", "conv"])
def test_without_memory_for_tiles_the_other_paths_serve_the_call(oracle, cuda_device, kind, monkeypatch):
    a = Layer(oracle, cuda_device, kind)
    empty = torch.empty

    def no_bytes(*args, **kwargs):
        if kwargs.get("dtype") == torch.uint8:
            raise torch.OutOfMemoryError("no memory (test)")
        return empty(*args, **kwargs)

    monkeypatch.setattr(torch, "empty", no_bytes)
    a.check(a.run())
    monkeypatch.undo()
    a.check(a.run())
