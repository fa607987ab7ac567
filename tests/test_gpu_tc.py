"""The tensor-core path (ds_tc_*) against the CPU oracle: all results are integers, all comparisons exact."""
import ctypes

import numpy as np
import pytest
import torch

from helpers import acts_q16, acts_wide, weights

pytestmark = pytest.mark.gpu


def _run(dev, x, shift, sign, bias, s, p, *, in_kind=0, act_bits=15, out_f32=False, relu=False, residual=None, I=4, F=12,
         round_f32=False, falls_back=None):
    """One call of any size through the C ABI, scratch and weights in buffers of exactly the asked size.
    ``falls_back`` (calls whose range is measured): whether the integer path must have given the answer."""
    from deepshift_b200 import _ffi, kernels, utils
    B, C, H, W = x.shape
    OC, _, KH, KW = shift.shape
    cw = utils.compress_bits(torch.from_numpy(shift).float(), torch.from_numpy(sign).float(), device=dev)
    geo = (B, C, H, W, OC, KH, KW, s[0], s[1], p[0], p[1])
    OH, OW = (H + 2 * p[0] - KH) // s[0] + 1, (W + 2 * p[1] - KW) // s[1] + 1
    xt = torch.from_numpy(x).to(dev)
    bt = torch.from_numpy(bias).to(dev) if bias is not None else None
    rt = torch.from_numpy(residual).to(dev) if residual is not None else None
    f = kernels._fuse(in_kind, 1 if out_f32 else 0, I, F, relu=relu, act_bits=act_bits, residual=rt, round_f32=round_f32)
    act, wt = kernels.tc_bytes(geo, cw, f, any_size=True)
    assert act > 0 and wt > 0
    weights_ = kernels.tc_expand(geo, cw, f, wt, dev)
    scratch = torch.full((act + 64,), 0xA5, dtype=torch.uint8, device=dev)
    out = torch.full((B * OC * OH * OW + 16,), 0x5EADBEE, dtype=torch.int32, device=dev)
    rc = _ffi.lib().ds_tc_conv2d(xt.data_ptr(), cw.data.data_ptr(), bt.data_ptr() if bt is not None else None,
                                 out.data_ptr(), *geo, cw.bits, cw.base, f, scratch.data_ptr(), act, weights_.data_ptr(),
                                 wt, torch.cuda.current_stream(dev).cuda_stream)
    assert rc == 0
    torch.cuda.synchronize(dev)
    assert kernels.last_kernel_error() == 0
    assert bool((scratch[act:] == 0xA5).all()) and bool((out[-16:] == 0x5EADBEE).all())
    if falls_back is not None:   # the range flag, first word of the scratch
        assert int(scratch[:4].view(torch.int32)) == int(falls_back)
    y = out[:-16].reshape(B, OC, OH, OW)
    return (y.view(torch.float32) if out_f32 else y).cpu().numpy()


# (B, C, H, W, OC, KH, KW, stride, pad): edges of the 128-row blocks and of the 32 / 64 / 128-column tiles,
# pixel widths of 4, 8 and 16 bytes, windows whose rows are no multiple of 16 bytes, K split over CTAs
SHAPES = [(1, 16, 4, 4, 16, 1, 1, (1, 1), (0, 0)), (2, 3, 9, 11, 5, 3, 3, (1, 1), (1, 1)), (1, 1, 28, 28, 20, 5, 5, (1, 1), (0, 0)),
          (3, 20, 12, 12, 50, 5, 5, (1, 1), (0, 0)), (2, 45, 31, 29, 70, 3, 3, (2, 2), (1, 1)),
          (2, 3, 32, 32, 64, 7, 7, (2, 2), (3, 3)), (1, 64, 16, 8, 128, 3, 3, (1, 1), (1, 1)),
          (1, 64, 16, 8, 129, 3, 3, (1, 1), (1, 1)), (5, 33, 13, 10, 257, 1, 1, (2, 2), (0, 0)),
          (2, 512, 7, 7, 512, 3, 3, (1, 1), (1, 1)), (3, 17, 6, 9, 33, 2, 3, (1, 2), (1, 0)),
          (40, 32, 28, 28, 64, 3, 3, (1, 1), (1, 1)), (33, 16, 32, 32, 16, 3, 3, (1, 1), (1, 1))]


@pytest.mark.parametrize("shape", SHAPES)
def test_conv(oracle, cuda_device, shape):
    B, C, H, W, OC, KH, KW, s, p = shape
    rng = np.random.default_rng(sum(shape[:7]))
    x = rng.integers(-16384, 16385, (B, C, H, W)).astype(np.int32)
    shift, sign = weights(rng, (OC, C, KH, KW))
    bias = rng.integers(-2000, 2000, OC).astype(np.int32)
    got = _run(cuda_device, x, shift, sign, bias, s, p)
    assert np.array_equal(got, oracle.conv2d(x, shift, sign, bias, s, p))


# (B, C, H, W, OC, KH, stride, pad) of 3-wide windows that move by one pixel: rows of 1 to 70 pixels that end with a
# warp's 32 lanes or do not, warps of which the first or last lane lends its sums only, outputs fewer than pixels, every
# width of tile with all and with few of its channels live, K split over CTAs
FOLDED = [(3, 16, 5, 1, 16, 3, 1, (1, 1)), (2, 32, 4, 3, 20, 3, 1, (1, 0)), (70, 16, 6, 8, 16, 3, 1, (1, 1)),
          (5, 49, 9, 15, 33, 3, 1, (1, 1)), (3, 48, 7, 16, 32, 3, 2, (1, 1)), (4, 50, 11, 30, 9, 1, 1, (0, 1)),
          (2, 64, 13, 31, 64, 3, 1, (1, 1)), (120, 16, 16, 16, 64, 3, 1, (1, 1)), (80, 16, 16, 16, 32, 3, 1, (1, 1)), (2, 33, 8, 33, 63, 2, 1, (0, 0)),
          (1, 256, 9, 56, 50, 3, 1, (1, 1)), (1, 130, 6, 70, 17, 5, 1, (2, 1))]


@pytest.mark.parametrize("shape", FOLDED)
@pytest.mark.parametrize("residual", [False, True])
def test_folded_windows(oracle, cuda_device, shape, residual):
    from deepshift_b200 import _ffi, kernels
    B, C, H, W, OC, KH, s, p = shape
    rng = np.random.default_rng(sum(shape[:7]))
    x = rng.integers(-16384, 16385, (B, C, H, W)).astype(np.int32)
    shift, sign = weights(rng, (OC, C, KH, 3))
    bias = rng.integers(-2000, 2000, OC).astype(np.int32)
    want = oracle.conv2d(x, shift, sign, bias, (s, 1), p)
    add = rng.integers(-2 ** 22, 2 ** 22, want.shape).astype(np.int32) if residual else None
    geo = (B, C, H, W, OC, KH, 3, s, 1, p[0], p[1])
    assert _ffi.lib().ds_tc_columns(*geo, 6, 0, kernels._fuse(0, act_bits=15)) in (48, 96, 192)
    got = _run(cuda_device, x, shift, sign, bias, (s, 1), p, residual=add, relu=residual)
    assert np.array_equal(got, np.maximum(want + add, 0) if residual else want)   # exact in fp32: below 2^24


@pytest.mark.parametrize("mkn", [(1, 64, 10), (127, 100, 31), (128, 2047, 1001), (129, 16, 64), (300, 4096, 130),
                                 (1000, 33, 65), (640, 800, 500)])
def test_linear_full_16_bit_range(oracle, cuda_device, mkn):
    """Codes over the whole 16-bit range, its ends among them, found to fit while packing."""
    M, K, N = mkn
    rng = np.random.default_rng(M + K + N)
    x = rng.integers(-32768, 32768, (M, K, 1, 1)).astype(np.int32)
    x.flat[::7] = -32768
    x.flat[3::11] = 32767
    shift, sign = weights(rng, (N, K, 1, 1))
    got = _run(cuda_device, x, shift, sign, None, (1, 1), (0, 0), act_bits=-1, falls_back=False)
    want = oracle.linear(x.reshape(M, K), shift.reshape(N, K), sign.reshape(N, K), None)
    assert np.array_equal(got.reshape(M, N), want)


@pytest.mark.parametrize("rows", [1, 130])
@pytest.mark.parametrize("fp32", [False, True])
def test_sums_wrap_around_like_int32(oracle, cuda_device, fp32, rows):
    """Partial sums of one sign that leave int32: 16-bit codes reach 2^31 after 2^16 products without a shift, 24-bit
    codes after 2^8.  The accumulators must wrap, not saturate."""
    rng = np.random.default_rng(rows)
    K, N = 150_000, 33
    x = np.full((rows, K, 1, 1), -128.0 if fp32 else -32768, np.float32 if fp32 else np.int32)
    x.flat[::5] = 127.5 if fp32 else -32767
    shift = np.zeros((N, K, 1, 1), np.int32)
    sign = np.ones((N, K, 1, 1), np.int32)
    sign[1::2] = -1
    shift[3, ::2] = -1
    shift[4] = -rng.integers(0, 16, (K, 1, 1))
    got = _run(cuda_device, x, shift, sign, None, (1, 1), (0, 0), in_kind=2 if fp32 else 0, act_bits=0 if fp32 else -1, I=16,
               F=16, falls_back=False)
    codes = (x.astype(np.float64) * (65536 if fp32 else 1)).astype(np.int64).reshape(rows, K)
    w, r = sign.reshape(N, K).astype(np.int64), -shift.reshape(N, K).astype(np.int64)
    exact = np.stack([((codes >> r[n]) * w[n]).sum(1) for n in range(N)], 1)
    assert np.abs(exact).max() > 2 ** 32
    assert np.array_equal(got.reshape(rows, N), exact.astype(np.int32))


@pytest.mark.parametrize("value", [32768, -32769, 1 << 30])
def test_one_wide_code_sends_the_call_to_the_integer_path(oracle, cuda_device, value):
    rng = np.random.default_rng(5)
    x = acts_q16(rng, (3, 20, 9, 10))
    x[2, 19, 8, 9] = value
    shift, sign = weights(rng, (40, 20, 3, 3))
    got = _run(cuda_device, x, shift, sign, None, (1, 1), (1, 1), act_bits=-1, falls_back=True)
    assert np.array_equal(got, oracle.conv2d(x, shift, sign, None, (1, 1), (1, 1)))
    xl = acts_q16(rng, (90, 70, 1, 1))
    xl[89, 69] = value
    sl, gl = weights(rng, (33, 70, 1, 1))
    got = _run(cuda_device, xl, sl, gl, None, (1, 1), (0, 0), act_bits=-1, falls_back=True)
    assert np.array_equal(got.reshape(90, 33), oracle.linear(xl.reshape(90, 70), sl.reshape(33, 70), gl.reshape(33, 70), None))


@pytest.mark.parametrize("out_f32", [False, True])
@pytest.mark.parametrize("geo", [(4, 24, 10, 10, 70, 3), (200, 96, 1, 1, 40, 1), (3, 256, 5, 5, 130, 3)])
def test_clamped_input_residual_relu_rounding(oracle, cuda_device, geo, out_f32):
    B, C, H, W, OC, k = geo
    rng = np.random.default_rng(sum(geo))
    x = acts_wide(rng, (B, C, H, W), 20)
    shift, sign = weights(rng, (OC, C, k, k))
    bias = rng.integers(-2000, 2000, OC).astype(np.int32)
    res = rng.integers(-50000, 50000, (B, OC, H, W)).astype(np.int32)
    got = _run(cuda_device, x, shift, sign, bias, (1, 1), (k // 2, k // 2), in_kind=3, act_bits=0, relu=True, residual=res,
               out_f32=out_f32, round_f32=True)
    acc = oracle.conv2d(np.clip(x, -32768, 28672), shift, sign, bias, (1, 1), (k // 2, k // 2))
    v = np.maximum((acc.astype(np.float32) + res.astype(np.float32)).astype(np.int32), 0)
    want = v.astype(np.float32) / np.float32(4096) if out_f32 else v
    assert np.array_equal(got, want)


@pytest.mark.parametrize("IF", [(4, 12), (1, 14), (3, 8)])
def test_fp32_input_is_quantised_while_packing(oracle, cuda_device, IF):
    I, F = IF
    rng = np.random.default_rng(I * 100 + F)
    x = (rng.normal(0, 3, (3, 18, 11, 7))).astype(np.float32)
    x[0, 0, 0, :4] = [0.0, -0.0, np.inf, -np.inf]
    shift, sign = weights(rng, (35, 18, 3, 3))
    codes = (np.sign(x) - 1) * 2 ** F if I == 1 else np.clip(np.floor(x * 2.0 ** F), -2 ** (I - 1 + F), (2 ** (I - 1) - 1) * 2 ** F)
    got = _run(cuda_device, x, shift, sign, None, (1, 1), (1, 1), in_kind=1, act_bits=0, I=I, F=F)
    assert np.array_equal(got, oracle.conv2d(codes.astype(np.int32), shift, sign, None, (1, 1), (1, 1)))


@pytest.mark.parametrize("bits", [2, 3, 4, 5])
def test_every_packing(oracle, cuda_device, bits):
    """All field widths, without zero weights, and every right shift of the width."""
    rng = np.random.default_rng(bits)
    x = rng.integers(-32768, 32768, (70, 96, 1, 1)).astype(np.int32)
    shift = -rng.integers(0, 2 ** bits, (48, 96, 1, 1)).astype(np.int32)
    sign = rng.choice([-1, 1], (48, 96, 1, 1)).astype(np.int32)
    shift[0, 0] = -(2 ** bits - 1)
    got = _run(cuda_device, x, shift, sign, None, (1, 1), (0, 0), act_bits=-1, falls_back=False)
    assert np.array_equal(got.reshape(70, 48), oracle.linear(x.reshape(70, 96), shift.reshape(48, 96), sign.reshape(48, 96), None))


def test_sizes_and_refusals(cuda_device):
    from deepshift_b200 import _ffi, kernels, utils
    rng = np.random.default_rng(1)
    shift, sign = weights(rng, (64, 64, 3, 3))
    cw = utils.compress_bits(torch.from_numpy(shift).float(), torch.from_numpy(sign).float(), device=cuda_device)
    geo = (64, 64, 28, 28, 64, 3, 3, 1, 1, 1, 1)
    assert kernels.tc_bytes(geo, cw, kernels._fuse(0, 0, act_bits=-1))[0] > 0
    tiny = (1, 64, 7, 7, 64, 3, 3, 2, 2, 1, 1)
    assert kernels.tc_bytes(tiny, cw, kernels._fuse(0, 0, act_bits=-1))[0] == 0      # too little work
    for f in (kernels._fuse(0, 0, act_bits=16), kernels._fuse(0, 0, act_bits=0), kernels._fuse(3, 0, 5, 12),
              kernels._fuse(2, 0, 16, 16)):   # 24-bit codes: linear layers only
        assert kernels.tc_bytes(geo, cw, f, any_size=True) == (0, 0)
    left = utils.ConcWeight(cw.data, -1, cw.bits)
    assert kernels.tc_bytes(geo, left, kernels._fuse(0, 0, act_bits=-1), any_size=True) == (0, 0)
    f = kernels._fuse(0, 0, act_bits=-1)
    act, wt = kernels.tc_bytes(geo, cw, f)
    buf = torch.empty(max(act, wt), dtype=torch.uint8, device=cuda_device)
    st = torch.cuda.current_stream(cuda_device).cuda_stream
    assert _ffi.lib().ds_tc_expand(cw.data.data_ptr(), *geo, cw.bits, 0, f, buf.data_ptr(), wt - 1, st) == 6
    assert _ffi.lib().ds_tc_expand(cw.data.data_ptr(), *geo, cw.bits, -1, f, buf.data_ptr(), wt, st) == 2
    x = torch.zeros(geo[:4], dtype=torch.int32, device=cuda_device)
    assert _ffi.lib().ds_tc_conv2d(x.data_ptr(), cw.data.data_ptr(), None, x.data_ptr(), *geo, cw.bits, 0, f, buf.data_ptr(),
                                   act - 1, buf.data_ptr(), wt, st) == 6


@pytest.mark.parametrize("geo", [(3, 16, 9, 11, 48, 3, 1, 1, 1), (2, 64, 14, 14, 32, 1, 2, 0, 1), (2, 512, 7, 7, 16, 3, 1, 1, 2),
                                 (5, 32, 8, 8, 144, 3, 2, 1, 1)])
@pytest.mark.parametrize("codes", [True, False])
def test_planes_in_and_out(oracle, cuda_device, geo, codes):
    """Planes packed with a border wider than the padding, read by a convolution that writes the next layer's
    planes; a second convolution reads those.  The border of the second tensor stays as it was filled."""
    from deepshift_b200 import _ffi, kernels, utils
    B, C, H, W, OC, k, s, p, halo = geo
    rng = np.random.default_rng(sum(geo))
    x = acts_wide(rng, (B, C, H, W), 17)
    shift, sign = weights(rng, (OC, C, k, k))
    bias = rng.integers(-2000, 2000, OC).astype(np.int32)
    OH, OW = (H + 2 * p - k) // s + 1, (W + 2 * p - k) // s + 1
    res = rng.integers(-50000, 50000, (B, OC, OH, OW)).astype(np.int32)
    s2, g2 = weights(rng, (20, OC, 3, 3))
    lib, st = _ffi.lib(), torch.cuda.current_stream(cuda_device).cuda_stream
    cw = utils.compress_bits(torch.from_numpy(shift).float(), torch.from_numpy(sign).float(), device=cuda_device)
    cw2 = utils.compress_bits(torch.from_numpy(s2).float(), torch.from_numpy(g2).float(), device=cuda_device)
    xt, bt, rt = (torch.from_numpy(a).to(cuda_device) for a in (x, bias, res))
    src, nxt = kernels.Planes(B, C, H, W, halo, cuda_device), kernels.Planes(B, OC, OH, OW, 1, cuda_device)
    assert lib.ds_planes_pack(xt.data_ptr(), _ffi.IN_I32_CLAMP, 4, 12, src.c, st) == 0
    f = kernels._fuse(_ffi.IN_I32_CLAMP, 0, 4, 12, relu=True, residual=rt, round_f32=True)
    g1 = (B, C, H, W, OC, k, k, s, s, p, p)
    gg2 = (B, OC, OH, OW, 20, 3, 3, 1, 1, 1, 1)
    a1, w1 = kernels.tc_bytes(g1, cw, f, any_size=True)
    a2, w2 = kernels.tc_bytes(gg2, cw2, f, any_size=True)
    act = torch.zeros(max(a1, a2), dtype=torch.uint8, device=cuda_device)
    out = torch.full((B, OC, OH, OW), -7, dtype=torch.int32, device=cuda_device)
    out2 = torch.empty((B, 20, OH, OW), dtype=torch.int32, device=cuda_device)
    e1, e2 = kernels.tc_expand(g1, cw, f, w1, cuda_device), kernels.tc_expand(gg2, cw2, f, w2, cuda_device)
    f2 = kernels._fuse(_ffi.IN_I32_CLAMP, 0, 4, 12)
    for _ in range(2):   # the second pass finds the scratch header as the first left it
        rc = lib.ds_tc_conv2d_ex(None, src.c, cw.data.data_ptr(), bt.data_ptr(), out.data_ptr() if codes else None, nxt.c, *g1,
                                 cw.bits, 0, f, act.data_ptr(), a1, e1.data_ptr(), w1, st)
        assert rc == 0
        rc = lib.ds_tc_conv2d_ex(None, nxt.c, cw2.data.data_ptr(), None, out2.data_ptr(), None, *gg2, cw2.bits, 0, f2,
                                 act.data_ptr(), a2, e2.data_ptr(), w2, st)
        assert rc == 0
    torch.cuda.synchronize(cuda_device)
    assert kernels.last_kernel_error() == 0
    acc = oracle.conv2d(np.clip(x, -32768, 28672), shift, sign, bias, (s, s), (p, p))
    v = np.maximum((acc.astype(np.float32) + res.astype(np.float32)).astype(np.int32), 0)
    if codes:
        assert np.array_equal(out.cpu().numpy(), v)
    else:
        assert bool((out == -7).all())
    assert np.array_equal(out2.cpu().numpy(), oracle.conv2d(np.clip(v, -32768, 28672), s2, g2, None, (1, 1), (1, 1)))
    assert int(act[:2048].sum()) == 0


@pytest.mark.parametrize("mkn", [(17, 128, 10), (64, 784, 512), (128, 2047, 65), (130, 300, 64), (1000, 513, 130)])
@pytest.mark.parametrize("scale", [1.0, 3e4, 1.27e5])
def test_linear_fp32_input_24_bit_codes(oracle, cuda_device, mkn, scale):
    """16.16 codes of up to 24 bits, both ends of the range among them; fp32 output and ReLU."""
    M, K, N = mkn
    rng = np.random.default_rng(M + K + N)
    x = (rng.uniform(-1, 1, (M, K, 1, 1)) * scale / 1e3).astype(np.float32)
    x.flat[::17], x.flat[5::31] = -128.0, np.float32(8388607 / 65536)
    shift, sign = weights(rng, (N, K, 1, 1))
    bias = rng.integers(-2000, 2000, N).astype(np.int32)
    got = _run(cuda_device, x, shift, sign, bias, (1, 1), (0, 0), in_kind=2, act_bits=0, I=16, F=16, relu=True,
               falls_back=False)
    codes = np.trunc(x.astype(np.float64) * 65536).astype(np.int32).reshape(M, K)
    want = np.maximum(oracle.linear(codes, shift.reshape(N, K), sign.reshape(N, K), bias), 0)
    assert np.array_equal(got.reshape(M, N), want)


@pytest.mark.parametrize("what", ["code", "shift"])
def test_linear_fp32_input_falls_back(oracle, cuda_device, what):
    """A code beyond 24 bits, or a right shift of 16..31 somewhere in the weights: the integer path."""
    rng = np.random.default_rng(8)
    M, K, N = 90, 200, 70
    x = rng.normal(0, 1, (M, K, 1, 1)).astype(np.float32)
    shift, sign = weights(rng, (N, K, 1, 1))
    sign[sign == 0] = 1
    sign[0, 0] = 0
    if what == "code":
        x[89, 199] = 128.0
    else:
        shift[69, 199] = -17
    got = _run(cuda_device, x, shift, sign, None, (1, 1), (0, 0), in_kind=2, act_bits=0, I=16, F=16, falls_back=True)
    codes = np.trunc(x.astype(np.float64) * 65536).astype(np.int32).reshape(M, K)
    assert np.array_equal(got.reshape(M, N), oracle.linear(codes, shift.reshape(N, K), sign.reshape(N, K), None))


def test_the_range_flag_belongs_to_the_call(oracle, cuda_device):
    """Threads may enqueue calls on one stream at once, launch by launch in any order; the workspace is the stream's,
    so a flag there would be cleared by one call between the packing and the product of another."""
    from deepshift_b200 import _ffi, kernels, utils
    rng = np.random.default_rng(9)
    M, K, N = 70, 400, 60
    shift, sign = weights(rng, (N, K))
    cw = utils.compress_bits(torch.from_numpy(shift).float(), torch.from_numpy(sign).float(), device=cuda_device)
    geo = (M, K, 1, 1, N, 1, 1, 1, 1, 0, 0)
    ws = torch.full((16384,), 77, dtype=torch.int32, device=cuda_device)
    f = kernels._fuse(_ffi.IN_F32_LINEAR, 0, 16, 16, workspace=ws)
    act, wt = kernels.tc_bytes(geo, cw, f, any_size=True)
    tiles = kernels.tc_expand(geo, cw, f, wt, cuda_device)
    scratch = torch.empty(act, dtype=torch.uint8, device=cuda_device)
    out = torch.empty((M, N), dtype=torch.int32, device=cuda_device)
    for wide in (0, 1):
        x = rng.normal(0, 1, (M, K)).astype(np.float32)
        if wide:
            x[M - 1, K - 1] = 200.0
        xt = torch.from_numpy(x).to(cuda_device)
        assert _ffi.lib().ds_tc_conv2d(xt.data_ptr(), cw.data.data_ptr(), None, out.data_ptr(), *geo, cw.bits, 0, f,
                                       scratch.data_ptr(), act, tiles.data_ptr(), wt,
                                       torch.cuda.current_stream(cuda_device).cuda_stream) == 0
        codes = np.trunc(x.astype(np.float64) * 65536).astype(np.int32)
        assert np.array_equal(out.cpu().numpy(), oracle.linear(codes, shift, sign, None))
        assert int(scratch[:4].view(torch.int32)) == wide
        assert bool((ws == 77).all())


@pytest.mark.parametrize("what", ["fits", "code", "shift"])
@pytest.mark.parametrize("kind", ["linear", "conv", "linear fp32"])
def test_calls_that_expand_their_weights(oracle, cuda_device, kind, what):
    """Weights expanded in the call, which may itself send it to the integer path (24-bit form, a shift of 16..31).  The
    scratch comes filled, as an allocator hands it out."""
    from deepshift_b200 import _ffi, kernels, utils
    rng = np.random.default_rng(3)
    fp32 = kind == "linear fp32"
    B, C, H, OC, k = (3, 40, 9, 70, 3) if kind == "conv" else (90, 400, 1, 70, 1)
    shift, sign = weights(rng, (OC, C, k, k))
    sign.flat[0] = 0
    if what == "shift":
        sign[OC - 1, C - 1], shift[OC - 1, C - 1] = 1, -17
    cw = utils.compress_bits(torch.from_numpy(shift).float(), torch.from_numpy(sign).float(), device=cuda_device)
    geo = (B, C, H, H, OC, k, k, 1, 1, k // 2, k // 2)
    f = kernels._fuse(_ffi.IN_F32_LINEAR, 0, 16, 16) if fp32 else kernels._fuse(act_bits=-1)
    act, wt = kernels.tc_bytes(geo, cw, f, any_size=True)
    scratch = torch.full((act + wt,), 0xA5, dtype=torch.uint8, device=cuda_device)
    out = torch.empty((B, OC, H, H), dtype=torch.int32, device=cuda_device)
    x = rng.normal(0, 1, (B, C, H, H)).astype(np.float32)
    if what == "code":
        x.flat[-1] = 200.0
    codes = np.trunc(x.astype(np.float64) * (65536 if fp32 else 4096)).astype(np.int32)
    xt = torch.from_numpy(x if fp32 else codes).to(cuda_device)
    assert _ffi.lib().ds_tc_conv2d_packed(xt.data_ptr(), cw.data.data_ptr(), None, out.data_ptr(), *geo, cw.bits, 0, f,
                                          scratch.data_ptr(), act, scratch.data_ptr() + act, wt, 0,
                                          torch.cuda.current_stream(cuda_device).cuda_stream) == 0
    assert np.array_equal(out.cpu().numpy(), oracle.conv2d(codes, shift, sign, None, (1, 1), (k // 2, k // 2)))
    assert int(scratch[:4].view(torch.int32)) == int(what == "code" or (fp32 and what == "shift"))


# (M, K, N, weight bits, zeros): rows at the edges of the 80- and 144-column tiles and of two of them, columns at those of
# 128, every packed field width that has a whole kernel of its own, words and groups that K does not fill, K shared
FEW = [(1, 16, 10, 5, True), (17, 300, 127, 5, True), (79, 1000, 128, 4, False), (80, 1024, 129, 3, False),
       (143, 257, 300, 2, False), (144, 100, 31, 6, True), (200, 4096, 130, 5, False), (64, 47, 64, 6, False)]


@pytest.mark.parametrize("case", FEW)
@pytest.mark.parametrize("wide", [False, True])
def test_linear_with_weights_expanded_in_the_kernel(oracle, cuda_device, case, wide):
    """Codes over the whole 16-bit range; one beyond it sends the call to the integer path, found in the scratch's first word."""
    from deepshift_b200 import _ffi, kernels, utils
    M, K, N, wb, zeros = case
    rng = np.random.default_rng(M + K + N)
    x = rng.integers(-32768, 32768, (M, K)).astype(np.int32)
    x.flat[::7] = -32768
    x.flat[3::11] = 32767
    if wide:
        x[M - 1, K - 1] = -32769
    shift = rng.integers(-(2 ** (wb - 1) - 1), 1, (N, K)).astype(np.int32)
    shift[0, 0] = -(2 ** (wb - 1) - 1)   # the widest field of this case
    sign = rng.choice([-1, 0, 1] if zeros else [-1, 1], (N, K)).astype(np.int32)
    bias = rng.integers(-2000, 2000, N).astype(np.int32)
    cw = utils.compress_bits(torch.from_numpy(shift).float(), torch.from_numpy(sign).float(), device=cuda_device)
    f = kernels._fuse(act_bits=-1)
    n = ctypes.c_longlong(0)
    assert _ffi.lib().ds_tc_few_bytes(M, K, N, cw.bits, cw.base, f, 1, ctypes.byref(n)) == 0 and n.value > 0
    xt, bt = torch.from_numpy(x).to(cuda_device), torch.from_numpy(bias).to(cuda_device)
    act = torch.full((n.value + 64,), 0xA5, dtype=torch.uint8, device=cuda_device)
    out = torch.full((M * N + 16,), 0x5EADBEE, dtype=torch.int32, device=cuda_device)
    rc = _ffi.lib().ds_tc_linear_few(xt.data_ptr(), cw.data.data_ptr(), bt.data_ptr(), out.data_ptr(), M, K, N, cw.bits, cw.base,
                                     f, act.data_ptr(), n.value, torch.cuda.current_stream(cuda_device).cuda_stream)
    torch.cuda.synchronize(cuda_device)
    assert rc == 0 and kernels.last_kernel_error() == 0
    assert bool((act[n.value:] == 0xA5).all()) and bool((out[-16:] == 0x5EADBEE).all())
    assert int(act[:4].view(torch.int32)) == int(wide)
    assert np.array_equal(out[:-16].reshape(M, N).cpu().numpy(), oracle.linear(x, shift, sign, bias))


def test_which_linear_calls_expand_their_weights_in_the_kernel(cuda_device):
    from deepshift_b200 import kernels
    assert kernels._few_bytes(64, 4096, 4096, 6, -1) > 0 and kernels._few_bytes(64, 4096, 4096, 6, 15) > 0
    assert kernels._few_bytes(16, 4096, 4096, 6, -1) == 0 and kernels._few_bytes(8192, 4096, 4096, 6, -1) == 0
    assert kernels._few_bytes(64, 4096, 4096, 6, 0) == 0 and kernels._few_bytes(64, 4096, 4096, 6, 16) == 0   # other promises
