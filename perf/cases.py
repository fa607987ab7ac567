"""The work a user of this package has it do, as cases that can be timed: whole networks through the
integer pipeline and through the drop-in modules, single layers through the operator API, and the
packing of a layer's weights.  Sizes are those of the benchmark networks and of the shift-GEMM /
shift-convolution sweep, plus ragged ones.  Every result is an integer code or an integer code
divided by a power of two, so all comparisons are exact."""
import math

import torch

from deepshift_b200 import kernels, modules, utils, workloads


def listed():
    return [
        # Serving: ImageNet-shape ResNet-18, the benchmark's batch, one captured forward pass per batch.
        dict(name="resnet18_b256_pipeline", kind="pipeline", net="resnet18", batch=256),
        # The same network as an nn.Module in a user's own evaluation loop, fused glue, a smaller batch.
        dict(name="resnet18_b64_modules", kind="modules", net="resnet18", batch=64, fuse=True),
        # One image at a time: the latency a single request sees.
        dict(name="resnet18_b1_pipeline", kind="pipeline", net="resnet18", batch=1),
        # CIFAR-shape network with few channels (16/32/64), large batch.
        dict(name="resnet20_b4096_pipeline", kind="pipeline", net="resnet20", batch=4096),
        # MNIST convolution network as drop-in modules with torch's own glue: 5x5 windows, odd channel
        # counts (1, 20, 50), unclamped linear layers.
        dict(name="mnist_conv_b1024_modules", kind="modules", net="mnist_conv", batch=1024, fuse=False),
        # The smallest network of all: three linear layers, a test loop's batch; launches and host work count.
        dict(name="mnist_fc_b64_modules", kind="modules", net="mnist_fc", batch=64, fuse=False),
        # Shift-GEMM through the reference's operator signature: one row (decode-like, the weights are the traffic),
        dict(name="gemm_m1_k4096_n4096", kind="gemm", M=1, K=4096, N=4096, weight_bits=5, zeros=True),
        # a small batch,
        dict(name="gemm_m64_k4096_n4096", kind="gemm", M=64, K=4096, N=4096, weight_bits=5, zeros=True),
        # and a large one.
        dict(name="gemm_m8192_k4096_n4096", kind="gemm", M=8192, K=4096, N=4096, weight_bits=5, zeros=True),
        # Shift-convolution through the operator signature at sizes nothing is a multiple of anything,
        # 3-bit weights without zeros.
        dict(name="conv3x3s2_b37_c45_31x29_o70", kind="conv", B=37, C=45, H=31, W=29, O=70, k=3, stride=2, pad=1,
             weight_bits=3, zeros=False),
        # A classifier layer as a module with the default 16.16 activations (32-bit codes), ragged sizes.
        dict(name="linear_shift_m1000_k2047_n1001", kind="linear_shift", M=1000, K=2047, N=1001, I=16, F=16,
             weight_bits=5),
        # Packing a layer's (shift, sign) parameters, as every load or change of weights does.
        dict(name="pack_n4096_k4096", kind="pack", O=4096, C=4096, k=1, weight_bits=5, zeros=True),
    ]


def _log(rng, lo, hi):
    """An integer between lo and hi, spread over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def draw(rng):
    kind = rng.choice(["pipeline", "modules", "gemm", "gemm", "conv", "conv", "linear_shift", "pack"])
    if kind in ("pipeline", "modules"):
        net = rng.choice(["resnet18", "resnet20", "mnist_conv", "mnist_fc"])
        most = {"resnet18": 256, "resnet20": 4096, "mnist_conv": 4096, "mnist_fc": 8192}[net]
        if kind == "pipeline":
            return dict(kind=kind, net=net, batch=_log(rng, 1, most))
        return dict(kind=kind, net=net, batch=_log(rng, 1, most // 2), fuse=rng.random() < 0.5)
    bits = rng.choice([2, 3, 4, 5, 5])
    zeros = rng.random() < 0.6
    if kind == "gemm":
        return dict(kind=kind, M=_log(rng, 1, 8192), K=_log(rng, 256, 4096), N=_log(rng, 256, 4096), weight_bits=bits,
                    zeros=zeros)
    if kind == "conv":
        while True:
            k = rng.choice([1, 3, 3, 3, 5, 7])
            hw = _log(rng, 7, 112)
            c = dict(kind=kind, B=_log(rng, 1, 256), C=_log(rng, 3, 512), H=hw, W=max(7, hw - rng.choice([0, 0, 0, 1, 3])),
                     O=_log(rng, 16, 512), k=k, stride=rng.choice([1, 1, 2]), pad=rng.choice([k // 2, k // 2, 0]),
                     weight_bits=bits, zeros=zeros)
            if work(c)["flops"] <= 3e11 and c["B"] * max(c["C"], c["O"]) * hw * hw <= 1 << 28:
                return c
    if kind == "linear_shift":
        I, F = rng.choice([(16, 16), (4, 12), (8, 8)])
        return dict(kind=kind, M=_log(rng, 1, 4096), K=_log(rng, 64, 4096), N=_log(rng, 10, 4096), I=I, F=F,
                    weight_bits=bits)
    return dict(kind=kind, O=_log(rng, 16, 4096), C=_log(rng, 16, 4096), k=1, weight_bits=bits, zeros=zeros)


# ------------------------------------------------------------------------------------------------ inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _weights(g, shape, weight_bits, zeros):
    """(shift, sign) int32: shift uniform in [-(2^(b-1)-1), 0], sign -1/0/+1 with P = 0.45/0.10/0.45
    (-1/+1 when the layer has no zero weights)."""
    shift = torch.randint(-(2 ** (weight_bits - 1) - 1), 1, shape, generator=g, device="cuda", dtype=torch.int32)
    u = torch.rand(shape, generator=g, device="cuda")
    sign = torch.where(u < 0.5, -1, 1).to(torch.int32)
    if zeros:
        sign[(u >= 0.45) & (u < 0.55)] = 0
    return shift, sign


def _codes(g, shape):
    """N(0,1) activations as 4.12 fixed-point codes."""
    x = utils.round_to_fixed(torch.randn(shape, generator=g, device="cuda"), 4, 12)
    return (x * 4096).to(torch.int32)


def _bias_codes(g, n):
    return (torch.randn(n, generator=g, device="cuda") * 0.01 * 4096).to(torch.int32)


def _net_state(case, seed):
    g = _generator(seed)
    net = workloads.NETS[case["net"]]()
    ws = []
    for L in net.layers:
        shift, sign = _weights(g, L.weight_shape, net.weight_bits, True)
        bias = torch.randn(L.cout, generator=g, device="cuda") * 0.01
        ws.append(dict(shift=shift, sign=sign,
                       bias=utils.round_to_fixed(bias, net.act_integer_bits, net.act_fraction_bits)))
    shape = (case["batch"],) + net.in_shape
    if case["net"].startswith("mnist"):
        x = (torch.rand(shape, generator=g, device="cuda") - 0.1307) / 0.3081
    else:
        x = torch.randn(shape, generator=g, device="cuda")
    x = utils.round_to_fixed(x, net.act_integer_bits, net.act_fraction_bits)
    if case["kind"] == "pipeline":
        return dict(kind="pipeline", net=workloads.IntPipeline(net, ws, case["batch"]), x=x)
    return dict(kind="modules", net=workloads.ModuleNet(net, ws, fuse=case["fuse"]).eval(), x=x)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("pipeline", "modules"):
        return _net_state(case, seed)
    g = _generator(seed)
    if kind == "gemm":
        shift, sign = _weights(g, (case["N"], case["K"]), case["weight_bits"], case["zeros"])
        return dict(kind=kind, x=_codes(g, (case["M"], case["K"])), shift=shift, sign=sign, bias=_bias_codes(g, case["N"]),
                    packed=utils.compress_bits(shift.float(), sign.float()))
    if kind == "conv":
        shift, sign = _weights(g, (case["O"], case["C"], case["k"], case["k"]), case["weight_bits"], case["zeros"])
        return dict(kind=kind, x=_codes(g, (case["B"], case["C"], case["H"], case["W"])), shift=shift, sign=sign,
                    bias=_bias_codes(g, case["O"]), packed=utils.compress_bits(shift.float(), sign.float()),
                    stride=case["stride"], pad=case["pad"])
    if kind == "linear_shift":
        shift, sign = _weights(g, (case["N"], case["K"]), case["weight_bits"], True)
        m = modules.LinearShift(case["K"], case["N"], use_kernel=True, weight_bits=case["weight_bits"],
                                act_integer_bits=case["I"], act_fraction_bits=case["F"]).cuda().eval()
        m.shift.data, m.sign.data = shift.float(), sign.float()
        m.bias.data = torch.randn(case["N"], generator=g, device="cuda") * 0.01
        m.conc_weight = utils.compress_bits(m.shift.data, m.sign.data)
        return dict(kind=kind, net=m, x=torch.randn(case["M"], case["K"], generator=g, device="cuda"))
    shift, sign = _weights(g, (case["O"], case["C"], case["k"], case["k"]), case["weight_bits"], case["zeros"])
    return dict(kind=kind, shift=shift.float(), sign=sign.float())


def run(state):
    kind = state["kind"]
    if kind == "pipeline":
        return state["net"].run(state["x"])
    if kind in ("modules", "linear_shift"):
        with torch.no_grad():
            return state["net"](state["x"])
    if kind == "gemm":
        return kernels.linear(state["x"], state["shift"], state["sign"], state["bias"], state["packed"])
    if kind == "conv":
        return kernels.conv2d(state["x"], state["shift"], state["sign"], state["bias"], state["packed"], state["stride"],
                              state["pad"])
    cw = utils.compress_bits(state["shift"], state["sign"])
    return dict(data=cw.data, base=cw.base, bits=cw.bits)


def _field_bits(case):
    """Width of the packed shift field: 6 when a weight may be zero (encoded as a right shift by 32)."""
    return 6 if case.get("zeros", True) else case["weight_bits"] - 1


def _packed_bytes(rows, K, bits):
    return 4 * rows * math.ceil(K / (32 // (bits + 1)))


def work(case):
    """Inputs and packed weights read once, outputs written once; a shift-accumulate counts as two operations."""
    kind = case["kind"]
    if kind in ("pipeline", "modules"):
        net = workloads.NETS[case["net"]]()
        B = case["batch"]
        weights = sum(_packed_bytes(L.cout, math.prod(L.weight_shape[1:]), 6) + 4 * L.cout for L in net.layers)
        return dict(bytes=4 * B * (math.prod(net.in_shape) + net.layers[-1].cout) + weights, flops=2 * net.shift_ops(B))
    if kind in ("gemm", "linear_shift"):
        M, K, N = case["M"], case["K"], case["N"]
        return dict(bytes=4 * (M * K + N + M * N) + _packed_bytes(N, K, _field_bits(case)), flops=2 * M * K * N)
    if kind == "conv":
        k, s, p = case["k"], case["stride"], case["pad"]
        oh, ow = (case["H"] + 2 * p - k) // s + 1, (case["W"] + 2 * p - k) // s + 1
        K = case["C"] * k * k
        out = case["B"] * case["O"] * oh * ow
        return dict(bytes=4 * (case["B"] * case["C"] * case["H"] * case["W"] + case["O"] + out) +
                    _packed_bytes(case["O"], K, _field_bits(case)), flops=2 * out * K)
    K = case["C"] * case["k"] ** 2
    return dict(bytes=8 * case["O"] * K + _packed_bytes(case["O"], K, _field_bits(case)), flops=4 * case["O"] * K)


def tolerance(case):
    return "exact"
