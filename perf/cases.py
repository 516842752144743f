"""The work whose speed counts: what a program that uses this framework has it do, through the public entry points of
``tab_b200`` - ``Quantize`` and ``Conv2d`` (the reference's two operators, all four types), the prepared convolution
``nn.TABConv2d`` and the ResNet-18-shaped network ``chain.forward_prepared``.  Inference only: no path has a backward.

``listed()`` are fixed cases, ``draw(rng)`` gives another one of the same ranges.  A case is a dict:

    path     "quantize" | "conv" | "module" | "chain"
    N H W C  activations, fp32 NHWC (for "quantize" also weights, whose N is the filter count)
    bits     quantize: 2 ternary, 1 binary
    type     conv, module, chain: 0 TNN, 1 TBN, 2 BTN, 3 BNN
    KN K stride pad      conv, module: filters, square kernel, both strides, both paddings

Values are N(0,1) and thresholds 0.7 * mean|.| per image and per filter, as everywhere in this repository.
"""
import math

import torch

import tab_b200 as TAB
from tab_b200 import chain, nn as tab_nn

SCALE = 0.7


def listed():
    return [
        # One image through one small layer: the call's latency (the reference's CPU-runnable configuration).
        {"name": "conv_tnn_n1_32x32x64", "path": "conv", "type": 0, "N": 1, "H": 32, "W": 32, "C": 64, "KN": 64, "K": 3, "stride": 1, "pad": 1},
        # One image through a deep layer of a loaded model, thresholds found by the module: latency of interactive inference.
        {"name": "module_bnn_n1_7x7x512", "path": "module", "type": 3, "N": 1, "H": 7, "W": 7, "C": 512, "KN": 512, "K": 3, "stride": 1, "pad": 1},
        # Ragged everything: odd image, channels and filters that fill no word and no tile, a 5x5 kernel.
        {"name": "conv_tbn_ragged_45x37x70", "path": "conv", "type": 1, "N": 9, "H": 45, "W": 37, "C": 70, "KN": 130, "K": 5, "stride": 1, "pad": 2},
        # Binary quantisation of a batch whose channel count is no multiple of 64.
        {"name": "quantize_bin_n64_27x31x200", "path": "quantize", "bits": 1, "N": 64, "H": 27, "W": 31, "C": 200},
        # The standalone quantiser on a large batch: the memory-bound end.
        {"name": "quantize_ter_n256_56x56x256", "path": "quantize", "bits": 2, "N": 256, "H": 56, "W": 56, "C": 256},
        # A batch through the widest images of a ResNet-18, binary network.
        {"name": "conv_bnn_n64_56x56x64", "path": "conv", "type": 3, "N": 64, "H": 56, "W": 56, "C": 64, "KN": 64, "K": 3, "stride": 1, "pad": 1},
        # A batch through a downsampling layer, ternary activations and binary weights.
        {"name": "conv_tbn_s2_n64_28x28x128", "path": "conv", "type": 1, "N": 64, "H": 28, "W": 28, "C": 128, "KN": 256, "K": 3, "stride": 2, "pad": 1},
        # The large 1x1 convolution, a plain matrix product: 25088 x 1024 x 1024.
        {"name": "conv_tnn_1x1_n128_14x14x1024", "path": "conv", "type": 0, "N": 128, "H": 14, "W": 14, "C": 1024, "KN": 1024, "K": 1, "stride": 1, "pad": 0},
        # The largest problem of the reference's demonstration notebook, binary activations and ternary weights.
        {"name": "conv_btn_n16_112x112x256", "path": "conv", "type": 2, "N": 16, "H": 112, "W": 112, "C": 256, "KN": 64, "K": 3, "stride": 1, "pad": 1},
        # A batch through one prepared layer in the middle of a ResNet-18.
        {"name": "module_tnn_n64_14x14x256", "path": "module", "type": 0, "N": 64, "H": 14, "W": 14, "C": 256, "KN": 256, "K": 3, "stride": 1, "pad": 1},
        # The whole network on a serving batch: 19 convolutions, launches and host work count.
        {"name": "chain_tnn_n8", "path": "chain", "type": 0, "N": 8, "H": 56, "W": 56, "C": 64},
        # The whole network on the benchmark's batch.
        {"name": "chain_tnn_n256", "path": "chain", "type": 0, "N": 256, "H": 56, "W": 56, "C": 64},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _channels(rng, lo, hi):
    """Half of the time a whole number of 64-channel words, else any count."""
    c = _log_int(rng, lo, hi)
    return max(64, (c + 32) // 64 * 64) if rng.random() < 0.5 else c


def draw(rng):
    path = rng.choice(["quantize", "conv", "conv", "conv", "module", "module", "chain"])
    if path == "chain":
        return {"path": path, "type": rng.randrange(4), "N": _log_int(rng, 1, 128), "H": rng.randint(32, 64), "W": rng.randint(32, 64), "C": 64}
    while True:
        case = {"path": path}
        if path == "quantize":
            case["bits"] = rng.choice([1, 2])
        else:
            case["type"] = rng.randrange(4)
        case["N"] = _log_int(rng, 1, 256)
        case["H"] = _log_int(rng, 7, 224)
        case["W"] = case["H"] if rng.random() < 0.5 else _log_int(rng, 7, 224)
        case["C"] = _channels(rng, 3, 1024)
        if path == "quantize":
            if 4 * case["N"] * case["H"] * case["W"] * case["C"] <= 800e6:
                return case
            continue
        case["KN"] = _channels(rng, 16, 1024)
        case["K"] = rng.choice([1, 3, 3, 3, 5, 7])
        case["stride"] = rng.choice([1, 1, 2])
        case["pad"] = rng.choice([0, case["K"] // 2, case["K"] // 2])
        if case["K"] > min(case["H"], case["W"]):
            continue
        w = work(case)
        if w["bytes"] <= 300e6 and w["flops"] <= 60e9:
            return case


def _thresholds(t):
    return (SCALE * t.abs().reshape(t.shape[0], -1).mean(dim=1)).contiguous()


def _out_size(case):
    return tuple((case[d] + 2 * case["pad"] - case["K"] + 1) // case["stride"] for d in "HW")


def prepare(case, seed):
    """Activations and, for a convolution, what a program keeps of its weights: packed words, or a prepared module."""
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    N, H, W, C = (case[k] for k in "NHWC")
    state = {"case": case, "x": torch.randn(N, H, W, C, device=dev, generator=gen)}
    if case["path"] in ("quantize", "conv"):
        state["ths"] = _thresholds(state["x"])
    if case["path"] == "conv":
        KN, K = case["KN"], case["K"]
        w = torch.randn(KN, K, K, C, device=dev, generator=gen)
        state["QW"], state["btn"] = TAB.Quantize(w, _thresholds(w), tab_nn.weight_bitwidth(case["type"]), KN, K, K, C)
    elif case["path"] == "module":
        w = torch.randn(case["KN"], case["K"], case["K"], C, device=dev, generator=gen)
        state["conv"] = tab_nn.TABConv2d.from_float(w, case["type"], case["pad"], case["stride"], threshold_scale=SCALE)
    elif case["path"] == "chain":
        state["convs"] = {}
        for cs in chain.conv_specs():
            w = torch.randn(cs.KN, cs.K, cs.K, cs.C, device=dev, generator=gen)
            state["convs"][cs.name] = tab_nn.TABConv2d.from_float(w, case["type"], cs.pad, cs.stride, threshold_scale=SCALE)
    return state


def run(state):
    case, x = state["case"], state["x"]
    N, H, W, C = (case[k] for k in "NHWC")
    if case["path"] == "quantize":
        return TAB.Quantize(x, state["ths"], case["bits"], N, H, W, C)
    if case["path"] == "conv":
        p, s, K = case["pad"], case["stride"], case["K"]
        return TAB.Conv2d(x, state["QW"], state["ths"], state["btn"], case["type"], p, p, s, s, N, H, W, C, case["KN"], K, K)
    if case["path"] == "module":
        return state["conv"](x)
    convs = state["convs"]
    qx, ths = convs[chain.resnet18_blocks()[0].conv_a.name].quantize_auto(x)
    return chain.forward_prepared(convs, x, ths, N, H, W, compact_mid=True, fused_quant=True, qx0=qx)[0]


def work(case):
    """Inputs read once and outputs written once, weights as packed words; an operation is a multiply or an add."""
    N, H, W, C = (case[k] for k in "NHWC")
    words = (C + 63) // 64
    if case["path"] == "quantize":
        return {"bytes": 4 * N * H * W * C + 8 * N * H * W * words * case["bits"] + 8 * N, "flops": 2 * N * H * W * C}
    wbits = tab_nn.weight_bitwidth(case["type"])
    if case["path"] == "chain":
        h, w = H, W
        for _ in range(3):
            h, w = h // 2, w // 2
        wbytes = sum(8 * cs.KN * cs.K * cs.K * (cs.C // 64) * wbits for cs in chain.conv_specs())
        return {"bytes": 4 * N * H * W * C + wbytes + 4 * N * h * w * 512, "flops": chain.chain_binary_ops(N, H, W)}
    OH, OW = _out_size(case)
    taps = case["K"] * case["K"]
    return {"bytes": 4 * N * H * W * C + 8 * case["KN"] * taps * words * wbits + 4 * N * OH * OW * case["KN"],
            "flops": 2 * N * OH * OW * case["KN"] * taps * C}


def tolerance(case):
    """Bit-planes are bytes and every convolution result is a whole number (in the network, a whole number plus one fp32
    addition per value); thresholds come from sums in double precision, whose order does not show in the rounded result."""
    return "exact"
