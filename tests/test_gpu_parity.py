"""Parity of the CUDA path, called through the C ABI, with the CPU oracle: bit-exact (integer-valued
results; the comparison is array equality, tolerance 0)."""
import glob
import os

import numpy as np
import pytest
import torch

import tab_b200 as TAB
from tab_b200 import _cabi, chain, nn as tab_nn
from oracle import c_oracle, tab_oracle as O
from oracle.oracle_ops import OracleOps
from util import make_input

pytestmark = pytest.mark.gpu
GOLD = os.path.join(os.path.dirname(__file__), "golden")
NAMES = ["tnn", "tbn", "btn", "bnn"]


@pytest.fixture(autouse=True, params=["tensor", "popcount", "popcount-plain"])
def conv_path(request):
    """Every test of this module runs once per compute path of the convolution entry points: the persistent tcgen05
    kernel (shapes it does not cover fall back to the popcount kernel inside the call), the bit-packed popcount
    kernel with its carry-save tree, and the same with one POPC per word.  After each test the tensor-core kernel's
    record of expired waits must be clean."""
    l = _cabi.lib()
    prev = l.tab_conv2d_set_path({"tensor": 0, "popcount": 1, "popcount-plain": 2}[request.param])
    yield request.param
    l.tab_conv2d_set_path(prev)
    torch.cuda.synchronize()
    assert l.tab_device_status() == 0


def dev_t(a, cuda):
    return torch.from_numpy(np.ascontiguousarray(a)).to(cuda)


def gpu_conv(cuda, x, qw, ths, btn, t, p1, p2, s1, s2, N, H, W, C, KN, KH, KW):
    y = TAB.Conv2d(dev_t(x, cuda), dev_t(qw, cuda), dev_t(ths, cuda), dev_t(btn, cuda), t, p1, p2, s1, s2, N, H, W, C, KN, KH, KW)
    return y.cpu().numpy()


# ------------------------------------------------------------------------------------------ quantise

@pytest.mark.parametrize("bw", [2, 1])
@pytest.mark.parametrize("C", [3, 64, 65, 128, 200, 256])
@pytest.mark.parametrize("N,H,W", [(1, 1, 1), (3, 5, 7), (16, 9, 4)])
def test_quantize_matches_oracle(cuda, bw, C, N, H, W):
    x, ths = make_input(C * 7 + N, N, H, W, C)
    q, b = TAB.Quantize(dev_t(x, cuda), dev_t(ths, cuda), bw, N, H, W, C)
    qo, bo = O.quantize(x, ths, bw, N, H, W, C)
    assert q.dtype == torch.int64 and tuple(q.shape) == qo.shape and b.dtype == torch.int32
    assert np.array_equal(q.cpu().numpy(), qo) and np.array_equal(b.cpu().numpy(), bo)


def test_quantize_edge_values_golden(cuda):
    g = np.load(os.path.join(GOLD, "quantize_edges.npz"))
    x, ths = g["x"], g["ths"]
    N, H, W, C = x.shape
    for bw, qk, bk in ((2, "q2", "btn2"), (1, "q1", "btn1")):
        q, b = TAB.Quantize(dev_t(x, cuda), dev_t(ths, cuda), bw, N, H, W, C)
        assert np.array_equal(q.cpu().numpy(), g[qk]) and np.array_equal(b.cpu().numpy(), g[bk])
    # the same edge values through the vectorised path (C = 128)
    x2 = np.zeros((1, 2, 2, 128), np.float32)
    x2[0, 0, 0, :8] = x[0, 0, 0, :8]
    x2[0, 1, 1, 120:128] = x[0, 0, 0, :8]
    t2 = np.array([0.5], np.float32)
    for bw in (2, 1):
        q, b = TAB.Quantize(dev_t(x2, cuda), dev_t(t2, cuda), bw, 1, 2, 2, 128)
        qo, bo = O.quantize(x2, t2, bw, 1, 2, 2, 128)
        assert np.array_equal(q.cpu().numpy(), qo) and np.array_equal(b.cpu().numpy(), bo)


def test_quantize_empty_and_unaligned(cuda):
    q, b = TAB.Quantize(torch.empty(0, device=cuda), torch.empty(0, device=cuda), 2, 0, 4, 4, 64)
    assert tuple(q.shape) == (0, 4, 4, 1, 2) and tuple(b.shape) == (0,)
    q, b = TAB.Quantize(torch.empty(0, device=cuda), torch.zeros(3, device=cuda), 2, 3, 0, 4, 64)
    assert tuple(q.shape) == (3, 0, 4, 1, 2) and not b.cpu().numpy().any()
    # input that starts 4 bytes past a 16-byte boundary: the scalar path must take over
    N, H, W, C = 2, 3, 5, 64
    x, ths = make_input(9, N, H, W, C)
    buf = torch.zeros(x.size + 1, device=cuda)
    buf[1:] = dev_t(x.reshape(-1), cuda)
    q, b = TAB.Quantize(buf[1:], dev_t(ths, cuda), 2, N, H, W, C)
    qo, bo = O.quantize(x, ths, 2, N, H, W, C)
    assert np.array_equal(q.cpu().numpy(), qo) and np.array_equal(b.cpu().numpy(), bo)


def test_notebook_facts_on_device(cuda):
    g = torch.Generator(device=cuda)
    g.manual_seed(11)
    w = torch.rand(64, 3, 3, 256, device=cuda, generator=g)
    t = 0.7 * w.reshape(64, -1).mean(dim=1)
    # a value equal to its threshold is neither "< t" nor "> t": the complement relation below holds for all other values
    w = torch.where(w == t.reshape(64, 1, 1, 1), w + 0.25, w)
    q2, b2 = TAB.Quantize(w, t, 2, 64, 3, 3, 256)
    q1, b1 = TAB.Quantize(w, t, 1, 64, 3, 3, 256)
    assert tuple(q2.shape) == (64, 3, 3, 4, 2) and q2.dtype == torch.int64 and tuple(b2.shape) == (64,)
    assert not q2[..., 0].any().item()
    assert torch.equal(q1[..., 0], ~q2[..., 1])
    assert not b1.any().item()


@pytest.mark.parametrize("bw", [2, 1])
def test_quantize_full_size_configuration(cuda, bw):
    """N=256, 56x56x256 (822 MB): two images against the oracle, and the BTN_W counts against a popcount
    of the device's own magnitude plane (a checksum over everything that was written)."""
    N, H, W, C = 256, 56, 56, 256
    g = torch.Generator(device=cuda)
    g.manual_seed(1)
    x = torch.randn(N, H, W, C, device=cuda, generator=g)
    ths = (0.7 * x.abs().mean(dim=(1, 2, 3))).contiguous()
    q, b = TAB.Quantize(x, ths, bw, N, H, W, C)
    th = ths.cpu().numpy()
    for n in (0, 131, N - 1):
        qo, bo = c_oracle.quantize(x[n].cpu().numpy(), th[n:n + 1], bw, 1, H, W, C)
        assert np.array_equal(q[n].cpu().numpy(), qo[0])
        assert int(b[n].item()) == int(bo[0])
    if bw == 2:
        lut = torch.tensor([bin(i).count("1") for i in range(256)], dtype=torch.int32, device=cuda)
        mag_bytes = q[..., 1].contiguous().view(torch.uint8).reshape(N, -1)
        counts = lut[mag_bytes.long()].sum(dim=1, dtype=torch.int64)
        assert torch.equal(counts, b.long())
        assert not (q[..., 0] & ~q[..., 1]).any().item()      # a sign bit never without its magnitude bit
    else:
        assert not b.any().item()


# ------------------------------------------------------------------------------------------ convolution

def test_conv_cfg1_golden(cuda):
    g = np.load(os.path.join(GOLD, "conv_cfg1_tnn.npz"))
    p1, p2, s1, s2, N, H, W, C, KN, KH, KW = (int(v) for v in g["geom"])
    qw, btn = TAB.Quantize(dev_t(g["w"], cuda), dev_t(g["wths"], cuda), 2, KN, KH, KW, C)
    assert np.array_equal(qw.cpu().numpy(), g["qw"]) and np.array_equal(btn.cpu().numpy(), g["btn"])
    y = TAB.Conv2d(dev_t(g["x"], cuda), qw, dev_t(g["ths"], cuda), btn, 0, p1, p2, s1, s2, N, H, W, C, KN, KH, KW)
    assert tuple(y.shape) == (1, 64, 32, 32) and y.dtype == torch.float32
    assert np.array_equal(y.cpu().numpy(), g["y"].astype(np.float32))


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(GOLD, "conv_small_*.npz"))))
def test_conv_small_golden(cuda, path):
    g = np.load(path)
    geom = [int(v) for v in g["geom"]]
    for t, name in enumerate(NAMES):
        y = gpu_conv(cuda, g["x"], g["qw_" + name], g["ths"], g["btn_" + name], t, *geom)
        assert np.array_equal(y, g["y_" + name].astype(np.float32)), name


@pytest.mark.parametrize("t", range(4))
@pytest.mark.parametrize("K,p", [(1, 0), (1, 1), (3, 0), (3, 1)])
@pytest.mark.parametrize("s", [1, 2])
def test_conv_grid(cuda, t, K, p, s):
    """types x {1x1,3x3} x stride x pad, over channel counts with and without a tail word and batch sizes."""
    for C in (3, 64, 65, 128, 200, 256):
        for N, H, W, KN in ((1, 6, 6, 4), (3, 9, 5, 70)):
            x, ths = make_input(C + N, N, H, W, C)
            w, wths = make_input(C + N + 1, KN, K, K, C)
            qw, btn = O.quantize(w, wths, O.weight_bits(t), KN, K, K, C)
            y = gpu_conv(cuda, x, qw, ths, btn, t, p, p, s, s, N, H, W, C, KN, K, K)
            yo = c_oracle.conv2d(x, qw, ths, btn, t, p, p, s, s, N, H, W, C, KN, K, K)
            assert y.shape == yo.shape and np.array_equal(y, yo), (C, N, H, W, KN)


@pytest.mark.parametrize("t", range(4))
@pytest.mark.parametrize("geom", [
    # p1 p2 s1 s2  N   H   W    C   KN KH KW
    (2, 2, 1, 1, 2, 12, 12, 128, 130, 5, 5),
    (3, 3, 2, 2, 1, 15, 13, 64, 20, 7, 7),
    (1, 2, 3, 2, 2, 10, 7, 200, 6, 3, 5),       # non-square everything; stride does not divide
    (0, 0, 1, 1, 1, 2, 2, 64, 8, 3, 3),         # kernel larger than image: empty output
    (1, 1, 1, 1, 5, 13, 11, 64, 257, 3, 3),     # M and KN not multiples of the CTA tile
    (0, 0, 1, 1, 2, 3, 3, 1024, 1024, 1, 1),    # KN = 1024 (impossible on the reference launch shape)
    (1, 1, 1, 1, 1, 4, 4, 4608, 3, 3, 3),       # 72 words per tap
    (0, 0, 2, 3, 2, 11, 10, 128, 70, 1, 1),     # strided 1x1 without padding: only the pixels it reads are quantised
    (0, 0, 2, 2, 3, 14, 14, 256, 512, 1, 1),
    (0, 0, 1, 1, 2, 9, 9, 64, 64, 2, 2),        # 2x2 taps, no padding
])
def test_conv_shapes(cuda, t, geom):
    p1, p2, s1, s2, N, H, W, C, KN, KH, KW = geom
    x, ths = make_input(31, N, H, W, C)
    w, wths = make_input(32, KN, KH, KW, C)
    qw, btn = O.quantize(w, wths, O.weight_bits(t), KN, KH, KW, C)
    y = gpu_conv(cuda, x, qw, ths, btn, t, *geom)
    yo = c_oracle.conv2d(x, qw, ths, btn, t, *geom)
    assert y.shape == yo.shape and np.array_equal(y, yo)
    yd = O.conv2d_dense(x, qw, ths, t, *geom) if N * H * W * C * KN < 4e7 else yo
    assert np.array_equal(y, yd)


@pytest.mark.parametrize("t", range(4))
def test_selected_path_is_the_one_that_runs(cuda, t, conv_path):
    """The path setting is honoured: the tensor-core kernel reports its tile, the popcount paths report none."""
    N, H, W, C, KN = 4, 14, 14, 256, 96
    x, ths = make_input(5, N, H, W, C)
    w, wths = make_input(6, KN, 3, 3, C)
    qw, btn = O.quantize(w, wths, O.weight_bits(t), KN, 3, 3, C)
    y = gpu_conv(cuda, x, qw, ths, btn, t, 1, 1, 1, 1, N, H, W, C, KN, 3, 3)
    name = _cabi.lib().tab_last_conv_kernel().decode()
    assert name.startswith("conv_umma_persist_kernel<") if conv_path == "tensor" else name == "none"
    assert np.array_equal(y, c_oracle.conv2d(x, qw, ths, btn, t, 1, 1, 1, 1, N, H, W, C, KN, 3, 3))


RESNET_LAYERS = [
    # H   C   KN  K s p
    (56, 64, 64, 3, 1, 1), (28, 128, 128, 3, 1, 1), (14, 256, 256, 3, 1, 1), (7, 512, 512, 3, 1, 1),
    (56, 64, 128, 3, 2, 1), (28, 128, 256, 3, 2, 1), (14, 256, 512, 3, 2, 1),
]


@pytest.mark.parametrize("t", range(4))
@pytest.mark.parametrize("layer", RESNET_LAYERS)
def test_resnet_layers_full_batch_sampled_images(cuda, t, layer):
    """The N=64 ResNet-18-shaped layers at full size on the device; the oracle checks images 0, 37 and 63
    (every image is independent, so a sample of images is an exact check of those outputs)."""
    H, C, KN, K, s, p = layer
    N = 64
    g = torch.Generator(device=cuda)
    g.manual_seed(H * 1000 + C + t)
    x = torch.randn(N, H, H, C, device=cuda, generator=g)
    ths = (0.7 * x.abs().mean(dim=(1, 2, 3))).contiguous()
    w, wths = make_input(H + C, KN, K, K, C)
    qw, btn = TAB.Quantize(dev_t(w, cuda), dev_t(wths, cuda), O.weight_bits(t), KN, K, K, C)
    y = TAB.Conv2d(x, qw, ths, btn, t, p, p, s, s, N, H, H, C, KN, K, K)
    OH = (H + 2 * p - K + 1) // s
    assert tuple(y.shape) == (N, KN, OH, OH)
    yb = y.reshape(N, OH, OH, KN)
    qwh, btnh, thh = qw.cpu().numpy(), btn.cpu().numpy(), ths.cpu().numpy()
    for n in (0, 37, 63):
        yo = c_oracle.conv2d(x[n].cpu().numpy(), qwh, thh[n:n + 1], btnh, t, p, p, s, s, 1, H, H, C, KN, K, K)
        assert np.array_equal(yb[n].cpu().numpy().reshape(-1), yo.reshape(-1)), n
    # sharding property: the first 8 images alone give the same answer as inside the full batch
    y8 = TAB.Conv2d(x[:8].contiguous(), qw, ths[:8].contiguous(), btn, t, p, p, s, s, 8, H, H, C, KN, K, K)
    assert torch.equal(y8.reshape(-1), y.reshape(-1)[:y8.numel()])


@pytest.mark.parametrize("t", [3, 0])
def test_large_1x1_configuration(cuda, t):
    """N=128, 14x14x1024 -> 1024, 1x1 (M=25088, KN=1024, K=1024 bits), types BNN and TNN."""
    N, H, C, KN = 128, 14, 1024, 1024
    g = torch.Generator(device=cuda)
    g.manual_seed(4 + t)
    x = torch.randn(N, H, H, C, device=cuda, generator=g)
    ths = (0.7 * x.abs().mean(dim=(1, 2, 3))).contiguous()
    w, wths = make_input(77, KN, 1, 1, C)
    qw, btn = TAB.Quantize(dev_t(w, cuda), dev_t(wths, cuda), O.weight_bits(t), KN, 1, 1, C)
    y = TAB.Conv2d(x, qw, ths, btn, t, 0, 0, 1, 1, N, H, H, C, KN, 1, 1).reshape(N, -1)
    qwh, btnh, thh = qw.cpu().numpy(), btn.cpu().numpy(), ths.cpu().numpy()
    for n in (0, 64, 127):
        yo = c_oracle.conv2d(x[n].cpu().numpy(), qwh, thh[n:n + 1], btnh, t, 0, 0, 1, 1, 1, H, H, C, KN, 1, 1)
        assert np.array_equal(y[n].cpu().numpy(), yo.reshape(-1))


def test_packed_entry_point_equals_fused_call(cuda):
    N, H, W, C, KN = 3, 9, 8, 130, 33
    x, ths = make_input(1, N, H, W, C)
    w, wths = make_input(2, KN, 3, 3, C)
    for t in range(4):
        qw, btn = O.quantize(w, wths, O.weight_bits(t), KN, 3, 3, C)
        qx, _ = TAB.Quantize(dev_t(x, cuda), dev_t(ths, cuda), O.act_bits(t), N, H, W, C)
        y = TAB.conv2d_packed(qx, dev_t(qw, cuda), dev_t(btn, cuda), t, 1, 1, 2, 1, N, H, W, C, KN, 3, 3)
        yo = c_oracle.conv2d(x, qw, ths, btn, t, 1, 1, 2, 1, N, H, W, C, KN, 3, 3)
        assert np.array_equal(y.cpu().numpy(), yo)


def test_expand_weights(cuda):
    """expand_weights against the de-quantised oracle planes (channel padding 0)."""
    KN, K, C, Cp = 70, 3, 130, 192
    w, wths = make_input(2, KN, K, K, C)
    for wb in (2, 1):
        qw, _ = O.quantize(w, wths, wb, KN, K, K, C)
        w8 = TAB.ops.expand_weights(dev_t(qw, cuda), wb, KN, K, K, C)
        assert tuple(w8.shape) == (KN, K, K, Cp)
        exp_w = np.zeros((KN, K, K, Cp), np.int8)
        exp_w[..., :C] = O.dequantize(qw, C).astype(np.int8)
        assert np.array_equal(w8.cpu().numpy(), exp_w)


@pytest.mark.parametrize("geom", [
    # p1 p2 s1 s2  N  H  W   C   KN KH KW
    (1, 1, 2, 1, 3, 9, 8, 130, 70, 3, 3),
    (1, 2, 1, 1, 3, 9, 8, 130, 70, 3, 3),
    (1, 2, 2, 2, 3, 9, 8, 130, 70, 3, 3),
    (1, 2, 3, 2, 3, 9, 8, 130, 70, 3, 3),
    (0, 0, 2, 2, 5, 14, 14, 64, 128, 1, 1),
    (3, 3, 1, 1, 2, 6, 5, 64, 16, 3, 3),         # padding wider than the kernel reaches: the grid does not share padding
    (0, 0, 1, 1, 2, 9, 9, 200, 300, 3, 3),
    (1, 1, 1, 1, 5, 10, 12, 64, 192, 3, 3),       # filter count a multiple of 64: the grid quantises its own result
    (1, 1, 2, 2, 4, 12, 12, 128, 64, 3, 3),
])
def test_bits_stage_entry_point(cuda, geom):
    """Quantize -> expand_weights -> conv2d_bits (the tensor-core GEMM stage on its own, prepared weights) equals the
    oracle's Conv2d, plain and chained through one state block that every call leaves zeroed."""
    p1, p2, s1, s2, N, H, W, C, KN, KH, KW = geom
    x, ths = make_input(7, N, H, W, C)
    w, wths = make_input(8, KN, KH, KW, C)
    state = TAB.ops.new_state(N, cuda)
    for t in range(4):
        ab, wb = O.act_bits(t), O.weight_bits(t)
        qw, btn = O.quantize(w, wths, wb, KN, KH, KW, C)
        qx, _ = TAB.Quantize(dev_t(x, cuda), dev_t(ths, cuda), ab, N, H, W, C)
        w8 = TAB.ops.expand_weights(dev_t(qw, cuda), wb, KN, KH, KW, C)
        yo = c_oracle.conv2d(x, qw, ths, btn, t, *geom)
        y, nxt = TAB.ops.conv2d_bits(qx, w8, t, *geom)
        assert nxt is None and np.array_equal(y.cpu().numpy(), yo)
        r = torch.round(torch.randn(*yo.shape, device=cuda) * 5)
        y2, nxt = TAB.ops.conv2d_bits(qx, w8, t, *geom, residual=r, threshold_scale=0.7, state=state)
        y2o = yo + r.cpu().numpy()
        assert np.array_equal(y2.cpu().numpy(), y2o)
        assert np.array_equal(nxt.cpu().numpy(), OracleOps.residual_threshold(y2o.copy(), None, 0.7))
        assert not state.any().item()
        # the compact form for chained layers: the same integers as int16, and the quantiser that reads them
        y16, nxt16 = TAB.ops.conv2d_bits(qx, w8, t, *geom, threshold_scale=0.7, state=state, out_int16=True)
        assert y16.dtype == torch.int16 and np.array_equal(y16.cpu().numpy().astype(np.float32), yo)
        assert np.array_equal(nxt16.cpu().numpy(), OracleOps.residual_threshold(yo.copy(), None, 0.7))
        OH, OW = yo.shape[2], yo.shape[3]
        if OH * OW:
            for bw in (2, 1):
                # the same launch handing on the quantised result (in the kernel where KN is a multiple of 64, else behind it)
                for kw in (dict(residual=r), dict(out_int16=True)):
                    ya, na, qa = TAB.ops.conv2d_bits(qx, w8, t, *geom, threshold_scale=0.7, state=state, next_bitwidth=bw, **kw)
                    yb, nb_ = TAB.ops.conv2d_bits(qx, w8, t, *geom, threshold_scale=0.7, state=state, **kw)
                    assert torch.equal(ya, yb) and torch.equal(na, nb_) and not state.any().item()
                    want = (TAB.ops.quantize_i16(yb, nb_, bw, N, OH, OW, KN) if yb.dtype == torch.int16
                            else TAB.Quantize(yb, nb_, bw, N, OH, OW, KN)[0])
                    assert torch.equal(qa.reshape(-1), want.reshape(-1))
                q16 = TAB.ops.quantize_i16(y16, nxt16, bw, N, OH, OW, KN)
                qf, _ = TAB.Quantize(dev_t(yo, cuda), nxt16, bw, N, OH, OW, KN)
                assert torch.equal(q16, qf)
                assert np.array_equal(q16.cpu().numpy(), O.quantize(yo.reshape(N, OH, OW, KN), nxt16.cpu().numpy(), bw, N, OH, OW, KN)[0])
        assert _cabi.lib().tab_device_status() == 0


@pytest.mark.parametrize("t", range(4))
@pytest.mark.parametrize("geom", [
    # p1 p2 s1 s2  N   H   W   C   KN KH KW
    (1, 1, 1, 1, 48, 14, 14, 256, 320, 3, 3),    # two filter blocks, the second ragged
    (0, 0, 1, 1, 80, 16, 16, 100, 256, 3, 3),    # no padding, one ragged channel word
    (1, 1, 1, 1, 153, 7, 7, 192, 512, 3, 3),     # odd number of 128-row blocks: the last pair's second CTA has no rows
])
def test_cta_pair_kernel(cuda, t, geom, conv_path):
    """Wide filter blocks with many tiles run on clusters of two CTAs (tcgen05 cta_group::2): plain and with next thresholds
    and 16-bit output, against the oracle; the same shapes with a residual."""
    if conv_path != "tensor":
        pytest.skip("tensor-core path only")
    p1, p2, s1, s2, N, H, W, C, KN, KH, KW = geom
    x, ths = make_input(61, N, H, W, C)
    w, wths = make_input(62, KN, KH, KW, C)
    ab, wb = O.act_bits(t), O.weight_bits(t)
    qw, btn = O.quantize(w, wths, wb, KN, KH, KW, C)
    qx, _ = TAB.Quantize(dev_t(x, cuda), dev_t(ths, cuda), ab, N, H, W, C)
    w8 = TAB.ops.expand_weights(dev_t(qw, cuda), wb, KN, KH, KW, C)
    yo = c_oracle.conv2d(x, qw, ths, btn, t, *geom)
    state = TAB.ops.new_state(N, cuda)
    y, _ = TAB.ops.conv2d_bits(qx, w8, t, *geom)
    assert ",pair>" in _cabi.lib().tab_last_conv_kernel().decode()
    assert np.array_equal(y.cpu().numpy(), yo)
    r = torch.round(torch.randn(*yo.shape, device=cuda) * 5)
    y2, nxt = TAB.ops.conv2d_bits(qx, w8, t, *geom, residual=r, threshold_scale=0.7, state=state)   # (a residual layer runs on single CTAs)
    y2o = yo + r.cpu().numpy()
    assert np.array_equal(y2.cpu().numpy(), y2o)
    assert np.array_equal(nxt.cpu().numpy(), OracleOps.residual_threshold(y2o.copy(), None, 0.7))
    y16, nxt16 = TAB.ops.conv2d_bits(qx, w8, t, *geom, threshold_scale=0.7, state=state, out_int16=True)
    assert ",pair>" in _cabi.lib().tab_last_conv_kernel().decode()
    assert y16.dtype == torch.int16 and np.array_equal(y16.cpu().numpy().astype(np.float32), yo)
    assert np.array_equal(nxt16.cpu().numpy(), OracleOps.residual_threshold(yo.copy(), None, 0.7))
    assert not state.any().item()
    # the pairs' grid quantising its own result
    OH, OW = yo.shape[2], yo.shape[3]
    ya, na, qa = TAB.ops.conv2d_bits(qx, w8, t, *geom, threshold_scale=0.7, state=state, out_int16=True, next_bitwidth=ab)
    assert ",pair>" in _cabi.lib().tab_last_conv_kernel().decode()
    assert torch.equal(ya, y16) and torch.equal(na, nxt16) and not state.any().item()
    assert np.array_equal(qa.cpu().numpy().reshape(-1), O.quantize(yo.reshape(N, OH, OW, KN), nxt16.cpu().numpy(), ab, N, OH, OW, KN)[0].reshape(-1))
    assert _cabi.lib().tab_device_status() == 0


@pytest.mark.parametrize("t", [0, 3])
@pytest.mark.parametrize("geom", [
    # p1 p2 s1 s2  N   H   W   C   KN KH KW
    (1, 1, 2, 2, 200, 14, 14, 256, 512, 3, 3),   # strided: 200 tiles, a last round of 52
    (0, 0, 2, 2, 200, 14, 14, 256, 512, 1, 1),   # 1x1 stride 2: 154 tiles, a last round of 6
    (1, 1, 1, 1, 200, 7, 7, 128, 512, 3, 3),     # residual layer shape: 200 tiles
    (1, 1, 1, 1, 48, 14, 14, 192, 320, 3, 3),    # ragged filter count: the second half of the last filter block is empty
])
def test_last_round_in_halves(cuda, t, geom, conv_path):
    """A last round of 256-filter tiles that fills at most half of the persistent grid is worked as halves of 128 filters:
    plain, with a residual and next thresholds, and with 16-bit output plus the next layer's quantised input, against the
    oracle."""
    if conv_path != "tensor":
        pytest.skip("tensor-core path only")
    p1, p2, s1, s2, N, H, W, C, KN, KH, KW = geom
    x, ths = make_input(71, N, H, W, C)
    w, wths = make_input(72, KN, KH, KW, C)
    ab, wb = O.act_bits(t), O.weight_bits(t)
    qw, btn = O.quantize(w, wths, wb, KN, KH, KW, C)
    qx, _ = TAB.Quantize(dev_t(x, cuda), dev_t(ths, cuda), ab, N, H, W, C)
    w8 = TAB.ops.expand_weights(dev_t(qw, cuda), wb, KN, KH, KW, C)
    yo = c_oracle.conv2d(x, qw, ths, btn, t, *geom)
    OH, OW = yo.shape[2], yo.shape[3]
    state = TAB.ops.new_state(N, cuda)
    r = torch.round(torch.randn(*yo.shape, device=cuda) * 5)
    y2, nxt = TAB.ops.conv2d_bits(qx, w8, t, *geom, residual=r, threshold_scale=0.7, state=state)
    name = _cabi.lib().tab_last_conv_kernel().decode()
    if torch.cuda.get_device_properties(cuda).multi_processor_count == 148:
        assert " halves" in name and ",pair" not in name, name
    y2o = yo + r.cpu().numpy()
    assert np.array_equal(y2.cpu().numpy(), y2o)
    assert np.array_equal(nxt.cpu().numpy(), OracleOps.residual_threshold(y2o.copy(), None, 0.7))
    if KH * KW == 1 or s1 > 1:                                      # (unit-stride 3x3 layers without a residual run on CTA pairs)
        y, _ = TAB.ops.conv2d_bits(qx, w8, t, *geom)
        assert np.array_equal(y.cpu().numpy(), yo)
        ya, na, qa = TAB.ops.conv2d_bits(qx, w8, t, *geom, threshold_scale=0.7, state=state, out_int16=True, next_bitwidth=ab)
        tn = OracleOps.residual_threshold(yo.copy(), None, 0.7)
        assert ya.dtype == torch.int16 and np.array_equal(ya.cpu().numpy().astype(np.float32), yo) and np.array_equal(na.cpu().numpy(), tn)
        assert np.array_equal(qa.cpu().numpy().reshape(-1), O.quantize(yo.reshape(N, OH, OW, KN), tn, ab, N, OH, OW, KN)[0].reshape(-1))
    assert not state.any().item()
    assert _cabi.lib().tab_device_status() == 0


@pytest.mark.parametrize("t", [0, 3])
@pytest.mark.parametrize("geom", [
    # p1 p2 s1 s2  N   H    W    C   KN KH KW
    (3, 3, 2, 2, 2, 224, 224, 3, 64, 7, 7),      # ResNet stem: 49 taps over four parity planes
    (1, 1, 1, 1, 1, 224, 224, 64, 64, 3, 3),     # wide image: the patch only fits with one row block per tile
    (1, 1, 1, 1, 1, 300, 500, 64, 40, 3, 3),     # wide image: a 1 130-row patch
    (2, 1, 3, 2, 2, 33, 17, 192, 200, 5, 3),     # stride 3 x 2, six parity planes, ragged filter count
    (1, 1, 1, 1, 70, 3, 3, 64, 64, 3, 3),        # 25 grid positions per image: a 32-row slab spans three images
    (0, 0, 1, 1, 2, 28, 28, 128, 1000, 1, 1),    # 1x1, filter count not a multiple of 32
])
def test_large_and_odd_shapes_plain_and_chained(cuda, t, geom):
    """Shapes that steer the dispatch to every branch, as plain Conv2d and as the chained call (residual, |y| sums, next
    thresholds from the GEMM's last CTA)."""
    p1, p2, s1, s2, N, H, W, C, KN, KH, KW = geom
    x, ths = make_input(41, N, H, W, C)
    w, wths = make_input(42, KN, KH, KW, C)
    qw, btn = O.quantize(w, wths, O.weight_bits(t), KN, KH, KW, C)
    yo = c_oracle.conv2d(x, qw, ths, btn, t, *geom)
    xd, qd, td, bd = dev_t(x, cuda), dev_t(qw, cuda), dev_t(ths, cuda), dev_t(btn, cuda)
    y = TAB.Conv2d(xd, qd, td, bd, t, *geom)
    assert np.array_equal(y.cpu().numpy(), yo)
    r = torch.round(torch.randn(*yo.shape, device=cuda) * 5)
    y2, nxt = TAB.ops.Conv2dFused(xd, qd, td, bd, t, *geom, r, 0.7)
    y2o = yo + r.cpu().numpy()
    assert np.array_equal(y2.cpu().numpy(), y2o)
    exp = (np.float64(np.float32(0.7)) * (np.abs(y2o).astype(np.float64).reshape(N, -1).sum(1) / y2o[0].size)).astype(np.float32)
    assert np.array_equal(nxt.cpu().numpy(), exp)


def test_shapes_beyond_the_tensor_kernel_fall_back(cuda):
    """A 9x9 kernel on a 300-pixel-wide image needs a patch that does not fit shared memory: the call falls back to the
    popcount kernel and must still be exact; the same kernel on a narrow image stays on the tensor cores."""
    for N, H, W, C, KN, K in ((1, 12, 12, 64, 8, 9), (1, 20, 300, 64, 8, 9)):
        x, ths = make_input(3, N, H, W, C)
        w, wths = make_input(4, KN, K, K, C)
        for t in (0, 3):
            qw, btn = O.quantize(w, wths, O.weight_bits(t), KN, K, K, C)
            y = gpu_conv(cuda, x, qw, ths, btn, t, 4, 4, 1, 1, N, H, W, C, KN, K, K)
            assert np.array_equal(y, c_oracle.conv2d(x, qw, ths, btn, t, 4, 4, 1, 1, N, H, W, C, KN, K, K))


# ------------------------------------------------------------------------------------------ chain

def test_residual_threshold(cuda):
    rng = np.random.default_rng(3)
    for shape in ((3, 5, 4, 4), (2, 7, 3, 3), (4, 64, 7, 7)):
        y = np.round(rng.standard_normal(shape) * 50).astype(np.float32)
        r = np.round(rng.standard_normal(shape) * 50).astype(np.float32)
        yd = dev_t(y, cuda)
        t0 = TAB.ops.residual_threshold(yd, None, 0.7)
        assert np.array_equal(t0.cpu().numpy(), OracleOps.residual_threshold(y.copy(), None, 0.7))
        t1 = TAB.ops.residual_threshold(yd, dev_t(r, cuda), 0.7)
        yo = y.copy()
        to = OracleOps.residual_threshold(yo, r, 0.7)
        assert np.array_equal(yd.cpu().numpy(), yo) and np.array_equal(t1.cpu().numpy(), to)


@pytest.mark.parametrize("bw", [2, 1])
@pytest.mark.parametrize("shape", [(3, 5, 7, 64), (16, 9, 4, 128), (2, 56, 56, 64), (5, 3, 3, 70), (300, 2, 2, 64)])
def test_quantize_auto(cuda, bw, shape):
    """Thresholds scale * mean|x[n]| and the bit-planes against them from one call: the thresholds equal the double-precision
    reference (integer-valued data: every summation order gives the same sum), the bit-planes are the oracle's for those
    thresholds, and the state block comes back zeroed; also with real-valued data against the device's own thresholds."""
    N, H, W, C = shape
    rng = np.random.default_rng(N + C)
    state = TAB.ops.new_state(N, cuda)
    for integer in (True, False):
        x = rng.standard_normal((N, H, W, C)).astype(np.float32)
        if integer:
            x = np.round(x * 40).astype(np.float32)
        for rep in range(2):                                           # twice through the same state block
            qx, ths = TAB.ops.quantize_auto(dev_t(x, cuda), 0.7, bw, N, H, W, C, state)
            t = ths.cpu().numpy()
            if integer:
                assert np.array_equal(t, OracleOps.residual_threshold(x.reshape(N, -1).copy(), None, 0.7))
            else:
                assert np.allclose(t, 0.7 * np.abs(x).reshape(N, -1).mean(1), rtol=1e-6)
            assert np.array_equal(qx.cpu().numpy(), O.quantize(x, t, bw, N, H, W, C)[0])
            assert not state.any().item()
    assert _cabi.lib().tab_device_status() == 0


def test_next_layer_quantisation_with_many_images(cuda):
    """More images than the kernel's second phase keeps thresholds for (8192): the quantiser runs behind the GEMM stage and the
    call returns the same three results."""
    N, H, W, C, KN = 8200, 2, 2, 64, 64
    x, ths = make_input(71, N, H, W, C)
    w, wths = make_input(72, KN, 1, 1, C)
    qw, btn = O.quantize(w, wths, 2, KN, 1, 1, C)
    qx, _ = TAB.Quantize(dev_t(x, cuda), dev_t(ths, cuda), 2, N, H, W, C)
    w8 = TAB.ops.expand_weights(dev_t(qw, cuda), 2, KN, 1, 1, C)
    state = TAB.ops.new_state(N, cuda)
    y, nxt, qn = TAB.ops.conv2d_bits(qx, w8, 0, 0, 0, 1, 1, N, H, W, C, KN, 1, 1, threshold_scale=0.7, state=state, next_bitwidth=2)
    assert "+next" not in _cabi.lib().tab_last_conv_kernel().decode()
    yo = c_oracle.conv2d(x, qw, ths, btn, 0, 0, 0, 1, 1, N, H, W, C, KN, 1, 1)
    assert np.array_equal(y.cpu().numpy(), yo)
    to = OracleOps.residual_threshold(yo.copy(), None, 0.7)
    assert np.array_equal(nxt.cpu().numpy(), to)
    assert np.array_equal(qn.cpu().numpy(), O.quantize(yo.reshape(N, H, W, KN), to, 2, N, H, W, KN)[0])
    assert not state.any().item() and _cabi.lib().tab_device_status() == 0


@pytest.mark.parametrize("C", [64, 70])
def test_quantize_i16_threshold_edge_values(cuda, C):
    """The 16-bit quantiser must agree with the fp32 quantiser (and the oracle) for every kind of threshold: fractions, exact
    integers, negative, zero, beyond the 16-bit range, infinities and NaN - on values that include the extremes and every
    integer around the thresholds."""
    ths = np.array([0.0, -0.0, 0.5, 5.0, 5.5, -3.0, -3.2, 32766.5, 32767.0, 40000.0, -40000.0, 1e30, -1e30, np.inf, -np.inf, np.nan, 1e-30, 7.999999],
                   dtype=np.float32)
    N, H, W = len(ths), 4, 8
    rng = np.random.default_rng(C)
    v = rng.integers(-12, 13, size=(N, H, W, C)).astype(np.int16)
    v[:, 0, 0, :8] = np.array([-32767, 32767, -32766, 32766, 0, 1, -1, 8], dtype=np.int16)
    v[:, 0, 1, :6] = np.array([5, 6, -5, -6, -3, -4], dtype=np.int16)
    vd = torch.from_numpy(v).to(cuda)
    td = torch.from_numpy(ths).to(cuda)
    xf = v.astype(np.float32)
    for bw in (2, 1):
        q16 = TAB.ops.quantize_i16(vd, td, bw, N, H, W, C)
        qf, _ = TAB.Quantize(torch.from_numpy(xf).to(cuda), td, bw, N, H, W, C)
        assert torch.equal(q16, qf)
        assert np.array_equal(q16.cpu().numpy(), O.quantize(xf, ths, bw, N, H, W, C)[0])


def test_fused_conv_matches_unfused(cuda):
    """tab_conv2d_fused_launch: residual and per-image |y| statistics in the epilogue == separate passes."""
    rng = np.random.default_rng(11)
    for geom in ((1, 1, 1, 1, 5, 7, 7, 128, 130, 3, 3), (0, 0, 2, 2, 3, 14, 14, 64, 33, 1, 1), (1, 1, 1, 1, 2, 56, 56, 64, 64, 3, 3)):
        p1, p2, s1, s2, N, H, W, C, KN, KH, KW = geom
        x, ths = make_input(5, N, H, W, C)
        w, wths = make_input(6, KN, KH, KW, C)
        OH, OW = (H + 2 * p1 - KH + 1) // s1, (W + 2 * p2 - KW + 1) // s2
        r = np.round(rng.standard_normal((N, KN, OH, OW)) * 20).astype(np.float32)
        for t in range(4):
            qw, btn = O.quantize(w, wths, O.weight_bits(t), KN, KH, KW, C)
            args = (dev_t(x, cuda), dev_t(qw, cuda), dev_t(ths, cuda), dev_t(btn, cuda), t, *geom)
            yo = c_oracle.conv2d(x, qw, ths, btn, t, *geom)
            y0, n0 = TAB.Conv2dFused(*args, None, None)
            assert n0 is None and np.array_equal(y0.cpu().numpy(), yo)
            y1, t1 = TAB.Conv2dFused(*args, None, 0.7)
            assert np.array_equal(y1.cpu().numpy(), yo)
            assert np.array_equal(t1.cpu().numpy(), OracleOps.residual_threshold(yo.copy(), None, 0.7))
            y2, t2 = TAB.Conv2dFused(*args, dev_t(r, cuda), 0.7)
            yr = yo.copy()
            tr = OracleOps.residual_threshold(yr, r, 0.7)
            assert np.array_equal(y2.cpu().numpy(), yr) and np.array_equal(t2.cpu().numpy(), tr)


@pytest.mark.parametrize("t", [0, 3])
def test_chain_matches_oracle(cuda, t):
    """The 19-convolution ResNet-18-shaped chain, N=3, integer-valued input so that every threshold is an
    exact function of the data on both sides."""
    N = 3
    rng = np.random.default_rng(8)
    x = np.round(rng.standard_normal((N, 56, 56, 64)) * 4).astype(np.float32)
    weights = chain.make_weights(2000, t)
    qo = chain.quantize_weights(weights, t, OracleOps.Quantize)
    ths = OracleOps.residual_threshold(x.copy(), None, chain.THRESHOLD_SCALE)
    yo, oh, ow, kn = chain.forward(OracleOps, x, ths, qo, t, N)
    qd = chain.quantize_weights(weights, t, TAB.Quantize, lambda a: dev_t(a, cuda))
    for k in qo:
        assert np.array_equal(qd[k][0].cpu().numpy(), qo[k][0]) and np.array_equal(qd[k][1].cpu().numpy(), qo[k][1])
    xd = dev_t(x, cuda)
    thd = TAB.ops.residual_threshold(xd, None, chain.THRESHOLD_SCALE)
    assert np.array_equal(thd.cpu().numpy(), ths)
    yd, oh2, ow2, kn2 = chain.forward(TAB.ops, xd, thd, qd, t, N)        # fused epilogues
    assert (oh, ow, kn) == (oh2, ow2, kn2) == (7, 7, 512)
    assert np.array_equal(yd.cpu().numpy().reshape(-1), yo.reshape(-1))

    class Unfused:
        Conv2d = staticmethod(TAB.ops.Conv2d)
        residual_threshold = staticmethod(TAB.ops.residual_threshold)
    yu, _, _, _ = chain.forward(Unfused, xd, thd, qd, t, N)              # separate passes
    assert np.array_equal(yu.cpu().numpy().reshape(-1), yo.reshape(-1))


# ------------------------------------------------------------------------------------------ errors

def test_error_behaviour(cuda):
    x = torch.zeros(1, 4, 4, 64, device=cuda)
    t = torch.zeros(1, device=cuda)
    qw2 = torch.zeros(4, 3, 3, 1, 2, dtype=torch.int64, device=cuda)
    qw1 = torch.zeros(4, 3, 3, 1, 1, dtype=torch.int64, device=cuda)
    btn = torch.zeros(4, dtype=torch.int32, device=cuda)
    with pytest.raises(RuntimeError, match="must be a CUDA tensor"):
        TAB.Conv2d(x.cpu(), qw2, t, btn, 0, 1, 1, 1, 1, 1, 4, 4, 64, 4, 3, 3)
    with pytest.raises(RuntimeError, match="must be contiguous"):
        TAB.Conv2d(x.permute(0, 2, 1, 3), qw2, t, btn, 0, 1, 1, 1, 1, 1, 4, 4, 64, 4, 3, 3)
    with pytest.raises(RuntimeError, match="bitwidth 2"):
        TAB.Conv2d(x, qw1, t, btn, 0, 1, 1, 1, 1, 1, 4, 4, 64, 4, 3, 3)       # 1-bit weights given to TNN
    with pytest.raises(RuntimeError, match="type must be"):
        TAB.Conv2d(x, qw2, t, btn, 4, 1, 1, 1, 1, 1, 4, 4, 64, 4, 3, 3)
    l = _cabi.lib()
    y = torch.zeros(64, device=cuda)
    ws = torch.zeros(64, dtype=torch.uint8, device=cuda)          # too small
    rc = l.tab_conv2d_launch(x.data_ptr(), qw2.data_ptr(), t.data_ptr(), btn.data_ptr(), y.data_ptr(), ws.data_ptr(), 64,
                             0, 1, 1, 1, 1, 1, 4, 4, 64, 4, 3, 3, None)
    assert rc == -3
    # after the rejected calls the device path still works
    yy = TAB.Conv2d(x, qw2, t, btn, 0, 1, 1, 1, 1, 1, 4, 4, 64, 4, 3, 3)
    assert not yy.any().item()


# ------------------------------------------------------------------- quantisers: channel counts that fill no word, odd alignments

@pytest.mark.parametrize("off", [0, 1, 2, 4])
@pytest.mark.parametrize("C", [1, 2, 3, 4, 6, 8, 9, 12, 40, 64, 66, 72, 127, 196])
def test_quantize_any_width_and_alignment(cuda, conv_path, C, off):
    """Every load width (8, 4, 2, 1 elements by C and by the start of x), one and eight lanes per word, one and several
    CTAs per image, special values; bit-planes and counts are compared exactly."""
    if conv_path != "tensor":
        pytest.skip("no convolution in this test")
    for N, H, W in ((3, 5, 7), (2, 40, 31)):
        x, ths = make_input(C + off, N, H, W, C)
        x.reshape(-1)[: 5] = np.array([np.nan, np.inf, -np.inf, ths[0], -ths[0]], np.float32)[: x.size]
        ths[-1] = -0.25                                                    # zeros of channel tails must not count as above it
        buf = torch.empty(x.size + off, device=cuda)
        buf[off:] = dev_t(x, cuda).reshape(-1)
        for bw in (2, 1):
            q, b = TAB.Quantize(buf[off:], dev_t(ths, cuda), bw, N, H, W, C)
            qo, bo = O.quantize(x, ths, bw, N, H, W, C)
            assert np.array_equal(q.cpu().numpy(), qo) and np.array_equal(b.cpu().numpy(), bo)


@pytest.mark.parametrize("C", [3, 8, 40, 64, 66, 100, 127])
@pytest.mark.parametrize("N,H,W", [(1, 3, 2), (5, 40, 31), (700, 3, 3)])
def test_quantize_auto_any_channels(cuda, conv_path, N, H, W, C):
    """Thresholds and bit-planes from one launch for every load width.  The thresholds are double sums rounded once to
    float, so another order of summation gives the same float unless the sum sits within 1e-13 of a rounding boundary."""
    if conv_path != "tensor":
        pytest.skip("no convolution in this test")
    from tab_b200 import ops
    x, _ = make_input(C + N, N, H, W, C)
    ths = (np.float64(np.float32(0.7)) * np.abs(x).reshape(N, -1).sum(axis=1, dtype=np.float64) / (H * W * C)).astype(np.float32)
    state = ops.new_state(N, cuda)
    for bw in (2, 1):
        for _ in range(2):                                                 # the state block is left zero
            q, t = ops.quantize_auto(dev_t(x, cuda), 0.7, bw, N, H, W, C, state)
            assert np.array_equal(t.cpu().numpy(), ths)
            qo, _b = O.quantize(x, ths, bw, N, H, W, C)
            assert np.array_equal(q.cpu().numpy(), qo)
    assert not state.cpu().numpy().any()


@pytest.mark.parametrize("C", [5, 24, 65, 72])
def test_quantize_i16_any_channels(cuda, conv_path, C):
    if conv_path != "tensor":
        pytest.skip("no convolution in this test")
    from tab_b200 import ops
    rng = np.random.default_rng(C)
    x = rng.integers(-40, 41, size=(3, 9, 11, C)).astype(np.int16)
    ths = np.array([3.0, 0.0, 17.5], np.float32)
    for bw in (2, 1):
        q = ops.quantize_i16(dev_t(x, cuda), dev_t(ths, cuda), bw, 3, 9, 11, C)
        assert np.array_equal(q.cpu().numpy(), O.quantize(x.astype(np.float32), ths, bw, 3, 9, 11, C)[0])


# ------------------------------------------------------------------- tiles whose width follows the filter count, ragged rows

@pytest.mark.parametrize("geom", [
    # p1 p2 s1 s2  N  H  W   C   KN KH KW       KN odd / even / multiple of 4; 1 to 4 K steps of the last channel word pair
    (1, 1, 1, 1, 2, 9, 8, 3, 1, 3, 3),
    (1, 1, 1, 1, 2, 9, 8, 33, 2, 3, 3),
    (0, 0, 1, 1, 3, 9, 8, 96, 31, 1, 1),
    (1, 1, 1, 1, 2, 20, 13, 97, 33, 3, 3),
    (1, 1, 1, 1, 2, 20, 13, 160, 36, 3, 3),
    (1, 1, 1, 1, 2, 20, 13, 161, 97, 3, 3),
    (2, 2, 1, 1, 2, 20, 13, 70, 130, 5, 5),
    (1, 1, 2, 2, 2, 20, 13, 64, 161, 3, 3),
    (1, 1, 1, 1, 40, 3, 3, 64, 67, 3, 3),        # a 32-row slab spans three images: |y| sums row by row
    (1, 1, 1, 1, 2, 14, 14, 256, 259, 3, 3),
    (1, 1, 1, 1, 90, 14, 14, 130, 300, 3, 3),    # CTA pairs of 160-filter tiles
    (1, 1, 1, 1, 60, 14, 14, 64, 450, 3, 3),
    (0, 0, 1, 1, 30, 28, 28, 64, 384, 1, 1),     # two tiles of 192 filters
    (0, 0, 1, 1, 75, 16, 16, 64, 250, 1, 1),     # 150 tiles, the last block partial (filters resident: no halves)
    (0, 0, 1, 1, 75, 16, 16, 64, 222, 1, 1),     # the same with 224-wide tiles
    (1, 1, 1, 1, 1, 12, 12, 64, 60, 3, 3),       # the TMA epilogue with a partial block
    (1, 1, 1, 1, 1, 12, 12, 64, 28, 3, 3),
])
def test_filter_counts_and_channel_steps(cuda, geom, conv_path):
    if conv_path != "tensor":
        pytest.skip("the tensor-core kernel's own entry point")
    test_bits_stage_entry_point(cuda, geom)
    p1, p2, s1, s2, N, H, W, C, KN, KH, KW = geom
    x, ths = make_input(7, N, H, W, C)
    w, wths = make_input(8, KN, KH, KW, C)
    for t in (0, 3):
        qw, btn = O.quantize(w, wths, O.weight_bits(t), KN, KH, KW, C)
        assert np.array_equal(gpu_conv(cuda, x, qw, ths, btn, t, *geom), c_oracle.conv2d(x, qw, ths, btn, t, *geom))


@pytest.mark.parametrize("C", [64, 70, 512])
@pytest.mark.parametrize("N,KN,K", [(1, 5, 3), (1, 512, 3), (700, 16, 1)])
def test_weight_expansion_inside_a_call(cuda, conv_path, N, KN, K, C):
    """One-image calls (the launch has more CTAs than the tensor needs, for the weights) and many-image calls."""
    if conv_path != "tensor":
        pytest.skip("only the tensor-core path expands weights")
    x, ths = make_input(5, N, 4, 5, C)
    w, wths = make_input(6, KN, K, K, C)
    for t in range(4):
        qw, btn = O.quantize(w, wths, O.weight_bits(t), KN, K, K, C)
        g = (K // 2, K // 2, 1, 1, N, 4, 5, C, KN, K, K)
        assert np.array_equal(gpu_conv(cuda, x, qw, ths, btn, t, *g), c_oracle.conv2d(x, qw, ths, btn, t, *g))


# ------------------------------------------------------------------- 4-bit operands

@pytest.mark.parametrize("geom", [
    # p1 p2 s1 s2  N  H  W   C   KN KH KW       1 to 5 words per pixel (1, 2, 4 taps per filter row), each tile and grid form
    (1, 1, 1, 1, 2, 9, 8, 3, 1, 3, 3),
    (1, 1, 1, 1, 2, 20, 13, 64, 64, 3, 3),
    (2, 2, 1, 1, 2, 20, 13, 70, 130, 5, 5),
    (1, 1, 1, 1, 3, 14, 14, 128, 128, 3, 3),
    (1, 1, 1, 1, 2, 14, 14, 129, 97, 3, 3),
    (1, 1, 1, 1, 2, 14, 14, 256, 259, 3, 3),
    (1, 1, 1, 1, 2, 14, 14, 260, 36, 3, 3),
    (1, 1, 2, 2, 2, 20, 13, 64, 161, 3, 3),
    (1, 1, 2, 2, 64, 14, 14, 320, 256, 3, 3),
    (1, 2, 3, 2, 3, 9, 8, 130, 70, 3, 3),
    (1, 1, 1, 1, 40, 3, 3, 64, 67, 3, 3),        # a 32-row slab spans three images
    (1, 1, 1, 1, 40, 3, 3, 64, 64, 3, 3),
    (0, 0, 1, 1, 75, 16, 16, 64, 250, 1, 1),     # a second round of two tiles
    (1, 1, 1, 1, 200, 14, 14, 64, 256, 3, 3),    # several tiles per CTA: accumulators that overlap, one row block
    (1, 1, 1, 1, 200, 14, 14, 64, 456, 3, 3),    # 256-filter tiles, the last block of the second one without filters
    (1, 1, 1, 1, 60, 28, 28, 128, 128, 3, 3),    # the same with two row blocks
    (1, 1, 1, 1, 48, 14, 14, 192, 320, 3, 3),
    (1, 1, 2, 2, 200, 14, 14, 256, 512, 3, 3),
    (1, 1, 1, 1, 8, 56, 56, 64, 60, 3, 3),       # the TMA epilogue, several tiles per CTA, a partial block
    (1, 1, 1, 1, 1, 100, 150, 200, 40, 3, 3),    # long patches: several chunks of items
    (1, 1, 1, 1, 1, 7, 7, 512, 512, 3, 3),       # one small image, a long sum: tiles of 32 filters
    (1, 1, 1, 1, 1, 7, 7, 300, 72, 3, 3),
    (3, 3, 2, 2, 2, 224, 224, 3, 64, 7, 7),
])
@pytest.mark.parametrize("t", [0, 1, 2, 3])
def test_packed4_weights(cuda, geom, t, conv_path):
    """The GEMM stage on 4-bit weights against the oracle - plain, with residual and thresholds (a residual that is no
    integer included), 16-bit output, next layer's input - and against the byte form for what the oracle does not give."""
    if conv_path != "tensor":
        pytest.skip("the tensor-core kernel's own entry point")
    p1, p2, s1, s2, N, H, W, C, KN, KH, KW = geom
    x, ths = make_input(91, N, H, W, C)
    w, wths = make_input(92, KN, KH, KW, C)
    ab, wb = O.act_bits(t), O.weight_bits(t)
    qw, btn = O.quantize(w, wths, wb, KN, KH, KW, C)
    qx, _ = TAB.Quantize(dev_t(x, cuda), dev_t(ths, cuda), ab, N, H, W, C)
    w8 = TAB.ops.expand_weights(dev_t(qw, cuda), wb, KN, KH, KW, C)
    w4 = TAB.ops.pack_weights(w8, KN, KH, KW, C)
    state = TAB.ops.new_state(N, cuda)
    y, _ = TAB.ops.conv2d_bits(qx, w4, t, *geom)
    assert ",e2m1>" in _cabi.lib().tab_last_conv_kernel().decode()
    some = sorted({0, N // 2, N - 1})                                   # images are independent
    OH, OW = y.shape[2], y.shape[3]
    for n in some:
        yo = c_oracle.conv2d(x[n:n + 1], qw, ths[n:n + 1], btn, t, p1, p2, s1, s2, 1, H, W, C, KN, KH, KW)
        assert np.array_equal(y.reshape(N, -1)[n].cpu().numpy(), yo.reshape(-1))
    y8, _ = TAB.ops.conv2d_bits(qx, w8, t, *geom)
    assert torch.equal(y, y8) and not torch.signbit(y[y == 0]).any().item()
    r = torch.randn(*y.shape, device=cuda) * 5
    for bw in (None, 2, 1):
        for kw in (dict(residual=r), dict(residual=torch.round(r)), dict(out_int16=True), dict()):
            a = TAB.ops.conv2d_bits(qx, w4, t, *geom, threshold_scale=0.7, state=state, next_bitwidth=bw, **kw)
            b = TAB.ops.conv2d_bits(qx, w8, t, *geom, threshold_scale=0.7, state=state, next_bitwidth=bw, **kw)
            assert len(a) == len(b) and all(torch.equal(u, v) for u, v in zip(a, b)) and not state.any().item()
    # a 16-bit residual, the result as fp32 and as 16-bit integers
    r16 = torch.round(r).to(torch.int16)
    for bw in (None, 2, 1):
        b = TAB.ops.conv2d_bits(qx, w8, t, *geom, residual=r16.float(), threshold_scale=0.7, state=state, next_bitwidth=bw)
        for out16 in (False, True):
            a = TAB.ops.conv2d_bits(qx, w4, t, *geom, residual=r16, threshold_scale=0.7, state=state, next_bitwidth=bw, out_int16=out16)
            assert a[0].dtype == (torch.int16 if out16 else torch.float32) and torch.equal(a[0].float(), b[0])
            assert all(torch.equal(u, v) for u, v in zip(a[1:], b[1:]) if u is not None) and not state.any().item()
    assert torch.equal(TAB.ops.conv2d_bits(qx, w4, t, *geom, residual=r16, out_int16=True)[0].float(), b[0])
    y3, _ = TAB.ops.conv2d_bits(qx, w4, t, *geom, residual=r)
    assert torch.equal(y3, y8 + r)
    assert _cabi.lib().tab_device_status() == 0


def test_packed4_sums_are_exact_at_large_magnitude(cuda, conv_path):
    """All operands +1 but a few: sums near KH*KW*C = 401408 and differing in the last unit."""
    if conv_path != "tensor":
        pytest.skip("the tensor-core kernel's own entry point")
    N, H, W, C, KN, K = 1, 14, 14, 2048, 40, 14
    x = torch.ones(N, H, W, C, device=cuda)
    x[0, 3, 5, :7] = -1.0
    w = torch.ones(KN, K, K, C, device=cuda)
    for f in range(KN):
        w[f].view(-1)[: 3 * f] = -1.0
    one = torch.full((N,), 0.5, device=cuda)
    q = TAB.Quantize(w, torch.full((KN,), 0.5, device=cuda), 2, KN, K, K, C)
    y = TAB.Conv2d(x, q[0], one, q[1], 0, 0, 0, 1, 1, N, H, W, C, KN, K, K)
    want = (x.double().reshape(1, -1) @ w.double().reshape(KN, -1).T).reshape(-1)
    assert torch.equal(y.double().reshape(-1), want)


@pytest.mark.parametrize("geom", [
    # p1 p2 s1 s2  N  H  W   C   KN KH KW       two tiles of 32 filters (a small image, 33 to 64 filters, 32 words or more per sum)
    (3, 3, 1, 1, 1, 16, 16, 20, 64, 7, 7),
    (3, 3, 1, 1, 1, 16, 16, 20, 36, 7, 7),
    (3, 3, 1, 1, 1, 28, 28, 16, 64, 7, 7),
    (3, 3, 1, 1, 1, 9, 13, 3, 60, 7, 7),
])
@pytest.mark.parametrize("t", [0, 3])
def test_tma_epilogue_on_tiles_of_32_filters(cuda, geom, t, conv_path):
    """The TMA epilogue where only half of its warps have columns: fp32 residuals, next thresholds, the next layer's input, and
    the same without a residual (the other epilogue)."""
    if conv_path != "tensor":
        pytest.skip("the tensor-core kernel's own entry point")
    test_packed4_weights(cuda, geom, t, conv_path)
    p1, p2, s1, s2, N, H, W, C, KN, KH, KW = geom
    x, ths = make_input(93, N, H, W, C)
    w, wths = make_input(94, KN, KH, KW, C)
    qw, btn = O.quantize(w, wths, O.weight_bits(t), KN, KH, KW, C)
    m = tab_nn.TABConv2d(dev_t(qw, cuda), dev_t(btn, cuda), t, KN, KH, KW, C, (p1, p2), (s1, s2))
    yo = c_oracle.conv2d(x, qw, ths, btn, t, *geom)
    r = np.random.default_rng(3).standard_normal(yo.shape).astype(np.float32)
    for _ in range(3):
        y, nxt = m.conv_bits(m.quantize(dev_t(x, cuda), dev_t(ths, cuda)), N, H, W, residual=dev_t(r, cuda), next_threshold_scale=0.7)
        assert np.array_equal(y.cpu().numpy(), yo + r)
        want = np.float32(np.float64(np.float32(0.7)) * np.abs((yo + r).astype(np.float64)).sum() / yo.size)
        assert abs(nxt.item() - want) <= 2 * np.spacing(want)              # compensated sums: good to far less than the last place
    assert ",2,1" in _cabi.lib().tab_last_conv_kernel().decode()           # residual, TMA epilogue


@pytest.mark.parametrize("H,KN", [(2, 128), (2, 33), (2, 72), (1, 100)])
def test_thresholds_of_small_images_with_extreme_residuals(cuda, H, KN, conv_path):
    """Images of so few positions that 32 rows of the grid span three, residuals that are infinite or whose sum leaves the range of
    float: the sums of |y| are taken in double, so the next thresholds are infinite there and finite here."""
    if conv_path != "tensor":
        pytest.skip("the tensor-core kernel's own entry point")
    N, C, K = 40, 64, 3
    x, ths = make_input(5, N, H, H, C)
    w, wths = make_input(6, KN, K, K, C)
    qw, btn = O.quantize(w, wths, 2, KN, K, K, C)
    geom = (1, 1, 1, 1, N, H, H, C, KN, K, K)
    yo = c_oracle.conv2d(x, qw, ths, btn, 0, *geom).reshape(N, -1)
    r = np.random.default_rng(1).standard_normal(yo.shape).astype(np.float32)
    r[1, 5] = np.inf
    r[2, :] = 3e38
    r[3, 0], r[3, 1] = -np.inf, np.inf
    want = (np.float64(np.float32(0.7)) * np.abs((yo + r).astype(np.float64)).sum(axis=1) / yo.shape[1]).astype(np.float32)
    qx = TAB.Quantize(dev_t(x, cuda), dev_t(ths, cuda), 2, N, H, H, C)[0]
    w8 = TAB.ops.expand_weights(dev_t(qw, cuda), 2, KN, K, K, C)
    for weights in (w8, TAB.ops.pack_weights(w8, KN, K, K, C)):
        y, nxt = TAB.ops.conv2d_bits(qx, weights, 0, *geom, residual=dev_t(r, cuda), threshold_scale=0.7, state=TAB.ops.new_state(N, cuda))
        assert np.array_equal(y.cpu().numpy().reshape(N, -1), yo + r)
        assert np.array_equal(np.isinf(nxt.cpu().numpy()), np.isinf(want)) and np.allclose(nxt.cpu().numpy(), want, rtol=2e-7, atol=0)


@pytest.mark.parametrize("C", [64, 70])
def test_meeting_point_whose_wait_runs_out(cuda, conv_path, C):
    """A counter that can never reach the number of CTAs: the wait ends by itself, the next calls say so until the status is read,
    and the state block is zero again, so that a caller who keeps it goes on with right results."""
    if conv_path != "tensor":
        pytest.skip("no convolution in this test")
    N, H, W, KN = 2, 4, 4, 64
    lib = _cabi.lib()
    assert lib.tab_device_status() == 0
    m = tab_nn.TABConv2d.from_float(torch.randn(KN, 3, 3, C, device=cuda), 0, 1, 1)
    x = torch.randn(N, H, W, C, device=cuda)
    want, qwant = m(x), m.quantize(x)
    state = m.state(N, cuda)
    try:
        state.view(torch.int32)[2 * N + 1] = -1                             # the meeting point, behind the sums and the completion counter: two CTAs take it to 1
        m.quantize_auto(x)
        torch.cuda.synchronize()
        with pytest.raises(_cabi.TabError, match="bounded wait") as stop:
            m(x)
        assert stop.value.code == -7
        with pytest.raises(_cabi.TabError, match="bounded wait"):
            m.conv_bits(qwant, N, H, W)
    finally:
        assert lib.tab_device_status() == 22
    assert lib.tab_device_status() == 0 and not state.any().item()
    assert torch.equal(m(x), want) and torch.equal(m.quantize(x), qwant)


def test_meeting_points_on_several_streams(cuda, conv_path):
    """The quantiser that finds its thresholds, whose CTAs wait for one another, on four streams at once and behind work that holds
    SMs: its launches are placed whole (cooperative ones), captured ones too."""
    if conv_path != "tensor":
        pytest.skip("the tensor-core kernel's own entry point")
    N, H, W, C = 16, 28, 28, 130
    layers = [tab_nn.TABConv2d.from_float(torch.randn(128, 3, 3, C, device=cuda), 0, 1, 1) for _ in range(4)]
    x = torch.randn(N, H, W, C, device=cuda)
    a = torch.randn(2048, 2048, device=cuda)

    def one(m):
        qx, ths = m.quantize_auto(x)
        return m.conv_bits(qx, N, H, W)[0], qx, ths

    want = [one(m) for m in layers]
    streams = [torch.cuda.Stream() for _ in layers]
    torch.cuda.synchronize()
    got = [[] for _ in layers]
    for _ in range(20):
        for m, s, g in zip(layers, streams, got):
            with torch.cuda.stream(s):
                a @ a
                g.append(one(m))
    torch.cuda.synchronize()
    for w, g in zip(want, got):
        assert all(torch.equal(u, v) for r in g for u, v in zip(r, w))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = one(layers[0])
    for _ in range(3):
        graph.replay()
    assert all(torch.equal(u, v) for u, v in zip(out, want[0]))
    assert _cabi.lib().tab_device_status() == 0


@pytest.mark.parametrize("KN", [4, 66, 100, 104, 128, 132, 99])
@pytest.mark.parametrize("N,H", [(40, 3), (3, 15)])                         # several images per 32 rows of the grid, or one
def test_rows_that_start_between_vectors(cuda, N, H, KN, conv_path):
    """Rows and residuals on 16-, 8-, 4- and 2-byte boundaries: filter counts that are multiples of four, two and one, a residual
    that starts 16 bytes into its allocation; fp32 and 16-bit residuals and results, byte and 4-bit operands."""
    if conv_path != "tensor":
        pytest.skip("the tensor-core kernel's own entry point")
    C, K = 130, 3
    x, ths = make_input(5, N, H, H, C)
    w, wths = make_input(6, KN, K, K, C)
    qw, btn = O.quantize(w, wths, 2, KN, K, K, C)
    geom = (1, 1, 1, 1, N, H, H, C, KN, K, K)
    yo = torch.from_numpy(c_oracle.conv2d(x, qw, ths, btn, 0, *geom)).to(cuda)
    qx = TAB.Quantize(dev_t(x, cuda), dev_t(ths, cuda), 2, N, H, H, C)[0]
    w8 = TAB.ops.expand_weights(dev_t(qw, cuda), 2, KN, K, K, C)
    w4 = TAB.ops.pack_weights(w8, KN, K, K, C)
    state = TAB.ops.new_state(N, cuda)

    def check(weights, r, **kw):
        y, nxt = TAB.ops.conv2d_bits(qx, weights, 0, *geom, residual=r, threshold_scale=0.7, state=state, **kw)
        want = yo if r is None else yo + r.float().reshape(yo.shape)
        assert torch.equal(y.float(), want) and not state.any().item()
        t = (float(np.float32(0.7)) * want.double().abs().reshape(N, -1).sum(dim=1) / want[0].numel()).float()
        assert torch.allclose(nxt, t, rtol=1.2e-7, atol=0)                 # both are roundings of sums good to far less than that
        assert torch.equal(TAB.ops.conv2d_bits(qx, weights, 0, *geom, residual=r, **kw)[0], y)

    for off in (0, 4):
        r = torch.round(torch.randn(yo.numel() + off, device=cuda) * 9)[off:].reshape(yo.shape)
        for weights in (w8, w4):
            check(weights, r)
            check(weights, r + 0.25 if off == 0 else r)
        r16 = torch.empty(yo.numel() + 2 * off, dtype=torch.int16, device=cuda)[2 * off:].reshape(yo.shape)
        r16.copy_(r)
        check(w4, r16)
        check(w4, r16, out_int16=True)
    for weights in (w8, w4):
        check(weights, None)
        check(weights, None, out_int16=True)
    assert _cabi.lib().tab_device_status() == 0


def _long_sums(cuda, C, KN, t):
    """A 1x1 layer of C channels whose operands are all +1 but for a few: filter f has -1 in its first f channels and, if t is
    ternary and f odd, 0 in channel 2000; pixel 0 is all +1, pixel 1 has -1 in the first 1000 channels, pixel 2 in the first half.
    Returns the result and what it has to be, as whole numbers."""
    PC, wb = C // 64, O.weight_bits(t)
    sign = np.zeros((KN, 32 * 64), bool)
    mag = np.ones((KN, 32 * 64), bool)
    for f in range(KN):
        sign[f, :f] = True
        mag[f, 2000] = wb == 1 or f % 2 == 0
    pack = lambda b: torch.from_numpy(np.packbits(b.reshape(KN, 32, 64), axis=2, bitorder="little").view(np.int64)[..., 0].copy()).to(cuda)
    QW = torch.zeros(KN, 1, 1, PC, wb, dtype=torch.int64, device=cuda)
    if wb == 2:
        QW[..., 1] = -1
        QW[:, 0, 0, :32, 1] = pack(mag)
    QW[:, 0, 0, :32, 0] = pack(sign & mag)
    x = torch.ones(1, 1, 3, C, device=cuda)
    x[0, 0, 1, :1000] = -1.0
    x[0, 0, 2, : C // 2] = -1.0
    y = TAB.Conv2d(x, QW, torch.full((1,), 0.0 if t >= 2 else 0.5, device=cuda), torch.zeros(KN, dtype=torch.int32, device=cuda), t, 0, 0, 1, 1, 1, 1, 3, C, KN, 1, 1)
    f = np.arange(KN, dtype=np.int64)
    zero = np.where(mag[:, 2000], 0, 1)
    want = np.stack([C - zero - 2 * f, C - zero - 2000 - 2 * f + 4 * np.minimum(f, 1000), C - 2 * (C // 2) + zero + 2 * f])
    return y.reshape(3, KN).cpu().numpy(), want


@pytest.mark.parametrize("KN", [17, 64, 128, 256])
def test_sums_just_below_two_to_the_24(cuda, KN, conv_path):
    """4-bit operands accumulate in fp32: exact up to the limit of the dispatch, on tiles of every width."""
    if conv_path != "tensor":
        pytest.skip("the tensor-core kernel")
    y, want = _long_sums(cuda, (1 << 24) - 64, KN, 0)
    assert "e2m1" in _cabi.lib().tab_last_conv_kernel().decode() and np.abs(want).max() > (1 << 24) - 128
    assert np.array_equal(y.astype(np.int64), want) and _cabi.lib().tab_device_status() == 0


@pytest.mark.parametrize("t", [0, 1])
def test_sums_from_two_to_the_24(cuda, t, conv_path):
    """Longer sums are multiplied as bytes on the tensor cores (int32 accumulators, rounded once to fp32)."""
    if conv_path != "tensor":
        pytest.skip("the tensor-core kernel")
    y, want = _long_sums(cuda, (1 << 24) + 64, 5, t)
    name = _cabi.lib().tab_last_conv_kernel().decode()
    assert name.startswith("conv_umma") and "e2m1" not in name
    assert np.array_equal(y, want.astype(np.float32)) and _cabi.lib().tab_device_status() == 0


@pytest.mark.parametrize("geom", [
    # p1 p2 s1 s2  N  H  W   C   KN KH KW       streamed filters, a last round that fills less than half of the SMs
    (1, 1, 1, 1, 90, 14, 14, 256, 256, 3, 3),
    (1, 1, 1, 1, 90, 14, 14, 256, 250, 3, 3),
    (1, 1, 1, 1, 90, 14, 14, 256, 192, 3, 3),
    (0, 0, 1, 1, 52, 14, 14, 512, 384, 1, 1),
])
def test_half_tiles_on_four_bit_operands(cuda, geom, conv_path):
    """Tiles worked as halves (overlapping accumulators for 256 filters): the reported kernel says so, plain and with an fp32 and a
    16-bit residual; results against the byte form, whose halves have a test of their own, and the oracle."""
    if conv_path != "tensor":
        pytest.skip("the tensor-core kernel's own entry point")
    p1, p2, s1, s2, N, H, W, C, KN, KH, KW = geom
    x, ths = make_input(95, N, H, W, C)
    w, wths = make_input(96, KN, KH, KW, C)
    qw, btn = O.quantize(w, wths, 2, KN, KH, KW, C)
    qx = TAB.Quantize(dev_t(x, cuda), dev_t(ths, cuda), 2, N, H, W, C)[0]
    w8 = TAB.ops.expand_weights(dev_t(qw, cuda), 2, KN, KH, KW, C)
    w4 = TAB.ops.pack_weights(w8, KN, KH, KW, C)
    y, _ = TAB.ops.conv2d_bits(qx, w8, 0, *geom)
    n = N - 1
    yo = c_oracle.conv2d(x[n:], qw, ths[n:], btn, 0, p1, p2, s1, s2, 1, H, W, C, KN, KH, KW)
    assert np.array_equal(y.reshape(N, -1)[n].cpu().numpy(), yo.reshape(-1))
    r = torch.round(torch.randn(*y.shape, device=cuda) * 5)
    state = TAB.ops.new_state(N, cuda)
    for residual in (None, r, r.to(torch.int16)):
        for scale in (None, 0.7):
            got = TAB.ops.conv2d_bits(qx, w4, 0, *geom, residual=residual, threshold_scale=scale, state=state)
            name = _cabi.lib().tab_last_conv_kernel().decode()
            assert "<1,256,4,0," in name and ",e2m1>" in name and " halves" in name, name
            want = y if residual is None else y + r
            assert torch.equal(got[0], want)
            if scale:
                t = (float(np.float32(0.7)) * (want.double().abs().reshape(N, -1).sum(dim=1) / want[0].numel())).float()
                assert torch.equal(got[1], t)                              # whole numbers: exact sums, rounded once
    assert _cabi.lib().tab_device_status() == 0


@pytest.mark.parametrize("H,C,KN,K,resident", [(14, 256, 64, 3, 1), (14, 128, 64, 5, 1), (16, 64, 64, 7, 1), (7, 512, 512, 3, 0), (7, 300, 100, 3, 0)])
def test_tile_rule_for_single_small_images(cuda, H, C, KN, K, resident, conv_path):
    """Narrower tiles are not taken where that would turn filters that stay in shared memory into streamed ones."""
    if conv_path != "tensor":
        pytest.skip("the tensor-core kernel")
    x, ths = make_input(21, 1, H, H, C)
    w, wths = make_input(22, KN, K, K, C)
    qw, btn = O.quantize(w, wths, 2, KN, K, K, C)
    geom = (K // 2, K // 2, 1, 1, 1, H, H, C, KN, K, K)
    assert np.array_equal(gpu_conv(cuda, x, qw, ths, btn, 0, *geom), c_oracle.conv2d(x, qw, ths, btn, 0, *geom))
    assert _cabi.lib().tab_last_conv_kernel().decode().startswith("conv_umma_persist_kernel<1,64,6,%d," % resident)


def test_sums_of_more_images_than_one_quantiser_launch_takes(cuda, conv_path):
    """|y| sums and next thresholds of 66000 one-pixel images, into a buffer that holds something else."""
    N, C, KN = 66000, 64, 5
    x, ths = make_input(31, N, 1, 1, C)
    w, wths = make_input(32, KN, 1, 1, C)
    qw, btn = O.quantize(w, wths, 2, KN, 1, 1, C)
    lib, geom = _cabi.lib(), (0, 0, 0, 1, 1, N, 1, 1, C, KN, 1, 1)
    xd, td, qd, bd = (dev_t(a, cuda) for a in (x, ths, qw, btn))
    y = torch.empty(N * KN, device=cuda)
    ws = torch.empty(lib.tab_conv2d_workspace_bytes(*geom), dtype=torch.uint8, device=cuda)
    sums, nxt = torch.full((N,), 1e9, dtype=torch.float64, device=cuda), torch.empty(N, device=cuda)
    stream = torch.cuda.current_stream(cuda).cuda_stream
    _cabi.check(lib.tab_conv2d_chain_launch(xd.data_ptr(), qd.data_ptr(), td.data_ptr(), bd.data_ptr(), y.data_ptr(), ws.data_ptr(), ws.numel(), *geom,
                                            None, sums.data_ptr(), nxt.data_ptr(), 0.7, stream), "chain")
    yo = c_oracle.conv2d(x, qw, ths, btn, *geom).reshape(N, KN)
    assert np.array_equal(y.cpu().numpy().reshape(N, KN), yo)
    total = np.abs(yo.astype(np.float64)).sum(axis=1)
    assert np.array_equal(sums.cpu().numpy(), total)
    assert np.array_equal(nxt.cpu().numpy(), (np.float64(np.float32(0.7)) * (total / KN)).astype(np.float32))
