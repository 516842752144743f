"""``tab_b200.nn.TABConv2d`` (prepared weights, the caller above the raw operators) and the chain written on it,
against the CPU oracle: bit-exact."""
import numpy as np
import pytest
import torch

import tab_b200 as TAB
from tab_b200 import _cabi, chain, nn as tab_nn
from oracle import c_oracle, tab_oracle as O
from oracle.oracle_ops import OracleOps
from util import make_input

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t", range(4))
@pytest.mark.parametrize("geom", [
    # pad stride N  H   W   C   KN K
    (1, 1, 3, 14, 14, 256, 96, 3),
    (0, 2, 2, 28, 28, 128, 256, 1),
    (1, 2, 2, 15, 11, 70, 33, 3),
    (3, 2, 1, 40, 40, 3, 16, 7),
])
def test_module_matches_oracle(cuda, t, geom):
    pad, stride, N, H, W, C, KN, K = geom
    x, ths = make_input(31, N, H, W, C)
    w, wths = make_input(32, KN, K, K, C)
    m = tab_nn.TABConv2d.from_float(torch.from_numpy(w).to(cuda), t, pad, stride, torch.from_numpy(wths).to(cuda))
    qw, btn = O.quantize(w, wths, O.weight_bits(t), KN, K, K, C)
    assert np.array_equal(m.QW.cpu().numpy().reshape(-1), qw.reshape(-1)) and np.array_equal(m.BTN_W.cpu().numpy(), btn)
    y = m(torch.from_numpy(x).to(cuda), torch.from_numpy(ths).to(cuda))
    yo = c_oracle.conv2d(x, qw, ths, btn, t, pad, pad, stride, stride, N, H, W, C, KN, K, K)
    assert tuple(y.shape) == yo.shape and np.array_equal(y.cpu().numpy(), yo)
    # thresholds computed by the module when none are passed: 0.7 * mean|x| per image, in double
    y2 = m(torch.from_numpy(x).to(cuda))
    tho = OracleOps.residual_threshold(x.copy(), None, 0.7)
    assert np.array_equal(y2.cpu().numpy(), c_oracle.conv2d(x, qw, tho, btn, t, pad, pad, stride, stride, N, H, W, C, KN, K, K))
    assert _cabi.lib().tab_device_status() == 0


def test_module_rejects_weights_of_the_wrong_bitwidth(cuda):
    """The reference's notebook passes 1-bit weights to 2-bit types (an out-of-bounds read there); here it is an error."""
    w, wths = make_input(1, 8, 3, 3, 64)
    q1, b1 = TAB.Quantize(torch.from_numpy(w).to(cuda), torch.from_numpy(wths).to(cuda), 1, 8, 3, 3, 64)
    with pytest.raises(ValueError, match="bitwidth 2"):
        tab_nn.TABConv2d(q1, b1, 0, 8, 3, 3, 64, 1, 1)
    tab_nn.TABConv2d(q1, b1, 1, 8, 3, 3, 64, 1, 1)          # the same weights are right for TBN


@pytest.mark.parametrize("t", [0, 3])
def test_prepared_chain_matches_oracle(cuda, t):
    """The 19-convolution chain on prepared modules (one quantised tensor per input, shared with the shortcut; residual and
    thresholds in the epilogue; one state block reused by every layer), N = 3, N(0,1) input like the benchmark's: the
    oracle gets the input thresholds the device computed, every later threshold follows from the data."""
    N = 3
    rng = np.random.default_rng(8)
    x = rng.standard_normal((N, 56, 56, 64), dtype=np.float32)
    weights = chain.make_weights(2000, t)
    specs = {cs.name: cs for cs in chain.conv_specs()}
    convs = {}
    for name, (w, wt) in weights.items():
        cs = specs[name]
        convs[name] = tab_nn.TABConv2d.from_float(torch.from_numpy(w).to(cuda), t, cs.pad, cs.stride, torch.from_numpy(wt).to(cuda))

    class Nhwc:
        def __init__(self, c):
            self.c = c
            self.conv_type = c.conv_type

        def quantize(self, xx, th):
            return self.c.quantize(xx, th)

        def conv_bits(self, *a, **k):
            out = self.c.conv_bits(*a, **k)
            y = out[0]
            return (y.view(y.shape[0], y.shape[2], y.shape[3], y.shape[1]),) + tuple(out[1:])

    xd = torch.from_numpy(x).to(cuda)
    thd = TAB.ops.residual_threshold(xd.reshape(N, -1), None, chain.THRESHOLD_SCALE)
    qo = chain.quantize_weights(weights, t, OracleOps.Quantize)
    yo, _, _, _ = chain.forward(OracleOps, x, thd.cpu().numpy(), qo, t, N)
    for compact in (False, True):                                      # fp32 everywhere / int16 between a block's two convolutions
        for fused_quant in (False, True):                              # quantiser launches / every convolution hands on its quantised result
            yd, oh, ow, kn = chain.forward_prepared({k: Nhwc(v) for k, v in convs.items()}, xd, thd, N, compact_mid=compact, fused_quant=fused_quant)
            assert (oh, ow, kn) == (7, 7, 512)
            assert np.array_equal(yd.cpu().numpy().reshape(-1), np.asarray(yo).reshape(-1)), (compact, fused_quant)
    # the modules themselves: 16-bit block results from the first strided shortcut on
    yd, _, _, _ = chain.forward_prepared(convs, xd, thd, N, compact_mid=True, fused_quant=True)
    assert yd.dtype == torch.float32 and np.array_equal(yd.cpu().numpy().reshape(-1), np.asarray(yo).reshape(-1))
    reps = 85                                                          # enough images for them to be used, against the fp32 hand-over
    xl, tl = xd.repeat(reps, 1, 1, 1).contiguous(), thd.repeat(reps).contiguous()
    seen = []
    plain = tab_nn.TABConv2d.conv_bits
    try:
        tab_nn.TABConv2d.conv_bits = lambda self, *a, **k: (seen.append(a[4] is not None and a[4].dtype == torch.int16 if len(a) > 4 else False), plain(self, *a, **k))[1]
        yl, _, _, _ = chain.forward_prepared(convs, xl, tl, N * reps, compact_mid=True, fused_quant=True)
    finally:
        tab_nn.TABConv2d.conv_bits = plain
    assert any(seen) and torch.equal(yl.reshape(reps, -1), yd.reshape(1, -1).expand(reps, -1))
    assert _cabi.lib().tab_device_status() == 0


def test_native_bodies_equal_the_python_ones(cuda):
    """``tab_b200._host`` against the Python bodies of the same operators, including what it leaves to them (sizes that are no
    plain integers, empty results, arguments that are refused)."""
    from tab_b200 import ops
    assert ops._host(), "tab_b200._host has not been built"

    def both(fn):
        native = fn()
        saved, ops._native = ops._native, False
        try:
            python = fn()
        finally:
            ops._native = saved
        flat = lambda r: [r] if isinstance(r, torch.Tensor) else list(r)
        a, b = flat(native), flat(python)
        assert type(native) is type(python) and len(a) == len(b)
        for u, v in zip(a, b):
            assert (u is None and v is None) or (u.dtype == v.dtype and u.shape == v.shape and u.device == v.device and torch.equal(u, v))
        return native

    N, H, W, C, KN, K = 3, 9, 8, 130, 70, 3
    x, ths = make_input(1, N, H, W, C)
    w, wths = make_input(2, KN, K, K, C)
    xd, td, wd, wtd = (torch.from_numpy(a).to(cuda) for a in (x, ths, w, wths))
    state = ops.new_state(N, cuda)
    for t in range(4):
        QW, btn = both(lambda: ops.Quantize(wd, wtd, O.weight_bits(t), KN, K, K, C))
        for geom in ((1, 1, 1, 1, N, H, W, C, KN, K, K), (0, 2, 2, 1, np.int64(N), H, float(W), C, KN, K, K)):
            both(lambda: ops.Conv2d(xd, QW, td, btn, t, *geom))
        QX, _ = both(lambda: ops.quantize_auto(xd, 0.7, O.act_bits(t), N, H, W, C, state))
        W4 = ops.pack_weights(ops.expand_weights(QW, O.weight_bits(t), KN, K, K, C), KN, K, K, C)
        g = (1, 1, 1, 1, N, H, W, C, KN, K, K)
        r = torch.randn(N, KN, H, W, device=cuda)
        for kw in (dict(), dict(residual=r), dict(threshold_scale=0.7, state=state), dict(threshold_scale=0.7, state=state, out_int16=True, next_bitwidth=2),
                   dict(residual=r, threshold_scale=0.7, state=state, next_bitwidth=1)):
            both(lambda: ops.conv2d_bits(QX, W4, t, *g, **kw))
    assert both(lambda: ops.Conv2d(xd, QW, td, btn, 3, 0, 0, 1, 1, N, H, W, C, KN, K, K)).numel() == N * KN * (H - 2) * (W - 2)
    assert ops.Quantize(torch.empty(0, device=cuda), torch.empty(0, device=cuda), 2, 0, 4, 4, 64)[0].numel() == 0
    with pytest.raises(RuntimeError, match="X has"):
        ops.Quantize(xd, td, 2, N, H, W + 1, C)
    with pytest.raises(RuntimeError, match="QX must have dtype"):
        ops.conv2d_bits(xd, W4, 3, *g)


def test_module_weights_follow_a_loaded_state(cuda):
    """``load_state_dict`` replaces the weights, the 4-bit form among them; the state itself holds what it always held."""
    N, H, W, C, KN = 2, 10, 9, 70, 40
    x = torch.randn(N, H, W, C, device=cuda)
    a = tab_nn.TABConv2d.from_float(torch.randn(KN, 3, 3, C, device=cuda), 0, 1, 1)
    b = tab_nn.TABConv2d.from_float(torch.randn(KN, 3, 3, C, device=cuda), 0, 1, 1)
    assert sorted(a.state_dict()) == ["BTN_W", "QW", "W8"] and not torch.equal(a(x), b(x))
    b.load_state_dict(a.state_dict())
    assert torch.equal(a(x), b(x))


def _pair(cuda, N=2, H=10, W=9, C=70, KN=40):
    """An input and two layers of one geometry with different weights."""
    make = lambda: tab_nn.TABConv2d.from_float(torch.randn(KN, 3, 3, C, device=cuda), 0, 1, 1)
    return torch.randn(N, H, W, C, device=cuda), make(), make()


@pytest.mark.parametrize("write", [
    lambda a, b: a.W8.copy_(b.W8),
    lambda a, b: a.state_dict()["W8"].copy_(b.W8),
    lambda a, b: a.W8.data.copy_(b.W8),                                    # no version counter sees this one
    lambda a, b: a.W8.data.view(torch.int64).copy_(b.W8.view(torch.int64)),
    lambda a, b: setattr(a, "W8", b.W8.clone()),
    lambda a, b: a._buffers.__setitem__("W8", b.W8),
], ids=["copy_", "state_dict", "data", "reinterpreted", "assigned", "buffers"])
def test_module_multiplies_the_registered_weights(cuda, write):
    """``W8`` is what a call multiplies, whoever wrote it and however; also the one pass that packs all layers at once."""
    x, a, b = _pair(cuda)
    old, want = a(x), b(x)
    assert not torch.equal(old, want)
    write(a, b)
    assert torch.equal(a(x), want)
    assert "e2m1" in _cabi.lib().tab_last_conv_kernel().decode()
    kw = tab_nn.TABConv2d.pack_together({"a": a, "b": b})
    qx = a.quantize(x)
    assert sorted(kw) == ["a", "b"]
    for k in kw:
        assert torch.equal(a.conv_bits(qx, 2, 10, 9, **kw[k])[0], want)
    from tab_b200 import ops
    saved, ops._native = ops._native, False
    try:                                                                   # the Python body of the same
        for w, k in zip(ops.pack_weights_many([a.W8, b.W8]), kw):
            assert torch.equal(w, kw[k]["packed"])
        assert torch.equal(a(x), want)
    finally:
        ops._native = saved
    assert ops.pack_weights_many([a.W8, b.W8.cpu()]) is None and ops.pack_weights_many([]) is None


def test_captured_module_follows_its_weights(cuda):
    """A captured pass multiplies what ``W8`` holds when it is replayed, as it did when ``W8`` itself was the operand."""
    x, a, b = _pair(cuda)
    want = b(x)
    a(x)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        y = a(x)
    a.W8.copy_(b.W8)
    g.replay()
    assert torch.equal(y, want)
    a.load_state_dict(tab_nn.TABConv2d.from_float(torch.randn(40, 3, 3, 70, device=cuda), 0, 1, 1).state_dict())
    g.replay()
    assert torch.equal(y, a(x)) and not torch.equal(y, want)


def test_module_copies_and_moves(cuda):
    """Deep copies, pickles (also ones that hold the derived form older versions kept) and weights that were loaded while the
    module was on the CPU give the same results on the same kernel."""
    import copy
    import pickle
    x, a, b = _pair(cuda)
    want = a(x)
    old = pickle.loads(pickle.dumps(a))
    old._buffers["W4"] = torch.zeros(8, dtype=torch.uint8, device=cuda)
    old._non_persistent_buffers_set.add("W4")
    b.cpu()
    b.load_state_dict(a.state_dict())
    b.to(cuda)
    for m in (copy.deepcopy(a), pickle.loads(pickle.dumps(old)), b):
        assert torch.equal(m(x), want) and "e2m1" in _cabi.lib().tab_last_conv_kernel().decode()
        assert [n for n, _ in m.named_buffers()] == ["QW", "BTN_W", "W8"]


def test_sizes_whose_product_leaves_64_bits_are_refused(cuda):
    """N*H*W*C = 2**64 + 96, and the bytes of its bit-planes are small modulo 2**64 too: a tensor of 96 elements is not taken for
    that.  (The checks are made on exact products; the call ends on the host, before anything is launched.)"""
    from tab_b200 import ops
    N, H, W, C = 1117667411, 5531, 373004, 8
    assert N * H * W * C - 2 ** 64 == 96
    ths = torch.empty(N, device=cuda)
    QW = torch.zeros(1, 1, 1, 1, 2, dtype=torch.int64, device=cuda)
    with pytest.raises(RuntimeError, match="X has 96 elements"):
        ops.Conv2d(torch.zeros(96, device=cuda), QW, ths, torch.zeros(1, dtype=torch.int32, device=cuda), 0, 0, 0, H, W, N, H, W, C, 1, 1, 1)
    with pytest.raises(RuntimeError, match="X has 96 elements"):
        ops.Quantize(torch.zeros(96, device=cuda), ths, 2, N, H, W, C)


@pytest.mark.parametrize("geom", [
    # pad stride N  H   W   C   KN K
    (1, 1, 1, 7, 7, 512, 512, 3),              # few words, many weights: CTAs that have only weights
    (1, 1, 2, 3, 5, 1, 1, 3),
    (0, 1, 70, 9, 9, 70, 20, 1),
    (1, 2, 64, 28, 28, 128, 96, 3),            # more words than CTAs
    (3, 1, 1, 150, 150, 64, 8, 7),             # not covered by the tensor-core kernel
])
@pytest.mark.parametrize("t", range(4))
def test_layer_in_two_launches_equals_its_stages(cuda, t, geom):
    pad, stride, N, H, W, C, KN, K = geom
    x = torch.randn(N, H, W, C, device=cuda)
    m = tab_nn.TABConv2d.from_float(torch.randn(KN, K, K, C, device=cuda), t, pad, stride)
    ths = torch.rand(N, device=cuda)
    for _ in range(2):
        assert torch.equal(m(x, ths), m.conv_bits(m.quantize(x, ths), N, H, W)[0])
        assert torch.equal(m(x), m.conv_bits(m.quantize(x), N, H, W)[0])
    W8 = m.W8
    y = TAB.ops.layer(x, W8, t, *m.geometry(N, H, W), ths, 0.7, None)
    assert (y is None) == (K == 7 and H == 150) and not m.state(N, cuda).any()
    qw = TAB.ops.pack_weights(W8, KN, K, K, C)
    assert torch.equal(TAB.ops.pack_weights_many([W8])[0], qw.view(-1))
    assert _cabi.lib().tab_device_status() == 0


def test_layer_with_stages_of_its_own(cuda):
    """A subclass that overrides a stage has it called."""
    calls = []

    class Mine(tab_nn.TABConv2d):
        def conv_bits(self, *a, **k):
            calls.append("conv_bits")
            return super().conv_bits(*a, **k)

    x = torch.randn(2, 6, 6, 64, device=cuda)
    w = torch.randn(8, 3, 3, 64, device=cuda)
    assert torch.equal(Mine.from_float(w, 0, 1, 1)(x), tab_nn.TABConv2d.from_float(w, 0, 1, 1)(x)) and calls == ["conv_bits"]
    m = tab_nn.TABConv2d.from_float(w, 0, 1, 1)
    for bad, message in ((x.double(), "float32"), (x.cpu(), "CUDA")):
        with pytest.raises(RuntimeError, match=message):
            m(bad, torch.ones(2, device=cuda))
    with pytest.raises(RuntimeError, match="thresholds has"):
        m(x, torch.ones(3, device=cuda))


def test_pack_together_asks_whether_a_layer_takes_it(cuda):
    """Subclasses whose ``conv_bits`` passes keywords on get the packed weights, ones with a signature of their own do not."""
    class Passing(tab_nn.TABConv2d):
        def conv_bits(self, *a, **k):
            return super().conv_bits(*a, **k)

    class Own(tab_nn.TABConv2d):
        def conv_bits(self, QX, N, H, W, residual=None, next_threshold_scale=None):
            return super().conv_bits(QX, N, H, W, residual, next_threshold_scale)

    w = torch.randn(8, 3, 3, 64, device=cuda)
    layers = {kind.__name__: kind.from_float(w, 0, 1, 1) for kind in (tab_nn.TABConv2d, Passing, Own)}
    kw = tab_nn.TABConv2d.pack_together(layers)
    assert sorted(kw) == ["Passing", "TABConv2d"]
    bare = tab_nn.TABConv2d.from_float(w, 0, 1, 1)
    w8 = bare.W8
    del bare.W8
    bare.__dict__["W8"] = w8                                               # no buffer any more: conv_bits packs it
    assert tab_nn.TABConv2d.pack_together({"bare": bare}) == {}
    qx = layers["Own"].quantize(torch.randn(2, 6, 6, 64, device=cuda))
    ys = [m.conv_bits(qx, 2, 6, 6, **kw.get(k, {}))[0] for k, m in layers.items()]
    assert torch.equal(ys[0], ys[1]) and torch.equal(ys[0], ys[2])
