// tab_b200._host: the bodies of tab_b200.ops' operators - checks, output and scratch allocation, one C-ABI call - in native code.
//
// A small convolution takes the device less time than the interpreter needs to check sixteen arguments, allocate two tensors
// and convert twenty values for a foreign call (about 20 us); here that is 2-3 us.  Every function returns None for arguments
// that are anything but plainly valid (wrong device, dtype, size; an empty result; an error code of the C ABI): the caller
// then runs its own body, which names what is wrong or does the rare case, so that there is one set of messages.
#include <torch/extension.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include "../../include/tab_b200.h"

namespace {

using at::Tensor;
using OptTensor = c10::optional<Tensor>;

bool plain(const Tensor& t, at::ScalarType dtype) { return t.defined() && t.is_cuda() && t.is_contiguous() && t.scalar_type() == dtype; }
tab_stream_t stream_of(const Tensor& t) { return reinterpret_cast<tab_stream_t>(at::cuda::getCurrentCUDAStream(t.get_device()).stream()); }
Tensor make(const Tensor& like, at::IntArrayRef size, at::ScalarType dtype) { return at::empty(size, like.options().dtype(dtype)); }

// n elements are the product of the sizes.  Sizes come from the caller one by one: their product may leave 64 bits, and a wrapped
// one must not pass for the size of a small tensor.
bool holds(int64_t n, std::initializer_list<int64_t> sizes) {
    int64_t product = 1;
    for (const int64_t s : sizes)
        if (__builtin_mul_overflow(product, s, &product)) return false;
    return n == product;
}

struct Conv {
    int type, p1, p2, s1, s2, N, H, W, C, KN, KH, KW;
    int64_t OH = 0, OW = 0, PC = 0;
    // Valid sizes with a result that is not empty.
    bool good() {
        if (type < 0 || type > 3 || N < 1 || H < 1 || W < 1 || C < 1 || KN < 1 || KH < 1 || KW < 1 || p1 < 0 || p2 < 0 || s1 < 1 || s2 < 1) return false;
        OH = ((int64_t)H + 2 * (int64_t)p1 - KH + 1) / s1;
        OW = ((int64_t)W + 2 * (int64_t)p2 - KW + 1) / s2;
        PC = ((int64_t)C + 63) / 64;
        return OH > 0 && OW > 0;
    }
    // n elements are `per_word` for each packed word of the weights, `per_pixel` for each pixel of the activations, the results.
    bool weights(int64_t n, int64_t per_word) const { return holds(n, {KN, KH, KW, PC, per_word}); }
    bool activations(int64_t n, int64_t per_pixel) const { return holds(n, {N, H, W, per_pixel}); }
    bool results(int64_t n) const { return holds(n, {N, KN, OH, OW}); }
};

py::object quantize(const Tensor& X, const Tensor& ths, int bitwidth, int N, int H, int W, int C) {
    Tensor QX, BTN;
    {
        py::gil_scoped_release nogil;
        if (plain(X, at::kFloat) && plain(ths, at::kFloat) && N >= 1 && H >= 1 && W >= 1 && C >= 1 && bitwidth >= 1 &&
            holds(X.numel(), {N, H, W, C}) && ths.numel() == N) {
            const c10::cuda::CUDAGuard guard(X.device());
            QX = make(X, {N, H, W, ((int64_t)C + 63) / 64, bitwidth == 1 ? 1 : 2}, at::kLong);
            BTN = make(X, {N}, at::kInt);
            if (tab_quantize_launch(X.data_ptr<float>(), ths.data_ptr<float>(), QX.data_ptr<int64_t>(), BTN.data_ptr<int32_t>(),
                                    bitwidth, N, H, W, C, stream_of(X)) != TAB_OK) QX.reset();
        }
    }
    if (!QX.defined()) return py::none();
    py::list out(2);
    out[0] = QX; out[1] = BTN;
    return out;
}

py::object conv2d(const Tensor& X, const Tensor& QW, const Tensor& ths, const Tensor& btn, int type, int p1, int p2, int s1, int s2,
                  int N, int H, int W, int C, int KN, int KH, int KW) {
    Tensor Y;
    {
        py::gil_scoped_release nogil;
        Conv g{type, p1, p2, s1, s2, N, H, W, C, KN, KH, KW};
        if (g.good() && plain(X, at::kFloat) && plain(QW, at::kLong) && plain(ths, at::kFloat) && plain(btn, at::kInt) &&
            g.weights(QW.numel(), type == 1 || type == 3 ? 1 : 2) && (type != 2 || btn.numel() == KN) &&
            g.activations(X.numel(), C) && ths.numel() == N) {
            const c10::cuda::CUDAGuard guard(X.device());
            Y = make(X, {N, KN, g.OH, g.OW}, at::kFloat);
            const size_t bytes = tab_conv2d_workspace_bytes(type, p1, p2, s1, s2, N, H, W, C, KN, KH, KW);
            Tensor ws = make(X, {(int64_t)std::max<size_t>(bytes, 256)}, at::kByte);
            if (tab_conv2d_launch(X.data_ptr<float>(), QW.data_ptr<int64_t>(), ths.data_ptr<float>(), btn.data_ptr<int32_t>(), Y.data_ptr<float>(),
                                  ws.data_ptr(), (size_t)ws.numel(), type, p1, p2, s1, s2, N, H, W, C, KN, KH, KW, stream_of(X)) != TAB_OK) Y.reset();
        }
    }
    return Y.defined() ? py::cast(Y) : py::none();
}

// state: zeroed, of tab_conv2d_state_bytes(N) bytes.
py::object quantize_auto(const Tensor& X, double scale, int bitwidth, int N, int H, int W, int C, const Tensor& state) {
    Tensor QX, ths;
    {
        py::gil_scoped_release nogil;
        if (plain(X, at::kFloat) && N >= 1 && H >= 1 && W >= 1 && C >= 1 && bitwidth >= 1 && holds(X.numel(), {N, H, W, C}) &&
            state.defined() && state.is_cuda()) {
            const c10::cuda::CUDAGuard guard(X.device());
            QX = make(X, {N, H, W, ((int64_t)C + 63) / 64, bitwidth == 1 ? 1 : 2}, at::kLong);
            ths = make(X, {N}, at::kFloat);
            if (tab_quantize_auto_launch(X.data_ptr<float>(), (float)scale, state.data_ptr(), ths.data_ptr<float>(), QX.data_ptr<int64_t>(), bitwidth,
                                         N, H, W, C, stream_of(X)) != TAB_OK) QX.reset();
        }
    }
    if (!QX.defined()) return py::none();
    return py::make_tuple(QX, ths);
}

// Byte weights of several layers -> their 4-bit operands, parts of one allocation.
py::object pack_weights(const std::vector<Tensor>& W8) {
    std::vector<Tensor> W4;
    {
        py::gil_scoped_release nogil;
        std::vector<int64_t> sizes;
        int64_t total = 0;
        for (const Tensor& w : W8) {
            if (!plain(w, at::kChar) || w.numel() == 0 || w.numel() % 64 != 0 || w.device() != W8[0].device()) break;
            sizes.push_back(w.numel() / 2);
            total += w.numel() / 2;
        }
        if (!W8.empty() && sizes.size() == W8.size()) {
            const c10::cuda::CUDAGuard guard(W8[0].device());
            W4 = make(W8[0], {total}, at::kByte).split_with_sizes(sizes);
            std::vector<const int8_t*> from;
            std::vector<uint8_t*> to;
            std::vector<long long> words;
            for (size_t i = 0; i < W8.size(); i++) {
                from.push_back(W8[i].data_ptr<int8_t>());
                to.push_back(W4[i].data_ptr<uint8_t>());
                words.push_back(sizes[i] / 32);
            }
            if (tab_pack_weights_many_launch((int)W8.size(), from.data(), to.data(), words.data(), stream_of(W8[0])) != TAB_OK) W4.clear();
        }
    }
    if (W4.empty()) return py::none();
    return py::cast(W4);
}

// The GEMM stage on 4-bit weights (ops.conv2d_bits with uint8 weights), or on byte weights that the call packs first.
py::object conv2d_packed4(const Tensor& QX, const Tensor& weights, int type, int p1, int p2, int s1, int s2, int N, int H, int W, int C, int KN, int KH, int KW,
                          const OptTensor& residual, c10::optional<double> threshold_scale, const OptTensor& state, bool out_int16,
                          c10::optional<int> next_bitwidth) {
    Tensor Y, nxt, QN;
    int rc = TAB_OK;
    {
        py::gil_scoped_release nogil;
        Conv g{type, p1, p2, s1, s2, N, H, W, C, KN, KH, KW};
        const bool want = threshold_scale.has_value();
        if (g.good() && plain(QX, at::kLong) && (plain(weights, at::kByte) || (plain(weights, at::kChar) && weights.device() == QX.device())) && g.activations(QX.numel(), g.PC * (type == 2 || type == 3 ? 1 : 2)) &&
            g.weights(weights.numel(), weights.scalar_type() == at::kByte ? 32 : 64) && (!residual.has_value() || ((plain(*residual, at::kShort) || (!out_int16 && plain(*residual, at::kFloat))) && g.results(residual->numel()))) &&
            (!want || (state.has_value() && state->defined() && state->is_cuda())) && (!next_bitwidth.has_value() || want)) {
            const c10::cuda::CUDAGuard guard(QX.device());
            const int nb = next_bitwidth.has_value() ? (*next_bitwidth == 1 ? 1 : 2) : 0;
            Y = make(QX, {N, KN, g.OH, g.OW}, out_int16 ? at::kShort : at::kFloat);
            if (want) nxt = make(QX, {N}, at::kFloat);
            if (nb) QN = make(QX, {N, g.OH, g.OW, ((int64_t)KN + 63) / 64, nb}, at::kLong);
            Tensor W4 = weights;
            if (weights.scalar_type() == at::kChar) {
                W4 = make(weights, {weights.numel() / 2}, at::kByte);
                rc = tab_pack_weights_launch(weights.data_ptr<int8_t>(), W4.data_ptr<uint8_t>(), KN, KH, KW, C, stream_of(QX));
            }
            if (rc == TAB_OK) rc = tab_conv2d_packed4_launch(QX.data_ptr<int64_t>(), W4.data_ptr<uint8_t>(), Y.data_ptr(), out_int16 ? 1 : 0, type, p1, p2, s1, s2,
                                          N, H, W, C, KN, KH, KW, residual.has_value() ? residual->data_ptr() : nullptr, residual.has_value() && residual->scalar_type() == at::kShort ? 1 : 0,
                                          want ? state->data_ptr() : nullptr, want ? nxt.data_ptr<float>() : nullptr,
                                          want ? (float)*threshold_scale : 0.f, nb ? QN.data_ptr<int64_t>() : nullptr, nb, stream_of(QX));
            if (rc != TAB_OK) Y.reset();
        }
    }
    if (rc == TAB_E_TOO_LARGE) return py::int_(rc);                         // the caller need not find that out again
    if (!Y.defined()) return py::none();
    py::object th = nxt.defined() ? py::cast(nxt) : py::none();
    if (QN.defined()) return py::make_tuple(Y, th, QN);
    return py::make_tuple(Y, th);
}

// Both launches of a layer kept as byte weights: quantiser (against the thresholds given, or against those it finds) with the
// weights packed on the side, then the GEMM stage.
py::object layer(const Tensor& X, const Tensor& W8, int type, int p1, int p2, int s1, int s2, int N, int H, int W, int C, int KN, int KH, int KW,
                 const OptTensor& thresholds, double scale, const OptTensor& state) {
    Tensor Y;
    {
        py::gil_scoped_release nogil;
        Conv g{type, p1, p2, s1, s2, N, H, W, C, KN, KH, KW};
        if (g.good() && plain(X, at::kFloat) && plain(W8, at::kChar) && W8.device() == X.device() && g.activations(X.numel(), C) && g.weights(W8.numel(), 64) &&
            (thresholds.has_value() ? plain(*thresholds, at::kFloat) && thresholds->numel() == N : state.has_value() && state->defined() && state->is_cuda())) {
            const c10::cuda::CUDAGuard guard(X.device());
            if (tab_conv2d_packed4_covers(type, p1, p2, s1, s2, N, H, W, C, KN, KH, KW)) {
                const int bits = type == 2 || type == 3 ? 1 : 2;
                const bool find = !thresholds.has_value();
                Tensor QX = make(X, {N, H, W, g.PC, bits}, at::kLong), W4 = make(X, {W8.numel() / 2}, at::kByte), found;
                if (find) found = make(X, {N}, at::kFloat);
                Y = make(X, {N, KN, g.OH, g.OW}, at::kFloat);
                int rc = tab_quantize_pack_launch(X.data_ptr<float>(), find ? nullptr : thresholds->data_ptr<float>(), (float)scale, find ? state->data_ptr() : nullptr,
                                                  find ? found.data_ptr<float>() : nullptr, QX.data_ptr<int64_t>(), bits, N, H, W, C, W8.data_ptr<int8_t>(),
                                                  W4.data_ptr<uint8_t>(), W8.numel() / 64, stream_of(X));
                if (rc == TAB_OK) rc = tab_conv2d_packed4_launch(QX.data_ptr<int64_t>(), W4.data_ptr<uint8_t>(), Y.data_ptr(), 0, type, p1, p2, s1, s2, N, H, W, C,
                                                                 KN, KH, KW, nullptr, 0, nullptr, nullptr, 0.f, nullptr, 0, stream_of(X));
                if (rc != TAB_OK) Y.reset();
            }
        }
    }
    return Y.defined() ? py::cast(Y) : py::none();
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
    m.def("quantize", &quantize);
    m.def("conv2d", &conv2d);
    m.def("quantize_auto", &quantize_auto);
    m.def("layer", &layer);
    m.def("pack_weights", &pack_weights);
    m.def("conv2d_packed4", &conv2d_packed4);
}
