// Threshold-quantise fp32 NHWC data into bit-planes packed 64 channels per 64-bit word, in one pass,
// with the per-n popcount of the magnitude plane folded in.
//
// Replaces the reference's TerOnlyKernel (TAB_GEMM.cu:163-208), BinOnlyKernel (:211-247) and
// BTN_Weight (:150-160).  Encoding (TAB_GEMM.cu:184-206, :231-245): ternary x > t -> (sign 0, mag 1),
// else x < -t -> (1, 1), else (0, 0); binary bit = (x < t); channel c is bit c%64 of word c/64.
//
// The kernel is HBM-bound: 4 bytes read per element, 2 or 1 bits written.  Fast path (C % 64 == 0,
// 32-byte aligned input): eight lanes own one 64-channel word; each lane issues QUNROLL independent
// 256-bit loads before it touches any of them, so a resident SM keeps > 200 KB in flight; a lane turns
// its 8 channels into one byte per plane with compares and predicated ORs and stores those bytes
// itself - no shuffles, votes or redux (a first version merged nibbles with redux.sync and was bound
// by that instruction's pipe at 37 % of DRAM bandwidth).
// Any other C or alignment: the same division of labour with the widest loads the rows allow (quantize_any_kernel).
//
// Inside a convolution call the same launch also does the call's small set-up jobs (QuantExtras), so that they cost no
// launch of their own: all CTAs share the expansion of the packed weights to the bytes the tensor-core kernel
// multiplies, and the first CTA of every image clears that image's |y| sum (the first of all the completion counter).
#include <algorithm>
#include <mutex>
#include "tab_kernels.cuh"
#include "umma_common.cuh"

namespace tab {

constexpr int QTHREADS = 256;
constexpr int QUNROLL = 4;                                   // independent 256-bit loads per lane
constexpr int QWORDS_PER_ITER = (QTHREADS / 8) * QUNROLL;    // 128 words = 32 KB of fp32 per CTA step

struct f8 { float v[8]; };

// One thread per (filter, word k, 16-channel group) of packed weights [KN][KH*KW*PC][WB]: 16 bytes of {-1,0,+1}
// into [KN][KH*KW*PC][64]; channels beyond C become 0.
template <int WB>
__device__ __forceinline__ void expand_group(const uint64_t* __restrict__ qw, int8_t* __restrict__ w8, long long idx, int PC, int C) {
    const long long word = idx >> 2;
    const int grp = (int)(idx & 3);
    uint32_t s16, m16;
    if (WB == 2) {
        const uint64_t sg = __ldg(qw + word * 2), mg = __ldg(qw + word * 2 + 1);
        m16 = (uint32_t)(mg >> (grp * 16)) & 0xFFFFu;
        s16 = (uint32_t)(sg >> (grp * 16));
    } else {
        m16 = 0xFFFFu;
        s16 = (uint32_t)(__ldg(qw + word) >> (grp * 16));                  // bit = 1 means -1
    }
    if (C & 63) {                                                          // only then is there a word with a tail, the last of PC
        const int pc = word < (1LL << 31) ? (int)((uint32_t)word % (uint32_t)PC) : (int)(word % PC);
        const int real = C - (pc * 64 + grp * 16);
        if (real < 16) m16 &= real > 0 ? (1u << real) - 1u : 0u;
    }
    s16 &= m16;
    *reinterpret_cast<uint4*>(w8 + word * 64 + grp * 16) =
        make_uint4(expand4(m16 & 15u, s16 & 15u), expand4((m16 >> 4) & 15u, (s16 >> 4) & 15u),
                   expand4((m16 >> 8) & 15u, (s16 >> 8) & 15u), expand4(m16 >> 12, s16 >> 12));
}

// One thread per 32 channels of packed weights: 16 bytes of e2m1 nibbles into [KN][KH*KW*PC][32], in the order nibbles32 gives
// them; channels beyond C become 0.
template <int WB>
__device__ __forceinline__ void expand_half(const uint64_t* __restrict__ qw, uint8_t* __restrict__ w4, long long idx, int PC, int C) {
    const long long word = idx >> 1;
    const int h = (int)(idx & 1);
    const uint32_t* q = reinterpret_cast<const uint32_t*>(qw + word * WB) + h;
    uint32_t s = __ldg(q), m = WB == 2 ? __ldg(q + 2) : 0xFFFFFFFFu;
    if (C & 63) {
        const int pc = word < (1LL << 31) ? (int)((uint32_t)word % (uint32_t)PC) : (int)(word % PC);
        const int real = C - (pc * 64 + h * 32);
        if (real < 32) m &= real > 0 ? (1u << real) - 1u : 0u;
    }
    *reinterpret_cast<uint4*>(w4 + word * 32 + h * 16) = nibbles32(m, s & m);
}

// One thread per 32 channels of byte weights: 32 bytes -> 16 bytes of e2m1 nibbles.
__device__ __forceinline__ void pack_half(const int8_t* __restrict__ w8, uint8_t* __restrict__ w4, long long idx) {
    uint32_t m = 0, s = 0;
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const uint4 v = __ldg(reinterpret_cast<const uint4*>(w8 + idx * 32) + k);
        const uint32_t q[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 16; i++) {
            const uint32_t b = (q[i >> 2] >> (8 * (i & 3))) & 0xFFu;
            m |= (b & 1u) << (16 * k + i);
            s |= (b >> 7) << (16 * k + i);
        }
    }
    *reinterpret_cast<uint4*>(w4 + idx * 16) = nibbles32(m, s & m);
}

// Byte weights -> 4-bit operands, several layers in one launch: a CTA takes 256 halves (32 channels: 32 bytes in, 16 out) of the
// layer whose range of CTAs it lies in.  Bound by the launch: a prepared layer's bytes are the registered weights and are
// packed again by every pass, so that whoever writes them is followed; a network does that once per pass for all its layers.
// B200, GPU time of a call with / without it: 3x3 64x14x14x256->256 19.4 / 18.1 us, the ResNet-18-shaped network's 19 layers
// (11 MB) in one launch 268 / 265 us at 8 images (one launch per layer adds about 1.2 us each).
constexpr int PACK_LAYERS = 32;
struct PackList {
    const int8_t* w8[PACK_LAYERS];
    uint8_t* w4[PACK_LAYERS];
    long long halves[PACK_LAYERS];
    unsigned first[PACK_LAYERS + 1];     // first CTA of each layer
    int count;
};
__global__ void __launch_bounds__(256) pack_weights_kernel(const __grid_constant__ PackList list) {
    pdl_launch_dependents();                                               // the convolution sets itself up meanwhile; this grid leaves it room
    pdl_wait();                                                            // the bytes may be the previous launch's, the nibbles its operands
    int l = 0;
    while (l + 1 < list.count && blockIdx.x >= list.first[l + 1]) l++;
    const long long idx = (long long)(blockIdx.x - list.first[l]) * 256 + threadIdx.x;
    if (idx < list.halves[l]) pack_half(list.w8[l], list.w4[l], idx);
}

template <int WB>
__global__ void expand_weights_kernel(const uint64_t* __restrict__ qw, int8_t* __restrict__ w8, long long words, int PC, int C) {
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= words * 4) return;
    expand_group<WB>(qw, w8, idx, PC, C);
}

// Runs at the top of both quantiser kernels.  Programmatic launch: nothing is read or written before the previous
// kernel of the stream (which produced x and the thresholds, and may still be reading the scratch this launch
// overwrites) has completed.
__device__ __forceinline__ void quant_prologue(const QuantExtras& ex, int n) {
    pdl_wait();
    if (ex.qw != nullptr) {                                                // the weights, spread over all CTAs of the launch
        const long long stride = (long long)gridDim.x * gridDim.y * blockDim.x;
        for (long long idx = ((long long)blockIdx.y * gridDim.x + blockIdx.x) * blockDim.x + threadIdx.x; idx < ex.words * 2; idx += stride) {
            if (ex.wbits == 2) expand_half<2>(ex.qw, ex.w4, idx, ex.PC, ex.C);
            else expand_half<1>(ex.qw, ex.w4, idx, ex.PC, ex.C);
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (ex.zero_sums) ex.zero_sums[n] = 0.0;
        if (n == 0 && ex.zero_counter) *ex.zero_counter = 0u;
    }
}

// Sixteen consecutive channels held as 16-bit integers (the compact output of a convolution): one 256-bit load.
struct u8w { uint32_t v[8]; };
__device__ __forceinline__ u8w ld_stream_u8(const int16_t* p) {
    u8w r;
    asm volatile("ld.global.nc.L1::no_allocate.v8.u32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]), "=r"(r.v[7]) : "l"(p));
    return r;
}

// 256-bit streaming load (sm_100): a lane reads 8 consecutive channels, a warp 1 KB contiguous.
__device__ __forceinline__ f8 ld_stream_f8(const float* p) {
    f8 r;
    asm volatile("ld.global.nc.L1::no_allocate.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(r.v[0]), "=f"(r.v[1]), "=f"(r.v[2]), "=f"(r.v[3]),
                   "=f"(r.v[4]), "=f"(r.v[5]), "=f"(r.v[6]), "=f"(r.v[7]) : "l"(p));
    return r;
}

// grid = (ctas_per_image, N).  words_per_image = H*W*PC with PC = C/64.
// Eight lanes own one 64-channel word: lane b of the group quantises channels 8b..8b+7 and stores byte b
// of the sign and of the magnitude word itself, so no cross-lane traffic is needed at all.
// IN16: x holds 16-bit integers instead of floats (same element order).
template <int BITS, bool IN16>
__global__ void __launch_bounds__(QTHREADS)
quantize_c64_kernel(const void* __restrict__ x, const float* __restrict__ ths,
                    uint64_t* __restrict__ qx, int* __restrict__ btn, long long words_per_image, const QuantExtras ex) {
    // Last image first, and within an image the last chunk first: the tensor usually was written front to back by the
    // kernel before this one, so its end is what the L2 still holds.
    const int n = (int)(gridDim.y - 1u - blockIdx.y);
    const unsigned bx = gridDim.x - 1u - blockIdx.x;
    quant_prologue(ex, n);
    const float t = __ldg(ths + n);
    const float nt = -t;
    const int byte = threadIdx.x & 7;
    const int grp = threadIdx.x >> 3;                         // word slot within the CTA: 0..31
    const float* xi = reinterpret_cast<const float*>(x) + (IN16 ? 0 : (long long)n * words_per_image * 64);
    const int16_t* xs = reinterpret_cast<const int16_t*>(x) + (IN16 ? (long long)n * words_per_image * 64 : 0);
    unsigned char* qi = reinterpret_cast<unsigned char*>(qx + (long long)n * words_per_image * BITS);
    int cnt = 0;

    if (IN16) {
        // 16-bit input: four lanes own a word, a lane loads its 16 channels as one 256-bit load (the same bytes per load and
        // per thread in flight as the fp32 path) and stores 16 bits per plane.  Inside the chain this form measured 1 us per
        // launch faster than 128-bit loads, twice as many of them, by eight lanes per word.
        constexpr int WORDS16 = (QTHREADS / 4) * QUNROLL;                  // 256 words per CTA step
        const int q4 = threadIdx.x & 3, g4 = threadIdx.x >> 2;
        for (long long w0 = (long long)bx * WORDS16; w0 < words_per_image; w0 += (long long)gridDim.x * WORDS16) {
            u8w raw[QUNROLL];
#pragma unroll
            for (int u = 0; u < QUNROLL; u++) {
                const long long w = w0 + u * (QTHREADS / 4) + g4;
                if (w < words_per_image) raw[u] = ld_stream_u8(xs + w * 64 + q4 * 16);
            }
#pragma unroll
            for (int u = 0; u < QUNROLL; u++) {
                const long long w = w0 + u * (QTHREADS / 4) + g4;
                if (w >= words_per_image) continue;
                unsigned pos = 0, neg = 0, bin = 0;
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const float lo = (float)(int16_t)(raw[u].v[i] & 0xFFFFu), hi = (float)(int16_t)(raw[u].v[i] >> 16);
                    if (BITS == 2) {
                        pos |= (lo > t) ? (1u << (2 * i)) : 0u;      neg |= (lo < nt) ? (1u << (2 * i)) : 0u;
                        pos |= (hi > t) ? (1u << (2 * i + 1)) : 0u;  neg |= (hi < nt) ? (1u << (2 * i + 1)) : 0u;
                    } else {
                        bin |= (lo < t) ? (1u << (2 * i)) : 0u;      bin |= (hi < t) ? (1u << (2 * i + 1)) : 0u;
                    }
                }
                if (BITS == 2) {
                    neg &= ~pos;
                    const unsigned mag = pos | neg;
                    unsigned short* o = reinterpret_cast<unsigned short*>(qi + w * 16) + q4;
                    o[0] = (unsigned short)neg;
                    o[4] = (unsigned short)mag;
                    cnt += __popc(mag);
                } else {
                    reinterpret_cast<unsigned short*>(qi + w * 8)[q4] = (unsigned short)bin;
                }
            }
        }
    }
    constexpr int UN = QUNROLL;
    constexpr int WORDS = (QTHREADS / 8) * UN;
    for (long long w0 = (long long)bx * WORDS; !IN16 && w0 < words_per_image; w0 += (long long)gridDim.x * WORDS) {
        f8 v[UN];
        long long w[UN];
#pragma unroll
        for (int u = 0; u < UN; u++) {
            w[u] = w0 + u * (QTHREADS / 8) + grp;
            if (w[u] < words_per_image) v[u] = ld_stream_f8(xi + w[u] * 64 + byte * 8);
        }
#pragma unroll
        for (int u = 0; u < UN; u++) {
            if (w[u] >= words_per_image) continue;
            const f8 val = v[u];
            if (BITS == 2) {
                unsigned pos = 0, neg = 0;
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    pos |= (val.v[i] > t) ? (1u << i) : 0u;
                    neg |= (val.v[i] < nt) ? (1u << i) : 0u;
                }
                neg &= ~pos;                                   // the "+1" branch is tested first
                const unsigned mag = pos | neg;
                unsigned char* o = qi + w[u] * 16 + byte;
                o[0] = (unsigned char)neg;                     // sign plane, byte `byte` of the word
                o[8] = (unsigned char)mag;                     // magnitude plane
                cnt += __popc(mag);
            } else {
                unsigned b = 0;
#pragma unroll
                for (int i = 0; i < 8; i++) b |= (val.v[i] < t) ? (1u << i) : 0u;
                qi[w[u] * 8 + byte] = (unsigned char)b;
            }
        }
    }

    if (BITS == 2 && btn != nullptr) {
        __shared__ int wsum[QTHREADS / 32];
        cnt = __reduce_add_sync(0xFFFFFFFFu, cnt);
        if ((threadIdx.x & 31) == 0) wsum[threadIdx.x >> 5] = cnt;
        __syncthreads();
        if (threadIdx.x == 0) {
            int tot = 0;
#pragma unroll
            for (int i = 0; i < QTHREADS / 32; i++) tot += wsum[i];
            if (gridDim.x == 1) btn[n] = tot;                 // the image's only CTA
            else if (tot) atomicAdd(btn + n, tot);            // integer: order-independent, exact
        }
    }
    if (BITS == 1 && btn != nullptr && blockIdx.x == 0 && threadIdx.x == 0) btn[n] = 0;
    pdl_launch_dependents();                                  // the next kernel may be scheduled once every CTA got here
}

// ---- any channel count, any alignment ------------------------------------------------------------------------------------
// Eight consecutive channels of one pixel, as many elements per load as the rows' alignment allows: V = 8 (C % 8 == 0), 4, 2
// or 1.  Channels from `valid` on are not read and come back as 0.  Rows whose length is no multiple of 32 bytes share
// sectors between lanes and between the loads of one lane, so these loads may stay in L1 (no streaming hint).
template <int V>
__device__ __forceinline__ f8 ld8(const float* p, int valid) {
    f8 r;
#pragma unroll
    for (int i = 0; i < 8; i++) r.v[i] = 0.f;
    if (V == 8) {
        if (valid > 0) r = ld_stream_f8(p);
    } else if (V == 4) {
#pragma unroll
        for (int i = 0; i < 8; i += 4)
            if (valid > i) { const float4 q = __ldg(reinterpret_cast<const float4*>(p + i)); r.v[i] = q.x; r.v[i + 1] = q.y; r.v[i + 2] = q.z; r.v[i + 3] = q.w; }
    } else if (V == 2) {
#pragma unroll
        for (int i = 0; i < 8; i += 2)
            if (valid > i) { const float2 q = __ldg(reinterpret_cast<const float2*>(p + i)); r.v[i] = q.x; r.v[i + 1] = q.y; }
    } else {
#pragma unroll
        for (int i = 0; i < 8; i++)
            if (valid > i) r.v[i] = __ldg(p + i);
    }
    return r;
}
template <int V>
__device__ __forceinline__ f8 ld8(const int16_t* p, int valid) {                   // V is 8 or 1 here
    f8 r;
#pragma unroll
    for (int i = 0; i < 8; i++) r.v[i] = 0.f;
    if (V == 8) {
        if (valid > 0) {
            const uint4 q = __ldg(reinterpret_cast<const uint4*>(p));
            const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int i = 0; i < 4; i++) { r.v[2 * i] = (float)(int16_t)(w[i] & 0xFFFFu); r.v[2 * i + 1] = (float)(int16_t)(w[i] >> 16); }
        }
    } else {
#pragma unroll
        for (int i = 0; i < 8; i++)
            if (valid > i) r.v[i] = (float)__ldg(p + i);
    }
    return r;
}

// How lanes share the words of an image.  L = 8: lane `byte` of a group of eight owns channels 8*byte .. 8*byte + 7 of a
// word and writes that byte of every plane; L = 1 (C <= 8, a network's first layer): one lane per word.  A pass of a CTA
// is QTHREADS / L words, a step QUNROLL passes.
template <int L> __host__ __device__ constexpr int words_per_pass() { return QTHREADS / L; }
struct WordAt { long long off; int valid; };                                       // element offset in the image, real channels of the lane's eight
template <int L>
__device__ __forceinline__ WordAt word_at(long long w, int C, int PC, const FastDiv& dPC, bool wide) {
    const long long pix = L == 1 ? w : (wide ? w / PC : (long long)dPC.div((uint32_t)w));
    const int c0 = L == 1 ? 0 : (int)(w - pix * PC) * 64 + (int)(threadIdx.x & 7) * 8;
    WordAt a;
    a.off = pix * C + c0;
    a.valid = C - c0;
    return a;
}
// Quantises a lane's eight channels and writes its share of word w; returns the number of nonzero ternary values.
template <int BITS, int L>
__device__ __forceinline__ int put8(const f8& x, int valid, float t, uint64_t* qi, long long w) {
    const unsigned mask = valid >= 8 ? 0xFFu : (valid <= 0 ? 0u : (1u << valid) - 1u);
    unsigned pos = 0, neg = 0;
    const float nt = -t;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        if (BITS == 2) {
            pos |= (x.v[i] > t) ? (1u << i) : 0u;
            neg |= (x.v[i] < nt) ? (1u << i) : 0u;
        } else {
            neg |= (x.v[i] < t) ? (1u << i) : 0u;
        }
    }
    pos &= mask;
    neg &= mask & ~pos;                                                            // ternary: the "+1" branch is tested first
    if (L == 1) {
        qi[w * BITS] = neg;
        if (BITS == 2) qi[w * BITS + 1] = pos | neg;
    } else {
        unsigned char* o = reinterpret_cast<unsigned char*>(qi) + w * (8 * BITS) + (threadIdx.x & 7);
        o[0] = (unsigned char)neg;
        if (BITS == 2) o[8] = (unsigned char)(pos | neg);
    }
    return BITS == 2 ? __popc(pos | neg) : 0;
}

// Same division of labour as quantize_c64_kernel for every other C and alignment.  grid = (ctas_per_image, N).
// Bound by HBM where rows are vectors, by the L1's load path where they are not; the pixel of a word comes from a
// multiply-high, every lane has QUNROLL * 8 channels in flight.  It replaces a warp-per-word ballot kernel, which had two
// loads in flight per lane behind a 64-bit division.  B200, us before / after: binary 64x27x31x200 31.0 / 8.6 (5.2 TB/s),
// ternary 64x56x56x70 57.4 / 22.8, 64x28x28x511 65.8 / 33.2 (single-element loads, 3.3 TB/s), 64x224x224x3 296 / 22.8.
template <int BITS, bool IN16, int V, int L>
__global__ void __launch_bounds__(QTHREADS, 4)
quantize_any_kernel(const void* __restrict__ x, const float* __restrict__ ths, uint64_t* __restrict__ qx, int* __restrict__ btn,
                    long long words_per_image, long long elems_per_image, int C, int PC, const FastDiv dPC, const QuantExtras ex) {
    const int n = (int)(gridDim.y - 1u - blockIdx.y);         // back to front, as above
    const unsigned bx = gridDim.x - 1u - blockIdx.x;
    quant_prologue(ex, n);
    const float t = __ldg(ths + n);
    const bool wide = words_per_image >= (1LL << 31);
    const int slot = threadIdx.x / L;
    const float* xf = reinterpret_cast<const float*>(x) + (IN16 ? 0 : (long long)n * elems_per_image);
    const int16_t* xs = reinterpret_cast<const int16_t*>(x) + (IN16 ? (long long)n * elems_per_image : 0);
    uint64_t* qi = qx + (long long)n * words_per_image * BITS;
    constexpr int PASS = words_per_pass<L>(), STEP = PASS * QUNROLL;
    int cnt = 0;
    for (long long w0 = (long long)bx * STEP + slot; w0 < words_per_image; w0 += (long long)gridDim.x * STEP) {
        f8 v[QUNROLL];
        int valid[QUNROLL];
#pragma unroll
        for (int u = 0; u < QUNROLL; u++) {
            const long long w = w0 + u * PASS;
            valid[u] = 0;
            if (w < words_per_image) {
                const WordAt a = word_at<L>(w, C, PC, dPC, wide);
                valid[u] = a.valid;
                if (IN16) v[u] = ld8<(V == 8 ? 8 : 1)>(xs + a.off, a.valid);
                else v[u] = ld8<V>(xf + a.off, a.valid);
            }
        }
#pragma unroll
        for (int u = 0; u < QUNROLL; u++) {
            const long long w = w0 + u * PASS;
            if (w < words_per_image) cnt += put8<BITS, L>(v[u], valid[u], t, qi, w);
        }
    }
    if (BITS == 2 && btn != nullptr) {
        __shared__ int wsum[QTHREADS / 32];
        cnt = __reduce_add_sync(0xFFFFFFFFu, cnt);
        if ((threadIdx.x & 31) == 0) wsum[threadIdx.x >> 5] = cnt;
        __syncthreads();
        if (threadIdx.x == 0) {
            int tot = 0;
#pragma unroll
            for (int i = 0; i < QTHREADS / 32; i++) tot += wsum[i];
            if (gridDim.x == 1) btn[n] = tot;                 // the image's only CTA
            else if (tot) atomicAdd(btn + n, tot);            // integer: order-independent, exact
        }
    }
    if (BITS == 1 && btn != nullptr && blockIdx.x == 0 && threadIdx.x == 0) btn[n] = 0;
    pdl_launch_dependents();
}

// Elements per load that C and the address of x allow (rows start at multiples of C elements): 8, 4, 2 or 1.
static int load_width(const void* x, int C, bool in16) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(x);
    if (in16) return C % 8 == 0 && (a & 15) == 0 ? 8 : 1;
    if (C % 8 == 0 && (a & 31) == 0) return 8;
    if (C % 4 == 0 && (a & 15) == 0) return 4;
    return C % 2 == 0 && (a & 7) == 0 ? 2 : 1;
}

// CTAs per image: every CTA the same whole number of steps (a ragged last step, or a nearly empty extra wave, costs a
// whole step's time), at most about six waves of eight CTAs per SM over all images.
static unsigned ctas_per_image(long long words_per_image, long long words_per_step, int N) {
    const long long steps = (words_per_image + words_per_step - 1) / words_per_step;
    const long long cap = 148LL * 8 * 6;
    const long long iters = ((long long)N * steps + cap - 1) / cap;        // steps per CTA
    const long long per_image = (steps + iters - 1) / iters;
    return (unsigned)(per_image < 1 ? 1 : per_image);
}

// A launch that also prepares weights gets enough CTAs for that, 32 channels per thread up to four CTAs per SM: the tensor of a
// single image fills 4 CTAs, which took 65 us for the weights of a 3x3x512 -> 512 layer.
static long long ctas_for_weights(long long words) {
    const long long groups = (words * 2 + QTHREADS - 1) / QTHREADS;
    return groups < 148 * 4 ? groups : 148 * 4;
}
static dim3 quantize_grid(unsigned per_image, int N, const QuantExtras& ex) {
    if (ex.qw) {
        const unsigned share = (unsigned)((ctas_for_weights(ex.words) + N - 1) / N);
        if (per_image < share) per_image = share;
    }
    return dim3(per_image, (unsigned)N);
}

// BTN_W is cleared by a memset only where several CTAs add to an image's count; else the kernel writes it.
static int clear_counts(int32_t* btn, int bits, dim3 grid, cudaStream_t stream) {
    if (!btn || bits == 1 || grid.x == 1) return TAB_OK;
    const cudaError_t e = cudaMemsetAsync(btn, 0, sizeof(int32_t) * (size_t)grid.y, stream);
    return e == cudaSuccess ? TAB_OK : record_cuda_error(e);
}

template <int BITS, bool IN16>
static int launch_quantize_any(const void* x, const float* ths, uint64_t* q, int32_t* btn, int N, long long pixels, int C,
                               cudaStream_t stream, const QuantExtras& ex) {
    const int PC = (C + 63) / 64;
    const long long wpi = pixels * PC;
    const FastDiv dPC = make_fastdiv((uint32_t)PC);
    const int V = load_width(x, C, IN16);
    const bool one = C <= 8;                                               // one lane per word
    const dim3 grid = quantize_grid(ctas_per_image(wpi, (long long)QTHREADS / (one ? 1 : 8) * QUNROLL, N), N, ex);
    const int rc = clear_counts(btn, BITS, grid, stream);
    if (rc != TAB_OK) return rc;
#define TAB_QANY(VV) (one ? launch_pdl(quantize_any_kernel<BITS, IN16, VV, 1>, grid, dim3(QTHREADS), 0, stream, x, ths, q, btn, wpi, pixels * C, C, PC, dPC, ex) \
                          : launch_pdl(quantize_any_kernel<BITS, IN16, VV, 8>, grid, dim3(QTHREADS), 0, stream, x, ths, q, btn, wpi, pixels * C, C, PC, dPC, ex))
    if (V == 8) return TAB_QANY(8);
    if (IN16 || V == 1) return TAB_QANY(1);
    return V == 4 ? TAB_QANY((IN16 ? 1 : 4)) : TAB_QANY((IN16 ? 1 : 2));
#undef TAB_QANY
}

int quantize_dispatch(const void* x, const float* ths, int64_t* qx, int32_t* btn, int bits,
                      int N, int H, int W, int C, cudaStream_t stream, const QuantExtras* extras, bool in16) {
    const QuantExtras ex = extras ? *extras : QuantExtras{};
    const long long pixels = (long long)H * W;
    const int PC = (C + 63) / 64;
    const long long wpi = pixels * PC;
    if (N == 0 || wpi == 0) return TAB_OK;
    if (N > 65535) {
        // grid.y is limited to 65535: process in slabs of images.
        for (int n0 = 0; n0 < N; n0 += 65535) {
            const int nn = (N - n0 < 65535) ? (N - n0) : 65535;
            int rc = quantize_dispatch(reinterpret_cast<const char*>(x) + (long long)n0 * pixels * C * (in16 ? 2 : 4), ths + n0,
                                       qx + (long long)n0 * wpi * bits, btn ? btn + n0 : nullptr,
                                       bits, nn, H, W, C, stream, n0 == 0 ? extras : nullptr, in16);
            if (rc != TAB_OK) return rc;
        }
        return TAB_OK;
    }
    const bool fast = (C % 64 == 0) && ((reinterpret_cast<uintptr_t>(x) & 31) == 0);
    uint64_t* q = reinterpret_cast<uint64_t*>(qx);
    if (fast) {
        const dim3 grid = quantize_grid(ctas_per_image(wpi, in16 ? 2 * QWORDS_PER_ITER : QWORDS_PER_ITER, N), N, ex);
        const int rc = clear_counts(btn, bits, grid, stream);
        if (rc != TAB_OK) return rc;
        if (in16) {
            if (bits == 2) return launch_pdl(quantize_c64_kernel<2, true>, grid, dim3(QTHREADS), 0, stream, x, ths, q, btn, wpi, ex);
            return launch_pdl(quantize_c64_kernel<1, true>, grid, dim3(QTHREADS), 0, stream, x, ths, q, btn, wpi, ex);
        }
        if (bits == 2) return launch_pdl(quantize_c64_kernel<2, false>, grid, dim3(QTHREADS), 0, stream, x, ths, q, btn, wpi, ex);
        return launch_pdl(quantize_c64_kernel<1, false>, grid, dim3(QTHREADS), 0, stream, x, ths, q, btn, wpi, ex);
    }
    if (in16) return bits == 2 ? launch_quantize_any<2, true>(x, ths, q, btn, N, pixels, C, stream, ex) : launch_quantize_any<1, true>(x, ths, q, btn, N, pixels, C, stream, ex);
    return bits == 2 ? launch_quantize_any<2, false>(x, ths, q, btn, N, pixels, C, stream, ex) : launch_quantize_any<1, false>(x, ths, q, btn, N, pixels, C, stream, ex);
}

// ---- thresholds and bit-planes of a tensor in one launch ----------------------------------------------------------------
// What every caller of Quantize does first - thresholds[n] = scale * mean|x[n]| (the reference leaves it to framework ops) -
// and the quantisation against them, as two phases of one persistent grid: per-image sums of |x| (double atomics), a
// grid-wide counter (all CTAs are resident: the grid is sized by the occupancy calculator and launched cooperatively; the wait is
// bounded and reports in *status), then every CTA quantises, last unit first, the units it has just summed - the end of its share is
// what the L2 still holds, and its last unit is still in registers.  A unit is one CTA step (QUNROLL passes) of one image; a
// CTA owns consecutive units, so that its sum leaves the registers once per image and not once per unit.
// The weights of the layer that reads the planes may be packed on the side (see PackJob).
// FULL: C % 64 == 0 and 32-byte rows (every lane has eight real channels); else V and L as in quantize_any_kernel.
constexpr uint32_t QA_WAIT_LIMIT = 1u << 21;                               // a second or two; the slowest CTA of 180 GB of input needs 30 ms

template <int BITS, int V, int L, bool FULL>
__global__ void __launch_bounds__(QTHREADS, 4)
quantize_auto_kernel(const float* __restrict__ x, float scale, double* __restrict__ sums, unsigned* __restrict__ bar,
                     float* __restrict__ ths_out, uint64_t* __restrict__ qx, long long words_per_image, long long elems_per_image, int C, int PC,
                     const FastDiv dPC, long long steps_per_image, long long units, int N, int* __restrict__ status, const PackJob pack) {
    pdl_wait();
    for (long long idx = (long long)blockIdx.x * QTHREADS + threadIdx.x; idx < pack.words * 2; idx += (long long)gridDim.x * QTHREADS) pack_half(pack.w8, pack.w4, idx);
    constexpr int PASS = words_per_pass<L>(), STEP = PASS * QUNROLL;
    const int slot = threadIdx.x / L;
    const bool wide = words_per_image >= (1LL << 31);
    const double per_image = (double)elems_per_image;
    __shared__ double wsum[QTHREADS / 32];
    __shared__ float s_t;
    auto at = [&](long long w) -> WordAt {
        if (FULL) return WordAt{w * 64 + (long long)(threadIdx.x & 7) * 8, 8};
        return word_at<L>(w, C, PC, dPC, wide);
    };
    f8 v[QUNROLL];
    auto load_unit = [&](long long n, long long st) {
        const float* xi = x + n * elems_per_image;
#pragma unroll
        for (int k = 0; k < QUNROLL; k++) {
            const long long w = st * STEP + k * PASS + slot;
#pragma unroll
            for (int i = 0; i < 8; i++) v[k].v[i] = 0.f;
            if (w < words_per_image) { const WordAt a = at(w); v[k] = ld8<V>(xi + a.off, a.valid); }
        }
    };
    // phase 1: sums
    const long long ub = units * blockIdx.x / gridDim.x, ue = units * (blockIdx.x + 1LL) / gridDim.x;     // empty where the grid is larger, for weights to prepare
    long long n = ub / steps_per_image, st = ub - n * steps_per_image;
    double acc = 0.0;
    for (long long u = ub; u < ue; u++) {
        load_unit(n, st);
#pragma unroll
        for (int k = 0; k < QUNROLL; k++) {
            const float* q = v[k].v;
            acc += (((double)fabsf(q[0]) + (double)fabsf(q[1])) + ((double)fabsf(q[2]) + (double)fabsf(q[3]))) +
                   (((double)fabsf(q[4]) + (double)fabsf(q[5])) + ((double)fabsf(q[6]) + (double)fabsf(q[7])));
        }
        const bool image_ends = st + 1 == steps_per_image;
        if (image_ends || u + 1 == ue) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xFFFFFFFFu, acc, o);
            __syncthreads();                                  // wsum of the previous image has been read
            if ((threadIdx.x & 31) == 0) wsum[threadIdx.x >> 5] = acc;
            __syncthreads();
            if (threadIdx.x == 0) {
                double t = 0.0;
#pragma unroll
                for (int i = 0; i < QTHREADS / 32; i++) t += wsum[i];
                atomicAdd(sums + n, t);
            }
            acc = 0.0;
        }
        if (u + 1 < ue) { if (image_ends) { n++; st = 0; } else st++; }
    }
    // grid-wide counter
    __threadfence();
    __syncthreads();
    int flag = 0;
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(bar, 1u);
        bool ok = false;
        for (uint32_t i = 0; i < QA_WAIT_LIMIT && !ok; i++) {
            unsigned seen;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(bar) : "memory");
            ok = seen >= gridDim.x;
            if (!ok) __nanosleep(100);
        }
        if (!ok && status) atomicExch(status, 22);
        flag = ok ? 1 : 0;
    }
    const bool met = __syncthreads_or(flag);                               // else the result of the launch is void; the status says so
    if (met && blockIdx.x == 0 && ths_out)
        for (int m = threadIdx.x; m < N; m += QTHREADS) ths_out[m] = (float)((double)scale * (__ldcg(sums + m) / per_image));
    // phase 2: the CTA's units again, last first (v still holds the last one)
    long long tn = -1;
    float t = 0.f;
    for (long long u = ue - 1; met && u >= ub; u--) {
        if (u != ue - 1) {
            if (st == 0) { n--; st = steps_per_image - 1; } else st--;
            load_unit(n, st);
        }
        if (n != tn) {
            __syncthreads();
            if (threadIdx.x == 0) s_t = (float)((double)scale * (__ldcg(sums + n) / per_image));
            __syncthreads();
            t = s_t;
            tn = n;
        }
        uint64_t* qi = qx + n * words_per_image * BITS;
#pragma unroll
        for (int k = 0; k < QUNROLL; k++) {
            const long long w = st * STEP + k * PASS + slot;
            if (w < words_per_image) put8<BITS, L>(v[k], FULL ? 8 : at(w).valid, t, qi, w);
        }
    }
    // the CTA that gets here last leaves the state block zero again (every CTA has read the sums it needs)
    __syncthreads();
    flag = 0;
    if (threadIdx.x == 0) flag = (atomicAdd(bar + 1, 1u) == gridDim.x - 1u) ? 1 : 0;
    if (__syncthreads_or(flag)) {
        for (int m = threadIdx.x; m < N; m += QTHREADS) sums[m] = 0.0;
        if (threadIdx.x == 0) { bar[0] = 0u; bar[1] = 0u; }
    }
    pdl_launch_dependents();
}

template <int BITS, int V, int L, bool FULL>
static int launch_quantize_auto(const float* x, float scale, double* sums, unsigned* bar, float* ths_out, int64_t* qx,
                                int N, int H, int W, int C, int* status, cudaStream_t stream, const PackJob& pack) {
    const int PC = (C + 63) / 64;
    const long long pixels = (long long)H * W, wpi = pixels * PC, step = (long long)words_per_pass<L>() * QUNROLL;
    const long long spi = (wpi + step - 1) / step, units = spi * N;
    static std::mutex mu;
    static int capacity[64] = {};                             // resident CTAs, per device
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return record_cuda_error(e);
    int cap = 0;
    {
        std::lock_guard<std::mutex> lock(mu);
        cap = dev < 64 ? capacity[dev] : 0;
        if (!cap) {
            int per_sm = 0, sms = 0;
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, quantize_auto_kernel<BITS, V, L, FULL>, QTHREADS, 0);
            if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
            if (e != cudaSuccess) return record_cuda_error(e);
            cap = per_sm * sms;
            if (dev < 64) capacity[dev] = cap;
        }
    }
    const long long want = std::max(units, ctas_for_weights(pack.words));
    const unsigned grid = (unsigned)(want < cap ? want : cap);
    return launch_pdl_as(true, 1, quantize_auto_kernel<BITS, V, L, FULL>, dim3(grid), dim3(QTHREADS), 0, stream, x, scale, sums, bar, ths_out,
                      reinterpret_cast<uint64_t*>(qx), wpi, pixels * C, C, PC, make_fastdiv((uint32_t)PC), spi, units, N, status, pack);
}

template <int BITS>
static int quantize_auto_by_width(const float* x, float scale, double* sums, unsigned* bar, float* ths_out, int64_t* qx,
                                  int N, int H, int W, int C, int* status, cudaStream_t s, const PackJob& pack) {
    const int V = load_width(x, C, false);
#define TAB_QAUTO(VV, LL, FF) return launch_quantize_auto<BITS, VV, LL, FF>(x, scale, sums, bar, ths_out, qx, N, H, W, C, status, s, pack)
    if (C <= 8) {
        if (V == 8) TAB_QAUTO(8, 1, false);
        if (V == 4) TAB_QAUTO(4, 1, false);
        if (V == 2) TAB_QAUTO(2, 1, false);
        TAB_QAUTO(1, 1, false);
    }
    if (V == 8 && C % 64 == 0) TAB_QAUTO(8, 8, true);
    if (V == 8) TAB_QAUTO(8, 8, false);
    if (V == 4) TAB_QAUTO(4, 8, false);
    if (V == 2) TAB_QAUTO(2, 8, false);
    TAB_QAUTO(1, 8, false);
#undef TAB_QAUTO
}

int quantize_auto_dispatch(const float* x, float scale, double* sums, unsigned* bar, float* ths_out, int64_t* qx, int bits,
                           int N, int H, int W, int C, int* status, cudaStream_t stream, const PackJob& pack) {
    return bits == 2 ? quantize_auto_by_width<2>(x, scale, sums, bar, ths_out, qx, N, H, W, C, status, stream, pack)
                     : quantize_auto_by_width<1>(x, scale, sums, bar, ths_out, qx, N, H, W, C, status, stream, pack);
}

int pack_weights_dispatch(int count, const int8_t* const* w8, uint8_t* const* w4, const long long* words, cudaStream_t stream) {
    for (int done = 0; done < count;) {
        PackList list = {};
        long long blocks = 0;
        for (; done < count && list.count < PACK_LAYERS; done++) {
            const long long more = (words[done] * 2 + 255) / 256;
            if (more >= (1LL << 31)) return TAB_E_TOO_LARGE;
            if (more == 0) continue;
            if (blocks + more >= (1LL << 31)) break;                       // the rest goes into another launch
            const int l = list.count++;
            list.w8[l] = w8[done]; list.w4[l] = w4[done]; list.halves[l] = words[done] * 2;
            list.first[l] = (unsigned)blocks;
            blocks += more;
        }
        if (list.count == 0) continue;
        const int rc = launch_pdl(pack_weights_kernel, dim3((unsigned)blocks), dim3(256), 0, stream, list);
        if (rc != TAB_OK) return rc;
    }
    return TAB_OK;
}

int expand_weights_dispatch(const int64_t* qw, int8_t* w8, int wbits, int KN, int KH, int KW, int C, cudaStream_t stream) {
    const int PC = packed_channels(C);
    const long long words = (long long)KN * KH * KW * PC;
    if (words == 0) return TAB_OK;
    if (words * 4 >= (1LL << 31) * 256) return TAB_E_TOO_LARGE;
    const unsigned blocks = (unsigned)((words * 4 + 255) / 256);
    const uint64_t* q = reinterpret_cast<const uint64_t*>(qw);
    if (wbits == 2) expand_weights_kernel<2><<<blocks, 256, 0, stream>>>(q, w8, words, PC, C);
    else expand_weights_kernel<1><<<blocks, 256, 0, stream>>>(q, w8, words, PC, C);
    return check_launch();
}

}  // namespace tab
