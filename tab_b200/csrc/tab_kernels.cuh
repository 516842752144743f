// Shared declarations for the sm_100a kernels behind the C ABI in include/tab_b200.h.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>
#include "../../include/tab_b200.h"

namespace tab {

// Records a CUDA failure for tab_last_cuda_error() and maps it to TAB_E_CUDA.
int record_cuda_error(cudaError_t e);

// cudaGetLastError() right after a launch -> TAB_OK or TAB_E_CUDA.
inline int check_launch() {
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? TAB_OK : record_cuda_error(e);
}

// Launch with programmatic stream serialisation: the kernel may be scheduled while its predecessor in the stream is
// still draining (the predecessor executed griddepcontrol.launch_dependents in every CTA); it must execute
// griddepcontrol.wait before it touches anything a predecessor wrote or may still read.  Works under stream capture
// (the dependency becomes a programmatic edge of the graph).
// resident: every CTA of the grid runs at the same time or the launch fails (cooperative launch) - for kernels whose CTAs wait for
// one another, which other streams' work must not keep from being placed.
// cluster: CTAs per thread-block cluster along x (grid.x a multiple of it).
template <typename... KArgs, typename... Args>
inline int launch_pdl_as(bool resident, unsigned cluster, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = stream;
    cudaLaunchAttribute attr[3];
    unsigned n = 0;
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n++].val.programmaticStreamSerializationAllowed = 1;
    if (resident) {
        attr[n].id = cudaLaunchAttributeCooperative;
        attr[n++].val.cooperative = 1;
    }
    if (cluster > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = cluster; attr[n].val.clusterDim.y = 1; attr[n++].val.clusterDim.z = 1;
    }
    cfg.attrs = attr; cfg.numAttrs = n;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
    return e == cudaSuccess ? TAB_OK : record_cuda_error(e);
}
template <typename... KArgs, typename... Args>
inline int launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args... args) {
    return launch_pdl_as(false, 1, kernel, grid, block, smem, stream, args...);
}

#ifdef __CUDACC__
// Device side of the above.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
#endif

inline int packed_channels(int C) { return (C + 63) / 64; }
inline int act_bits(int type) { return (type == 2 || type == 3) ? 1 : 2; }      // TAB_GEMM.cu:367-372
inline int weight_bits(int type) { return (type == 1 || type == 3) ? 1 : 2; }   // TAB_GEMM.cu:374-379

// Small jobs a quantiser launch does on the side for the convolution that follows it (all optional).
struct QuantExtras {
    double* zero_sums = nullptr;         // [N]: cleared
    unsigned* zero_counter = nullptr;    // cleared
    const uint64_t* qw = nullptr;        // packed weights [KN][KH*KW*PC][wbits] to expand into w4 [KN][KH*KW*PC][32] (4-bit operands)
    uint8_t* w4 = nullptr;
    long long words = 0;                 // KN*KH*KW*PC
    int wbits = 2, PC = 1, C = 64;       // of the weights
};

// Byte weights [words][64] for the quantiser that finds its thresholds to pack into 4-bit operands [words][32] on the side.
struct PackJob {
    const int8_t* w8 = nullptr;
    uint8_t* w4 = nullptr;
    long long words = 0;
};

// quantize_sm100.cu: bits is 1 or 2; btn may be null, else it receives the per-image counts (zeros for bits 1).  in16: x holds int16 instead of float.
int quantize_dispatch(const void* x, const float* ths, int64_t* qx, int32_t* btn, int bits,
                      int N, int H, int W, int C, cudaStream_t stream, const QuantExtras* extras = nullptr, bool in16 = false);
int expand_weights_dispatch(const int64_t* qw, int8_t* w8, int wbits, int KN, int KH, int KW, int C, cudaStream_t stream);
// Byte weights {-1,0,+1} of `count` layers -> the 4-bit operands of the same words (words[i] = KN*KH*KW*PC of layer i).
int pack_weights_dispatch(int count, const int8_t* const* w8, uint8_t* const* w4, const long long* words, cudaStream_t stream);
// Thresholds scale * mean|x[n]| and the bit-planes against them in one launch (sums: N doubles, bar: two words, all zero
// before and after).
int quantize_auto_dispatch(const float* x, float scale, double* sums, unsigned* bar, float* ths_out, int64_t* qx, int bits,
                           int N, int H, int W, int C, int* status, cudaStream_t stream, const PackJob& pack = PackJob{});
// Word of the current device that records a bounded wait that ran out (shared with the tensor-core kernel); null if unavailable.
// It lies in pinned host memory, so that the launches that follow see it without synchronising.
int* device_status_word();
inline bool stalled(const int* status) { return status && *static_cast<const volatile int*>(status) != 0; }

// conv_sm100.cu: implicit-im2col popcount GEMM on packed activations.  csa: carry-save popcount tree (else one POPC per word).
int conv_packed_dispatch(const int64_t* qx, const int64_t* qw, const int32_t* btn, float* y, int type,
                         int p1, int p2, int s1, int s2, int N, int H, int W, int C,
                         int KN, int KH, int KW, cudaStream_t stream, bool csa = true);

}  // namespace tab
