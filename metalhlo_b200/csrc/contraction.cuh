// Problem descriptions shared by the contraction dispatcher and the tcgen05 kernels.
#pragma once

#include "common.cuh"

namespace mhlo {

struct GemmProblem {
    const void* a;
    const void* b;
    void* c;
    const void* bias;
    const void* residual = nullptr;  // added to the product after the bias: same type, pitch and column offset as C; no activation
    int64_t as[4], bs[4];  // {batch0, batch1, row, col} element strides
    int64_t batch0, batch1, m, n, k;
    int32_t in_dtype, out_dtype, epilogue;
    // Output placement. ldc = elements between rows of C (0: dense, = n); c_col0 = first column this product fills
    // inside a wider matrix; copies[] = further matrices (peers' memory) that receive the same tile stores.
    int64_t ldc = 0, c_col0 = 0;
    void* copies[7] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
    int32_t n_copies = 0;
    int32_t copy_stores = 0;  // how the copies are written: 0 / 1 = 16-byte stores per lane, 2 = bulk tensor stores (one map per copy)
    // Launch knobs of the tensor-core kernel; 0 = chosen by the library. tile_n: 128 or 256 columns per tile; stages: depth
    // of the TMA ring; cta_group: 1 = one CTA per 128-row tile, 2 = a pair of CTAs per 256-row tile.
    int32_t tile_n = 0, stages = 0, cta_group = 0;
    int32_t split_k = 0;  // 1: the sum over K may be split (see mhlo_cuda_gemm_tuning)
    int32_t exact_act = 0;  // 1: the activation in fp32 with the CUDA library's functions, as the elementwise programs have it
};

// The limits of mhlo_cuda_dot_strided: a product beyond them is no one else's to hand over.
inline bool general_kernel_takes(const GemmProblem& p) { return p.batch0 * p.batch1 <= 65535 && (p.m + 63) / 64 <= 65535; }

// How the tensor-core kernels read a 16-bit operand [rows, cols] with element strides {batch0, batch1, row, col} in place: which
// dimension its tensor map has as the contiguous one, kNoMajor if neither can be (TMA wants every other stride to be a positive
// multiple of 16 bytes). A dimension of extent 1 is contiguous and on every grid, whatever its stride says. K comes first where
// both would do. Support, packing and launch all go by this rule.
enum OperandMajor : int32_t { kNoMajor = -1, kMajorK = 0, kMajorMN = 1 };
inline bool tma_stride(int64_t elems) { return elems > 0 && elems % 8 == 0; }
inline bool contiguous_along(int64_t stride, int64_t extent, int64_t other_stride, int64_t other_extent) {
    return (stride == 1 || extent == 1) && (other_extent == 1 || tma_stride(other_stride));
}
inline OperandMajor a_major(const GemmProblem& p) {
    return contiguous_along(p.as[3], p.k, p.as[2], p.m) ? kMajorK : contiguous_along(p.as[2], p.m, p.as[3], p.k) ? kMajorMN : kNoMajor;
}
inline OperandMajor b_major(const GemmProblem& p) {
    return contiguous_along(p.bs[2], p.k, p.bs[3], p.n) ? kMajorK : contiguous_along(p.bs[3], p.n, p.bs[2], p.k) ? kMajorMN : kNoMajor;
}
// Base and batch strides of an operand on the grid. A batch stride of 0 (one matrix for every entry) is: the tensor map then has
// extent 1 in that dimension and every entry reads coordinate 0.
inline bool operand_on_grid(const GemmProblem& p, const void* base, const int64_t* st) {
    return aligned16(base) && (p.batch0 == 1 || st[0] == 0 || tma_stride(st[0])) && (p.batch1 == 1 || st[1] == 0 || tma_stride(st[1]));
}
inline int64_t operand_batch(int64_t extent, int64_t stride) { return stride == 0 ? 1 : extent; }

// A 2-D convolution of dense NHWC input with dense HWIO filters into dense NHWC output, stride 1, one feature group: the
// form the tensor-core kernel reads without a patch matrix.
struct ConvProblem {
    const void* x;
    const void* wgt;
    void* out;
    const void* bias = nullptr;  // one value per output feature, of the output's type
    int32_t dtype, out_dtype, epilogue = 0;
    int64_t images, h, w, channels, kh, kw, features, oh, ow, pad_h, pad_w, dil_h, dil_w;
    int64_t stride_h = 1, stride_w = 1;
};
bool conv_tc_supported(const ConvProblem& c);
int conv_tc_launch(const ConvProblem& c, cudaStream_t stream);

struct AttnShape {
    int64_t qs[3], ks[3], vs[3], os[3];  // {batch, head, sequence} element strides; head_dim is contiguous
    int64_t batch, heads, seq_q, seq_k, head_dim;
    float scale;
    int32_t causal;
    int32_t tile_order = 0;  // tensor-core kernel: 0 = chosen by the library, 1 = long/short pairs per (batch, head), 2 = longest tiles first
};

// Tensor-core (tcgen05 + TMA + TMEM) paths; *_supported() says whether the problem meets their layout rules.
bool gemm_tc_supported(const GemmProblem& p);
int gemm_tc_launch(const GemmProblem& p, cudaStream_t stream);
// 16-bit operands that have to be copied onto the 16-byte grid first. False: not a product this applies to, nothing was queued and
// the general kernel takes it; true: *status is the result of the launches.
// scratch: the caller's own memory (256-byte aligned; too little: false), null: from the library's pool.
struct PackScratch {
    void* base;
    size_t bytes;
};
bool gemm_pack_launch(GemmProblem p, const PackScratch* scratch, cudaStream_t stream, int* status);
bool gemm_fp32_sums(const GemmProblem& p);  // whether a 16-bit product read in place is kept from the tensor cores' sums
size_t gemm_pack_bytes(GemmProblem p);  // what that takes when both operands start on the grid; 0: nothing is packed
// mhlo_cuda_gemm_tuned with the scratch of packed operands from the caller.
int gemm_entry(int32_t in_dtype, int32_t out_dtype, const void* a, const int64_t* a_strides, const void* b, const int64_t* b_strides, void* c,
               int64_t batch0, int64_t batch1, int64_t m, int64_t n, int64_t k, const void* bias, int32_t epilogue,
               const mhlo_cuda_gemm_tuning* tuning, const PackScratch* scratch, cudaStream_t stream);
// fp32 operands and results on the FMA units, any strides.
bool gemm_fp32_supported(const GemmProblem& p);
int gemm_fp32_launch(const GemmProblem& p, cudaStream_t stream);
int gemm_device_error();       // synchronises; returns and clears the GEMM kernel's error word (-1: CUDA error)
int attention_device_error();  // same for the attention kernel
// Stream-ordered copies of the error words into pinned host memory, and host stores into them (clearing, or the test hook).
bool gemm_error_fetch_async(int* pinned_dst, cudaStream_t stream);
bool attention_error_fetch_async(int* pinned_dst, cudaStream_t stream);
bool gemm_error_store(int code);
bool attention_error_store(int code);
bool gemm_wait_expiry_probe(uint64_t limit_ns, cudaStream_t stream);
// One CTA: stores `epoch` into word `rank` of every other rank's flag array, then waits (at most limit_ns) until every word
// of this rank's own array has reached `epoch`; an expired wait records code 95 in the GEMM error word.
bool gemm_peer_barrier_launch(uint64_t* const* flag_arrays, int n_ranks, int rank, uint64_t epoch, uint64_t limit_ns, cudaStream_t stream);
// fp32 on the FMA units: any strides, optional additive mask, head dimensions up to 128.
bool attention_fp32_supported(int dtype, const AttnShape& s);
int attention_fp32_launch(const void* q, const void* k, const void* v, const void* mask, void* o, const AttnShape& s, cudaStream_t stream);
bool attention_tc_supported(int dtype, const AttnShape& s, const void* mask);
int attention_tc_launch(int dtype, const void* q, const void* k, const void* v, void* o, const AttnShape& s,
                        cudaStream_t stream);

}  // namespace mhlo
