// fp32 attention on the FMA units: softmax(scale . Q K^T + mask) V with fp32 products and sums, any strides with the head
// dimension contiguous, head dimensions up to 128. Bound by the packed FMA rate (73 TFLOP/s measured), like the fp32 GEMM.
//
// A CTA walks the keys of one (batch, head) for 32 x RG query rows, 32 keys at a time (64 with two warps per row group). A
// warp owns 32 rows: its scores are an 8 x 4 register tile per thread (4 threads along the rows x 8 along the keys, so a row
// lives in 8 lanes and its maximum takes three shuffles), the probabilities go through shared memory as [key][row] - the layout the product with V reads like
// any other left operand - and O stays in registers, 8 rows x 8 columns per thread, rescaled when a row's maximum moves.
// Head dimensions above 64 take two warps per 32 rows (HALVES = 2): each scores half of the keys and then accumulates half
// of the head dimension; they exchange row maxima and probabilities through shared memory and a barrier of their own, which
// keeps two warps' worth of accumulators out of one register file.
// K is transposed on the way in (4-byte cp.async, 8 elements x 4 keys per warp instruction), V arrives in 16-byte copies;
// the next K is in flight during the softmax and the product with V, the next V during the next scores.
// 32 keys and at most 168 registers let three CTAs of four warps share an SM: [8,12,512,64] is one wave of 384 CTAs and runs
// in 174 us (37 TFLOP/s); with 64 keys, two CTAs and two waves it took 210 us against 188. Tiles too few for the machine share their
// keys among a cluster of up to 8 CTAs, whose sums, maxima and partial O meet through distributed shared memory: one head of
// 1024 causal rows 198 us without, 31 us with it. One warp per query row with scalar loads, the former kernel, took 6.94 ms
// and 571 us.
#include <cooperative_groups.h>

#include <atomic>

#include "contraction.cuh"

namespace cg = cooperative_groups;

namespace mhlo {
namespace {

struct Fp32Attention {
    const float *q, *k, *v, *mask;
    float* o;
    int64_t qs[3], ks[3], vs[3], os[3];  // {batch, head, sequence}
    int32_t heads, seq_q, seq_k, head_dim, causal;
    int32_t splits;        // CTAs of a cluster that share a tile's keys
    int32_t v_vec, o_vec;  // 16-byte copies of V rows, 16-byte stores of O rows
    float scale;
};

__device__ __forceinline__ void cp4(uint32_t dst, const void* src, bool valid) {
    const int bytes = valid ? 4 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp16(uint32_t dst, const void* src, bool valid) {
    const int bytes = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <int RG, int HALVES, int KEYS>
struct Fp32AttentionTile {
    static constexpr int kThreads = 32 * RG * HALVES, kRows = 32 * RG, kDim = 64 * HALVES;
    static constexpr int kQPitch = kRows + 4, kKPitch = KEYS + 4, kVPitch = kDim + 4, kPPitch = 36;
    static constexpr int kQ = kDim * kQPitch, kK = kDim * kKPitch, kV = KEYS * kVPitch, kP = RG * KEYS * kPPitch, kM = 2 * kRows;
    // registers for three CTAs of four warps on an SM; two warps per row group hold fewer accumulators each
    static constexpr int kMinCtas = RG == 4 && HALVES == 1 ? 3 : 1;
    static_assert(kRows * (kDim + 4) <= kQ + kK + kV, "the partial results fit where the operands were");
    static constexpr size_t kShared = sizeof(float) * (kQ + kK + kV + kP + kM);
};

// Rows [r0, r0 + R) of a [rows, dim] matrix (row stride `stride`) to shared memory as [d][row], zeros outside.
template <int R, int PITCH, int DIM, int WARPS>
__device__ __forceinline__ void load_transposed(uint32_t dst, const float* base, int64_t stride, int r0, int rows, int dim) {
    const int w = threadIdx.x / 32, l = threadIdx.x % 32;
    constexpr int kAlong = DIM / 8 / WARPS;  // 8-element blocks of the head dimension a warp takes
    static_assert(DIM / 8 % WARPS == 0, "a warp takes whole blocks");
    const int d = w * kAlong * 8 + l % 8;
    int r = r0 + l / 8;
    const float* s = base + static_cast<int64_t>(r) * stride + d;
    uint32_t to = dst + static_cast<uint32_t>((d * PITCH + l / 8) * 4);
#pragma unroll 4
    for (int i = 0; i < R / 4; ++i, r += 4, s += 4 * stride, to += 16) {
#pragma unroll
        for (int a = 0; a < kAlong; ++a) {
            const bool ok = r < rows && d + a * 8 < dim;
            cp4(to + a * 8 * PITCH * 4, ok ? s + a * 8 : base, ok);
        }
    }
}

template <int R, int DIM, int PITCH, int NT>
__device__ __forceinline__ void load_rows(uint32_t dst, const float* base, int64_t stride, int r0, int rows, int dim, int vec) {
    if (vec) {
        constexpr int kPerRow = DIM / 4;
#pragma unroll 4
        for (int e = threadIdx.x; e < R * kPerRow; e += NT) {
            const int r = e / kPerRow, d = e % kPerRow * 4;
            const bool ok = r0 + r < rows && d < dim;
            cp16(dst + (r * PITCH + d) * 4, ok ? base + static_cast<int64_t>(r0 + r) * stride + d : base, ok);
        }
    } else {
#pragma unroll 4
        for (int e = threadIdx.x; e < R * DIM; e += NT) {
            const int r = e / DIM, d = e % DIM;
            const bool ok = r0 + r < rows && d < dim;
            cp4(dst + (r * PITCH + d) * 4, ok ? base + static_cast<int64_t>(r0 + r) * stride + d : base, ok);
        }
    }
}

// acc[8][2C] += a . b for one step: 8 values of the left operand (two groups of four rows) against C groups of four columns.
// MASKED: only the rows whose place in the warp's rows (less the thread's first) is at least `first` take part.
template <int C, bool MASKED = false>
__device__ __forceinline__ void step(float2 (*acc)[2 * C], const float* a, const float* b, int b_apart, int first = 0) {
    const float4 a0 = *reinterpret_cast<const float4*>(a), a1 = *reinterpret_cast<const float4*>(a + 16);
    const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
    for (int c = 0; c < C; ++c) {
        const float4 x = *reinterpret_cast<const float4*>(b + c * b_apart);
        const float2 lo = make_float2(x.x, x.y), hi = make_float2(x.z, x.w);
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            if (MASKED && r / 4 * 16 + r % 4 < first) continue;
            const float2 d = make_float2(av[r], av[r]);
            acc[r][2 * c] = __ffma2_rn(d, lo, acc[r][2 * c]);
            acc[r][2 * c + 1] = __ffma2_rn(d, hi, acc[r][2 * c + 1]);
        }
    }
}

template <int RG, int HALVES, int kKeys, bool CAUSAL>
__global__ void __launch_bounds__((Fp32AttentionTile<RG, HALVES, kKeys>::kThreads), (Fp32AttentionTile<RG, HALVES, kKeys>::kMinCtas))
attention_fp32_kernel(const __grid_constant__ Fp32Attention p) {
    using T = Fp32AttentionTile<RG, HALVES, kKeys>;
    constexpr int NT = T::kThreads, C = kKeys / (32 * HALVES);  // C: groups of four keys a thread scores
    extern __shared__ __align__(16) float smem[];
    float* const sq = smem;
    float* const sk = sq + T::kQ;
    float* const sv = sk + T::kK;
    float* const sp = sv + T::kV;
    float* const sm = sp + T::kP;
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, group = warp % RG, half = warp / RG;
    const int ty = lane / 8, tx = lane % 8;
    const int rank = static_cast<int>(blockIdx.x) % p.splits, head = static_cast<int>(blockIdx.x) / p.splits;
    // the tiles that see most keys under a causal mask first, those of all heads before the next: every SM gets some of each
    const int tile = CAUSAL ? static_cast<int>(gridDim.y) - 1 - static_cast<int>(blockIdx.y) : static_cast<int>(blockIdx.y);
    const int q0 = tile * T::kRows;
    const int64_t b = head / p.heads, h = head % p.heads;
    const float* q = p.q + b * p.qs[0] + h * p.qs[1];
    const float* k = p.k + b * p.ks[0] + h * p.ks[1];
    const float* v = p.v + b * p.vs[0] + h * p.vs[1];
    float* o = p.o + b * p.os[0] + h * p.os[1];
    const uint32_t aq = static_cast<uint32_t>(__cvta_generic_to_shared(sq)), ak = static_cast<uint32_t>(__cvta_generic_to_shared(sk)),
                   av = static_cast<uint32_t>(__cvta_generic_to_shared(sv));
    int limit = p.seq_k;  // keys any row of this tile sees
    if (CAUSAL && q0 + T::kRows < limit) limit = q0 + T::kRows;
    const int n_blocks = (limit + kKeys - 1) / kKeys;
    // the two warps of a row group
    auto pair_sync = [&]() {
        if constexpr (HALVES == 1) __syncwarp();
        else asm volatile("bar.sync %0, 64;" ::"r"(1 + group) : "memory");
    };

    if (rank < n_blocks) {
        load_transposed<T::kRows, T::kQPitch, T::kDim, NT / 32>(aq, q, p.qs[2], q0, p.seq_q, p.head_dim);
        load_transposed<kKeys, T::kKPitch, T::kDim, NT / 32>(ak, k, p.ks[2], rank * kKeys, p.seq_k, p.head_dim);
    }
    cp_commit();
    if (rank < n_blocks) load_rows<kKeys, T::kDim, T::kVPitch, NT>(av, v, p.vs[2], rank * kKeys, p.seq_k, p.head_dim, p.v_vec);
    cp_commit();

    // thread's rows: ty * 4 + {0..3} and 16 + ty * 4 + {0..3} of the warp's 32
    float2 out[8][4];
    float m[8], l[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        m[r] = -INFINITY;
        l[r] = 0.f;
#pragma unroll
        for (int c = 0; c < 4; ++c) out[r][c] = make_float2(0.f, 0.f);
    }
    auto row_of = [&](int r) { return q0 + group * 32 + (r / 4) * 16 + ty * 4 + r % 4; };
    const float* qa = sq + group * 32 + ty * 4;
    const float* kb = sk + half * 32 + tx * 4;
    float* const pw = sp + group * kKeys * T::kPPitch;
    const float* vb = sv + half * 64 + tx * 4;

    for (int j = rank; j < n_blocks; j += p.splits) {
        cp_wait<1>();  // K of this block (and Q); V may still be on its way
        __syncthreads();
        float2 s[8][2 * C];
#pragma unroll
        for (int r = 0; r < 8; ++r)
#pragma unroll
            for (int c = 0; c < 2 * C; ++c) s[r][c] = make_float2(0.f, 0.f);
#pragma unroll 8
        for (int d = 0; d < T::kDim; ++d) step<C>(s, qa + d * T::kQPitch, kb + d * T::kKPitch, 32);
        __syncthreads();  // every warp is done with K
        if (j + p.splits < n_blocks) load_transposed<kKeys, T::kKPitch, T::kDim, NT / 32>(ak, k, p.ks[2], (j + p.splits) * kKeys, p.seq_k, p.head_dim);
        cp_commit();

        const int key0 = j * kKeys + half * 32 + tx * 4;  // this thread's keys: key0 + {0..3} (+ 32)
        const bool ragged = (j + 1) * kKeys > p.seq_k || (CAUSAL && (j + 1) * kKeys - 1 > q0 + group * 32);
        float* sf = reinterpret_cast<float*>(s);
#pragma unroll
        for (int r = 0; r < 8; ++r)
#pragma unroll
            for (int e = 0; e < 4 * C; ++e) {
                float x = sf[r * 4 * C + e] * p.scale;
                const int key = key0 + e / 4 * 32 + e % 4;
                if (p.mask != nullptr) {
                    const int row = row_of(r);
                    if (row < p.seq_q && key < p.seq_k) x += p.mask[static_cast<int64_t>(row) * p.seq_k + key];
                }
                if (ragged && (key >= p.seq_k || (CAUSAL && key > row_of(r)))) x = -INFINITY;
                sf[r * 4 * C + e] = x;
            }
        float top[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            float x = sf[r * 4 * C];
#pragma unroll
            for (int e = 1; e < 4 * C; ++e) x = fmaxf(x, sf[r * 4 * C + e]);
#pragma unroll
            for (int w = 4; w > 0; w >>= 1) x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, w));
            top[r] = x;
        }
        if constexpr (HALVES == 2) {
            if (tx == 0)
#pragma unroll
                for (int r = 0; r < 8; ++r) sm[half * T::kRows + group * 32 + r / 4 * 16 + ty * 4 + r % 4] = top[r];
            pair_sync();
#pragma unroll
            for (int r = 0; r < 8; ++r) top[r] = fmaxf(top[r], sm[(1 - half) * T::kRows + group * 32 + r / 4 * 16 + ty * 4 + r % 4]);
        }
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const float mn = fmaxf(m[r], top[r]);
            const float corr = m[r] == -INFINITY ? 0.f : __expf(m[r] - mn);
            m[r] = mn;
            float sum = 0.f;
#pragma unroll
            for (int e = 0; e < 4 * C; ++e) {
                const float x = sf[r * 4 * C + e];
                const float pr = x == -INFINITY ? 0.f : __expf(x - mn);  // a maximum of -inf leaves -inf and NaN: NaN stays NaN
                sf[r * 4 * C + e] = pr;
                sum += pr;
            }
            l[r] = l[r] * corr + sum;
            const float2 c2 = make_float2(corr, corr);
#pragma unroll
            for (int c = 0; c < 4; ++c) out[r][c] = __fmul2_rn(out[r][c], c2);
        }
#pragma unroll
        for (int e = 0; e < 4 * C; ++e) {
            float* to = pw + (half * 32 + e / 4 * 32 + tx * 4 + e % 4) * T::kPPitch + ty * 4;
            *reinterpret_cast<float4*>(to) = make_float4(sf[e], sf[4 * C + e], sf[8 * C + e], sf[12 * C + e]);
            *reinterpret_cast<float4*>(to + 16) = make_float4(sf[16 * C + e], sf[20 * C + e], sf[24 * C + e], sf[28 * C + e]);
        }
        cp_wait<1>();  // V of this block; the next K may still be on its way
        __syncthreads();
        // keys of this block that some of the warp's rows do not see: those rows leave the key's V alone, which need not be finite
        const int behind = j * kKeys - (q0 + group * 32);  // key - row of the block's first key and the warp's first row
        if (!CAUSAL || behind + kKeys - 1 <= 0) {
#pragma unroll 8
            for (int key = 0; key < kKeys; ++key) step<2>(out, pw + key * T::kPPitch + ty * 4, vb + key * T::kVPitch, 32);
        } else {
            const int seen = 32 - behind < kKeys ? 32 - behind : kKeys;  // by the warp's last row
#pragma unroll 8
            for (int key = 0; key < seen; ++key)
                step<2, true>(out, pw + key * T::kPPitch + ty * 4, vb + key * T::kVPitch, 32, behind + key - ty * 4);
        }
        __syncthreads();  // every warp is done with V (and with its probabilities)
        if (j + p.splits < n_blocks) load_rows<kKeys, T::kDim, T::kVPitch, NT>(av, v, p.vs[2], (j + p.splits) * kKeys, p.seq_k, p.head_dim, p.v_vec);
        cp_commit();
    }
    cp_wait<0>();
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int w = 4; w > 0; w >>= 1) l[r] += __shfl_xor_sync(0xffffffffu, l[r], w);
    if constexpr (HALVES == 2) {
        if (tx == 0)
#pragma unroll
            for (int r = 0; r < 8; ++r) sm[half * T::kRows + group * 32 + r / 4 * 16 + ty * 4 + r % 4] = l[r];
        pair_sync();
#pragma unroll
        for (int r = 0; r < 8; ++r) l[r] += sm[(1 - half) * T::kRows + group * 32 + r / 4 * 16 + ty * 4 + r % 4];
    }
    auto store4 = [&](int row, int d, float4 x) {
        float* to = o + static_cast<int64_t>(row) * p.os[2] + d;
        if (p.o_vec && d + 3 < p.head_dim) {
            *reinterpret_cast<float4*>(to) = x;
            return;
        }
        if (d < p.head_dim) to[0] = x.x;
        if (d + 1 < p.head_dim) to[1] = x.y;
        if (d + 2 < p.head_dim) to[2] = x.z;
        if (d + 3 < p.head_dim) to[3] = x.w;
    };
    auto inverse = [](float sum) { return sum > 0.f ? 1.0f / sum : (sum != sum ? sum : 0.f); };
    if (p.splits > 1) {
        // partial sums, row maxima and row sums of this CTA's keys, then an equal part of the rows from all of them
        constexpr int kPitch = T::kDim + 4;
        __syncthreads();
        float* const so = smem;
        float* const sl = sm + T::kRows;
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const int row = group * 32 + r / 4 * 16 + ty * 4 + r % 4;
#pragma unroll
            for (int c = 0; c < 2; ++c)
                *reinterpret_cast<float4*>(so + row * kPitch + half * 64 + c * 32 + tx * 4) =
                    make_float4(out[r][2 * c].x, out[r][2 * c].y, out[r][2 * c + 1].x, out[r][2 * c + 1].y);
            if (tx == 0 && half == 0) {
                sm[row] = m[r];
                sl[row] = l[r];
            }
        }
        cg::cluster_group cluster = cg::this_cluster();
        cluster.sync();
        const int rows = T::kRows / p.splits;
        for (int e = threadIdx.x; e < rows * (T::kDim / 4); e += NT) {
            const int row = rank * rows + e / (T::kDim / 4), d = e % (T::kDim / 4) * 4;
            float top = -INFINITY;
            for (int c = 0; c < p.splits; ++c) top = fmaxf(top, cluster.map_shared_rank(sm, c)[row]);
            float sum = 0.f;
            float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int c = 0; c < p.splits; ++c) {
                const float mc = cluster.map_shared_rank(sm, c)[row];
                const float w = mc == -INFINITY ? 0.f : __expf(mc - top);
                sum += w * cluster.map_shared_rank(sl, c)[row];
                const float4 y = *reinterpret_cast<const float4*>(cluster.map_shared_rank(so, c) + row * kPitch + d);
                x.x += w * y.x; x.y += w * y.y; x.z += w * y.z; x.w += w * y.w;
            }
            const float inv = inverse(sum);
            if (q0 + row < p.seq_q) store4(q0 + row, d, make_float4(x.x * inv, x.y * inv, x.z * inv, x.w * inv));
        }
        cluster.sync();  // nobody leaves while its shared memory is being read
        return;
    }
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const int row = row_of(r);
        if (row >= p.seq_q) continue;
        const float inv = inverse(l[r]);
#pragma unroll
        for (int c = 0; c < 2; ++c)
            store4(row, half * 64 + c * 32 + tx * 4,
                   make_float4(out[r][2 * c].x * inv, out[r][2 * c].y * inv, out[r][2 * c + 1].x * inv, out[r][2 * c + 1].y * inv));
    }
}

template <int RG, int HALVES, int KEYS>
int launch(Fp32Attention p, int64_t batch_heads, cudaStream_t stream) {
    using T = Fp32AttentionTile<RG, HALVES, KEYS>;
    // A kernel of its own for causal masks: as a run-time condition their rows' limits cost the others 3 to 6 % (without them and with
    // the mask known at compile time [8,12,512,64] 174 us, one query against 1024 keys of 12 heads 26). Under a mask the limits cost
    // nothing up to head dimension 64 and 4 to 6 % above.
    auto kernel = p.causal ? attention_fp32_kernel<RG, HALVES, KEYS, true> : attention_fp32_kernel<RG, HALVES, KEYS, false>;
    static std::atomic<uint64_t> configured{0};  // devices whose copies of the kernels may use this much shared memory
    int dev = 0;
    MHLO_CUDA_TRY(cudaGetDevice(&dev), MHLO_CUDA_NO_DEVICE);
    const uint64_t bit = uint64_t{1} << (dev & 63);
    if (!(configured.load(std::memory_order_relaxed) & bit)) {
        for (auto each : {attention_fp32_kernel<RG, HALVES, KEYS, true>, attention_fp32_kernel<RG, HALVES, KEYS, false>})
            MHLO_CUDA_TRY(cudaFuncSetAttribute(each, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(T::kShared)), MHLO_CUDA_EXECUTION_FAILED);
        configured.fetch_or(bit, std::memory_order_relaxed);
    }
    const int64_t tiles = (p.seq_q + T::kRows - 1) / T::kRows;
    // few query rows and many keys: the keys of a tile are shared by a cluster
    const int64_t blocks = (p.seq_k + KEYS - 1) / KEYS;
    p.splits = 1;
    while (RG == 1 && p.splits < 8 && tiles * batch_heads * p.splits * 2 <= 2 * kNumSMs && blocks >= p.splits * 2) p.splits *= 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(batch_heads * p.splits), static_cast<unsigned>(tiles));
    cfg.blockDim = dim3(T::kThreads);
    cfg.dynamicSmemBytes = T::kShared;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<unsigned>(p.splits);
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = p.splits > 1 ? 1 : 0;
    MHLO_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, p), MHLO_CUDA_EXECUTION_FAILED);
    return MHLO_CUDA_OK;
}

}  // namespace

// Whether the tiles are quicker than the general kernel's warp per query row. A tile costs the same whether 1 or 32 of its rows exist:
// one query against many keys of many heads (a decoding step), or a handful of keys, is the general kernel's. The times (us) are
// fits to 508 measured shapes (1 to 4096 heads, 1 to 32 queries, 1 to 512 keys, head dimensions 4 to 128); none of them is sent to
// the tiles to take longer there. 4096 heads of one query and 128 keys of 64: 236 us there, 411 here; 8 queries: 1319 and 420.
static bool tiles_pay(const AttnShape& s) {
    const int64_t heads = s.batch * s.heads, rows = heads * s.seq_q, keys = s.causal && s.seq_q < s.seq_k ? s.seq_q : s.seq_k;
    const double dim = static_cast<double>(s.head_dim), seen = s.causal ? 0.5 * static_cast<double>(keys + 1) : static_cast<double>(keys);
    const double one_row = 3.0 + static_cast<double>(keys) * (0.13 + 0.0045 * dim);              // a warp's chain over its keys
    const double all_rows = static_cast<double>(rows) * (0.45 + seen * (0.034 + 0.0036 * dim)) * 1e-3;  // the machine full of warps
    const int64_t tiles = heads * ((s.seq_q + 31) / 32), per = s.head_dim <= 64 ? 32 : 64, blocks = (keys + per - 1) / per;
    int64_t splits = 1;
    while (splits < 8 && tiles * splits * 2 <= 2 * kNumSMs && blocks >= splits * 2) splits *= 2;
    const double longest = static_cast<double>((blocks + splits - 1) / splits), exchange = splits > 1 ? 4.0 : 0.0;
    double one_tile, all_tiles;
    if (s.head_dim <= 64) {
        one_tile = 3.5 + 5.2 * longest + exchange;
        all_tiles = static_cast<double>(tiles) * (3.5 + 24.5 * static_cast<double>(blocks)) * 1e-3;
    } else {  // one CTA to an SM
        one_tile = 2.0 + 10.3 * longest + exchange;
        all_tiles = tiles > kNumSMs ? (2.0 + 13.5 * static_cast<double>(blocks)) * static_cast<double>((tiles + kNumSMs - 1) / kNumSMs) : 0.0;
    }
    return (one_tile > all_tiles ? one_tile : all_tiles) <= (one_row > all_rows ? one_row : all_rows);
}

bool attention_fp32_supported(int dtype, const AttnShape& s) {
    const bool general = s.batch * s.heads * s.seq_q <= int64_t{4} * 0x7fffffff;  // rows the general kernel's grid holds
    if (general && !tiles_pay(s)) return false;
    return dtype == MHLO_DT_F32 && s.head_dim <= 128 && s.batch * s.heads < (int64_t{1} << 27) && s.seq_q <= 32 * int64_t{65535} &&
           s.seq_k < (int64_t{1} << 30);
}

int attention_fp32_launch(const void* q, const void* k, const void* v, const void* mask, void* o, const AttnShape& s, cudaStream_t stream) {
    Fp32Attention p;
    p.q = static_cast<const float*>(q); p.k = static_cast<const float*>(k); p.v = static_cast<const float*>(v);
    p.mask = static_cast<const float*>(mask); p.o = static_cast<float*>(o);
    bool v_grid = aligned16(v) && s.head_dim % 4 == 0, o_grid = aligned16(o) && s.head_dim % 4 == 0;
    for (int i = 0; i < 3; ++i) {
        p.qs[i] = s.qs[i]; p.ks[i] = s.ks[i]; p.vs[i] = s.vs[i]; p.os[i] = s.os[i];
        v_grid = v_grid && s.vs[i] % 4 == 0;
        o_grid = o_grid && s.os[i] % 4 == 0;
    }
    p.heads = static_cast<int32_t>(s.heads); p.seq_q = static_cast<int32_t>(s.seq_q); p.seq_k = static_cast<int32_t>(s.seq_k);
    p.head_dim = static_cast<int32_t>(s.head_dim); p.causal = s.causal;
    p.v_vec = v_grid; p.o_vec = o_grid;
    p.scale = s.scale;
    // as many query rows per CTA as still give every SM one
    const int64_t bh = s.batch * s.heads;
    const auto ctas = [&](int64_t rows) { return (s.seq_q + rows - 1) / rows * bh; };
    if (s.head_dim <= 64) {
        if (ctas(128) >= 2 * kNumSMs) return launch<4, 1, 32>(p, bh, stream);
        if (ctas(64) >= kNumSMs) return launch<2, 1, 32>(p, bh, stream);
        return launch<1, 1, 32>(p, bh, stream);
    }
    if (ctas(128) >= kNumSMs) return launch<4, 2, 64>(p, bh, stream);
    if (ctas(64) >= kNumSMs) return launch<2, 2, 64>(p, bh, stream);
    return launch<1, 2, 64>(p, bh, stream);
}

}  // namespace mhlo
