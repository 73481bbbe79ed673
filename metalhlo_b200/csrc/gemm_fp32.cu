// fp32 products C = act(A . B + bias) on the FMA units, every operand layout. fp32 programs keep fp32 products and fp32
// accumulation, which the tensor cores do not offer, so the bound is the packed FMA rate (fma.rn.f32x2): 73 TFLOP/s
// measured over 148 SMs, against 59 TFLOP/s for scalar FMAs.
//
// A CTA of 256 threads owns a BM x BN tile and a thread 8 x 8 outputs, as 32 packed pairs along N; per step of K it reads
// 8 values of A (broadcast inside the warp) and 8 of B in four 16-byte shared-memory accesses for 32 packed FMAs. Panels
// are staged [k][m] and [k][n] by cp.async in a ring of three: 16-byte copies where the operand is contiguous along M (or
// N), 4-byte copies that transpose on the way otherwise, whole 32-byte sectors on the global side and 32 different banks
// on the shared side; a thread's addresses advance by constants (recomputing them cost 15 %). Two CTAs share an SM: with
// one (pairs along K instead, no duplicated operand, 254 registers) 4096^3 ran at 40 TFLOP/s, with two it runs at 54 to 59.
//
// Three shapes of the same CTA:  128 x 128, one group of threads;  64 x 64, four groups that take a quarter of every K
// panel each;  16 x 64, sixteen groups. Smaller tiles trade operand reuse for CTAs: the dispatch takes the largest whose
// tiles fill the 148 SMs and are mostly filled themselves. When even 64 x 64 (or 16 x 64) tiles are too few, K is split over a cluster of 2, 4 or 8 CTAs
// whose partial tiles meet through distributed shared memory - no workspace, no atomics, the same sum on every run.
#include <cooperative_groups.h>

#include <atomic>

#include "contraction.cuh"

namespace cg = cooperative_groups;

namespace mhlo {
namespace {

struct Fp32Gemm {
    const float* a;
    const float* b;
    float* c;
    const float* bias;
    int64_t as[4], bs[4];  // {batch0, batch1, row, col} element strides
    int64_t batch1, m, n, k;
    int32_t tiles_n, epilogue;
    int32_t a_mode, b_mode;  // how the panel is copied
    int32_t c_vec;           // rows of C on the 16-byte grid
};

enum PanelMode : int32_t {
    kRows16 = 0,  // contiguous along the rows, on the 16-byte grid: 16-byte copies
    kAcross = 1,  // contiguous along the rows: 4-byte copies, consecutive rows in consecutive lanes
    kAlongK = 2   // anything else: 4-byte copies that transpose, a warp takes 8 k x 4 rows
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool valid) {
    const int bytes = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src, bool valid) {
    const int bytes = valid ? 4 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ float fp32_epilogue(float x, int epilogue) {
    switch (epilogue) {
        case MHLO_EPILOGUE_RELU: return x > 0.f ? x : (x != x ? x : 0.f);
        case MHLO_EPILOGUE_GELU_TANH: return 0.5f * x * (1.f + tanhf(0.7978845608028654f * (x + 0.044715f * x * x * x)));
        case MHLO_EPILOGUE_GELU_ERF: return 0.5f * x * (1.f + erff(x * 0.70710678118654752440f));
        case MHLO_EPILOGUE_SILU: return x / (1.f + expf(-x));
        case MHLO_EPILOGUE_TANH: return tanhf(x);
        case MHLO_EPILOGUE_SIGMOID: return 1.f / (1.f + expf(-x));
        default: return x;
    }
}

// The panel of R rows x BK steps of one operand (element (r, k) at base + r * sr + k * sk) as a thread copies it to
// [k][row] in shared memory: which element it starts at and how it goes on.
template <int R, int BK>
struct Panel {
    static constexpr int kPitch = R + 4;  // floats per k; 4 mod 16, so 8 k x 4 rows hit 32 banks
    const float* src;   // this thread's first element of the panel in flight
    int64_t dsrc;       // to its next element
    int64_t next;       // to the next panel
    int64_t k;          // its k
    uint32_t dst;       // byte offset inside the stage
    int32_t mode, row;

    __device__ __forceinline__ void init(const float* base, int64_t sr, int64_t sk, int64_t r0, int64_t k0, int m) {
        int kk, rr;
        mode = m;
        if (m == kRows16) {
            kk = threadIdx.x / (R / 4);
            rr = threadIdx.x % (R / 4) * 4;
            dsrc = sk * (1024 / R);
        } else if (m == kAcross) {
            kk = threadIdx.x / R;
            rr = threadIdx.x % R;
            dsrc = sk * (256 / R);
        } else {
            const int w = threadIdx.x / 32, l = threadIdx.x % 32;
            kk = w % (BK / 8) * 8 + l % 8;
            rr = w / (BK / 8) * 4 + l / 8;
            dsrc = sr * (32 / (BK / 8));
        }
        row = static_cast<int32_t>(r0) + rr;
        k = k0 + kk;
        src = base + (r0 + rr) * sr + (k0 + kk) * sk;
        next = sk * BK;
        dst = static_cast<uint32_t>((kk * kPitch + rr) * 4);
    }
    // Copies the current panel to shared memory at `stage`; what lies outside the operand becomes zero. `base`: any
    // address of the operand, for copies of no bytes.
    __device__ __forceinline__ void load(uint32_t stage, const float* base, int32_t rows, int64_t k_end) {
        const float* s = src;
        if (mode == kRows16) {
            constexpr int kStep = 1024 / R;
            const int32_t left = row < rows ? static_cast<int32_t>(k_end - k < BK ? k_end - k : BK) : 0;  // rows is a multiple of 4
#pragma unroll
            for (int i = 0; i < BK / kStep; ++i, s += dsrc)
                cp_async16(stage + dst + i * kStep * kPitch * 4, i * kStep < left ? s : base, i * kStep < left);
        } else if (mode == kAcross) {
            constexpr int kStep = 256 / R;
            const int32_t left = row < rows ? static_cast<int32_t>(k_end - k < BK ? k_end - k : BK) : 0;
#pragma unroll
            for (int i = 0; i < BK / kStep; ++i, s += dsrc)
                cp_async4(stage + dst + i * kStep * kPitch * 4, i * kStep < left ? s : base, i * kStep < left);
        } else {
            constexpr int kStep = 32 / (BK / 8);
            const int32_t left = k < k_end ? rows - row : 0;
#pragma unroll
            for (int i = 0; i < R / kStep; ++i, s += dsrc)
                cp_async4(stage + dst + i * kStep * 4, i * kStep < left ? s : base, i * kStep < left);
        }
        src += next;
        k += BK;
    }
};

template <int BM, int BN, int BK, int KG>
struct Fp32Tile {
    static constexpr int kThreads = BM / 8 * (BN / 8) * KG;
    static constexpr int kStages = 3;
    static constexpr int kStageFloats = BK * (Panel<BM, BK>::kPitch + Panel<BN, BK>::kPitch);
    static constexpr size_t kRing = sizeof(float) * kStages * kStageFloats;
    static constexpr size_t kPartials = KG > 1 ? sizeof(float) * KG * BM * BN : 0;
    static constexpr size_t kShared = kRing > kPartials ? kRing : kPartials;
};

// SPLIT: the CTAs of a cluster share one tile and take equal ranges of K.
template <int BM, int BN, int BK, int KG, bool SPLIT>
__global__ void __launch_bounds__((Fp32Tile<BM, BN, BK, KG>::kThreads), 2) gemm_fp32_kernel(const __grid_constant__ Fp32Gemm p, int splits) {
    using Tile = Fp32Tile<BM, BN, BK, KG>;
    constexpr int NT = Tile::kThreads, S = Tile::kStages;
    constexpr int kGroup = NT / KG;       // threads of one K group
    constexpr int kCols = BN / 8;         // threads along N
    constexpr int kPerGroup = BK / KG;    // steps of K a group takes of every panel
    static_assert(NT == 256 && BK % KG == 0 && BK % 8 == 0 && BM % 16 == 0, "tile shape");
    extern __shared__ __align__(16) float smem[];
    const int tile = SPLIT ? blockIdx.x / splits : blockIdx.x;
    const int rank = SPLIT ? blockIdx.x % splits : 0;
    const int64_t m0 = static_cast<int64_t>(tile / p.tiles_n) * BM, n0 = static_cast<int64_t>(tile % p.tiles_n) * BN;
    const int64_t z = blockIdx.z, z0 = z / p.batch1, z1 = z % p.batch1;
    const float* a = p.a + z0 * p.as[0] + z1 * p.as[1];
    const float* b = p.b + z0 * p.bs[0] + z1 * p.bs[1];
    int64_t k_begin = 0, k_end = p.k;
    if (SPLIT) {  // whole panels per CTA
        const int64_t panels = (p.k + BK - 1) / BK, each = (panels + splits - 1) / splits;
        k_begin = rank * each * BK < p.k ? rank * each * BK : p.k;
        k_end = k_begin + each * BK < p.k ? k_begin + each * BK : p.k;
    }
    const int n_panels = static_cast<int>((k_end - k_begin + BK - 1) / BK);
    const uint32_t ring = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
    Panel<BM, BK> panel_a;
    Panel<BN, BK> panel_b;
    panel_a.init(a, p.as[2], p.as[3], m0, k_begin, p.a_mode);
    panel_b.init(b, p.bs[3], p.bs[2], n0, k_begin, p.b_mode);
    const int32_t rows_m = static_cast<int32_t>(p.m), rows_n = static_cast<int32_t>(p.n);
    auto load = [&](int stage) {
        const uint32_t at = ring + static_cast<uint32_t>(stage) * Tile::kStageFloats * 4;
        panel_a.load(at, a, rows_m, k_end);
        panel_b.load(at + BK * Panel<BM, BK>::kPitch * 4, b, rows_n, k_end);
    };
#pragma unroll
    for (int i = 0; i < S - 1; ++i) {
        if (i < n_panels) load(i);
        cp_async_commit();
    }
    const int group = threadIdx.x / kGroup, in_group = threadIdx.x % kGroup;
    // a warp is 4 threads along M x 8 along N where the group is that large: its reads of B are one 128-byte row
    int tm, tn;
    if constexpr (kGroup >= 32) {
        constexpr int kWarpsN = kCols / 8;
        const int warp = in_group / 32, lane = in_group % 32;
        tm = warp / kWarpsN * 4 + lane / 8;
        tn = warp % kWarpsN * 8 + lane % 8;
    } else {
        tm = in_group / kCols;
        tn = in_group % kCols;
    }
    float2 acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = make_float2(0.f, 0.f);
    int stage = 0;
    for (int i = 0; i < n_panels; ++i) {
        cp_async_wait<S - 2>();
        __syncthreads();
        if (i + S - 1 < n_panels) load(stage == 0 ? S - 1 : stage - 1);
        cp_async_commit();
        const float* pa = smem + stage * Tile::kStageFloats + group * kPerGroup * Panel<BM, BK>::kPitch + tm * 4;
        const float* pb = smem + stage * Tile::kStageFloats + BK * Panel<BM, BK>::kPitch + group * kPerGroup * Panel<BN, BK>::kPitch + tn * 4;
#pragma unroll
        for (int kk = 0; kk < kPerGroup; ++kk) {
            const float4 a0 = *reinterpret_cast<const float4*>(pa + kk * Panel<BM, BK>::kPitch);
            const float4 a1 = *reinterpret_cast<const float4*>(pa + kk * Panel<BM, BK>::kPitch + BM / 2);
            const float4 b0 = *reinterpret_cast<const float4*>(pb + kk * Panel<BN, BK>::kPitch);
            const float4 b1 = *reinterpret_cast<const float4*>(pb + kk * Panel<BN, BK>::kPitch + BN / 2);
            const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
            const float2 bv[4] = {make_float2(b0.x, b0.y), make_float2(b0.z, b0.w), make_float2(b1.x, b1.y), make_float2(b1.z, b1.w)};
#pragma unroll
            for (int r = 0; r < 8; ++r)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[r][q] = __ffma2_rn(make_float2(av[r], av[r]), bv[q], acc[r][q]);
        }
        stage = stage == S - 1 ? 0 : stage + 1;
    }
    cp_async_wait<0>();
    float* c = p.c + z * p.m * p.n;
    if constexpr (KG == 1) {
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const int64_t gm = m0 + r / 4 * (BM / 2) + tm * 4 + r % 4;
            if (gm >= p.m) continue;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int64_t gn = n0 + h * (BN / 2) + tn * 4;
                float v[4] = {acc[r][2 * h].x, acc[r][2 * h].y, acc[r][2 * h + 1].x, acc[r][2 * h + 1].y};
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (gn + e < p.n) v[e] = fp32_epilogue(p.bias != nullptr ? v[e] + p.bias[gn + e] : v[e], p.epilogue);
                if (p.c_vec && gn + 3 < p.n) {
                    *reinterpret_cast<float4*>(c + gm * p.n + gn) = make_float4(v[0], v[1], v[2], v[3]);
                } else {
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (gn + e < p.n) c[gm * p.n + gn + e] = v[e];
                }
            }
        }
        return;
    }
    // the groups' partial tiles meet in shared memory (over the ring, which nobody reads any more)
    __syncthreads();
    float* mine = smem + group * BM * BN;
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int h = 0; h < 2; ++h)
            *reinterpret_cast<float4*>(mine + (r / 4 * (BM / 2) + tm * 4 + r % 4) * BN + h * (BN / 2) + tn * 4) =
                make_float4(acc[r][2 * h].x, acc[r][2 * h].y, acc[r][2 * h + 1].x, acc[r][2 * h + 1].y);
    __syncthreads();
    auto finish = [&](int e, float4 v) {  // 4 outputs from tile element e on
        const int64_t gm = m0 + e / BN, gn = n0 + e % BN;
        if (gm >= p.m) return;
        float x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (gn + q < p.n) x[q] = fp32_epilogue(p.bias != nullptr ? x[q] + p.bias[gn + q] : x[q], p.epilogue);
        if (p.c_vec && gn + 3 < p.n) {
            *reinterpret_cast<float4*>(c + gm * p.n + gn) = make_float4(x[0], x[1], x[2], x[3]);
        } else {
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (gn + q < p.n) c[gm * p.n + gn + q] = x[q];
        }
    };
    auto sum_groups = [&](int e) {
        float4 s = *reinterpret_cast<const float4*>(smem + e);
#pragma unroll
        for (int g = 1; g < KG; ++g) {
            const float4 t = *reinterpret_cast<const float4*>(smem + g * BM * BN + e);
            s.x += t.x; s.y += t.y; s.z += t.z; s.w += t.w;
        }
        return s;
    };
    if constexpr (!SPLIT) {
        for (int e = threadIdx.x * 4; e < BM * BN; e += NT * 4) finish(e, sum_groups(e));
    } else {
        // this CTA's sum over its groups goes to the front of its shared memory; every CTA then finishes an equal part of
        // the tile from all of them
        for (int e = threadIdx.x * 4; e < BM * BN; e += NT * 4) *reinterpret_cast<float4*>(smem + e) = sum_groups(e);
        cg::cluster_group cluster = cg::this_cluster();
        cluster.sync();
        const int part = BM * BN / splits;
        for (int e = rank * part + threadIdx.x * 4; e < (rank + 1) * part; e += NT * 4) {
            float4 s = *reinterpret_cast<const float4*>(cluster.map_shared_rank(smem, 0) + e);
            for (int r = 1; r < splits; ++r) {
                const float4 t = *reinterpret_cast<const float4*>(cluster.map_shared_rank(smem, r) + e);
                s.x += t.x; s.y += t.y; s.z += t.z; s.w += t.w;
            }
            finish(e, s);
        }
        cluster.sync();  // nobody leaves while its shared memory is being read
    }
}

int panel_mode(const float* base, int64_t rows, int64_t row_stride, int64_t k_stride, const int64_t* batch_strides) {
    if (row_stride != 1) return kAlongK;
    const bool grid16 = aligned16(base) && rows % 4 == 0 && k_stride % 4 == 0 && batch_strides[0] % 4 == 0 && batch_strides[1] % 4 == 0;
    return grid16 ? kRows16 : kAcross;
}

template <int BM, int BN, int BK, int KG, bool SPLIT>
int launch(const Fp32Gemm& p, int64_t tiles, int64_t batches, int splits, cudaStream_t stream) {
    using Tile = Fp32Tile<BM, BN, BK, KG>;
    auto kernel = gemm_fp32_kernel<BM, BN, BK, KG, SPLIT>;
    static std::atomic<uint64_t> configured{0};  // devices whose copy of the kernel may use this much shared memory
    int dev = 0;
    MHLO_CUDA_TRY(cudaGetDevice(&dev), MHLO_CUDA_NO_DEVICE);
    const uint64_t bit = uint64_t{1} << (dev & 63);
    if (!(configured.load(std::memory_order_relaxed) & bit)) {
        MHLO_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(Tile::kShared)), MHLO_CUDA_EXECUTION_FAILED);
        configured.fetch_or(bit, std::memory_order_relaxed);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(tiles * splits), 1, static_cast<unsigned>(batches));
    cfg.blockDim = dim3(Tile::kThreads);
    cfg.dynamicSmemBytes = Tile::kShared;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<unsigned>(splits);
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = SPLIT ? 1 : 0;
    MHLO_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, p, splits), MHLO_CUDA_EXECUTION_FAILED);
    return MHLO_CUDA_OK;
}

// Tiles are made smaller, and K is split, until four fifths of the SMs have two CTAs: one CTA (8 warps) does not cover the
// latency of its shared-memory reads (2048 x 1024 x 256 in 128 tiles of 128 x 128: 46.6 us, in 512 of 64 x 64: 37.0 us;
// 512 x 1024 x 1024: 39.0 us as 128 CTAs, 38.1 us as 256, 42.4 us as 512 with panels too few per CTA).
constexpr int64_t kFill = 236;

template <int BM, int BN, int BK, int KG>
int launch_split(Fp32Gemm p, int64_t batches, cudaStream_t stream) {
    p.tiles_n = static_cast<int32_t>((p.n + BN - 1) / BN);
    const int64_t tiles = (p.m + BM - 1) / BM * p.tiles_n, panels = (p.k + BK - 1) / BK;
    // enough CTAs for the machine, as long as each has a panel of its own (a 64 x 64 tile: two, so that copies overlap)
    int splits = 1;
    while (splits < 8 && tiles * batches * splits < kFill && panels >= splits * 2 * (BM >= 64 ? 2 : 1)) splits *= 2;
    if (tiles * splits > 0x7fffffff) return fail(MHLO_CUDA_UNSUPPORTED, "gemm: more than 2^31 tiles");
    if (splits == 1) return launch<BM, BN, BK, KG, false>(p, tiles, batches, 1, stream);
    return launch<BM, BN, BK, KG, true>(p, tiles, batches, splits, stream);
}

}  // namespace

// Few steps of K in many tiles: a CTA's prologue (addresses, the ring's first two panels) is then most of its work and the general
// kernel is quicker: 4096 products of [64,4] . [4,4] 41 us there, 67 here; [262144,8] . [8,32] 42 and 68. At K = 32 the second takes
// 69 and 70, at K = 64 120 and 80; with two tiles per SM or fewer this kernel leads at any K.
static bool short_sums(const GemmProblem& g) {
    const int64_t tiles = (g.m <= 16 ? 1 : (g.m + 63) / 64) * ((g.n + 63) / 64) * g.batch0 * g.batch1;
    return g.k <= 16 && tiles > 2 * kNumSMs && general_kernel_takes(g);
}

bool gemm_fp32_supported(const GemmProblem& g) {
    if (g.batch0 <= 0 || g.batch1 <= 0 || g.m <= 0 || g.n <= 0 || short_sums(g)) return false;
    return g.in_dtype == MHLO_DT_F32 && g.out_dtype == MHLO_DT_F32 && g.residual == nullptr && g.n_copies == 0 && (g.ldc == 0 || g.ldc == g.n) &&
           g.c_col0 == 0 && g.batch0 * g.batch1 <= 65535 && g.m * g.n > 0 && g.k > 0 && g.m < (int64_t{1} << 31) && g.n < (int64_t{1} << 31);
}

int gemm_fp32_launch(const GemmProblem& g, cudaStream_t stream) {
    if (g.a == nullptr || g.b == nullptr || g.c == nullptr) return fail(MHLO_CUDA_INVALID_ARGUMENT, "gemm: null pointer");
    Fp32Gemm p;
    p.a = static_cast<const float*>(g.a);
    p.b = static_cast<const float*>(g.b);
    p.c = static_cast<float*>(g.c);
    p.bias = static_cast<const float*>(g.bias);
    for (int i = 0; i < 4; ++i) { p.as[i] = g.as[i]; p.bs[i] = g.bs[i]; }
    p.batch1 = g.batch1; p.m = g.m; p.n = g.n; p.k = g.k;
    p.epilogue = g.epilogue;
    p.a_mode = panel_mode(p.a, g.m, g.as[2], g.as[3], g.as);
    p.b_mode = panel_mode(p.b, g.n, g.bs[3], g.bs[2], g.bs);
    p.c_vec = aligned16(g.c) && g.n % 4 == 0;
    const int64_t batches = g.batch0 * g.batch1;
    if (g.m <= 16) return launch_split<16, 64, 64, 16>(p, batches, stream);
    p.tiles_n = static_cast<int32_t>((p.n + 127) / 128);
    const int64_t large = (p.m + 127) / 128 * p.tiles_n;
    if (large > 0x7fffffff) return fail(MHLO_CUDA_UNSUPPORTED, "gemm: more than 2^31 tiles");
    // Large tiles only where at least 0.6 of them is results (a row or column block of 64 of the 128 takes no less time than a
    // whole one: [65536,64] . [64,32] 47 us, 24 in tiles of 64 x 64) and K is more than two panels of the small tile.
    const bool filled = 5 * p.m * p.n >= 3 * large * 128 * 128;
    if (large * batches >= kFill && filled && p.k > 64) return launch<128, 128, 16, 1, false>(p, large, batches, 1, stream);
    return launch_split<64, 64, 32, 4>(p, batches, stream);
}

}  // namespace mhlo
