// Products with few output tiles (small batches, short prompts, narrow layers): K is split over a cluster of CTAs.
//
// A 128 x 128 tile with K = 3072 is 48 steps of 32 KB through one SM's port to L2 (about 0.3 us each), so a product of a
// dozen tiles ran for 12 to 16 us on a dozen SMs. Here 2, 4 or 8 CTAs of a cluster take equal ranges of K of one tile, each
// with its own TMA ring and TMEM accumulator; the fp32 partial tiles are written to shared memory over the ring, and every
// CTA finishes an equal share of the rows: it sums them out of all the cluster's shared memories in rank order (the same
// result on every run), applies bias and activation and stores. No workspace, no second kernel, no atomics.
// Included by gemm_sm100.cu, whose error word and epilogue functions it uses.

constexpr int kClusterThreads = 256;
constexpr int kClusterStages = 3;  // six measured the same; three leave room for the next kernel's CTA beside this one

template <int BN>
struct ClusterLayout {
    static constexpr int kABytes = BM * BK * 2, kBBytes = BN * BK * 2, kStageBytes = kABytes + kBBytes;
    static constexpr int kPitch = BN + 4;  // floats per row of the partial tile: eight rows cover the 32 banks
    static constexpr int kRing = kClusterStages * kStageBytes, kPartial = BM * kPitch * 4;
    static_assert(kPartial <= kRing, "the partial tile lies over the ring");
    static constexpr int kBarrierOff = kRing;
    static constexpr int kTotal = kBarrierOff + 256 + 1024;  // + slack for 1024-byte alignment
};

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}

// `epilogue` with or without kExactAct; four results a thread, so that a switch per result costs nothing beside the exchange.
__device__ __forceinline__ float cluster_act(float v, int epilogue) {
    switch (epilogue) {
        case MHLO_EPILOGUE_GELU_TANH: return epilogue_act<MHLO_EPILOGUE_GELU_TANH>(v);
        case MHLO_EPILOGUE_SILU: return epilogue_act<MHLO_EPILOGUE_SILU>(v);
        case MHLO_EPILOGUE_SIGMOID: return epilogue_act<MHLO_EPILOGUE_SIGMOID>(v);
        default: break;
    }
    switch (epilogue & ~kExactAct) {
        case MHLO_EPILOGUE_RELU: return epilogue_act<MHLO_EPILOGUE_RELU>(v);
        case MHLO_EPILOGUE_GELU_TANH: return epilogue_act<MHLO_EPILOGUE_GELU_TANH | kExactAct>(v);
        case MHLO_EPILOGUE_GELU_ERF: return epilogue_act<MHLO_EPILOGUE_GELU_ERF>(v);
        case MHLO_EPILOGUE_SILU: return epilogue_act<MHLO_EPILOGUE_SILU | kExactAct>(v);
        case MHLO_EPILOGUE_TANH: return epilogue_act<MHLO_EPILOGUE_TANH>(v);
        case MHLO_EPILOGUE_SIGMOID: return epilogue_act<MHLO_EPILOGUE_SIGMOID | kExactAct>(v);
        default: return v;
    }
}

template <int BN>
__global__ void __launch_bounds__(kClusterThreads, 1) gemm_cluster_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                                                                          const __grid_constant__ GemmParams p, int splits) {
    using L = ClusterLayout<BN>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + L::kBarrierOff);
    uint64_t* empty_bar = full_bar + kClusterStages;
    uint64_t* done_bar = empty_bar + kClusterStages;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done_bar + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = static_cast<int>(cluster_cta_rank());
    const int64_t tile = blockIdx.x / splits;
    int bz, tm, tn;
    tile_coords(tile, p, &bz, &tm, &tn);
    const int k_blocks = static_cast<int>((p.k + BK - 1) / BK), each = (k_blocks + splits - 1) / splits;
    const int kb_begin = min(k_blocks, rank * each), kb_end = min(k_blocks, kb_begin + each);

    if (warp == 0 && lane == 0) {
        prefetch_tmap(&map_a);
        prefetch_tmap(&map_b);
        for (int s = 0; s < kClusterStages; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
        mbar_init(done_bar, 1);
        fence_barrier_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, BN);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    grid_dependency_wait();
    grid_dependency_release();

    if (warp == 0) {
        if (lane == 0) {
            const int b0 = bz / static_cast<int>(p.batch1), b1 = bz % static_cast<int>(p.batch1);
            const int a0 = b0 * p.a_batch[0], a1 = b1 * p.a_batch[1], w0 = b0 * p.b_batch[0], w1 = b1 * p.b_batch[1];
            int stage = 0;
            uint32_t phase = 0;
            for (int kb = kb_begin; kb < kb_end; ++kb) {
                if (!mbar_wait(&empty_bar[stage], phase ^ 1)) { atomicExch(&g_gemm_error, 11); break; }
                uint8_t* sa = smem + stage * L::kStageBytes;
                uint8_t* sb = sa + L::kABytes;
                mbar_expect_tx(&full_bar[stage], L::kStageBytes);
                if (!p.a_mn_major) {
                    tma_load_4d(sa, &map_a, &full_bar[stage], kb * BK, tm * BM, a1, a0);
                } else {
#pragma unroll
                    for (int j = 0; j < BM / 64; ++j) tma_load_4d(sa + j * 64 * BK * 2, &map_a, &full_bar[stage], tm * BM + j * 64, kb * BK, a1, a0);
                }
                if (!p.b_mn_major) {
                    tma_load_4d(sb, &map_b, &full_bar[stage], kb * BK, tn * BN, w1, w0);
                } else {
#pragma unroll
                    for (int j = 0; j < BN / 64; ++j) tma_load_4d(sb + j * 64 * BK * 2, &map_b, &full_bar[stage], tn * BN + j * 64, kb * BK, w1, w0);
                }
                if (++stage == kClusterStages) { stage = 0; phase ^= 1; }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        const uint32_t fmt = p.in_bf16 ? 1u : 0u;
        const uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | (static_cast<uint32_t>(p.a_mn_major) << 15) | (static_cast<uint32_t>(p.b_mn_major) << 16) |
                               (static_cast<uint32_t>(BN >> 3) << 17) | (static_cast<uint32_t>(BM >> 4) << 24);
        int stage = 0;
        uint32_t phase = 0;
        for (int kb = kb_begin; kb < kb_end; ++kb) {
            if (!mbar_wait(&full_bar[stage], phase)) { atomicExch(&g_gemm_error, 12); break; }
            tc_fence_after();
            const uint32_t sa = smem_u32(smem + stage * L::kStageBytes), sb = sa + L::kABytes;
#pragma unroll
            for (int k = 0; k < BK / UMMA_K; ++k) {
                const uint64_t da = p.a_mn_major ? make_smem_desc(sa + k * UMMA_K * 128, 64 * BK * 2, 1024) : make_smem_desc(sa + k * UMMA_K * 2, 16, 1024);
                const uint64_t db = p.b_mn_major ? make_smem_desc(sb + k * UMMA_K * 128, 64 * BK * 2, 1024) : make_smem_desc(sb + k * UMMA_K * 2, 16, 1024);
                if (elect_one()) umma_f16(tmem_base, da, db, idesc, kb != kb_begin || k != 0 ? 1u : 0u);
            }
            if (elect_one()) umma_commit(&empty_bar[stage]);
            __syncwarp();
            if (++stage == kClusterStages) { stage = 0; phase ^= 1; }
        }
        if (elect_one()) umma_commit(done_bar);
        __syncwarp();
    }
    // bias of the four columns this thread finishes, asked for while the tile is being accumulated
    const int64_t gn = static_cast<int64_t>(tn) * BN + threadIdx.x % (BN / 4) * 4;
    float bias[4] = {0.f, 0.f, 0.f, 0.f};
    if (p.bias != nullptr) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (gn + q >= p.n) continue;
            if (p.out_dtype == MHLO_DT_F32) bias[q] = static_cast<const float*>(p.bias)[gn + q];
            else if (p.out_dtype == MHLO_DT_BF16) bias[q] = __bfloat162float(static_cast<const __nv_bfloat16*>(p.bias)[gn + q]);
            else bias[q] = __half2float(static_cast<const __half*>(p.bias)[gn + q]);
        }
    }
    // every thread: this CTA's partial tile to shared memory
    const bool any = kb_end > kb_begin;
    if (any && !mbar_wait(done_bar, 0)) atomicExch(&g_gemm_error, 13);
    __syncwarp();
    tc_fence_after();
    float* partial = reinterpret_cast<float*>(smem);
    {
        const int quarter = warp & 3, row = quarter * 32 + lane, col0 = (warp >> 2) * (BN / 2);
        float* to = partial + row * L::kPitch + col0;
#pragma unroll
        for (int c = 0; c < BN / 2; c += 32) {
            uint32_t r[32];
            if (any) {
                tmem_ld32(tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + static_cast<uint32_t>(col0 + c), r);
                tmem_ld_wait();
            } else {
#pragma unroll
                for (int j = 0; j < 32; ++j) r[j] = 0u;
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) *reinterpret_cast<uint4*>(to + c + 4 * j) = make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
        }
    }
    tc_fence_before();
    cluster_arrive();
    cluster_wait();
    tc_fence_after();
    if (warp == 1) tmem_dealloc(tmem_base, BN);  // every warp has read its share (the cluster barrier above)

    // This CTA's rows, eight per iteration of the block (four with 64 columns twice as many): a thread keeps its four columns.
    constexpr int kColThreads = BN / 4, kRowsAtOnce = kClusterThreads / kColThreads;
    const int rows = BM / splits, col = threadIdx.x % kColThreads * 4, row0 = rank * rows + threadIdx.x / kColThreads;
    const uint32_t base = smem_u32(partial) + static_cast<uint32_t>(col * 4);
    uint8_t* cbase = static_cast<uint8_t*>(p.c);
    auto finish = [&](int row, float4 x) {
        const int64_t gm = static_cast<int64_t>(tm) * BM + row;
        if (gm >= p.m || gn >= p.n) return;
        float v[4] = {x.x + bias[0], x.y + bias[1], x.z + bias[2], x.w + bias[3]};
        if (p.epilogue != MHLO_EPILOGUE_NONE) {
#pragma unroll
            for (int q = 0; q < 4; ++q) v[q] = cluster_act(v[q], p.epilogue);
        }
        const int64_t off = (static_cast<int64_t>(bz) * p.m + gm) * p.n + gn;
        if (p.out_dtype == MHLO_DT_F32) {
            float* to = reinterpret_cast<float*>(cbase) + off;
            if (p.c_vec_ok) {
                *reinterpret_cast<float4*>(to) = make_float4(v[0], v[1], v[2], v[3]);
            } else {
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (gn + q < p.n) to[q] = v[q];
            }
            return;
        }
        uint32_t w[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            if (p.out_dtype == MHLO_DT_BF16) {
                const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * q], v[2 * q + 1]);
                w[q] = *reinterpret_cast<const uint32_t*>(&h);
            } else {
                const __half2 h = __floats2half2_rn(v[2 * q], v[2 * q + 1]);
                w[q] = *reinterpret_cast<const uint32_t*>(&h);
            }
        }
        uint16_t* to = reinterpret_cast<uint16_t*>(cbase) + off;
        if (p.c_vec_ok) {
            *reinterpret_cast<uint2*>(to) = make_uint2(w[0], w[1]);
        } else {
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (gn + q < p.n) to[q] = static_cast<uint16_t>(w[q / 2] >> (16 * (q % 2)));
        }
    };
    // S CTAs' partial rows, U rows at a time: S * U reads of distributed shared memory are in flight together
    auto reduce = [&](auto s_const, auto u_const) {
        constexpr int S = decltype(s_const)::value, U = decltype(u_const)::value;
        uint32_t at[S];
#pragma unroll
        for (int r = 0; r < S; ++r) at[r] = map_to_cta(base, static_cast<uint32_t>(r));
        for (int i = 0; i < rows / kRowsAtOnce; i += U) {
            float4 part[U][S];
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int r = 0; r < S; ++r) part[u][r] = ld_cluster_f4(at[r] + static_cast<uint32_t>((row0 + (i + u) * kRowsAtOnce) * L::kPitch * 4));
#pragma unroll
            for (int u = 0; u < U; ++u) {
                float4 x = part[u][0];
#pragma unroll
                for (int r = 1; r < S; ++r) { x.x += part[u][r].x; x.y += part[u][r].y; x.z += part[u][r].z; x.w += part[u][r].w; }
                finish(row0 + (i + u) * kRowsAtOnce, x);
            }
        }
    };
    if (splits == 2) reduce(std::integral_constant<int, 2>(), std::integral_constant<int, 4>());
    else if (splits == 4) reduce(std::integral_constant<int, 4>(), std::integral_constant<int, 2>());
    else reduce(std::integral_constant<int, 8>(), std::integral_constant<int, 1>());
    cluster_arrive();
    cluster_wait();  // nobody leaves while its shared memory is being read
}
