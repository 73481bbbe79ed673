// 16-bit products whose operands the tensor-core kernels cannot read in place: rows off the 16-byte grid (an odd pitch),
// bases off it, or no contiguous dimension. Such an operand is copied once into a buffer whose rows are on the grid (one
// launch for both operands, stream-ordered scratch) and the product then runs on the tensor cores. The copy reads and
// writes the operand once, 2 (MK + KN) * 2 bytes from HBM or L2, against 2 MNK operations that otherwise ran as scalar
// fp32 FMAs over scalar loads: [1021,1111] . [1111,3001] + bias + GELU took 509 us that way.
//
// Products with an fp32 result that are to have fp32 sums (the tensor cores add more coarsely) have both operands widened to fp32
// on the same way and run on the packed FMAs: [301,1023] . [1023,1001] f16 -> f32 37 us, 208 on the general kernel, with errors
// against fp64 of 1.4e-7 and 5.6e-7.
#include <type_traits>

#include "contraction.cuh"

namespace mhlo {
namespace {

struct PackJob {
    const uint16_t* src;
    void* dst;                                 // the same elements, or floats
    int64_t s_batch0, s_batch1, s_row, s_col;  // element strides of the source
    int64_t batch1, rows, cols, pitch;         // destination: [batch0][batch1][rows][pitch]
    int64_t all_rows;                          // batch0 * batch1 * rows
    int64_t pieces;                            // of kPackColumns columns per row
};
struct PackJobs {
    PackJob job[2];
    int64_t blocks0;  // blocks of the first job
};

// A warp per row, or per 512 columns of a longer row, consecutive lanes on consecutive columns (64 bytes per load and store
// instruction). 512 columns are 16 trips of a warp: with whole rows, an operand of few long rows kept few warps busy
// ([768, 50257], the weights of a product of one row: 543 us with it, 89 in pieces).
constexpr int kPackColumns = 512;

template <typename From, typename To>
__global__ void __launch_bounds__(256) pack_operands_kernel(const __grid_constant__ PackJobs jobs) {
    const bool second = blockIdx.x >= jobs.blocks0;
    const PackJob& j = jobs.job[second];
    const int64_t block = blockIdx.x - (second ? jobs.blocks0 : 0);
    const int lane = threadIdx.x & 31;
    const int64_t unit = block * 8 + (threadIdx.x >> 5), row = unit / j.pieces;
    if (row >= j.all_rows) return;
    const int64_t c0 = unit % j.pieces * kPackColumns, c1 = c0 + kPackColumns < j.cols ? c0 + kPackColumns : j.cols;
    const int64_t b = row / j.rows, r = row % j.rows;
    const From* s = reinterpret_cast<const From*>(j.src) + b / j.batch1 * j.s_batch0 + b % j.batch1 * j.s_batch1 + r * j.s_row;
    To* d = static_cast<To*>(j.dst) + row * j.pitch;
#pragma unroll 8
    for (int64_t c = c0 + lane; c < c1; c += 32) {
        if constexpr (std::is_same<From, To>::value) d[c] = s[c * j.s_col];
        else d[c] = VecTraits<From>::to_float(s[c * j.s_col]);
    }
}

// Packs along whichever dimension is contiguous (if neither is, the columns; a single column as one row) and rewrites the
// operand's strides. A matrix that every entry of a batch dimension shares is packed once.
void plan(PackJob* j, const void* p, int64_t* st, int64_t batch0, int64_t batch1, int64_t rows, int64_t cols) {
    const bool along_rows = cols == 1 || (st[3] != 1 && st[2] == 1 && rows > 1);
    batch0 = operand_batch(batch0, st[0]);
    batch1 = operand_batch(batch1, st[1]);
    j->src = static_cast<const uint16_t*>(p);
    j->s_batch0 = st[0]; j->s_batch1 = st[1];
    j->s_row = along_rows ? st[3] : st[2];
    j->s_col = along_rows ? st[2] : st[3];
    j->batch1 = batch1;
    j->rows = along_rows ? cols : rows;
    j->cols = along_rows ? rows : cols;
    j->pitch = (j->cols + 7) / 8 * 8;
    j->all_rows = batch0 * batch1 * j->rows;
    j->pieces = (j->cols + kPackColumns - 1) / kPackColumns;
    const int64_t matrix = j->rows * j->pitch;
    if (st[0] != 0) st[0] = batch1 * matrix;
    if (st[1] != 0) st[1] = matrix;
    st[2] = along_rows ? 1 : j->pitch;
    st[3] = along_rows ? j->pitch : 1;
}

struct PackWork {
    PackJobs jobs;
    int count;
    int packed[2];  // 0 = A, 1 = B
    bool widen;     // to floats
    size_t bytes, offset[2];
    int64_t blocks[2];
};

// Whether *p has operands to pack, and how; rewrites their strides and leaves their addresses null.
bool lay_out(GemmProblem* p, PackWork* w) {
    memset(w, 0, sizeof *w);
    int n = 0;
    if (p->in_dtype != MHLO_DT_F16 && p->in_dtype != MHLO_DT_BF16) return false;
    if (p->out_dtype != p->in_dtype && p->out_dtype != MHLO_DT_F32) return false;
    const bool elsewhere = general_kernel_takes(*p);
    w->widen = p->out_dtype == MHLO_DT_F32 && elsewhere;
    if (p->a == nullptr || p->b == nullptr || p->n_copies > 0 || p->m <= 0 || p->n <= 0 || p->k <= 0 || p->batch0 <= 0 || p->batch1 <= 0) return false;
    if (p->m > 0x7fffffff || p->n > 0x7fffffff || p->k > 0x7fffffff || p->batch0 * p->batch1 > 0x7fffffff) return false;
    // Copy and product cost 10 to 14 us before the first panel; the general kernel does 32 steps of K in 10, whatever the number of
    // results up to about eight million ([33,31] . [31,4001] 14 us packed, 10 there; with K = 63 14 and 15; [301,15] . [15,50257]
    // 37 and 46).
    if (p->m * p->n * p->k < 32 * 1024 || (p->k <= 32 && elsewhere && p->m * p->n * p->batch0 * p->batch1 < int64_t{1} << 23))
        return false;
    for (const bool is_a : {true, false}) {
        const void** base = is_a ? &p->a : &p->b;
        int64_t* st = is_a ? p->as : p->bs;
        if (!w->widen && operand_on_grid(*p, *base, st) && (is_a ? a_major(*p) : b_major(*p)) != kNoMajor) continue;
        plan(&w->jobs.job[n], *base, st, p->batch0, p->batch1, is_a ? p->m : p->k, is_a ? p->k : p->n);
        w->offset[n] = w->bytes;
        w->packed[n] = is_a ? 0 : 1;
        *base = nullptr;  // on the grid; its address comes with the scratch
        w->bytes += static_cast<size_t>(w->jobs.job[n].all_rows * w->jobs.job[n].pitch * (w->widen ? 4 : 2) + 255) / 256 * 256;
        ++n;
    }
    for (int i = 0; i < 2; ++i) w->blocks[i] = (w->jobs.job[i].all_rows * w->jobs.job[i].pieces + 7) / 8;
    w->count = n;
    p->exact_act = 1;
    if (n == 0 || w->blocks[0] + w->blocks[1] > 0x7fffffff) return false;
    if (!w->widen) return gemm_tc_supported(*p);
    p->in_dtype = MHLO_DT_F32;
    return gemm_fp32_supported(*p);
}

}  // namespace

size_t gemm_pack_bytes(GemmProblem p) {
    PackWork w;
    p.a = p.b = reinterpret_cast<const void*>(uintptr_t{256});  // any address on the grid
    if (!gemm_fp32_sums(p) && gemm_tc_supported(p)) return 0;
    return lay_out(&p, &w) ? w.bytes : 0;
}

bool gemm_pack_launch(GemmProblem p, const PackScratch* own, cudaStream_t stream, int* status) {
    PackWork w;
    const bool half = p.in_dtype == MHLO_DT_F16;
    if (!lay_out(&p, &w)) return false;
    void* scratch = own != nullptr ? own->base : nullptr;
    if (own != nullptr && own->bytes < w.bytes) return false;
    int st = own != nullptr ? MHLO_CUDA_OK : scratch_alloc(&scratch, w.bytes, stream);
    if (st != MHLO_CUDA_OK) {  // no memory to pack into: the general kernel reads the operands where they are
        clear_error();
        return false;
    }
    for (int i = 0; i < w.count; ++i) {
        w.jobs.job[i].dst = static_cast<char*>(scratch) + w.offset[i];
        (w.packed[i] == 0 ? p.a : p.b) = w.jobs.job[i].dst;
    }
    w.jobs.blocks0 = w.blocks[0];
    auto kernel = !w.widen ? pack_operands_kernel<uint16_t, uint16_t>
                  : half   ? pack_operands_kernel<__half, float>
                           : pack_operands_kernel<__nv_bfloat16, float>;
    kernel<<<static_cast<unsigned>(w.blocks[0] + w.blocks[1]), 256, 0, stream>>>(w.jobs);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) st = fail(MHLO_CUDA_EXECUTION_FAILED, "launch of pack_operands failed: %s", cudaGetErrorString(e));
    if (st == MHLO_CUDA_OK) st = w.widen ? gemm_fp32_launch(p, stream) : gemm_tc_launch(p, stream);
    const int freed = own != nullptr ? MHLO_CUDA_OK : scratch_free(scratch, stream);
    *status = st != MHLO_CUDA_OK ? st : freed;
    return true;
}

}  // namespace mhlo
