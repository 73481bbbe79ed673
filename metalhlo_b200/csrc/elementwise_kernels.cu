// Elementwise programs over strided views: every unary / binary / compare / select / clamp / convert / iota operator,
// data movement expressed as a strided copy, and fused elementwise chains. Bound by HBM (each operand read once, the
// result written once) as long as decoding the program costs less than the bytes of the elements it is decoded for.
//
// A thread works on V consecutive elements of the innermost dimension (16 bytes of a 16-bit or 32-bit operand), so that the
// opcode switch, the coordinate arithmetic (multiply-high divisions by the extents) and the type switch of a load are paid
// once per V elements and dense operands move in 16-byte accesses. Where the elements are too few to fill the machine a thread
// takes one (kFewElements): its chain of work is then what a call lasts. Rows whose length is no multiple of V end in a partial
// vector. A program of one instruction keeps its operands in registers; a longer one keeps the values that more than the
// next instruction reads in shared-memory slots, one private column of 16-byte words per thread (no conflicts, no
// barriers), assigned by liveness on the host.
// One element per iteration with 64-bit divisions and a dynamically indexed register file in local memory, the former
// shape of this kernel, ran a seven-instruction chain over 4.2 M bf16 elements in 75 us and a scalar multiply over
// 134 M bf16 elements in 208 us (HBM time: 4 us and 82 us).
#include <atomic>

#include "common.cuh"
#include "element_access.cuh"

namespace mhlo {
namespace {

// ---- the operators ---------------------------------------------------------------------------------------------------

// stablehlo.reduce_precision on the bits of a float (8 / 23) or a double (11 / 52): round the mantissa to nearest even at
// `mant` bits, then clamp the exponent range to `expo` bits (overflow -> infinity, underflow -> signed zero).
template <typename U, int kExpBits, int kMantBits>
__device__ __forceinline__ U reduce_precision_bits(U bits, int expo, int mant) {
    const U one = 1;
    const U exp_mask = ((one << kExpBits) - 1) << kMantBits, mant_mask = (one << kMantBits) - 1, sign = bits & (one << (kExpBits + kMantBits));
    const bool is_nan = (bits & exp_mask) == exp_mask && (bits & mant_mask) != 0;
    if (is_nan) return mant > 0 ? bits : (sign | exp_mask);  // a format without mantissa bits has no NaN: it becomes infinity
    if (mant < kMantBits) {
        const U last = one << (kMantBits - mant);
        const U bias = (last >> 1) - 1 + ((bits & last) >> (kMantBits - mant));
        bits = (bits + bias) & ~(last - 1);
    }
    if (expo < kExpBits) {
        const long long full_bias = (1ll << (kExpBits - 1)) - 1, reduced_bias = (1ll << (expo - 1)) - 1;
        const U max_exp = static_cast<U>(full_bias + reduced_bias) << kMantBits, min_exp = static_cast<U>(full_bias - reduced_bias) << kMantBits;
        const U e = bits & exp_mask;
        if (e > max_exp) bits = sign | exp_mask;
        else if (e <= min_exp) bits = sign;
    }
    return bits;
}
__device__ __forceinline__ float reduce_precision_value(float a, int expo, int mant) {
    return __uint_as_float(reduce_precision_bits<uint32_t, 8, 23>(__float_as_uint(a), expo, mant));
}
__device__ __forceinline__ double reduce_precision_value(double a, int expo, int mant) {
    return __longlong_as_double(static_cast<long long>(reduce_precision_bits<unsigned long long, 11, 52>(static_cast<unsigned long long>(__double_as_longlong(a)), expo, mant)));
}

template <typename C>
__device__ __forceinline__ C ew_float_op(int op, C a, C b, C c, double imm) {
    switch (op) {
        case MHLO_EW_COPY: return a;
        case MHLO_EW_IMM: return static_cast<C>(imm);
        case MHLO_EW_ADD: return a + b;
        case MHLO_EW_SUB: return a - b;
        case MHLO_EW_MUL: return a * b;
        case MHLO_EW_DIV: return a / b;
        case MHLO_EW_REM: return fmod(a, b);
        case MHLO_EW_MAX: return (a != a || b != b) ? C(NAN) : (a > b ? a : b);
        case MHLO_EW_MIN: return (a != a || b != b) ? C(NAN) : (a < b ? a : b);
        case MHLO_EW_POW: return pow(a, b);
        case MHLO_EW_ATAN2: return atan2(a, b);
        case MHLO_EW_AND: return C(a != C(0) && b != C(0));
        case MHLO_EW_OR: return C(a != C(0) || b != C(0));
        case MHLO_EW_XOR: return C((a != C(0)) != (b != C(0)));
        case MHLO_EW_NEG: return -a;
        case MHLO_EW_ABS: return fabs(a);
        case MHLO_EW_EXP: return exp(a);
        case MHLO_EW_EXPM1: return expm1(a);
        case MHLO_EW_LOG: return log(a);
        case MHLO_EW_LOG1P: return log1p(a);
        case MHLO_EW_SQRT: return sqrt(a);
        case MHLO_EW_RSQRT: return C(1) / sqrt(a);
        case MHLO_EW_CBRT: return cbrt(a);
        case MHLO_EW_TANH: return tanh(a);
        case MHLO_EW_LOGISTIC: return C(1) / (C(1) + exp(-a));
        case MHLO_EW_SIN: return sin(a);
        case MHLO_EW_COS: return cos(a);
        case MHLO_EW_TAN: return tan(a);
        case MHLO_EW_FLOOR: return floor(a);
        case MHLO_EW_CEIL: return ceil(a);
        case MHLO_EW_ROUND_AFZ: return round(a);
        case MHLO_EW_ROUND_EVEN: return rint(a);
        case MHLO_EW_SIGN: return a != a ? a : C((a > C(0)) - (a < C(0)));
        case MHLO_EW_NOT: return C(a == C(0));
        case MHLO_EW_IS_FINITE: return C(isfinite(a) ? 1 : 0);
        case MHLO_EW_CMP_EQ: return C(a == b);
        case MHLO_EW_CMP_NE: return C(a != b);
        case MHLO_EW_CMP_LT: return C(a < b);
        case MHLO_EW_CMP_LE: return C(a <= b);
        case MHLO_EW_CMP_GT: return C(a > b);
        case MHLO_EW_CMP_GE: return C(a >= b);
        case MHLO_EW_SELECT: return a != C(0) ? b : c;
        case MHLO_EW_CLAMP: {  // minimum(maximum(operand, min), max), each of which hands a NaN on
            if (a != a || b != b || c != c) return C(NAN);
            C lo = b < a ? a : b;
            return lo > c ? c : lo;
        }
        case MHLO_EW_GELU_TANH: {
            const C inner = C(0.7978845608028654) * (a + C(0.044715) * a * a * a);
            return C(0.5) * a * (C(1) + tanh(inner));
        }
        case MHLO_EW_GELU_ERF: return C(0.5) * a * (C(1) + erf(a * C(0.70710678118654752440)));
        case MHLO_EW_SILU: return a / (C(1) + exp(-a));
        case MHLO_EW_RELU: return a > C(0) ? a : (a != a ? a : C(0));
        case MHLO_EW_ROUND_TO: {
            const int dt = static_cast<int>(imm);
            if (dt == MHLO_DT_F16) return C(__half2float(__float2half_rn(static_cast<float>(a))));
            if (dt == MHLO_DT_BF16) return C(__bfloat162float(__float2bfloat16_rn(static_cast<float>(a))));
            if (dt == MHLO_DT_F32) return C(static_cast<float>(a));
            return a;
        }
        case MHLO_EW_ERF: return erf(a);
        case MHLO_EW_REDUCE_PRECISION: return reduce_precision_value(a, static_cast<int>(imm) / 64, static_cast<int>(imm) % 64);
        default: return a;
    }
}

__device__ __forceinline__ int64_t ew_int_op(int op, int64_t a, int64_t b, int64_t c, double imm, bool uns, bool boolean,
                                             int bits) {
    const uint64_t ua = static_cast<uint64_t>(a), ub = static_cast<uint64_t>(b);
    const uint64_t wmask = bits >= 64 ? ~0ull : ((1ull << bits) - 1);  // operand width: shifts and bit counts are per type
    switch (op) {
        case MHLO_EW_COPY: return a;
        case MHLO_EW_IMM: return static_cast<int64_t>(imm);
        case MHLO_EW_ADD: return static_cast<int64_t>(ua + ub);
        case MHLO_EW_SUB: return static_cast<int64_t>(ua - ub);
        case MHLO_EW_MUL: return static_cast<int64_t>(ua * ub);
        case MHLO_EW_DIV: return b == 0 ? -1 : (uns ? static_cast<int64_t>(ua / ub) : (b == -1 ? static_cast<int64_t>(0 - ua) : a / b));
        case MHLO_EW_REM: return b == 0 ? a : (uns ? static_cast<int64_t>(ua % ub) : (b == -1 ? 0 : a % b));
        case MHLO_EW_MAX: return uns ? static_cast<int64_t>(ua > ub ? ua : ub) : (a > b ? a : b);
        case MHLO_EW_MIN: return uns ? static_cast<int64_t>(ua < ub ? ua : ub) : (a < b ? a : b);
        case MHLO_EW_POW: {
            if (b < 0 && !uns) return a == 1 ? 1 : (a == -1 ? ((b & 1) ? -1 : 1) : 0);
            uint64_t r = 1, base = ua, e = ub;
            while (e) { if (e & 1) r *= base; base *= base; e >>= 1; }
            return static_cast<int64_t>(r);
        }
        case MHLO_EW_AND: return a & b;
        case MHLO_EW_OR: return a | b;
        case MHLO_EW_XOR: return a ^ b;
        case MHLO_EW_SHL: return ub >= static_cast<uint64_t>(bits) ? 0 : static_cast<int64_t>(ua << ub);
        case MHLO_EW_SHR_A: return ub >= static_cast<uint64_t>(bits) ? (a < 0 ? -1 : 0) : (a >> ub);
        case MHLO_EW_SHR_L: return ub >= static_cast<uint64_t>(bits) ? 0 : static_cast<int64_t>((ua & wmask) >> ub);
        case MHLO_EW_NEG: return static_cast<int64_t>(0 - ua);
        case MHLO_EW_ABS: return a < 0 ? static_cast<int64_t>(0 - ua) : a;
        case MHLO_EW_SIGN: return (a > 0) - (a < 0);
        case MHLO_EW_NOT: return boolean ? (a == 0) : ~a;
        case MHLO_EW_POPCNT: return __popcll(ua & wmask);
        case MHLO_EW_CLZ: return __clzll(static_cast<int64_t>(ua & wmask)) - (64 - bits);
        case MHLO_EW_CMP_EQ: return a == b;
        case MHLO_EW_CMP_NE: return a != b;
        case MHLO_EW_CMP_LT: return uns ? ua < ub : a < b;
        case MHLO_EW_CMP_LE: return uns ? ua <= ub : a <= b;
        case MHLO_EW_CMP_GT: return uns ? ua > ub : a > b;
        case MHLO_EW_CMP_GE: return uns ? ua >= ub : a >= b;
        case MHLO_EW_SELECT: return a != 0 ? b : c;
        case MHLO_EW_CLAMP: {
            if (uns) { uint64_t lo = ub < ua ? ua : ub; uint64_t uc = static_cast<uint64_t>(c); return static_cast<int64_t>(lo > uc ? uc : lo); }
            int64_t lo = b < a ? a : b; return lo > c ? c : lo;
        }
        case MHLO_EW_RELU: return a > 0 ? a : 0;
        case MHLO_EW_IS_FINITE: return 1;
        default: return a;
    }
}

// Operators whose inline expansion would cost every other program its registers.
template <typename C>
__device__ __noinline__ C ew_outlined(int op, C a, C b, C c, double imm) {
    return ew_float_op<C>(op, a, b, c, imm);
}
__device__ __noinline__ int64_t ew_int_outlined(int op, int64_t a, int64_t b, int64_t c, double imm, bool uns, bool boolean, int bits) {
    return ew_int_op(op, a, b, c, imm, uns, boolean, bits);
}

// (powf from a call of its own: behind the switch of ew_outlined 16.8 M elements took 77 us, so 68)
__device__ __noinline__ float ew_pow(float a, float b) { return powf(a, b); }

// ---- launch parameters -------------------------------------------------------------------------------------------------

enum EwAccess : int32_t { kSplat = 0, kVector = 1, kStrided = 2 };  // the operand along the innermost dimension

struct EwOperand {
    void* base;
    int32_t dtype, access;
    int64_t inner;                          // element stride of the innermost dimension
    int64_t outer[MHLO_CUDA_MAX_RANK - 1];  // and of the outer ones, outermost first
};

struct EwInstr {
    double imm;
    int16_t op;
    int8_t a, b, c;  // shared-memory slot of each operand, kPrevious = result of the instruction before
    int8_t dst;      // slot the result is kept in, kNowhere = only the next instruction (or the store) reads it
};
constexpr int8_t kPrevious = -1, kNowhere = -1;

struct EwParams {
    EwOperand in[MHLO_CUDA_EW_MAX_INPUTS];
    EwOperand out;
    EwInstr prog[MHLO_CUDA_EW_MAX_INSTS];
    int64_t extent[MHLO_CUDA_MAX_RANK];   // collapsed output shape
    FastDiv div[MHLO_CUDA_MAX_RANK - 1];  // by the outer extents
    FastDiv per_row_div;                  // by the vectors of one innermost row
    int64_t n_vec, per_row;
    int32_t n_inputs, n_insts, n_outer;
    int32_t wide;           // 2^31 vectors and more: 64-bit divisions
    int32_t unsigned_mode;  // integer domain: treat values as uint64 for div / rem / shift / compare / min / max
    int32_t bool_mode;      // integer domain: NOT is logical (i1)
    int32_t int_bits;       // integer domain: width of the operand type (shifts, popcnt, clz)
};

// ---- operand access ------------------------------------------------------------------------------------------------------

template <typename T, typename C, int V>
__device__ __forceinline__ void load_strided(const void* base, int64_t at, int64_t stride, int count, C* x) {
    const T* p = static_cast<const T*>(base) + at;
#pragma unroll
    for (int e = 0; e < V; ++e)
        if (e < count) {
            if constexpr (std::is_same<T, __half>::value) x[e] = static_cast<C>(__half2float(p[e * stride]));
            else if constexpr (std::is_same<T, __nv_bfloat16>::value) x[e] = static_cast<C>(__bfloat162float(p[e * stride]));
            else if constexpr (std::is_same<T, bool>::value) x[e] = static_cast<C>(reinterpret_cast<const uint8_t*>(p)[e * stride] != 0);
            else x[e] = static_cast<C>(p[e * stride]);
        }
}

template <typename C, int V>
__device__ __forceinline__ void load_operand(const EwOperand& o, int64_t at, int count, C* x) {
    if (o.access == kSplat) {
        const C v = load_as<C>(o.base, o.dtype, at);
#pragma unroll
        for (int e = 0; e < V; ++e) x[e] = v;
        return;
    }
    if constexpr (std::is_same<C, float>::value && V >= 4) {
        if (o.access == kVector && count == V) {
            if (o.dtype == MHLO_DT_F32) {
#pragma unroll
                for (int q = 0; q < V / 4; ++q) {
                    const float4 f = reinterpret_cast<const float4*>(static_cast<const float*>(o.base) + at)[q];
                    x[4 * q] = f.x; x[4 * q + 1] = f.y; x[4 * q + 2] = f.z; x[4 * q + 3] = f.w;
                }
                return;
            }
            if constexpr (V == 8) {
                if (o.dtype == MHLO_DT_F16) return VecTraits<__half>::unpack(*reinterpret_cast<const uint4*>(static_cast<const __half*>(o.base) + at), x);
                if (o.dtype == MHLO_DT_BF16)
                    return VecTraits<__nv_bfloat16>::unpack(*reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(o.base) + at), x);
            }
        }
    }
#pragma unroll
    for (int e = 0; e < V; ++e) x[e] = C(0);
    switch (o.dtype) {
        case MHLO_DT_F32: return load_strided<float, C, V>(o.base, at, o.inner, count, x);
        case MHLO_DT_F16: return load_strided<__half, C, V>(o.base, at, o.inner, count, x);
        case MHLO_DT_BF16: return load_strided<__nv_bfloat16, C, V>(o.base, at, o.inner, count, x);
        case MHLO_DT_F64: return load_strided<double, C, V>(o.base, at, o.inner, count, x);
        case MHLO_DT_I1: return load_strided<bool, C, V>(o.base, at, o.inner, count, x);
        case MHLO_DT_I8: return load_strided<int8_t, C, V>(o.base, at, o.inner, count, x);
        case MHLO_DT_UI8: return load_strided<uint8_t, C, V>(o.base, at, o.inner, count, x);
        case MHLO_DT_I16: return load_strided<int16_t, C, V>(o.base, at, o.inner, count, x);
        case MHLO_DT_UI16: return load_strided<uint16_t, C, V>(o.base, at, o.inner, count, x);
        case MHLO_DT_I32:
            if constexpr (std::is_same<C, int64_t>::value && V == 4) {
                if (o.access == kVector && count == V) {
                    const int4 f = *reinterpret_cast<const int4*>(static_cast<const int32_t*>(o.base) + at);
                    x[0] = f.x; x[1] = f.y; x[2] = f.z; x[3] = f.w;
                    return;
                }
            }
            return load_strided<int32_t, C, V>(o.base, at, o.inner, count, x);
        case MHLO_DT_UI32: return load_strided<uint32_t, C, V>(o.base, at, o.inner, count, x);
        case MHLO_DT_I64: return load_strided<int64_t, C, V>(o.base, at, o.inner, count, x);
        default: return load_strided<uint64_t, C, V>(o.base, at, o.inner, count, x);
    }
}

template <typename C, int V>
__device__ __forceinline__ void store_result(const EwOperand& o, int64_t at, int count, const C* x) {
    if constexpr (std::is_same<C, float>::value && V >= 4) {
        if (o.access == kVector && count == V) {
            if (o.dtype == MHLO_DT_F32) {
#pragma unroll
                for (int q = 0; q < V / 4; ++q)
                    reinterpret_cast<float4*>(static_cast<float*>(o.base) + at)[q] = make_float4(x[4 * q], x[4 * q + 1], x[4 * q + 2], x[4 * q + 3]);
                return;
            }
            if constexpr (V == 8) {
                if (o.dtype == MHLO_DT_F16) {
                    *reinterpret_cast<uint4*>(static_cast<__half*>(o.base) + at) = VecTraits<__half>::pack(x);
                    return;
                }
                if (o.dtype == MHLO_DT_BF16) {
                    *reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(o.base) + at) = VecTraits<__nv_bfloat16>::pack(x);
                    return;
                }
            }
        }
    }
    if constexpr (std::is_same<C, int64_t>::value && V == 4) {
        if (o.access == kVector && count == V && o.dtype == MHLO_DT_I32) {
            *reinterpret_cast<int4*>(static_cast<int32_t*>(o.base) + at) =
                make_int4(static_cast<int>(x[0]), static_cast<int>(x[1]), static_cast<int>(x[2]), static_cast<int>(x[3]));
            return;
        }
    }
#pragma unroll 1
    for (int e = 0; e < count; ++e) {
        C v = x[0];
#pragma unroll
        for (int q = 1; q < V; ++q) v = q == e ? x[q] : v;  // a register select: indexing x by e would put it in local memory
        store_as<C>(o.base, o.dtype, at + e * o.inner, v);
    }
}

// ---- one instruction on V elements -----------------------------------------------------------------------------------------

#define MHLO_EW_EACH(expr)                        \
    {                                             \
        _Pragma("unroll") for (int e = 0; e < V; ++e) { \
            const C x = a[e], y = b[e], z = c[e]; \
            (void)x; (void)y; (void)z;            \
            r[e] = (expr);                        \
        }                                         \
        return;                                   \
    }

template <typename C, int V>
__device__ __forceinline__ void ew_apply(const EwParams& p, int op, double imm, const C* a, const C* b, const C* c, C* r) {
    if constexpr (std::is_floating_point<C>::value) {
        switch (op) {
            case MHLO_EW_COPY: MHLO_EW_EACH(x)
            case MHLO_EW_IMM: MHLO_EW_EACH(static_cast<C>(imm))
            case MHLO_EW_ADD: MHLO_EW_EACH(x + y)
            case MHLO_EW_SUB: MHLO_EW_EACH(x - y)
            case MHLO_EW_MUL: MHLO_EW_EACH(x * y)
            case MHLO_EW_DIV: MHLO_EW_EACH(x / y)
            case MHLO_EW_MAX: MHLO_EW_EACH((x != x || y != y) ? C(NAN) : (x > y ? x : y))
            case MHLO_EW_MIN: MHLO_EW_EACH((x != x || y != y) ? C(NAN) : (x < y ? x : y))
            case MHLO_EW_NEG: MHLO_EW_EACH(-x)
            case MHLO_EW_ABS: MHLO_EW_EACH(fabs(x))
            case MHLO_EW_SQRT: MHLO_EW_EACH(sqrt(x))
            case MHLO_EW_RSQRT: MHLO_EW_EACH(C(1) / sqrt(x))
            case MHLO_EW_CMP_EQ: MHLO_EW_EACH(C(x == y))
            case MHLO_EW_CMP_NE: MHLO_EW_EACH(C(x != y))
            case MHLO_EW_CMP_LT: MHLO_EW_EACH(C(x < y))
            case MHLO_EW_CMP_LE: MHLO_EW_EACH(C(x <= y))
            case MHLO_EW_CMP_GT: MHLO_EW_EACH(C(x > y))
            case MHLO_EW_CMP_GE: MHLO_EW_EACH(C(x >= y))
            case MHLO_EW_SELECT: MHLO_EW_EACH(x != C(0) ? y : z)
            case MHLO_EW_RELU: MHLO_EW_EACH(x > C(0) ? x : (x != x ? x : C(0)))
            default: break;
        }
        if constexpr (std::is_same<C, float>::value) {
            switch (op) {
                case MHLO_EW_POW: MHLO_EW_EACH(ew_pow(x, y))
                case MHLO_EW_EXP: MHLO_EW_EACH(expf(x))
                case MHLO_EW_TANH: MHLO_EW_EACH(tanhf(x))
                case MHLO_EW_LOGISTIC: MHLO_EW_EACH(1.f / (1.f + expf(-x)))
                case MHLO_EW_SILU: MHLO_EW_EACH(x / (1.f + expf(-x)))
                case MHLO_EW_GELU_TANH: MHLO_EW_EACH(0.5f * x * (1.f + tanhf(0.7978845608028654f * (x + 0.044715f * x * x * x))))
                case MHLO_EW_ROUND_TO:
                    if (static_cast<int>(imm) == MHLO_DT_F16) MHLO_EW_EACH(__half2float(__float2half_rn(x)))
                    if (static_cast<int>(imm) == MHLO_DT_BF16) MHLO_EW_EACH(__bfloat162float(__float2bfloat16_rn(x)))
                    MHLO_EW_EACH(x)
                default: break;
            }
        }
#pragma unroll
        for (int e = 0; e < V; ++e) r[e] = ew_outlined<C>(op, a[e], b[e], c[e], imm);
    } else {
        const bool uns = p.unsigned_mode != 0;
        switch (op) {
            case MHLO_EW_COPY: MHLO_EW_EACH(x)
            case MHLO_EW_IMM: MHLO_EW_EACH(static_cast<int64_t>(imm))
            case MHLO_EW_ADD: MHLO_EW_EACH(static_cast<int64_t>(static_cast<uint64_t>(x) + static_cast<uint64_t>(y)))
            case MHLO_EW_SUB: MHLO_EW_EACH(static_cast<int64_t>(static_cast<uint64_t>(x) - static_cast<uint64_t>(y)))
            case MHLO_EW_AND: MHLO_EW_EACH(x & y)
            case MHLO_EW_OR: MHLO_EW_EACH(x | y)
            case MHLO_EW_XOR: MHLO_EW_EACH(x ^ y)
            case MHLO_EW_CMP_EQ: MHLO_EW_EACH(x == y)
            case MHLO_EW_CMP_NE: MHLO_EW_EACH(x != y)
            case MHLO_EW_SELECT: MHLO_EW_EACH(x != 0 ? y : z)
            default: break;
        }
#pragma unroll
        for (int e = 0; e < V; ++e) r[e] = ew_int_outlined(op, a[e], b[e], c[e], imm, uns, p.bool_mode != 0, p.int_bits);
    }
}
#undef MHLO_EW_EACH

// ---- the kernel ------------------------------------------------------------------------------------------------------------

// Vector number v -> outer row, first innermost index, and the offset of that row in every operand on request.
struct EwPlace {
    int64_t row;
    int32_t count;  // elements of this vector that exist
    int64_t j;      // innermost index of the first
};

template <int V>
__device__ __forceinline__ EwPlace ew_place(const EwParams& p, int64_t v) {
    EwPlace w;
    if (p.n_outer == 0) {
        w.row = 0;
        w.j = v * V;
    } else if (!p.wide) {
        uint32_t q, r;
        p.per_row_div.divmod(static_cast<uint32_t>(v), &q, &r);
        w.row = q;
        w.j = static_cast<int64_t>(r) * V;
    } else {
        w.row = v / p.per_row;
        w.j = (v % p.per_row) * V;
    }
    const int64_t left = p.extent[p.n_outer] - w.j;
    w.count = left < V ? static_cast<int32_t>(left) : V;
    return w;
}

// Coordinates of a row along the outer dimensions, innermost of them first: calls f(d, coordinate).
template <typename F>
__device__ __forceinline__ void ew_coords(const EwParams& p, int64_t row, F f) {
    if (!p.wide) {
        uint32_t rem = static_cast<uint32_t>(row);
        for (int d = p.n_outer - 1; d >= 0; --d) {
            uint32_t q, r;
            p.div[d].divmod(rem, &q, &r);
            f(d, static_cast<int64_t>(r));
            rem = q;
        }
    } else {
        for (int d = p.n_outer - 1; d >= 0; --d) {
            f(d, row % p.extent[d]);
            row /= p.extent[d];
        }
    }
}

template <typename C, int V>
__device__ __forceinline__ void ew_iota(const EwParams& p, const EwPlace& w, int dim, C* r) {
    if (dim == p.n_outer) {
#pragma unroll
        for (int e = 0; e < V; ++e) r[e] = static_cast<C>(w.j + e);
        return;
    }
    int64_t at = 0;
    ew_coords(p, w.row, [&](int d, int64_t x) { at = d == dim ? x : at; });
#pragma unroll
    for (int e = 0; e < V; ++e) r[e] = static_cast<C>(at);
}

// One instruction: operands straight from memory to registers. N = inputs (0 to 3), read before any of them is used.
template <typename C, int V, int N>
__global__ void __launch_bounds__(256) ew_single_kernel(const __grid_constant__ EwParams p) {
    const int64_t step = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t v = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; v < p.n_vec; v += step) {
        const EwPlace w = ew_place<V>(p, v);
        int64_t at[N > 0 ? N : 1] = {}, to = 0;
        if (p.n_outer > 0)
            ew_coords(p, w.row, [&](int d, int64_t x) {
#pragma unroll
                for (int k = 0; k < N; ++k) at[k] += x * p.in[k].outer[d];
                to += x * p.out.outer[d];
            });
        C x[N > 0 ? N : 1][V], r[V];
#pragma unroll
        for (int k = 0; k < N; ++k) load_operand<C, V>(p.in[k], at[k] + w.j * p.in[k].inner, w.count, x[k]);
        if (p.prog[0].op == MHLO_EW_IOTA) ew_iota<C, V>(p, w, static_cast<int>(p.prog[0].imm), r);
        else ew_apply<C, V>(p, p.prog[0].op, p.prog[0].imm, x[0], x[N > 1 ? 1 : 0], x[N > 2 ? 2 : 0], r);
        store_result<C, V>(p.out, to + w.j * p.out.inner, w.count, r);
    }
}

constexpr int kProgramThreads = 128;

template <typename C, int V>
__global__ void __launch_bounds__(kProgramThreads) ew_program_kernel(const __grid_constant__ EwParams p) {
    // slot s of a thread: V elements as words of 16 bytes (or the one element), word q at [s][q][thread]
    extern __shared__ __align__(16) unsigned char slots[];
    using Word = typename std::conditional<V == 1, C, uint4>::type;
    constexpr int W = V * static_cast<int>(sizeof(C)) / static_cast<int>(sizeof(Word));
    Word* const mine = reinterpret_cast<Word*>(slots) + threadIdx.x;
    auto put = [&](int s, const C* x) {
#pragma unroll
        for (int q = 0; q < W; ++q) {
            Word u;
            memcpy(&u, x + q * (V / W), sizeof u);
            mine[(s * W + q) * kProgramThreads] = u;
        }
    };
    auto get = [&](int s, C* x) {
#pragma unroll
        for (int q = 0; q < W; ++q) {
            const Word u = mine[(s * W + q) * kProgramThreads];
            memcpy(x + q * (V / W), &u, sizeof u);
        }
    };
    const int64_t step = static_cast<int64_t>(gridDim.x) * kProgramThreads;
    for (int64_t v = static_cast<int64_t>(blockIdx.x) * kProgramThreads + threadIdx.x; v < p.n_vec; v += step) {
        const EwPlace w = ew_place<V>(p, v);
        auto offset = [&](const EwOperand& o) {
            int64_t at = w.j * o.inner;
            if (p.n_outer > 0) ew_coords(p, w.row, [&](int d, int64_t x) { at += x * o.outer[d]; });
            return at;
        };
        // inputs, two at a time in flight
        int k = 0;
        for (; k + 1 < p.n_inputs; k += 2) {
            C x[V], y[V];
            load_operand<C, V>(p.in[k], offset(p.in[k]), w.count, x);
            load_operand<C, V>(p.in[k + 1], offset(p.in[k + 1]), w.count, y);
            put(k, x);
            put(k + 1, y);
        }
        if (k < p.n_inputs) {
            C x[V];
            load_operand<C, V>(p.in[k], offset(p.in[k]), w.count, x);
            put(k, x);
        }
        C r[V];
#pragma unroll
        for (int e = 0; e < V; ++e) r[e] = C(0);
        for (int i = 0; i < p.n_insts; ++i) {
            const EwInstr in = p.prog[i];
            C a[V], b[V], c[V], t[V];
            auto fetch = [&](int s, C* x) {
                if (s == kPrevious) {
#pragma unroll
                    for (int e = 0; e < V; ++e) x[e] = r[e];
                } else {
                    get(s, x);
                }
            };
            if (in.op == MHLO_EW_IOTA) {
                ew_iota<C, V>(p, w, static_cast<int>(in.imm), t);
            } else {
                fetch(in.a, a);
                if (in.b == in.a) {
#pragma unroll
                    for (int e = 0; e < V; ++e) b[e] = a[e];
                } else {
                    fetch(in.b, b);
                }
                if (in.op == MHLO_EW_SELECT || in.op == MHLO_EW_CLAMP) {
                    fetch(in.c, c);
                } else {
#pragma unroll
                    for (int e = 0; e < V; ++e) c[e] = a[e];
                }
                ew_apply<C, V>(p, in.op, in.imm, a, b, c, t);
            }
#pragma unroll
            for (int e = 0; e < V; ++e) r[e] = t[e];
            if (in.dst != kNowhere) put(in.dst, r);
        }
        store_result<C, V>(p.out, offset(p.out), w.count, r);
    }
}

// ---- host side -------------------------------------------------------------------------------------------------------------

struct EwShape {  // the output shape and the strides of every operand (index n_inputs: the output), before and after collapsing
    int rank = 0;
    int64_t extent[MHLO_CUDA_MAX_RANK];
    int64_t stride[MHLO_CUDA_EW_MAX_INPUTS + 1][MHLO_CUDA_MAX_RANK];
    bool pinned[MHLO_CUDA_MAX_RANK];  // an iota reads this coordinate: the dimension stays as it is
    int dim_of[MHLO_CUDA_MAX_RANK];   // original dimension -> collapsed one, -1 = extent 1
};

// Drops dimensions of extent 1 and merges neighbours that every operand walks with one stride.
void collapse(EwShape* s, int n_operands) {
    int r = 0;
    bool last_pinned = false;
    for (int d = 0; d < s->rank; ++d) {
        s->dim_of[d] = -1;
        if (s->extent[d] == 1) continue;
        bool merge = r > 0 && !last_pinned && !s->pinned[d];
        for (int k = 0; k < n_operands && merge; ++k) merge = s->stride[k][r - 1] == s->stride[k][d] * s->extent[d];
        if (merge) {
            s->extent[r - 1] *= s->extent[d];
            for (int k = 0; k < n_operands; ++k) s->stride[k][r - 1] = s->stride[k][d];
        } else {
            s->extent[r] = s->extent[d];
            for (int k = 0; k < n_operands; ++k) s->stride[k][r] = s->stride[k][d];
            ++r;
        }
        last_pinned = s->pinned[d];
        s->dim_of[d] = r - 1;
    }
    if (r == 0) {  // one element
        s->extent[0] = 1;
        for (int k = 0; k < n_operands; ++k) s->stride[k][0] = 0;
        r = 1;
    }
    s->rank = r;
}

void fill_operand(EwOperand* o, void* base, int dtype, const EwShape& s, int k, int vec) {
    const int inner = s.rank - 1;
    const int64_t es = static_cast<int64_t>(mhlo_cuda_dtype_size(dtype));
    o->base = base;
    o->dtype = dtype;
    o->inner = s.stride[k][inner];
    // a 16-byte access needs a dense innermost dimension and every row on the grid of V elements
    bool on_grid = vec > 1 && o->inner == 1 && (reinterpret_cast<uintptr_t>(base) % static_cast<uintptr_t>(vec * es < 16 ? vec * es : 16)) == 0;
    for (int d = 0; d < inner; ++d) {
        o->outer[d] = s.stride[k][d];
        on_grid = on_grid && s.stride[k][d] % vec == 0;
    }
    o->access = o->inner == 0 ? kSplat : on_grid ? kVector : kStrided;
}

// Operand registers (inputs, then one per instruction) -> shared-memory slots. Inputs take the first slots; a result gets
// one only when something other than the next instruction reads it, and gives it back behind its last reader.
int assign_slots(const mhlo_cuda_ew_inst* prog, int n_inputs, int n_insts, EwInstr* out) {
    constexpr int kRegs = MHLO_CUDA_EW_MAX_INPUTS + MHLO_CUDA_EW_MAX_INSTS;
    int last_use[kRegs], slot[kRegs];
    bool kept[kRegs];
    for (int r = 0; r < kRegs; ++r) { last_use[r] = -1; slot[r] = -1; kept[r] = false; }
    auto reads = [&](int i, int* regs) {
        const mhlo_cuda_ew_inst& in = prog[i];
        if (in.op == MHLO_EW_IMM || in.op == MHLO_EW_IOTA) return 0;
        regs[0] = in.a; regs[1] = in.b; regs[2] = in.c;
        return in.op == MHLO_EW_SELECT || in.op == MHLO_EW_CLAMP ? 3 : 2;
    };
    for (int i = 0; i < n_insts; ++i) {
        int regs[3];
        const int n = reads(i, regs);
        for (int k = 0; k < n; ++k) {
            last_use[regs[k]] = i;
            if (regs[k] >= n_inputs && regs[k] != n_inputs + i - 1) kept[regs[k]] = true;
        }
    }
    bool used[kRegs] = {};
    int high = n_inputs;
    for (int r = 0; r < n_inputs; ++r) { slot[r] = r; used[r] = true; }
    for (int i = 0; i < n_insts; ++i) {
        int regs[3] = {0, 0, 0};
        const int n = reads(i, regs);
        auto place = [&](int k) -> int8_t {
            if (k >= n) return kPrevious;
            return regs[k] == n_inputs + i - 1 && i > 0 ? kPrevious : static_cast<int8_t>(slot[regs[k]]);
        };
        out[i].op = static_cast<int16_t>(prog[i].op);
        out[i].imm = prog[i].imm;
        out[i].a = place(0); out[i].b = place(1); out[i].c = place(2);
        for (int k = 0; k < n; ++k)
            if (last_use[regs[k]] == i && slot[regs[k]] >= 0) used[slot[regs[k]]] = false;
        out[i].dst = kNowhere;
        const int r = n_inputs + i;
        if (kept[r]) {
            int s = 0;
            while (used[s]) ++s;
            used[s] = true;
            slot[r] = s;
            out[i].dst = static_cast<int8_t>(s);
            high = s + 1 > high ? s + 1 : high;
        }
    }
    return high;
}

// Up to this many elements (two CTAs of 256 threads per SM) a thread takes one element of anything but a short program of cheap
// float operators over dense operands, whose 16-byte accesses are worth more. 10000 elements, V elements a thread -> one: bf16 power
// 5.1 -> 3.2 us, f64 exponential 3.6 -> 2.6, i32 divide 3.6 -> 3.0, f32 compare 3.4 -> 2.6, sixteen bf16 instructions 12.5 -> 9.0;
// f32 add 2.1 -> 2.6. At 320000 the vectors lead everywhere.
constexpr int64_t kFewElements = kNumSMs * 512;

// Float operators that ew_apply has inline: a few instructions each.
bool inlined_op(int op) {
    switch (op) {
        case MHLO_EW_COPY: case MHLO_EW_IMM: case MHLO_EW_ADD: case MHLO_EW_SUB: case MHLO_EW_MUL: case MHLO_EW_DIV: case MHLO_EW_MAX: case MHLO_EW_MIN:
        case MHLO_EW_NEG: case MHLO_EW_ABS: case MHLO_EW_SQRT: case MHLO_EW_RSQRT: case MHLO_EW_SELECT: case MHLO_EW_RELU: case MHLO_EW_EXP:
        case MHLO_EW_TANH: case MHLO_EW_LOGISTIC: case MHLO_EW_SILU: case MHLO_EW_GELU_TANH: case MHLO_EW_ROUND_TO: return true;
        default: return false;
    }
}

template <typename C, int V>
int launch_single(const EwParams& p, cudaStream_t s) {
    const int64_t blocks = (p.n_vec + 255) / 256;
    const int grid = static_cast<int>(blocks < kNumSMs * 32 ? blocks : kNumSMs * 32);
    switch (p.n_inputs) {
        case 0: ew_single_kernel<C, V, 0><<<grid, 256, 0, s>>>(p); break;
        case 1: ew_single_kernel<C, V, 1><<<grid, 256, 0, s>>>(p); break;
        case 2: ew_single_kernel<C, V, 2><<<grid, 256, 0, s>>>(p); break;
        default: ew_single_kernel<C, V, 3><<<grid, 256, 0, s>>>(p); break;
    }
    MHLO_CUDA_CHECK_LAUNCH("elementwise");
    return MHLO_CUDA_OK;
}

template <typename C, int V>
int launch_program(const EwParams& p, int n_slots, cudaStream_t s) {
    const size_t smem = static_cast<size_t>(n_slots) * V * sizeof(C) * kProgramThreads;  // at most 40 slots x 4 KB
    if (smem > 48 * 1024) {
        // The limit belongs to the kernel and not to a launch: once per device, for the largest program there is, so that one
        // thread's setting is never too small for what another is about to launch.
        constexpr int kMost = (MHLO_CUDA_EW_MAX_INPUTS + MHLO_CUDA_EW_MAX_INSTS) * V * static_cast<int>(sizeof(C)) * kProgramThreads;
        static std::atomic<uint64_t> configured{0};
        int dev = 0;
        MHLO_CUDA_TRY(cudaGetDevice(&dev), MHLO_CUDA_NO_DEVICE);
        const uint64_t bit = uint64_t{1} << (dev & 63);
        if (!(configured.load(std::memory_order_acquire) & bit)) {
            MHLO_CUDA_TRY(cudaFuncSetAttribute(ew_program_kernel<C, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMost), MHLO_CUDA_EXECUTION_FAILED);
            configured.fetch_or(bit, std::memory_order_release);
        }
    }
    const int64_t blocks = (p.n_vec + kProgramThreads - 1) / kProgramThreads;
    const int grid = static_cast<int>(blocks < kNumSMs * 64 ? blocks : kNumSMs * 64);
    ew_program_kernel<C, V><<<grid, kProgramThreads, smem, s>>>(p);
    MHLO_CUDA_CHECK_LAUNCH("elementwise");
    return MHLO_CUDA_OK;
}

}  // namespace
}  // namespace mhlo

using namespace mhlo;

extern "C" {

static int elementwise_impl(const mhlo_cuda_view* inputs, int32_t n_inputs, const mhlo_cuda_ew_inst* prog,
                            int32_t n_insts, void* out_dev, int32_t out_dtype, const int64_t* out_shape,
                            int32_t out_rank, const int64_t* out_strides, mhlo_cuda_stream_t stream) {
    if (n_inputs < 0 || n_inputs > MHLO_CUDA_EW_MAX_INPUTS || n_insts < 1 || n_insts > MHLO_CUDA_EW_MAX_INSTS)
        return fail(MHLO_CUDA_INVALID_ARGUMENT, "elementwise: %d inputs / %d instructions outside the limits (%d / %d)",
                    n_inputs, n_insts, MHLO_CUDA_EW_MAX_INPUTS, MHLO_CUDA_EW_MAX_INSTS);
    if (out_rank < 0 || out_rank > MHLO_CUDA_MAX_RANK)
        return fail(MHLO_CUDA_UNSUPPORTED, "elementwise: rank %d above %d", out_rank, MHLO_CUDA_MAX_RANK);
    if (mhlo_cuda_dtype_size(out_dtype) == 0) return fail(MHLO_CUDA_INVALID_ARGUMENT, "elementwise: bad output dtype %d", out_dtype);
    EwShape shape;
    shape.rank = out_rank;
    int64_t n = 1;
    for (int d = 0; d < out_rank; ++d) {
        if (out_shape[d] < 0) return fail(MHLO_CUDA_INVALID_ARGUMENT, "elementwise: negative extent");
        shape.extent[d] = out_shape[d];
        shape.pinned[d] = false;
        n *= out_shape[d];
    }
    if (n == 0) return MHLO_CUDA_OK;
    if (out_dev == nullptr) return fail(MHLO_CUDA_INVALID_ARGUMENT, "elementwise: null output");
    bool any_f64 = out_dtype == MHLO_DT_F64, any_float = is_float_dt(out_dtype), any_u64 = out_dtype == MHLO_DT_UI64;
    bool all_bool = out_dtype == MHLO_DT_I1, narrow = mhlo_cuda_dtype_size(out_dtype) < 4;
    for (int k = 0; k < n_inputs; ++k) {
        if (inputs[k].rank != out_rank)
            return fail(MHLO_CUDA_INVALID_ARGUMENT, "elementwise: input %d has rank %d, output has %d", k, inputs[k].rank, out_rank);
        if (inputs[k].base == nullptr) return fail(MHLO_CUDA_INVALID_ARGUMENT, "elementwise: input %d is null", k);
        if (mhlo_cuda_dtype_size(inputs[k].dtype) == 0) return fail(MHLO_CUDA_INVALID_ARGUMENT, "elementwise: bad dtype");
        for (int d = 0; d < out_rank; ++d) shape.stride[k][d] = inputs[k].stride[d];
        any_f64 |= inputs[k].dtype == MHLO_DT_F64;
        any_float |= is_float_dt(inputs[k].dtype);
        any_u64 |= inputs[k].dtype == MHLO_DT_UI64;
        all_bool &= inputs[k].dtype == MHLO_DT_I1;
        narrow |= mhlo_cuda_dtype_size(inputs[k].dtype) < 4;
    }
    int64_t dense = 1;
    for (int d = out_rank - 1; d >= 0; --d) {
        shape.stride[n_inputs][d] = out_strides != nullptr ? out_strides[d] : dense;
        dense *= out_shape[d];
    }
    mhlo_cuda_ew_inst insts[MHLO_CUDA_EW_MAX_INSTS];
    for (int k = 0; k < n_insts; ++k) {
        mhlo_cuda_ew_inst in = prog[k];
        const int limit = n_inputs + k;
        if (in.op < 0 || in.op >= MHLO_EW_OP_COUNT) return fail(MHLO_CUDA_INVALID_ARGUMENT, "elementwise: bad opcode %d", in.op);
        if (in.op == MHLO_EW_IOTA && (in.imm < 0 || in.imm >= out_rank))
            return fail(MHLO_CUDA_INVALID_ARGUMENT, "elementwise: iota dimension out of range");
        const bool nullary = in.op == MHLO_EW_IMM || in.op == MHLO_EW_IOTA;
        if (!nullary && (in.a < 0 || in.a >= limit || in.b < 0 || in.b >= (limit > 0 ? limit : 1) || in.c < 0 || in.c >= (limit > 0 ? limit : 1)))
            return fail(MHLO_CUDA_INVALID_ARGUMENT, "elementwise: instruction %d reads a register that is not defined yet", k);
        if (nullary) in.a = in.b = in.c = 0;
        if (in.op == MHLO_EW_IOTA) shape.pinned[static_cast<int>(in.imm)] = true;
        insts[k] = in;
    }
    collapse(&shape, n_inputs + 1);
    for (int k = 0; k < n_insts; ++k)
        if (insts[k].op == MHLO_EW_IOTA) {
            const int d = shape.dim_of[static_cast<int>(insts[k].imm)];
            if (d < 0) { insts[k].op = MHLO_EW_IMM; insts[k].imm = 0.0; }
            else insts[k].imm = d;
        }
    // eight elements per thread where a 16-bit (or narrower) tensor takes part, four otherwise: 16 bytes of the narrower type
    int vec = !any_f64 && any_float && narrow ? 8 : 4;
    EwParams p;
    memset(&p, 0, sizeof p);
    auto lay_out = [&] {
        auto wide = [](const EwOperand& o) { return o.access == kVector && is_float_dt(o.dtype); };
        bool all = true;  // operands move in 16-byte accesses
        for (int k = 0; k < n_inputs; ++k) {
            fill_operand(&p.in[k], const_cast<void*>(inputs[k].base), inputs[k].dtype, shape, k, vec);
            all = all && (p.in[k].access == kSplat || wide(p.in[k]));
        }
        fill_operand(&p.out, out_dev, out_dtype, shape, n_inputs, vec);
        return all && wide(p.out);
    };
    const bool in_vectors = lay_out();
    if (n <= kFewElements) {
        bool cheap = in_vectors && !any_f64 && (vec == 4 || n_insts == 1);
        for (int k = 0; k < n_insts; ++k) cheap = cheap && inlined_op(insts[k].op);
        if (!cheap) {
            vec = 1;
            lay_out();
        }
    }
    if (p.out.access == kSplat) p.out.access = kStrided;  // one innermost element
    p.n_outer = shape.rank - 1;
    p.per_row = (shape.extent[p.n_outer] + vec - 1) / vec;
    p.n_vec = p.per_row;
    for (int d = 0; d < shape.rank; ++d) p.extent[d] = shape.extent[d];
    for (int d = 0; d < p.n_outer; ++d) p.n_vec *= shape.extent[d];
    p.wide = p.n_vec >= (int64_t{1} << 31);
    if (!p.wide) {
        p.per_row_div = FastDiv(static_cast<uint32_t>(p.per_row));
        for (int d = 0; d < p.n_outer; ++d) p.div[d] = FastDiv(static_cast<uint32_t>(shape.extent[d]));
    }
    p.n_inputs = n_inputs;
    p.n_insts = n_insts;
    p.unsigned_mode = any_u64;
    p.int_bits = static_cast<int>(8 * mhlo_cuda_dtype_size(n_inputs > 0 ? inputs[0].dtype : out_dtype));
    p.bool_mode = all_bool;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    // one instruction whose operands are the inputs in order (how single operators are built; an operand a unary operator
    // does not read may name any of them). With two inputs the kernel hands the first one to the third operand.
    const mhlo_cuda_ew_inst& first = insts[0];
    const bool reads_c = first.op == MHLO_EW_SELECT || first.op == MHLO_EW_CLAMP;
    const bool in_order = n_inputs == 0 || (first.a == 0 && (n_inputs < 2 || first.b == 1) && (n_inputs < 3 || first.c == 2) &&
                                            (n_inputs != 2 || !reads_c || first.c == 0));
    if (n_insts == 1 && n_inputs <= 3 && in_order) {
        p.prog[0].op = static_cast<int16_t>(first.op);
        p.prog[0].imm = first.imm;
        if (vec == 1) return any_f64 ? launch_single<double, 1>(p, s) : !any_float ? launch_single<int64_t, 1>(p, s) : launch_single<float, 1>(p, s);
        if (any_f64) return launch_single<double, 4>(p, s);
        if (!any_float) return launch_single<int64_t, 4>(p, s);
        return vec == 8 ? launch_single<float, 8>(p, s) : launch_single<float, 4>(p, s);
    }
    const int slots = assign_slots(insts, n_inputs, n_insts, p.prog);
    if (vec == 1)
        return any_f64 ? launch_program<double, 1>(p, slots, s) : !any_float ? launch_program<int64_t, 1>(p, slots, s) : launch_program<float, 1>(p, slots, s);
    if (any_f64) return launch_program<double, 4>(p, slots, s);
    if (!any_float) return launch_program<int64_t, 4>(p, slots, s);
    return vec == 8 ? launch_program<float, 8>(p, slots, s) : launch_program<float, 4>(p, slots, s);
}

int mhlo_cuda_elementwise(const mhlo_cuda_view* inputs, int32_t n_inputs, const mhlo_cuda_ew_inst* prog,
                          int32_t n_insts, void* out_dev, int32_t out_dtype, const int64_t* out_shape,
                          int32_t out_rank, mhlo_cuda_stream_t stream) {
    return elementwise_impl(inputs, n_inputs, prog, n_insts, out_dev, out_dtype, out_shape, out_rank, nullptr, stream);
}

int mhlo_cuda_elementwise_to_view(const mhlo_cuda_view* inputs, int32_t n_inputs, const mhlo_cuda_ew_inst* prog,
                                  int32_t n_insts, const mhlo_cuda_view* out, mhlo_cuda_stream_t stream) {
    if (!out || out->rank < 0 || out->rank > MHLO_CUDA_MAX_RANK)
        return fail(MHLO_CUDA_INVALID_ARGUMENT, "elementwise_to_view: bad destination view");
    return elementwise_impl(inputs, n_inputs, prog, n_insts, const_cast<void*>(out->base), out->dtype, out->shape,
                            out->rank, out->stride, stream);
}

}  // extern "C"
