// Operands of the split-operand kernels: fp32 numbers as sums of three 16-bit ones.
#pragma once

#include "common.cuh"

namespace corope {

struct SplitRows {   // three bf16 copies [B, H, N, D], `plane` elements apart: hi, mid, lo
    __nv_bfloat16* rows;
    size_t plane;
};

#ifdef __CUDACC__
// How V and dO enter the MMAs: 16-bit tensors as they are, fp32 tensors as three bf16 parts; P in parts of the same type.
template <typename T> struct Plain {
    using Mma = T;
    static constexpr int kParts = 1, kDtype = Elem<T>::kDtype;
};
template <> struct Plain<float> {
    using Mma = __nv_bfloat16;
    static constexpr int kParts = 3, kDtype = COROPE_DTYPE_BF16;
};
// the products of two split operands, smallest first: parts of the one and of the other
constexpr int kProducts = 6;
__host__ __device__ constexpr int product_a(int i) { return i == 0 ? 1 : i == 2 ? 2 : i == 4 ? 1 : 0; }
__host__ __device__ constexpr int product_b(int i) { return i == 0 ? 1 : i == 1 ? 2 : i == 3 ? 1 : 0; }
// One product of a 64-row block of streamed rows as the K dimension, A from TMEM: a(kk), b(kk) for the k-step of 16 rows `kk`.  REL >= 0: a
// block on the diagonal, REL rows (0 or 64) behind the first owned one.  Owned rows that a k-step's 16 rows are all hidden from are then left
// out, because their 0 (P or dS) would make an infinity or a NaN of a row that they have no part in their own.  KEYS: the owned rows are
// keys, seen by the streamed rows behind them, else queries.  The step with the most owned rows comes first and is the one that may start the sum.
struct WholeBlock { static constexpr int kRel = -1; };
struct FirstOnDiagonal { static constexpr int kRel = 0; };
struct SecondOnDiagonal { static constexpr int kRel = 64; };
template <bool KEYS, typename Where, int X = 0, typename A, typename B>
__device__ __forceinline__ void block_product(Where where, bool leader, uint32_t d, A a, B b, uint32_t b_hi, uint32_t idesc, bool start) {
    constexpr int kk = KEYS && Where::kRel >= 0 ? 3 - X : X, rel = Where::kRel + 16 * kk;
    const uint32_t accumulate = start && X == 0 ? 0u : 1u;
    if constexpr (Where::kRel < 0) {
        if (leader) umma_ts2(d, a(kk), b(kk), b_hi, idesc, accumulate);
    } else {
        if (leader) umma_ts2_lanes<KEYS ? 0 : rel, KEYS ? rel + 16 : 128>(d, a(kk), b(kk), b_hi, idesc, accumulate);
    }
    if constexpr (X < 3) block_product<KEYS, Where, X + 1>(where, leader, d, a, b, b_hi, idesc, start);
}
// eight neighbouring numbers of a row, aligned to 16 bytes
template <typename T>
__device__ __forceinline__ void load8(const T* __restrict__ x, float2 (&to)[4]) {
    if constexpr (sizeof(T) == 4) {
        const float4 a = *reinterpret_cast<const float4*>(x), b = *reinterpret_cast<const float4*>(x + 4);
        to[0] = make_float2(a.x, a.y), to[1] = make_float2(a.z, a.w), to[2] = make_float2(b.x, b.y), to[3] = make_float2(b.z, b.w);
    } else {
        const uint4 a = *reinterpret_cast<const uint4*>(x);
        to[0] = unpack2<T>(a.x), to[1] = unpack2<T>(a.y), to[2] = unpack2<T>(a.z), to[3] = unpack2<T>(a.w);
    }
}
template <typename T>
__device__ __forceinline__ void store8(T* to, const float2 (&x)[4]) {
    if constexpr (sizeof(T) == 4) {
        *reinterpret_cast<float4*>(to) = make_float4(x[0].x, x[0].y, x[1].x, x[1].y);
        *reinterpret_cast<float4*>(to + 4) = make_float4(x[2].x, x[2].y, x[3].x, x[3].y);
    } else {
        *reinterpret_cast<uint4*>(to) = make_uint4(pack2<T>(x[0].x, x[0].y), pack2<T>(x[1].x, x[1].y), pack2<T>(x[2].x, x[2].y), pack2<T>(x[3].x, x[3].y));
    }
}

// (a, b) minus a pair of T: fp32 additions that take the 16-bit number as it is, so nothing is converted back
template <typename T>
__device__ __forceinline__ void subtract_pair(uint32_t pair, float& a, float& b) {
    if constexpr (Elem<T>::kDtype == COROPE_DTYPE_F16)
        asm("{\n\t.reg .f16 lo, hi;\n\tmov.b32 {lo, hi}, %2;\n\tadd.rn.f32.f16 %0, lo, %0;\n\tadd.rn.f32.f16 %1, hi, %1;\n\t}" : "+f"(a), "+f"(b) : "r"(pair ^ 0x80008000u));
    else
        asm("{\n\t.reg .b16 lo, hi;\n\tmov.b32 {lo, hi}, %2;\n\tadd.rn.f32.bf16 %0, lo, %0;\n\tadd.rn.f32.bf16 %1, hi, %1;\n\t}" : "+f"(a), "+f"(b) : "r"(pair ^ 0x80008000u));
}
// parts[] = hi, mid, lo of (a, b), each rounded to T; a non-finite number is its own hi
template <typename T>
__device__ __forceinline__ void split3(float a, float b, uint32_t (&parts)[3]) {
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        parts[x] = pack2<T>(a, b);
        if (x < 2) subtract_pair<T>(parts[x], a, b);
    }
}
// the same for two finite numbers, bf16 parts cut off instead of rounded (the three then hold the 24 bits exactly): byte permutes and
// masks instead of conversions
template <typename T>
__device__ __forceinline__ void split3_cut(float a, float b, uint32_t (&parts)[3]) {
    if constexpr (Elem<T>::kDtype == COROPE_DTYPE_BF16) {
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            const uint32_t ua = __float_as_uint(a), ub = __float_as_uint(b);
            parts[x] = __byte_perm(ua, ub, 0x7632);
            if (x < 2) f2_unpack(f2_sub(f2_pack(a, b), f2_pack_bits(ua & 0xffff0000u, ub & 0xffff0000u)), a, b);
        }
    } else {
        split3<T>(a, b, parts);
    }
}
// bf16 parts of operands of any value: three rounded ones hold the 24 bits of every number of its own, whatever the size of its neighbours.
// A finite number beyond the largest bf16 number, which would round to an infinity, has that one as its hi.  What is not finite is hi alone, or
// (`in_lo`, for V and dO) lo alone: of the six products lo only meets the leading part of the other operand, so an infinity never meets a
// part that is 0 where the number is not.
__device__ __forceinline__ void split3_any(float a, float b, uint32_t (&parts)[3], bool in_lo = false) {
    constexpr float kTop = 0x1.fep127f;
    const bool fa = fabsf(a) < INFINITY, fb = fabsf(b) < INFINITY;
    const float x = a, y = b;
    parts[0] = pack_bf162(fa ? fminf(fmaxf(a, -kTop), kTop) : in_lo ? 0.f : x, fb ? fminf(fmaxf(b, -kTop), kTop) : in_lo ? 0.f : y);
    float2 f = unpack_bf162(parts[0]);
    a = fa ? a - f.x : 0.f, b = fb ? b - f.y : 0.f;
    parts[1] = pack_bf162(a, b);
    f = unpack_bf162(parts[1]);
    parts[2] = pack_bf162(fa || !in_lo ? a - f.x : x, fb || !in_lo ? b - f.y : y);
}

// The leading products of two split operands (hi hi) are one chain of MMAs per 16 columns, whose adder drops bits towards zero: 2^-26 of the
// sum per step on average (measured through the LSE, N(0, 1) to N(0, 64) inputs: 1.07 2^-24 in the 4 steps of D = 64, 1.99 2^-24 in the 8 of
// D = 128).  This joins both sums and puts that mean back; the LSE's error at scores with a standard deviation of 16 goes from 6.9e-6 to 3.9e-6
// (D = 64), from 9.3e-6 to 4.7e-6 (D = 128).  (Leading parts on a common grid per row would make the chain exact, but cost the small elements of
// a row up to 8 of their 24 bits: with channels of different scale the results were off by up to 1e-3.)
template <int D>
__device__ __forceinline__ uint64_t join_products(uint64_t leading, uint64_t smaller) {
    constexpr float kDropped = D / 16 * 0x1p-26f;
    return f2_add(leading, f2_fma(leading, f2_pack(kDropped, kDropped), smaller));
}
// two rotation pairs (a.x, b.x), (a.y, b.y) by neighbouring table entries
__device__ __forceinline__ void rotate(float2& a, float2& b, const float* c, const float* s) {
    const float2 x = a, y = b;
    a = make_float2(x.x * c[0] - y.x * s[0], x.y * c[1] - y.y * s[1]);
    b = make_float2(y.x * c[0] + x.x * s[0], y.y * c[1] + x.y * s[1]);
}
// rows of both tables are aligned to 16 bytes
__host__ __device__ __forceinline__ bool tables_aligned(const RopeParams& p) {
    return (((uintptr_t)p.cos | (uintptr_t)p.sin) & 15) == 0 && (p.table_stride & 3) == 0;
}
__device__ __forceinline__ void load_table8(const float* __restrict__ src, bool vec, float (&x)[8]) {
    if (vec) {
        const float4 a = *reinterpret_cast<const float4*>(src), b = *reinterpret_cast<const float4*>(src + 4);
        x[0] = a.x, x[1] = a.y, x[2] = a.z, x[3] = a.w, x[4] = b.x, x[5] = b.y, x[6] = b.z, x[7] = b.w;
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = src[i];
    }
}
// Scores that joined to NaN: an infinity of an operand is its leading part alone, so the leading products have it with the sign it has in fp32
// (the smaller ones may be 0 times it).  `col`: their TMEM column, still as the MMAs left it; the whole warp comes here.
__device__ __forceinline__ void infinite_scores(uint32_t col, float (&s)[16]) {
#pragma unroll
    for (int half = 0; half < 16; half += 8) {
        uint32_t leading[8];
        COROPE_TMEM_LD8(col + half, leading);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 8; ++i) s[half + i] = fabsf(__uint_as_float(leading[i])) == INFINITY ? __uint_as_float(leading[i]) : s[half + i];
    }
}

// P of f16 tensors enters its products times this
template <typename T> constexpr float kPScale = Elem<T>::kDtype == COROPE_DTYPE_F16 ? 16384.f : 1.f;
#endif

// The split copies of a call in its workspace.  V and dO (rows null: not copied) of fp32 tensors only.
struct SplitCopies {
    SplitRows k, q, v, d_o;
};
SplitCopies split_copies(const RopeParams& p, void* ws, bool bwd, int dtype);
// Pre-pass: the copies whose `rows` are set, K and Q rotated by the tables of p (none: as they are), Q times sm_scale * log2e; with_delta:
// p.delta from p.o and p.d_o; the two words at p.sched_counter are zeroed.
int launch_split_rows(const RopeParams& p, const SplitCopies& to, bool with_delta, int dtype, cudaStream_t s);

}  // namespace corope
