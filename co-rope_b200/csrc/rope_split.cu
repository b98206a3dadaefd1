// Fused-RoPE / plain attention for 16-bit tensors at lengths that are not whole 128-row tiles, D = 64 or 128: tensor-core products
// (mma.sync m16n8k16) of fp32 operands.  Every fp32 operand x enters the MMAs as hi + mid + lo, hi = x rounded to 16 bits, mid = (x - hi)
// rounded, lo = the rest.  Three bf16 numbers hold the 24 bits of an fp32 number exactly, so nothing is lost in the operands:
//     S  = Q~ K~^T        Q~, K~ rotated in fp32, both split into bf16      6 MMAs (without mid lo, lo mid, lo lo: about 2^-24)
//     dP = dO V^T         inputs as they are                                1 MMA
//     O += P V, dV += P^T dO     P split into the inputs' own type          3 MMAs
//     dQ += dS K~, dK += dS^T Q~  dS split into bf16                        6 MMAs
// bf16 for everything that is not bounded, so that no magnitude of the inputs leaves the range.  P <= 1 of f16 tensors enters its
// products times 2^14: the three numbers then reach down to 2^-38 of the row's largest probability.  The adder of the MMAs does not round to
// nearest; the large products therefore go through one 16-wide step each (with the smaller ones in front for the sums over keys or
// queries), which fp32 additions join.
//
// Error against 64-bit arithmetic next to the CUDA-core kernels with fp32 operands (N(0, 1) inputs, B1 H4 N1777 D128 causal f16): LSE
// 3.75e-7 (3.87e-7), results that are not the exact one rounded: O 0.11 % (0.33 %), dV 0.21 % (0.36 %); with q and k times 4 (scores
// with a standard deviation of 16) LSE 4.5e-6 (1.2e-5), O 0.29 % (0.71 %).  Two parts per operand (16 bits; half the MMAs, half the time)
// had 2 to 10 times the error of the fp32 kernels.
//
// The forward below is what short sequences take; the others run on tcgen05 MMAs (rope_split_fwd_sm100.cu).  Backward: B1 H32 N1777 D128
// bf16 causal 1315 us (the CUDA-core kernel 5081 us), B4 H16 N1000 D64 bf16 full 777 us (2890 us).
// What bounds it: mma.sync, measured at 553 TFLOP/s with all operands in registers (B200, 8 warps per SM); with 8 warps per SM
// (D = 128: 255 registers; D = 64: 12 warps) the latency between a tile's ldmatrix, MMAs and softmax is not fully hidden, and the
// shared-memory port is close behind, a warp's 16 rows reading every streamed tile, all three parts of it, once per product.
// Infinities in Q or K keep the scores they have in fp32; beyond that non-finite operands give NaN, also where fp32 sums would
// have been infinite.
//
// Math: fused-rope/rope_attn_pytorch.py:108-155 (forward), :187-222 (backward); exp2-domain softmax and log2-domain LSE as
// fused-rope/fused_rope_attn.py:103-114, 316.
#include <type_traits>

#include "rope_split.cuh"

namespace corope {
namespace {

// ------------------------------------------------------------------------------------------------ operands
// row-major 16-bit tile in shared memory: rows of D elements + 16 bytes, so that 8 consecutive rows of an ldmatrix fall into
// distinct bank groups
template <int D> struct Pitch { static constexpr int kBytes = 2 * D + 16; };

__device__ __forceinline__ void ldm_x4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldm_x4_trans(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
// byte offsets of a lane's ldmatrix row inside a tile.  A operand (16 rows x 16 k): registers a0..a3.  B operand from a tile with
// k contiguous: (b0, b1) of columns 0-7, then of columns 8-15.  B operand from a tile with the columns contiguous (.trans): the same.
template <int D> __device__ __forceinline__ uint32_t lane_a(int lane) { return ((lane & 7) + ((lane >> 3) & 1) * 8) * Pitch<D>::kBytes + (lane >> 4) * 16; }
template <int D> __device__ __forceinline__ uint32_t lane_b(int lane) { return ((lane & 7) + (lane >> 4) * 8) * Pitch<D>::kBytes + ((lane >> 3) & 1) * 16; }
template <int D> __device__ __forceinline__ uint32_t lane_bt(int lane) { return ((lane & 7) + ((lane >> 3) & 1) * 8) * Pitch<D>::kBytes + (lane >> 4) * 16; }

template <typename T> __device__ __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1);
template <> __device__ __forceinline__ void mma<__nv_bfloat16>(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
template <> __device__ __forceinline__ void mma<__half>(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// four neighbouring accumulator tiles d += a b, b the two ldmatrix_x4 results of their columns: independent MMAs back to back
template <typename T>
__device__ __forceinline__ void mma4(float (*d)[4], const uint32_t (&a)[4], const uint32_t (&b0)[4], const uint32_t (&b1)[4]) {
    mma<T>(d[0], a, b0[0], b0[1]);
    mma<T>(d[1], a, b0[2], b0[3]);
    mma<T>(d[2], a, b1[0], b1[1]);
    mma<T>(d[3], a, b1[2], b1[3]);
}
// d += t for four neighbouring accumulator tiles, rounded to nearest
__device__ __forceinline__ void add4(float (*d)[4], const float (&t)[4][4]) {
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int x = 0; x < 4; ++x) d[n][x] += t[n][x];
}
// the products of two split operands (PA and PB parts) for four neighbouring accumulator tiles, b[part][two ldmatrix_x4 results]: hi hi
// into `d` by way of an fp32 addition, the others into `e`, smallest first
template <int PA, int PB>
__device__ __forceinline__ void mma4_split(float (*d)[4], float (*e)[4], const uint32_t (&a)[PA][4], const uint32_t (&b)[PB][2][4]) {
    using B = __nv_bfloat16;
    float t[4][4] = {};
    if constexpr (PA > 1 && PB > 1) mma4<B>(e, a[1], b[1][0], b[1][1]);
    if constexpr (PB > 2) mma4<B>(e, a[0], b[2][0], b[2][1]);
    if constexpr (PA > 2) mma4<B>(e, a[2], b[0][0], b[0][1]);
    mma4<B>(t, a[0], b[0][0], b[0][1]);
    if constexpr (PB > 1) mma4<B>(e, a[0], b[1][0], b[1][1]);
    if constexpr (PA > 1) mma4<B>(e, a[1], b[0][0], b[0][1]);
    add4(d, t);
}
// hi hi + the smaller products.  An infinity shows in hi hi with the sign it has in fp32; the other parts of such a product are
// meaningless (0 or either infinity).
__device__ __forceinline__ float join(float main, float small) { return fabsf(main) < INFINITY ? main + small : main; }
// two neighbouring 8-column accumulator tiles as the A operand of one k-step, split: a[part]
template <typename T>
__device__ __forceinline__ void split_a(const float (&c0)[4], const float (&c1)[4], float scale, uint32_t (&a)[3][4]) {
    uint32_t w[4][3];
    split3<T>(c0[0] * scale, c0[1] * scale, w[0]);
    split3<T>(c0[2] * scale, c0[3] * scale, w[1]);
    split3<T>(c1[0] * scale, c1[1] * scale, w[2]);
    split3<T>(c1[2] * scale, c1[3] * scale, w[3]);
#pragma unroll
    for (int x = 0; x < 3; ++x)
#pragma unroll
        for (int e = 0; e < 4; ++e) a[x][e] = w[e][x];
}
// d += P b for four neighbouring tiles of columns, one 16-row step: its own sum, then one fp32 addition
template <typename T>
__device__ __forceinline__ void add_products(float (*d)[4], const uint32_t (&a)[3][4], const uint32_t (&b0)[4], const uint32_t (&b1)[4]) {
    float t[4][4] = {};
    mma4<T>(t, a[2], b0, b1);
    mma4<T>(t, a[1], b0, b1);
    mma4<T>(t, a[0], b0, b1);
    add4(d, t);
}
// the same with both operands split
template <int PB>
__device__ __forceinline__ void add_products_split(float (*d)[4], const uint32_t (&a)[3][4], const uint32_t (&b)[PB][2][4]) {
    using B = __nv_bfloat16;
    float t[4][4] = {};
    if constexpr (PB > 1) mma4<B>(t, a[1], b[1][0], b[1][1]);
    if constexpr (PB > 2) mma4<B>(t, a[0], b[2][0], b[2][1]);
    mma4<B>(t, a[2], b[0][0], b[0][1]);
    if constexpr (PB > 1) mma4<B>(t, a[0], b[1][0], b[1][1]);
    mma4<B>(t, a[1], b[0][0], b[0][1]);
    mma4<B>(t, a[0], b[0][0], b[0][1]);
    add4(d, t);
}

// 16 bytes global -> shared, zeros when `have` is false (the address is then not read)
__device__ __forceinline__ void cp16(uint32_t dst, const void* src, bool have) {
    const int bytes = have ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// ROWS rows [r0, r0 + ROWS) of X (row stride xs elements) into a padded tile, rows at or beyond N as zeros
template <int D, int ROWS, int THREADS, typename E>
__device__ __forceinline__ void load_rows(uint32_t dst, const E* X, int64_t xs, int r0, int N) {
    constexpr int kPerRow = D / 8;
#pragma unroll
    for (int it = 0; it < ROWS * kPerRow / THREADS; ++it) {
        const int idx = threadIdx.x + it * THREADS, r = idx / kPerRow, ch = idx % kPerRow, pos = r0 + r;
        const bool have = pos < N;
        cp16(dst + r * Pitch<D>::kBytes + ch * 16, X + (int64_t)(have ? pos : 0) * xs + ch * 8, have);
    }
}

// the three parts of ROWS rows of head `head` into three tiles `step` bytes apart
template <int D, int ROWS, int THREADS>
__device__ __forceinline__ void load_split(uint32_t dst, uint32_t step, const SplitRows& x, int head, int r0, int N) {
#pragma unroll
    for (int part = 0; part < 3; ++part) load_rows<D, ROWS, THREADS>(dst + part * step, x.rows + part * x.plane + (size_t)head * N * D, D, r0, N);
}

// Rotated K: three parts.  K of plain attention on bf16 tensors is its own hi part and is read where the caller has it (KP = 1): 3 MMAs per
// score product and 3 for dQ instead of 6, no pass over K.  (f16 K would need two bf16 parts: 5 instead of 6.)
template <typename T, int D, int KP, int ROWS, int THREADS>
__device__ __forceinline__ void load_k(uint32_t dst, uint32_t step, const RopeParams& p, const SplitRows& ks, int head, int r0) {
    if constexpr (KP == 1)
        load_rows<D, ROWS, THREADS>(dst, reinterpret_cast<const T*>(p.k) + row_offset(p.sk, p.Hkv, head, 0), p.sk.n, r0, p.N);
    else
        load_split<D, ROWS, THREADS>(dst, step, ks, head, r0, p.N);
}

// ------------------------------------------------------------------------------------------------
// pre-pass: rows of X rotated in fp32, times `scale`, split.  One thread per 8 pairs; the threads of a row are neighbouring lanes.
// ------------------------------------------------------------------------------------------------
template <typename T, int D>
__global__ void __launch_bounds__(256) split_rotate_kernel(const T* __restrict__ X, RowAddr ax, const float* __restrict__ cosT, const float* __restrict__ sinT,
                                                           int64_t ts, float scale, SplitRows out, size_t rows, int* counter) {
    constexpr int kPerRow = D / 16;
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    pdl_trigger();
    if (idx == 0 && counter != nullptr) *counter = 0;
    const bool live = idx / kPerRow < rows;
    const size_t row = live ? idx / kPerRow : rows - 1;   // threads beyond the last row take part in the shuffles with it
    const int d = (int)(idx % kPerRow) * 8, n = (int)(row % (size_t)ax.N);
    const T* src = X + flat_row_offset(ax, row) + d;
    const uint4 xa = *reinterpret_cast<const uint4*>(src), xb = *reinterpret_cast<const uint4*>(src + D / 2);
    const uint32_t a[4] = {xa.x, xa.y, xa.z, xa.w}, b[4] = {xb.x, xb.y, xb.z, xb.w};
    float2 ra[4], rb[4];
    float largest = 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        ra[e] = unpack2<T>(a[e]), rb[e] = unpack2<T>(b[e]);
        if (cosT != nullptr) {   // null tables: plain attention
            const float *c = cosT + (int64_t)n * ts + d + 2 * e, *s = sinT + (int64_t)n * ts + d + 2 * e;
            rotate(ra[e], rb[e], c, s);
        }
        ra[e].x *= scale, ra[e].y *= scale, rb[e].x *= scale, rb[e].y *= scale;
        largest = fmax3_nan(largest, fmax3_nan(0.f, fabsf(ra[e].x), fabsf(ra[e].y)), fmax3_nan(0.f, fabsf(rb[e].x), fabsf(rb[e].y)));
    }
#pragma unroll
    for (int off = 1; off < kPerRow; off <<= 1) largest = fmax3_nan(0.f, largest, __shfl_xor_sync(0xffffffffu, largest, off));
    const RowUnit unit = row_unit(largest);
    uint32_t pa[4][3], pb[4][3];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        split_row_pair(ra[e].x, ra[e].y, unit, pa[e]);
        split_row_pair(rb[e].x, rb[e].y, unit, pb[e]);
    }
    if (!live) return;
#pragma unroll
    for (int part = 0; part < 3; ++part) {
        __nv_bfloat16* o = out.rows + part * out.plane + row * D + d;
        *reinterpret_cast<uint4*>(o) = make_uint4(pa[0][part], pa[1][part], pa[2][part], pa[3][part]);
        *reinterpret_cast<uint4*>(o + D / 2) = make_uint4(pb[0][part], pb[1][part], pb[2][part], pb[3][part]);
    }
}

// ------------------------------------------------------------------------------------------------
// forward: 64 query rows per CTA (4 warps of 16), double-buffered key tiles of 64 (D = 64) or 32 keys
// ------------------------------------------------------------------------------------------------
template <int D, int KP> struct Fwd {
    static constexpr int kThreads = 128, kRows = 64, kCtas = D == 64 ? 3 : 2;
    static constexpr int kBN = D == 64 ? 64 : 32;
    static constexpr uint32_t kTile = kBN * Pitch<D>::kBytes;
    static constexpr uint32_t kStage = (KP + 1) * kTile;   // parts of K~, V
    static constexpr size_t kSmem = 2 * kStage;
};

template <typename T, int D, int KP>
__global__ void __launch_bounds__(Fwd<D, KP>::kThreads, Fwd<D, KP>::kCtas) rope_fwd_split_kernel(RopeParams p, SplitRows ks) {
    using F = Fwd<D, KP>;
    constexpr int BN = F::kBN, KS = D / 16, NT = BN / 8, DT = D / 8;
    extern __shared__ __align__(16) uint8_t smem[];
    const uint32_t sm = smem_u32(smem);
    // heads run fastest and the longest causal rows come first
    const int N = p.N, heads = p.B * p.H, bh = blockIdx.x % heads, kvh = bh / (p.H / p.Hkv);
    const int m0 = (gridDim.x / heads - 1 - blockIdx.x / heads) * F::kRows;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, c2 = (lane & 3) * 2;
    const int row0 = m0 + warp * 16 + g;   // the lane's rows: row0 and row0 + 8
    const T* V = reinterpret_cast<const T*>(p.v) + row_offset(p.sv, p.Hkv, kvh, 0);
    auto load = [&](int j0, int buf) {
        const uint32_t st = sm + buf * F::kStage;
        load_k<T, D, KP, BN, F::kThreads>(st, F::kTile, p, ks, kvh, j0);
        load_rows<D, BN, F::kThreads>(st + KP * F::kTile, V, p.sv.n, j0, N);
        cp_commit();
    };
    load(0, 0);

    // Q~ = rotated q * sm_scale * log2e as A operands, split; both columns of a rotation pair belong to the same lane
    uint32_t qa[KS][3][4];
    {
        const T* Q = reinterpret_cast<const T*>(p.q) + row_offset(p.sq, p.H, bh, 0);
        const float scale = p.sm_scale * kLog2e;
        // rows beyond the head repeat its last one (their results are not stored): no branch stands between the loads
        auto load_q = [&](auto rot) {
#pragma unroll
            for (int k = 0; k < KS / 2; ++k)
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    const int pos = min(row0 + (x & 1) * 8, N - 1), d = k * 16 + (x >> 1) * 8 + c2;
                    const T* q = Q + (int64_t)pos * p.sq.n + d;
                    float2 a = unpack2<T>(*reinterpret_cast<const uint32_t*>(q)), b = unpack2<T>(*reinterpret_cast<const uint32_t*>(q + D / 2));
                    if constexpr (decltype(rot)::value) rotate(a, b, p.cos + (int64_t)pos * p.table_stride + d, p.sin + (int64_t)pos * p.table_stride + d);
                    uint32_t w[3];
                    split3_any<__nv_bfloat16>(a.x * scale, a.y * scale, w);
#pragma unroll
                    for (int part = 0; part < 3; ++part) qa[k][part][x] = w[part];
                    split3_any<__nv_bfloat16>(b.x * scale, b.y * scale, w);
#pragma unroll
                    for (int part = 0; part < 3; ++part) qa[k + KS / 2][part][x] = w[part];
                }
        };
        if (p.cos != nullptr)
            load_q(std::true_type{});
        else
            load_q(std::false_type{});   // plain attention
    }
    float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f}, o[DT][4];
#pragma unroll
    for (int n = 0; n < DT; ++n) o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f;

    const int n_end = p.causal ? min(N, m0 + F::kRows) : N;
    int buf = 0;
    for (int j0 = 0; j0 < n_end; j0 += BN, buf ^= 1) {
        cp_wait_all();
        __syncthreads();   // the tile has landed for every thread, and every warp is done with the other buffer
        if (j0 + BN < n_end) load(j0 + BN, buf ^ 1);
        if (p.causal && j0 > m0 + warp * 16 + 15) continue;   // no key of the tile is seen by the warp's rows
        const uint32_t st = sm + buf * F::kStage, kk = st + lane_b<D>(lane), vv = st + KP * F::kTile + lane_bt<D>(lane);
        float s[NT][4];
#pragma unroll
        for (int np = 0; np < NT / 4; ++np) {   // 32 keys
            float (*main)[4] = s + 4 * np, small[4][4];
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
                for (int x = 0; x < 4; ++x) main[n][x] = small[n][x] = 0.f;
#pragma unroll
            for (int k = 0; k < KS; ++k) {
                uint32_t b[KP][2][4];
#pragma unroll
                for (int part = 0; part < KP; ++part)
#pragma unroll
                    for (int y = 0; y < 2; ++y) ldm_x4(b[part][y], kk + part * F::kTile + (2 * np + y) * 16 * Pitch<D>::kBytes + k * 32);
                mma4_split(main, small, qa[k], b);
            }
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
                for (int x = 0; x < 4; ++x) main[n][x] = join(main[n][x], small[n][x]);
        }
        // keys the lane's rows do not see
        if (j0 + BN > N || (p.causal && j0 + BN - 1 > m0 + warp * 16)) {
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    const int key = j0 + n * 8 + c2 + (x & 1);
                    if (key >= N || (p.causal && key > row0 + (x >> 1) * 8)) s[n][x] = -INFINITY;
                }
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            float mx = m[r];
#pragma unroll
            for (int n = 0; n < NT; ++n) mx = fmax3(mx, s[n][2 * r], s[n][2 * r + 1]);
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
            const float ref = mx == -INFINITY ? 0.f : mx;   // a row that has seen no key yet
            const float alpha = exp2f(m[r] - ref);
            float sum = 0.f;
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    s[n][2 * r + x] = exp2f(s[n][2 * r + x] - ref);
                    sum += s[n][2 * r + x];
                }
            l[r] = l[r] * alpha + sum;   // this lane's columns only; the four lanes of a row are added at the end
            m[r] = mx;
#pragma unroll
            for (int n = 0; n < DT; ++n) o[n][2 * r] *= alpha, o[n][2 * r + 1] *= alpha;
        }
#pragma unroll
        for (int t = 0; t < BN / 16; ++t) {
            uint32_t pa[3][4];
            split_a<T>(s[2 * t], s[2 * t + 1], kPScale<T>, pa);
#pragma unroll
            for (int dp = 0; dp < DT / 2; dp += 2) {
                uint32_t b0[4], b1[4];
                ldm_x4_trans(b0, vv + t * 16 * Pitch<D>::kBytes + dp * 32);
                ldm_x4_trans(b1, vv + t * 16 * Pitch<D>::kBytes + dp * 32 + 32);
                add_products<T>(o + 2 * dp, pa, b0, b1);
            }
        }
    }
    T* O = reinterpret_cast<T*>(p.out_o) + row_offset(p.so, p.H, bh, 0);
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        float sum = l[r];
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        const int pos = row0 + 8 * r;
        if (pos >= N) continue;
        const float inv = sum > 0.f ? (1.f / kPScale<T>) / sum : 0.f;
        uint32_t* out = reinterpret_cast<uint32_t*>(O + (int64_t)pos * p.so.n + c2);
#pragma unroll
        for (int n = 0; n < DT; ++n) out[n * 4] = pack2<T>(o[n][2 * r] * inv, o[n][2 * r + 1] * inv);
        if (c2 == 0) p.lse2[(size_t)bh * N + pos] = m[r] + log2f(sum);
    }
}

// ------------------------------------------------------------------------------------------------
// backward: two kernels of one form.  KV = false: dQ of 64 query rows, sweeping the keys.  KV = true: dK, dV of 64 keys, sweeping
// the query rows of the group's heads (everything transposed).  The owned rows are the A operands, the streamed rows the B operands of
// both score products, and the streamed rotated rows again those of the gradient product.  The scores are formed twice (29 MMAs against
// 22), but every sum has one owner and one order: the same bits every time, and no fp32 accumulator of dQ.
// A warp owns 16 rows and takes 32 streamed rows per step.  D = 64: 4 warps, three CTAs per SM.  D = 128: the parts of the owned rows fill
// half of the shared memory, so 8 warps share them, two per 16 rows, each with its half of the streamed rows; their sums meet at the
// end: B1 H32 N1777 1315 us, B1 H2 N1023 244 us, forward + backward of B1 Hq8 Hkv2 N2400 without rotation 1349 us.  (8 warps on 128 owned
// rows, half the CTAs: 1262, 417 and 2776 us.)
// ------------------------------------------------------------------------------------------------
template <int D, int KP, bool KV> struct Bwd {
    static constexpr int kGroups = D == 64 ? 1 : 2, kThreads = 128 * kGroups, kCtas = D == 64 ? 3 : 1;
    static constexpr int kRows = 64, kStep = 32, kBS = kStep * kGroups;   // owned rows; streamed rows per step of a warp and of the CTA
    static constexpr int kOwnParts = KV ? KP : 3, kStrParts = KV ? 3 : KP;   // parts of the rotated rows; the plain rows follow them
    static constexpr uint32_t kOwn = kRows * Pitch<D>::kBytes, kTile = kBS * Pitch<D>::kBytes, kStage = (kStrParts + 1) * kTile;
    static constexpr size_t kSmem = (kOwnParts + 1) * kOwn + 2 * kStage;
    static_assert(kGroups == 1 || kSmem >= (KV ? 2 : 1) * kRows * (D + 4) * sizeof(float), "room for the sums of the second group");
};

template <typename T, int D, int KP, bool KV>
__global__ void __launch_bounds__(Bwd<D, KP, KV>::kThreads, Bwd<D, KP, KV>::kCtas) rope_bwd_split_kernel(RopeParams p, SplitRows qs, SplitRows ks) {
    using W = Bwd<D, KP, KV>;
    constexpr int BS = W::kBS, SR = W::kStep, KS = D / 16, NT = SR / 8, DT = D / 8, kThreads = W::kThreads, kRows = W::kRows, OP = W::kOwnParts, SP = W::kStrParts;
    static_assert(NT == 4, "the score products of a step are four accumulator tiles");
    extern __shared__ __align__(16) uint8_t smem[];
    const uint32_t sm = smem_u32(smem), stages = sm + (OP + 1) * W::kOwn;
    const int N = p.N, G = p.H / p.Hkv;
    const int warp = (threadIdx.x >> 5) & 3, group = threadIdx.x >> 7, lane = threadIdx.x & 31, g = lane >> 2, c2 = (lane & 3) * 2;
    const int heads = p.B * (KV ? p.Hkv : p.H), own_head = blockIdx.x % heads, block = blockIdx.x / heads;   // KV: a K / V head, otherwise a query head
    const int kvh = KV ? own_head : own_head / G;
    const int own0 = (KV ? block : gridDim.x / heads - 1 - block) * kRows;   // long causal sweeps first
    const int row0 = own0 + warp * 16 + g;                   // the lane's owned rows: row0 and row0 + 8
    const int first = KV && p.causal ? own0 : 0, end = !KV && p.causal ? min(N, own0 + kRows) : N;
    const int steps = (end - first + BS - 1) / BS, total = KV ? steps * G : steps;

    auto load = [&](int step, int buf) {
        const uint32_t st = stages + buf * W::kStage;
        const int r0 = first + (KV ? step % steps : step) * BS;
        if constexpr (KV) {
            const int qh = kvh * G + step / steps;
            load_split<D, BS, kThreads>(st, W::kTile, qs, qh, r0, N);
            load_rows<D, BS, kThreads>(st + SP * W::kTile, reinterpret_cast<const T*>(p.d_o) + row_offset(p.sdo, p.H, qh, 0), p.sdo.n, r0, N);
        } else {
            load_k<T, D, KP, BS, kThreads>(st, W::kTile, p, ks, kvh, r0);
            load_rows<D, BS, kThreads>(st + SP * W::kTile, reinterpret_cast<const T*>(p.v) + row_offset(p.sv, p.Hkv, kvh, 0), p.sv.n, r0, N);
        }
        cp_commit();
    };
    if constexpr (KV) {
        load_k<T, D, KP, kRows, kThreads>(sm, W::kOwn, p, ks, own_head, own0);
        load_rows<D, kRows, kThreads>(sm + OP * W::kOwn, reinterpret_cast<const T*>(p.v) + row_offset(p.sv, p.Hkv, own_head, 0), p.sv.n, own0, N);
    } else {
        load_split<D, kRows, kThreads>(sm, W::kOwn, qs, own_head, own0, N);
        load_rows<D, kRows, kThreads>(sm + OP * W::kOwn, reinterpret_cast<const T*>(p.d_o) + row_offset(p.sdo, p.H, own_head, 0), p.sdo.n, own0, N);
    }
    load(0, 0);
    float lse_r[2], dl_r[2];
    if (!KV) {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int pos = row0 + 8 * r;
            lse_r[r] = pos < N ? p.lse2[(size_t)own_head * N + pos] : INFINITY;   // P = 0 beyond the head
            dl_r[r] = pos < N ? p.delta[(size_t)own_head * N + pos] : 0.f;
        }
    }
    float acc[DT][4], dv[KV ? DT : 1][4];   // dQ~ / dK~ and dV
#pragma unroll
    for (int n = 0; n < DT; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
#pragma unroll
    for (int n = 0; n < (KV ? DT : 1); ++n) dv[n][0] = dv[n][1] = dv[n][2] = dv[n][3] = 0.f;
    const uint32_t a_addr = sm + warp * 16 * Pitch<D>::kBytes + lane_a<D>(lane);   // of the hi rows; the other parts and the plain rows follow

    for (int step = 0, buf = 0; step < total; ++step, buf ^= 1) {
        cp_wait_all();
        __syncthreads();   // the tile has landed for every thread, and every warp is done with the other buffer
        if (step + 1 < total) load(step + 1, buf ^ 1);
        const uint32_t st = stages + buf * W::kStage + group * SR * Pitch<D>::kBytes;
        const int r0 = first + (KV ? step % steps : step) * BS + group * SR;
        // no pair of the warp's owned and streamed rows is visible
        if (r0 >= N || (p.causal && (KV ? r0 + SR - 1 < own0 + warp * 16 : r0 > own0 + warp * 16 + 15))) continue;
        float s[NT][4], dp[NT][4], small[NT][4];
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int x = 0; x < 4; ++x) s[n][x] = dp[n][x] = small[n][x] = 0.f;
        const uint32_t b_addr = st + lane_b<D>(lane);
#pragma unroll
        for (int k = 0; k < KS; ++k) {
            uint32_t a[OP][4], ax[4], b[SP][2][4], bx[2][4];   // split and plain rows
#pragma unroll
            for (int y = 0; y < 2; ++y) ldm_x4(bx[y], b_addr + SP * W::kTile + y * 16 * Pitch<D>::kBytes + k * 32);
            ldm_x4(ax, a_addr + OP * W::kOwn + k * 32);
            {
                float t[4][4] = {};
                mma4<T>(t, ax, bx[0], bx[1]);
                add4(dp, t);
            }
#pragma unroll
            for (int x = 0; x < OP; ++x) ldm_x4(a[x], a_addr + x * W::kOwn + k * 32);
#pragma unroll
            for (int x = 0; x < SP; ++x)
#pragma unroll
                for (int y = 0; y < 2; ++y) ldm_x4(b[x][y], b_addr + x * W::kTile + y * 16 * Pitch<D>::kBytes + k * 32);
            mma4_split(s, small, a, b);
        }
        // P and dS = P (dP - delta), in place of S and dP
        const size_t head = KV ? (size_t)(kvh * G + step / steps) * N : 0;
        const bool edge = KV ? (p.causal && r0 < own0 + warp * 16 + 15) : (r0 + SR > N || (p.causal && r0 + SR - 1 > own0 + warp * 16));
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            float lse_c[2], dl_c[2];
            if (KV) {
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    const int pos = r0 + n * 8 + c2 + x;
                    lse_c[x] = pos < N ? p.lse2[head + pos] : INFINITY;
                    dl_c[x] = pos < N ? p.delta[head + pos] : 0.f;
                }
            }
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                float pv = exp2f(join(s[n][x], small[n][x]) - (KV ? lse_c[x & 1] : lse_r[x >> 1]));
                if (edge) {
                    const int own = row0 + (x >> 1) * 8, str = r0 + n * 8 + c2 + (x & 1);
                    const bool seen = KV ? (!p.causal || own <= str) : (str < N && (!p.causal || str <= own));
                    if (!seen) pv = 0.f;
                }
                dp[n][x] = pv * (dp[n][x] - (KV ? dl_c[x & 1] : dl_r[x >> 1]));
                s[n][x] = pv;
            }
        }
        const uint32_t t_addr = st + lane_bt<D>(lane);
#pragma unroll
        for (int t = 0; t < SR / 16; ++t) {
            uint32_t da[3][4], pa[3][4];
            split_a<__nv_bfloat16>(dp[2 * t], dp[2 * t + 1], 1.f, da);
            if (KV) split_a<T>(s[2 * t], s[2 * t + 1], kPScale<T>, pa);
#pragma unroll
            for (int d = 0; d < DT / 2; d += 2) {
                const uint32_t off = t * 16 * Pitch<D>::kBytes + d * 32;
                uint32_t b[SP][2][4];
#pragma unroll
                for (int x = 0; x < SP; ++x)
#pragma unroll
                    for (int y = 0; y < 2; ++y) ldm_x4_trans(b[x][y], t_addr + x * W::kTile + off + 32 * y);
                add_products_split(acc + 2 * d, da, b);
                if (KV) {
                    uint32_t bx0[4], bx1[4];
                    ldm_x4_trans(bx0, t_addr + SP * W::kTile + off);
                    ldm_x4_trans(bx1, t_addr + SP * W::kTile + off + 32);
                    add_products<T>(dv + (KV ? 2 * d : 0), pa, bx0, bx1);
                }
            }
        }
    }
    if constexpr (W::kGroups == 2) {   // the second group's sums to the first, in the layout of the accumulators: rows of D + 4 floats
        __syncthreads();               // every warp is done with the tiles
        float* sums = reinterpret_cast<float*>(smem) + (warp * 16 + g) * (D + 4) + c2;
        constexpr int kSecond = kRows * (D + 4);
        if (group == 1) {
#pragma unroll
            for (int n = 0; n < DT; ++n)
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    *reinterpret_cast<float2*>(sums + r * 8 * (D + 4) + n * 8) = make_float2(acc[n][2 * r], acc[n][2 * r + 1]);
                    if (KV) *reinterpret_cast<float2*>(sums + kSecond + r * 8 * (D + 4) + n * 8) = make_float2(dv[KV ? n : 0][2 * r], dv[KV ? n : 0][2 * r + 1]);
                }
        }
        __syncthreads();
        if (group == 1) return;
#pragma unroll
        for (int n = 0; n < DT; ++n)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const float2 x = *reinterpret_cast<const float2*>(sums + r * 8 * (D + 4) + n * 8);
                acc[n][2 * r] += x.x;
                acc[n][2 * r + 1] += x.y;
                if (KV) {
                    const float2 y = *reinterpret_cast<const float2*>(sums + kSecond + r * 8 * (D + 4) + n * 8);
                    dv[KV ? n : 0][2 * r] += y.x;
                    dv[KV ? n : 0][2 * r + 1] += y.y;
                }
            }
    }

    // gradients of the rotated rows turned back (both columns of a pair belong to the same lane); Q~ carries sm_scale * log2e, so
    // dK only takes the log2e off again
    const float scale = KV ? kLn2 : p.sm_scale;
    T* OUT = reinterpret_cast<T*>(KV ? p.dk : p.dq) + (KV ? row_offset(p.sdk, p.Hkv, own_head, 0) : row_offset(p.sdq, p.H, own_head, 0));
    const int64_t out_stride = KV ? p.sdk.n : p.sdq.n;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int pos = row0 + 8 * r;
        if (pos >= N) continue;
        uint32_t* out = reinterpret_cast<uint32_t*>(OUT + (int64_t)pos * out_stride + c2);
#pragma unroll
        for (int n = 0; n < DT / 2; ++n) {
            float c0 = 1.f, c1 = 1.f, s0 = 0.f, s1 = 0.f;
            if (p.cos != nullptr) {
                const float *c = p.cos + (int64_t)pos * p.table_stride + n * 8 + c2, *s = p.sin + (int64_t)pos * p.table_stride + n * 8 + c2;
                c0 = c[0], c1 = c[1], s0 = s[0], s1 = s[1];
            }
            const float a0 = acc[n][2 * r], a1 = acc[n][2 * r + 1], b0 = acc[n + DT / 2][2 * r], b1 = acc[n + DT / 2][2 * r + 1];
            out[n * 4] = pack2<T>((a0 * c0 + b0 * s0) * scale, (a1 * c1 + b1 * s1) * scale);
            out[n * 4 + D / 4] = pack2<T>((b0 * c0 - a0 * s0) * scale, (b1 * c1 - a1 * s1) * scale);
        }
        if (KV) {
            constexpr float kUnscale = 1.f / kPScale<T>;
            uint32_t* o2 = reinterpret_cast<uint32_t*>(reinterpret_cast<T*>(p.dv) + row_offset(p.sdv, p.Hkv, own_head, pos) + c2);
#pragma unroll
            for (int n = 0; n < DT; ++n) o2[n * 4] = pack2<T>(dv[KV ? n : 0][2 * r] * kUnscale, dv[KV ? n : 0][2 * r + 1] * kUnscale);
        }
    }
}

// ------------------------------------------------------------------------------------------------ launchers
template <typename T, int D>
int split_rows(const void* x, const Strides& st, int H, const RopeParams& p, float scale, SplitRows out, cudaStream_t s, int* counter = nullptr) {
    const size_t rows = (size_t)p.B * H * p.N;
    split_rotate_kernel<T, D><<<(unsigned)((rows * (D / 16) + 255) / 256), 256, 0, s>>>((const T*)x, row_addr(st, H, p.N), p.cos, p.sin, p.table_stride, scale,
                                                                                       out, rows, counter);
    count_launch();
    return (int)cudaGetLastError();
}
SplitRows take_rows(__nv_bfloat16*& ws, int B, int H, int N, int D) {
    const size_t n = (size_t)B * H * N * D;
    SplitRows r{ws, n};
    ws += 3 * n;
    return r;
}

template <typename T, int D, int KP>
int fwd(const RopeParams& p, void* ws, cudaStream_t s) {
    using F = Fwd<D, KP>;
    __nv_bfloat16* at = reinterpret_cast<__nv_bfloat16*>(ws);
    const SplitRows k = take_rows(at, p.B, p.Hkv, p.N, D);
    if (KP > 1)
        if (int e = split_rows<T, D>(p.k, p.sk, p.Hkv, p, 1.f, k, s)) return e;
    auto kern = rope_fwd_split_kernel<T, D, KP>;
    static std::atomic<uint64_t> smem_ok;
    if (int e = allow_smem(kern, F::kSmem, smem_ok)) return e;
    kern<<<rope_split_fwd_grid(p.B, p.H, p.N).blocks(), F::kThreads, F::kSmem, s>>>(p, k);
    count_launch();
    return (int)cudaGetLastError();
}
template <typename T, int D, int KP, bool KV>
int bwd_sweep(const RopeParams& p, const SplitRows& q, const SplitRows& k, cudaStream_t s) {
    using W = Bwd<D, KP, KV>;
    auto kern = rope_bwd_split_kernel<T, D, KP, KV>;
    static std::atomic<uint64_t> smem_ok;
    if (int e = allow_smem(kern, W::kSmem, smem_ok)) return e;
    kern<<<rope_split_bwd_grid(p.B, KV ? p.Hkv : p.H, p.N).blocks(), W::kThreads, W::kSmem, s>>>(p, q, k);
    count_launch();
    return (int)cudaGetLastError();
}
template <typename T, int D, int KP>
int bwd(const RopeParams& p, void* ws, cudaStream_t s) {
    __nv_bfloat16* at = reinterpret_cast<__nv_bfloat16*>(ws);
    const SplitRows k = take_rows(at, p.B, p.Hkv, p.N, D), q = take_rows(at, p.B, p.H, p.N, D);
    if (KP > 1)
        if (int e = split_rows<T, D>(p.k, p.sk, p.Hkv, p, 1.f, k, s)) return e;
    if (int e = split_rows<T, D>(p.q, p.sq, p.H, p, p.sm_scale * kLog2e, q, s)) return e;
    if (int e = bwd_sweep<T, D, KP, true>(p, q, k, s)) return e;
    return bwd_sweep<T, D, KP, false>(p, q, k, s);
}
template <typename T, int KP>
int run(bool backward, const RopeParams& p, void* ws, cudaStream_t s) {
    if (backward) return p.D == 64 ? bwd<T, 64, KP>(p, ws, s) : bwd<T, 128, KP>(p, ws, s);
    return p.D == 64 ? fwd<T, 64, KP>(p, ws, s) : fwd<T, 128, KP>(p, ws, s);
}
int run(bool backward, const RopeParams& p, void* ws, int dtype, cudaStream_t s) {
    if (dtype == COROPE_DTYPE_F16) return run<__half, 3>(backward, p, ws, s);
    return p.cos == nullptr ? run<__nv_bfloat16, 1>(backward, p, ws, s) : run<__nv_bfloat16, 3>(backward, p, ws, s);
}

}  // namespace

constexpr int kSplitRows = 64;   // rows per CTA, forward and backward
static_assert(Fwd<64, 3>::kRows == kSplitRows && Fwd<128, 3>::kRows == kSplitRows && Bwd<64, 3, true>::kRows == kSplitRows && Bwd<128, 3, true>::kRows == kSplitRows, "grids");
FlatGrid rope_split_fwd_grid(int B, int H, int N) { return {(unsigned)(B * H), ceil_div(N, kSplitRows)}; }
FlatGrid rope_split_bwd_grid(int B, int H, int N) { return {(unsigned)(B * H), ceil_div(N, kSplitRows)}; }

size_t rope_split_workspace_bytes(bool bwd, int B, int Hq, int Hkv, int N, int D) {
    return ((size_t)B * Hkv + (bwd ? (size_t)B * Hq : 0)) * N * D * 3 * sizeof(__nv_bfloat16);
}

int launch_split_rows(const void* x, const Strides& st, int H, const RopeParams& p, float scale, const SplitRows& out, int* counter, int dtype, cudaStream_t s) {
    if (dtype == COROPE_DTYPE_BF16)
        return p.D == 64 ? split_rows<__nv_bfloat16, 64>(x, st, H, p, scale, out, s, counter) : split_rows<__nv_bfloat16, 128>(x, st, H, p, scale, out, s, counter);
    return p.D == 64 ? split_rows<__half, 64>(x, st, H, p, scale, out, s, counter) : split_rows<__half, 128>(x, st, H, p, scale, out, s, counter);
}

// The forward on mma.sync where its short start counts more than its rate: one block of rows, and for bf16 keys without rotation, which it
// reads as they are, a few.  GPU time of it and of the tcgen05 kernel (pre-pass included): B1 H1 N50 D64 8.6 / 9.6 us, N50 D128 11.9 / 12.5,
// N129 D64 13.8 / 11.5, N129 D128 19.0 / 15.3; without rotation B1 H1 N129 D64 9.3 / 11.1, N200 D128 17.4 / 16.0, B4 H16 N300 D64 19.1 / 21.6,
// N500 D64 32.2 / 26.8, B2 H32 N200 D128 21.7 / 18.5.
bool short_forward(const RopeParams& p, int dtype) {
    if (p.cos == nullptr && dtype == COROPE_DTYPE_BF16) return p.N < (p.D == 64 ? 320 : 160);
    return p.N <= 64;
}
int launch_rope_fwd_split(const RopeParams& p, void* ws, int dtype, cudaStream_t s) {
    return short_forward(p, dtype) ? run(false, p, ws, dtype, s) : launch_rope_fwd_split_tc(p, ws, dtype, s);
}
int launch_rope_bwd_split(const RopeParams& p, void* ws, int dtype, cudaStream_t s) { return run(true, p, ws, dtype, s); }   // delta computed before

}  // namespace corope
