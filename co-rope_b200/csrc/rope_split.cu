// Fused-RoPE / plain attention forward of short sequences, 16-bit tensors at lengths that are not whole 128-row tiles, D = 64 or 128:
// tensor-core products (mma.sync m16n8k16) of fp32 operands.  Every fp32 operand x enters the MMAs as hi + mid + lo (rope_split.cuh):
//     S  = Q~ K~^T        Q~, K~ rotated in fp32, both split into bf16      6 MMAs (without mid lo, lo mid, lo lo: about 2^-24)
//     O += P V            P split into the inputs' own type                 3 MMAs
// bf16 for everything that is not bounded, so that no magnitude of the inputs leaves the range.  P <= 1 of f16 tensors enters its
// products times 2^14: the three numbers then reach down to 2^-38 of the row's largest probability.  The adder of the MMAs does not round to
// nearest; the large products therefore go through one 16-wide step each (with the smaller ones in front for the sums over keys), which
// fp32 additions join.  Infinities in Q or K keep the scores they have in fp32; beyond that non-finite operands of 16-bit tensors give NaN
// here and in the other split-operand kernels, also where fp32 sums would have been infinite (0 times an infinity where a part of P is 0).
//
// Longer sequences and the backward run on tcgen05 MMAs (rope_split_fwd_sm100.cu, rope_split_bwd_sm100.cu); the line is at short_forward.
// What bounds this one: mma.sync, measured at 553 TFLOP/s with all operands in registers (B200, 8 warps per SM); with 8 warps per SM
// (D = 128: 255 registers; D = 64: 12 warps) the latency between a tile's ldmatrix, MMAs and softmax is not fully hidden.
//
// Math: fused-rope/rope_attn_pytorch.py:108-155; exp2-domain softmax and log2-domain LSE as fused-rope/fused_rope_attn.py:103-114, 316.
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
// byte offsets of a lane's ldmatrix row inside a tile.  B operand from a tile with k contiguous: (b0, b1) of columns 0-7, then of columns
// 8-15.  B operand from a tile with the columns contiguous (.trans): the same.
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
// the products of two split operands (three and PB parts) for four neighbouring accumulator tiles, b[part][two ldmatrix_x4 results]: hi hi
// into `d` by way of an fp32 addition, the others into `e`, smallest first
template <int PB>
__device__ __forceinline__ void mma4_split(float (*d)[4], float (*e)[4], const uint32_t (&a)[3][4], const uint32_t (&b)[PB][2][4]) {
    using B = __nv_bfloat16;
    float t[4][4] = {};
    if constexpr (PB > 1) mma4<B>(e, a[1], b[1][0], b[1][1]);
    if constexpr (PB > 2) mma4<B>(e, a[0], b[2][0], b[2][1]);
    mma4<B>(e, a[2], b[0][0], b[0][1]);
    mma4<B>(t, a[0], b[0][0], b[0][1]);
    if constexpr (PB > 1) mma4<B>(e, a[0], b[1][0], b[1][1]);
    mma4<B>(e, a[1], b[0][0], b[0][1]);
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
                    split3_any(a.x * scale, a.y * scale, w);
#pragma unroll
                    for (int part = 0; part < 3; ++part) qa[k][part][x] = w[part];
                    split3_any(b.x * scale, b.y * scale, w);
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

// ------------------------------------------------------------------------------------------------ launchers
template <typename T, int D, int KP>
int fwd(const RopeParams& p, void* ws, cudaStream_t s) {
    using F = Fwd<D, KP>;
    const SplitRows k = split_copies(p, ws, false, Elem<T>::kDtype).k;
    if (KP > 1)
        if (int e = launch_split_rows(p, SplitCopies{k, {}, {}, {}}, false, Elem<T>::kDtype, s)) return e;
    auto kern = rope_fwd_split_kernel<T, D, KP>;
    static std::atomic<uint64_t> smem_ok;
    if (int e = allow_smem(kern, F::kSmem, smem_ok)) return e;
    kern<<<rope_split_fwd_grid(p.B, p.H, p.N).blocks(), F::kThreads, F::kSmem, s>>>(p, k);
    count_launch();
    return (int)cudaGetLastError();
}
template <typename T, int KP>
int fwd(const RopeParams& p, void* ws, cudaStream_t s) {
    return p.D == 64 ? fwd<T, 64, KP>(p, ws, s) : fwd<T, 128, KP>(p, ws, s);
}

}  // namespace

constexpr int kSplitRows = 64;   // rows per CTA
static_assert(Fwd<64, 3>::kRows == kSplitRows && Fwd<128, 3>::kRows == kSplitRows, "grids");
FlatGrid rope_split_fwd_grid(int B, int H, int N) { return {(unsigned)(B * H), ceil_div(N, kSplitRows)}; }

// The forward on mma.sync where its short start counts more than its rate: one block of rows, and for bf16 keys without rotation, which it
// reads as they are, a few.  GPU time of it and of the tcgen05 kernel (pre-pass included): B1 H1 N50 D64 8.6 / 9.6 us, N50 D128 11.9 / 12.5,
// N129 D64 13.8 / 11.5, N129 D128 19.0 / 15.3; without rotation B1 H1 N129 D64 9.3 / 11.1, N200 D128 17.4 / 16.0, B4 H16 N300 D64 19.1 / 21.6,
// N500 D64 32.2 / 26.8, B2 H32 N200 D128 21.7 / 18.5.
bool short_forward(const RopeParams& p, int dtype) {
    if (p.cos == nullptr && dtype == COROPE_DTYPE_BF16) return p.N < (p.D == 64 ? 320 : 160);
    return p.N <= 64;
}
int launch_rope_fwd_split(const RopeParams& p, void* ws, int dtype, cudaStream_t s) {
    // 16-bit V is read by TMA there, by plain copies here
    if (dtype == COROPE_DTYPE_F32 || (!short_forward(p, dtype) && no_shared_heads(p.sv, p.B, p.Hkv))) return launch_rope_fwd_split_tc(p, ws, dtype, s);
    if (dtype == COROPE_DTYPE_F16) return fwd<__half, 3>(p, ws, s);
    return p.cos == nullptr ? fwd<__nv_bfloat16, 1>(p, ws, s) : fwd<__nv_bfloat16, 3>(p, ws, s);
}
}  // namespace corope
