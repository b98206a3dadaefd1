// Fused-RoPE / plain attention in fp32 arithmetic on the CUDA cores: fp32 inputs (which must match the fp32 reference to 1e-4) where they do not
// run on split operands (rope_split_fp32: aligned rows of D = 64 from 256 rows on do), and the forward of every 16-bit shape the
// tensor-core kernels do not take (D = 32, strides that are no multiples of 16 bytes).  Any N, causal or full, D in {32, 64, 128}.
//
// Every product is a register-blocked tile product out of shared memory.  What bounds it is the rate at which shared memory fills
// registers, 128 bytes per clock and SM whatever is broadcast: a thread tile of m x n needs (m + n) / (m n) floats per FMA, so the
// 4 x 4 tiles of the 64-row CTA could use half of the FMA pipe, the 2 x 4 tiles of the 32-row CTA a third (ncu: 84 % of the
// shared-memory cycles in the backward).  B4 H8 N512 D64 fp32 causal: forward 119 -> 64 us, backward (seven products) 400 -> 196 us
// against one warp per 8 rows and 12 loads per 32 FMAs; B4 H8 N2048 D64 forward + backward 4.50 -> 3.15 ms.
//
// 256 threads = 16 x 16: thread (ty, tx) with 8 x 4 of them per warp, so that a 16-byte load of the row operand covers 8 and of
// the column operand 4 distinct rows.  Rows in shared memory are padded by 4 floats: consecutive rows start in consecutive
// 16-byte bank groups.
//
// Math: fused-rope/rope_attn_pytorch.py:108-155 (forward), :187-222 (backward); exp2-domain softmax and log2-domain LSE as
// fused-rope/fused_rope_attn.py:103-114, 316.
#include "common.cuh"

namespace corope {
namespace {

constexpr int kThreads = 256;

template <typename T>
__device__ __forceinline__ void load4(float (&x)[4], const T* p, bool vec) {
    if (vec) {
        if constexpr (sizeof(T) == 4) {
            const float4 v = *reinterpret_cast<const float4*>(p);
            x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
        } else {
            const uint2 v = *reinterpret_cast<const uint2*>(p);
            const float2 a = unpack2<T>(v.x), b = unpack2<T>(v.y);
            x[0] = a.x; x[1] = a.y; x[2] = b.x; x[3] = b.y;
        }
    } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) x[e] = Elem<T>::to_f32(p[e]);
    }
}

// ROWS rows [r0, r0 + ROWS) of X[N][D] to dst[ROWS][D + 4] as fp32, rotated (ROTATE and tables given) and scaled; rows >= N become
// 0.  In two parts: fetch() issues every global load, store() rotates and writes, so that a tile's loads can be in flight while
// the previous tile is worked on.
template <typename T, int D, int ROWS, bool ROTATE>
struct Tile {
    static constexpr int H2 = D / 2, kPerRow = H2 / 4, kItems = ROWS * kPerRow, kIter = (kItems + kThreads - 1) / kThreads;
    float x1[kIter][4], x2[kIter][4], c[ROTATE ? kIter : 1][4], s[ROTATE ? kIter : 1][4];

    __device__ __forceinline__ void fetch(const T* X, int64_t xs, int r0, int N, const float* cosT, const float* sinT, int64_t ts, bool vec, bool tvec) {
#pragma unroll
        for (int it = 0; it < kIter; ++it) {
            const int idx = threadIdx.x + it * kThreads, r = idx / kPerRow, d = (idx % kPerRow) * 4, pos = r0 + r;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                x1[it][e] = x2[it][e] = 0.f;
                if (ROTATE) c[it][e] = s[it][e] = 0.f;
            }
            if (pos < N && (kItems % kThreads == 0 || idx < kItems)) {
                load4<T>(x1[it], X + (int64_t)pos * xs + d, vec);
                load4<T>(x2[it], X + (int64_t)pos * xs + d + H2, vec);
                if (ROTATE && cosT != nullptr) {   // null tables: plain attention, no rotation
                    load4<float>(c[it], cosT + pos * ts + d, tvec);
                    load4<float>(s[it], sinT + pos * ts + d, tvec);
                }
            }
        }
    }
    __device__ __forceinline__ void store(float* dst, bool rotate, float scale) const {
#pragma unroll
        for (int it = 0; it < kIter; ++it) {
            const int idx = threadIdx.x + it * kThreads, r = idx / kPerRow, d = (idx % kPerRow) * 4;
            if (kItems % kThreads != 0 && idx >= kItems) break;
            float y1[4], y2[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                if (ROTATE && rotate) {
                    y1[e] = (x1[it][e] * c[it][e] - x2[it][e] * s[it][e]) * scale;
                    y2[e] = (x2[it][e] * c[it][e] + x1[it][e] * s[it][e]) * scale;
                } else {
                    y1[e] = x1[it][e] * scale;
                    y2[e] = x2[it][e] * scale;
                }
            }
            float* p = dst + r * (D + 4) + d;
            *reinterpret_cast<float4*>(p) = make_float4(y1[0], y1[1], y1[2], y1[3]);
            *reinterpret_cast<float4*>(p + H2) = make_float4(y2[0], y2[1], y2[2], y2[3]);
        }
    }
};

// acc[i][j] = sum_k A[row0 + 16 i][k] B[col0 + 16 j][k]: both operands with k contiguous, so the even and the odd k are the two lanes
// of packed multiply-adds (half the issue slots of scalar ones)
template <int MI, int NJ, int K>
__device__ __forceinline__ void dot_tile(float (&acc)[MI][NJ], const float* A, int lda, const float* B, int ldb, int row0, int col0) {
    const float* a = A + row0 * lda;
    const float* b = B + col0 * ldb;
    uint64_t s[MI][NJ];   // (even, odd) partial sums; all bits zero = (+0, +0)
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j) s[i][j] = 0;
#pragma unroll 4
    for (int k = 0; k < K; k += 4) {
        ulonglong2 av[MI], bv[NJ];
#pragma unroll
        for (int i = 0; i < MI; ++i) av[i] = *reinterpret_cast<const ulonglong2*>(a + i * 16 * lda + k);
#pragma unroll
        for (int j = 0; j < NJ; ++j) bv[j] = *reinterpret_cast<const ulonglong2*>(b + j * 16 * ldb + k);
#pragma unroll
        for (int i = 0; i < MI; ++i)
#pragma unroll
            for (int j = 0; j < NJ; ++j) s[i][j] = f2_fma(av[i].y, bv[j].y, f2_fma(av[i].x, bv[j].x, s[i][j]));
    }
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
            float lo, hi;
            f2_unpack(s[i][j], lo, hi);
            acc[i][j] = lo + hi;
        }
}

// The columns of a [.][D] tile that thread column tx of 16 owns: kVec consecutive ones, kNV times, 16 * kVec apart.
template <int D>
struct Cols {
    static constexpr int kVec = D >= 64 ? 4 : 2;
    static constexpr int kNV = D / (16 * kVec);
    static constexpr int kN = kVec * kNV;
    __device__ static __forceinline__ int col(int tx, int n) { return tx * kVec + (n / kVec) * 16 * kVec + n % kVec; }
    __device__ static __forceinline__ void load(float (&b)[kN], const float* row, int tx) {
#pragma unroll
        for (int v = 0; v < kNV; ++v) {
            if constexpr (kVec == 4) {
                const float4 x = *reinterpret_cast<const float4*>(row + tx * 4 + v * 64);
                b[4 * v] = x.x; b[4 * v + 1] = x.y; b[4 * v + 2] = x.z; b[4 * v + 3] = x.w;
            } else {
                const float2 x = *reinterpret_cast<const float2*>(row + tx * 2);
                b[0] = x.x; b[1] = x.y;
            }
        }
    }
};
// The same with rotation partners in one thread: thread column tx of D / 8 owns columns 4 tx .. 4 tx + 3 and those + D/2.
template <int D>
struct PairCols {
    static constexpr int kN = 8, kGroups = D / 8;
    __device__ static __forceinline__ void load(float (&b)[kN], const float* row, int tx) {
        const float4 x = *reinterpret_cast<const float4*>(row + tx * 4), y = *reinterpret_cast<const float4*>(row + tx * 4 + D / 2);
        b[0] = x.x; b[1] = x.y; b[2] = x.z; b[3] = x.w;
        b[4] = y.x; b[5] = y.y; b[6] = y.z; b[7] = y.w;
    }
};

// acc[i][n] += sum_k A[row0 + RS i][k] B[k][col n]: A with k contiguous, B with the columns contiguous
template <int MI, int RS, class C, int K>
__device__ __forceinline__ void row_tile(float (&acc)[MI][C::kN], const float* A, int lda, const float* B, int ldb, int row0, int tx) {
    const float* a = A + row0 * lda;
#pragma unroll 2
    for (int k = 0; k < K; k += 4) {
        float av[MI][4];
#pragma unroll
        for (int i = 0; i < MI; ++i) {
            const float4 v = *reinterpret_cast<const float4*>(a + i * RS * lda + k);
            av[i][0] = v.x; av[i][1] = v.y; av[i][2] = v.z; av[i][3] = v.w;
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            float b[C::kN];
            C::load(b, B + (k + e) * ldb, tx);
#pragma unroll
            for (int i = 0; i < MI; ++i)
#pragma unroll
                for (int n = 0; n < C::kN; ++n) acc[i][n] = fmaf(av[i][e], b[n], acc[i][n]);
        }
    }
}

struct Flags {
    bool q, k, v, o, d_o, tab;   // rows can be moved in vectors of four elements
};

// ------------------------------------------------------------------------------------------------
// forward: one CTA per BM query rows
// ------------------------------------------------------------------------------------------------
template <typename T, int D, int BM>
__global__ void __launch_bounds__(kThreads, 2) rope_fwd_fp32_kernel(RopeParams p, Flags f) {
    constexpr int BN = D == 128 ? 32 : 64, LDD = D + 4, LDS_ = BN + 4, MI = BM / 16, TPR = kThreads / BM, NS = BN / TPR;
    extern __shared__ __align__(16) float smem[];
    float* q_s = smem;               // [BM][D+4]  rotated * sm_scale * log2e
    float* k_s = q_s + BM * LDD;     // [BN][D+4]  rotated
    float* v_s = k_s + BN * LDD;     // [BN][D+4]
    float* s_s = v_s + BN * LDD;     // [BM][BN+4] scores, then P
    float* row_s = s_s + BM * LDS_;  // [BM] rescale factor of the row, at the end its sum

    // heads run fastest and the longest causal rows come first: dealt to the SMs in this order the CTAs balance
    const int N = p.N, heads = p.B * p.H, bh = blockIdx.x % heads;
    const int m0 = (gridDim.x / heads - 1 - blockIdx.x / heads) * BM;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ty = (warp >> 2) * 8 + (lane >> 2), tx = (warp & 3) * 4 + (lane & 3);
    const int kvh = bh / (p.H / p.Hkv);                 // the heads of a group are adjacent
    const T* Q = reinterpret_cast<const T*>(p.q) + row_offset(p.sq, p.H, bh, 0);
    const T* K = reinterpret_cast<const T*>(p.k) + row_offset(p.sk, p.Hkv, kvh, 0);
    const T* V = reinterpret_cast<const T*>(p.v) + row_offset(p.sv, p.Hkv, kvh, 0);
    T* O = reinterpret_cast<T*>(p.out_o) + row_offset(p.so, p.H, bh, 0);

    const bool rot = p.cos != nullptr;
    Tile<T, D, BN, true> kt;
    Tile<T, D, BN, false> vt;
    {
        Tile<T, D, BM, true> qt;
        qt.fetch(Q, p.sq.n, m0, N, p.cos, p.sin, p.table_stride, f.q, f.tab);
        kt.fetch(K, p.sk.n, 0, N, p.cos, p.sin, p.table_stride, f.k, f.tab);
        vt.fetch(V, p.sv.n, 0, N, nullptr, nullptr, 0, f.v, false);
        qt.store(q_s, rot, p.sm_scale * kLog2e);
    }
    const int srow = threadIdx.x / TPR, part = threadIdx.x % TPR;   // softmax: TPR neighbouring threads per row
    float m = -INFINITY, l = 0.f;
    float acc[MI][Cols<D>::kN];
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int n = 0; n < Cols<D>::kN; ++n) acc[i][n] = 0.f;

    const int n_end = p.causal ? min(N, m0 + BM) : N;
    for (int j0 = 0; j0 < n_end; j0 += BN) {
        __syncthreads();   // the previous tile has been used
        kt.store(k_s, rot, 1.f);
        vt.store(v_s, false, 1.f);
        __syncthreads();
        float s[MI][BN / 16];
        dot_tile<MI, BN / 16, D>(s, q_s, LDD, k_s, LDD, ty, tx);
#pragma unroll
        for (int i = 0; i < MI; ++i)
#pragma unroll
            for (int j = 0; j < BN / 16; ++j) s_s[(ty + 16 * i) * LDS_ + tx + 16 * j] = s[i][j];
        if (j0 + BN < n_end) {   // the next tile's loads fly during the softmax and the second product
            kt.fetch(K, p.sk.n, j0 + BN, N, p.cos, p.sin, p.table_stride, f.k, f.tab);
            vt.fetch(V, p.sv.n, j0 + BN, N, nullptr, nullptr, 0, f.v, false);
        }
        __syncthreads();
        {
            const int i = m0 + srow;
            const int last = min(p.causal ? i : N - 1, N - 1) - j0;   // last visible column of the tile
            float4* row = reinterpret_cast<float4*>(s_s + srow * LDS_);
            float x[NS], mx = m;
#pragma unroll
            for (int e = 0; e < NS / 4; ++e) {
                const float4 v = row[e * TPR + part];
                const int c = (e * TPR + part) * 4;
                x[4 * e] = c <= last ? v.x : -INFINITY;
                x[4 * e + 1] = c + 1 <= last ? v.y : -INFINITY;
                x[4 * e + 2] = c + 2 <= last ? v.z : -INFINITY;
                x[4 * e + 3] = c + 3 <= last ? v.w : -INFINITY;
#pragma unroll
                for (int y = 0; y < 4; ++y) mx = fmaxf(mx, x[4 * e + y]);
            }
#pragma unroll
            for (int off = 1; off < TPR; off <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
            const float ref = mx == -INFINITY ? 0.f : mx;   // a row that has seen no key yet
            const float alpha = exp2f(m - ref);
            float sum = 0.f;
#pragma unroll
            for (int e = 0; e < NS / 4; ++e) {
#pragma unroll
                for (int y = 0; y < 4; ++y) {
                    x[4 * e + y] = exp2f(x[4 * e + y] - ref);
                    sum += x[4 * e + y];
                }
                row[e * TPR + part] = make_float4(x[4 * e], x[4 * e + 1], x[4 * e + 2], x[4 * e + 3]);
            }
#pragma unroll
            for (int off = 1; off < TPR; off <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
            l = l * alpha + sum;
            m = mx;
            if (part == 0) row_s[srow] = alpha;
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < MI; ++i) {
            const float alpha = row_s[ty + 16 * i];
#pragma unroll
            for (int n = 0; n < Cols<D>::kN; ++n) acc[i][n] *= alpha;
        }
        row_tile<MI, 16, Cols<D>, BN>(acc, s_s, LDS_, v_s, LDD, ty, tx);
    }
    __syncthreads();
    if (part == 0) {
        row_s[srow] = l;
        if (m0 + srow < N) p.lse2[(size_t)bh * N + m0 + srow] = m + log2f(l);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < MI; ++i) {
        const int r = m0 + ty + 16 * i;
        if (r >= N) continue;
        const float sum = row_s[ty + 16 * i], inv = sum > 0.f ? 1.f / sum : 0.f;
        T* out = O + (int64_t)r * p.so.n;
#pragma unroll
        for (int v = 0; v < Cols<D>::kNV; ++v) {
            const int c = Cols<D>::col(tx, v * Cols<D>::kVec);
            if constexpr (sizeof(T) == 4 && Cols<D>::kVec == 4) {
                if (f.o) {
                    *reinterpret_cast<float4*>(out + c) = make_float4(acc[i][4 * v] * inv, acc[i][4 * v + 1] * inv, acc[i][4 * v + 2] * inv, acc[i][4 * v + 3] * inv);
                    continue;
                }
            }
#pragma unroll
            for (int e = 0; e < Cols<D>::kVec; ++e) out[c + e] = Elem<T>::from_f32(acc[i][v * Cols<D>::kVec + e] * inv);
        }
    }
}

// ------------------------------------------------------------------------------------------------
// backward, fp32 tensors.  Two kinds of CTA in one launch: dQ of 32 query rows (sweeping the keys) and dK, dV of 32 keys (sweeping
// the query rows of the group's heads).  The scores are formed twice (seven products against five), but every sum has one owner
// and one order: results are the same bits every time, which dQ summed across CTAs with reductions was not.
// ------------------------------------------------------------------------------------------------
constexpr int kBR = 32;   // rows a CTA owns
template <int D>
struct Bwd {
    static constexpr int kBS = D == 128 ? 32 : 64;   // rows streamed per step
    static constexpr int kLdd = D + 4;
    static constexpr size_t kSmem = sizeof(float) * (2 * kBR * kLdd + 2 * kBS * kLdd + 2 * kBS * (kBR + 4) + 2 * kBS);
    // the dQ CTA's P buffer is [kBR][kBS + 4], the other's are 2 x [kBS][kBR + 4]; the row statistics follow
    static_assert(kBR * (kBS + 4) <= 2 * kBS * (kBR + 4), "dS buffer");
};

template <int D>
__device__ void dq_block(const RopeParams& p, const Flags& f, float* smem, int bh, int m0) {
    constexpr int BM = kBR, BN = Bwd<D>::kBS, LDD = Bwd<D>::kLdd, LDP = BN + 4, MI = BM / 16, NJ = BN / 16;
    using P = PairCols<D>;
    constexpr int RG = kThreads / P::kGroups, MQ = BM >= RG ? BM / RG : 1, kWX = P::kGroups / 4;
    float* q_s = smem;                  // [BM][D+4] rotated * sm_scale * log2e
    float* do_s = q_s + BM * LDD;       // [BM][D+4]
    float* k_s = do_s + BM * LDD;       // [BN][D+4] rotated
    float* v_s = k_s + BN * LDD;        // [BN][D+4]
    float* ds_s = v_s + BN * LDD;       // [BM][BN+4]
    const int N = p.N, kvh = bh / (p.H / p.Hkv);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ty = (warp >> 2) * 8 + (lane >> 2), tx = (warp & 3) * 4 + (lane & 3);
    const int qy = (warp / kWX) * 8 + (lane >> 2), qx = (warp % kWX) * 4 + (lane & 3);   // thread grid of the dQ product
    const float* K = reinterpret_cast<const float*>(p.k) + row_offset(p.sk, p.Hkv, kvh, 0);
    const float* V = reinterpret_cast<const float*>(p.v) + row_offset(p.sv, p.Hkv, kvh, 0);
    const bool rot = p.cos != nullptr;
    Tile<float, D, BN, true> kt;
    Tile<float, D, BN, false> vt;
    auto fetch = [&](int j0) {
        kt.fetch(K, p.sk.n, j0, N, p.cos, p.sin, p.table_stride, f.k, f.tab);
        vt.fetch(V, p.sv.n, j0, N, nullptr, nullptr, 0, f.v, false);
    };
    {
        Tile<float, D, BM, true> qt;
        Tile<float, D, BM, false> dot;
        qt.fetch(reinterpret_cast<const float*>(p.q) + row_offset(p.sq, p.H, bh, 0), p.sq.n, m0, N, p.cos, p.sin, p.table_stride, f.q, f.tab);
        dot.fetch(reinterpret_cast<const float*>(p.d_o) + row_offset(p.sdo, p.H, bh, 0), p.sdo.n, m0, N, nullptr, nullptr, 0, f.d_o, false);
        fetch(0);
        qt.store(q_s, rot, p.sm_scale * kLog2e);
        dot.store(do_s, false, 1.f);
    }
    float lse[MI], dl[MI], dq[MQ][8];
#pragma unroll
    for (int i = 0; i < MI; ++i) {
        const int r = m0 + ty + 16 * i;
        lse[i] = r < N ? p.lse2[(size_t)bh * N + r] : INFINITY;   // P = 0 beyond the head
        dl[i] = r < N ? p.delta[(size_t)bh * N + r] : 0.f;
    }
#pragma unroll
    for (int i = 0; i < MQ; ++i)
#pragma unroll
        for (int n = 0; n < 8; ++n) dq[i][n] = 0.f;
    const int n_end = p.causal ? min(N, m0 + BM) : N;
    for (int j0 = 0; j0 < n_end; j0 += BN) {
        __syncthreads();   // the previous tile has been used
        kt.store(k_s, rot, 1.f);
        vt.store(v_s, false, 1.f);
        __syncthreads();
        float s[MI][NJ], dp[MI][NJ];
        dot_tile<MI, NJ, D>(s, q_s, LDD, k_s, LDD, ty, tx);
        dot_tile<MI, NJ, D>(dp, do_s, LDD, v_s, LDD, ty, tx);
#pragma unroll
        for (int i = 0; i < MI; ++i)
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
                const int c = j0 + tx + 16 * j;
                const bool ok = c < N && (!p.causal || c <= m0 + ty + 16 * i);
                const float pv = ok ? exp2f(s[i][j] - lse[i]) : 0.f;
                ds_s[(ty + 16 * i) * LDP + tx + 16 * j] = pv * (dp[i][j] - dl[i]);
            }
        if (j0 + BN < n_end) fetch(j0 + BN);
        __syncthreads();
        if (qy < BM) row_tile<MQ, RG, P, BN>(dq, ds_s, LDP, k_s, LDD, qy, qx);
    }
    float* DQ = reinterpret_cast<float*>(p.dq) + row_offset(p.sdq, p.H, bh, 0);
    if (qy < BM) {
#pragma unroll
        for (int i = 0; i < MQ; ++i) {
            const int pos = m0 + qy + RG * i;
            if (pos >= N) continue;
            float c[4] = {1.f, 1.f, 1.f, 1.f}, s[4] = {0.f, 0.f, 0.f, 0.f};
            if (rot) {
                load4<float>(c, p.cos + pos * p.table_stride + qx * 4, f.tab);
                load4<float>(s, p.sin + pos * p.table_stride + qx * 4, f.tab);
            }
            float* out = DQ + (int64_t)pos * p.sdq.n + qx * 4;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                out[e] = (dq[i][e] * c[e] + dq[i][4 + e] * s[e]) * p.sm_scale;
                out[e + D / 2] = (dq[i][4 + e] * c[e] - dq[i][e] * s[e]) * p.sm_scale;
            }
        }
    }
}

template <int D>
__device__ void dkdv_block(const RopeParams& p, const Flags& f, float* smem, int kvh, int n0) {
    constexpr int BK = kBR, BQ = Bwd<D>::kBS, LDD = Bwd<D>::kLdd, LDP = BK + 4, MI = BQ / 16, NJ = BK / 16, KK = BK / 16;   // KK keys per thread
    float* k_s = smem;                  // [BK][D+4] rotated
    float* v_s = k_s + BK * LDD;        // [BK][D+4]
    float* q_s = v_s + BK * LDD;        // [BQ][D+4] rotated * sm_scale * log2e
    float* do_s = q_s + BQ * LDD;       // [BQ][D+4]
    float* p_s = do_s + BQ * LDD;       // [BQ][BK+4]
    float* ds_s = p_s + BQ * LDP;       // [BQ][BK+4]
    float* lse_s = ds_s + BQ * LDP;     // [BQ]
    float* dl_s = lse_s + BQ;           // [BQ]
    const int N = p.N, G = p.H / p.Hkv;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ty = (warp >> 2) * 8 + (lane >> 2), tx = (warp & 3) * 4 + (lane & 3);
    const bool rot = p.cos != nullptr;
    const int i_first = p.causal ? n0 / BQ * BQ : 0;
    Tile<float, D, BQ, true> qt;
    Tile<float, D, BQ, false> dot;
    auto fetch = [&](int g, int i0) {
        qt.fetch(reinterpret_cast<const float*>(p.q) + row_offset(p.sq, p.H, kvh * G + g, 0), p.sq.n, i0, N, p.cos, p.sin, p.table_stride, f.q, f.tab);
        dot.fetch(reinterpret_cast<const float*>(p.d_o) + row_offset(p.sdo, p.H, kvh * G + g, 0), p.sdo.n, i0, N, nullptr, nullptr, 0, f.d_o, false);
    };
    {
        Tile<float, D, BK, true> kt;
        Tile<float, D, BK, false> vt;
        kt.fetch(reinterpret_cast<const float*>(p.k) + row_offset(p.sk, p.Hkv, kvh, 0), p.sk.n, n0, N, p.cos, p.sin, p.table_stride, f.k, f.tab);
        vt.fetch(reinterpret_cast<const float*>(p.v) + row_offset(p.sv, p.Hkv, kvh, 0), p.sv.n, n0, N, nullptr, nullptr, 0, f.v, false);
        fetch(0, i_first);
        kt.store(k_s, rot, 1.f);
        vt.store(v_s, false, 1.f);
    }
    float dk[KK][Cols<D>::kN], dv[KK][Cols<D>::kN];   // keys KK ty .. KK ty + KK - 1
#pragma unroll
    for (int i = 0; i < KK; ++i)
#pragma unroll
        for (int n = 0; n < Cols<D>::kN; ++n) dk[i][n] = dv[i][n] = 0.f;
    for (int g = 0; g < G; ++g) {
        const int bh = kvh * G + g;
        for (int i0 = i_first; i0 < N; i0 += BQ) {
            __syncthreads();   // the previous tile has been used
            qt.store(q_s, rot, p.sm_scale * kLog2e);
            dot.store(do_s, false, 1.f);
            if (threadIdx.x < BQ) {
                const int i = i0 + threadIdx.x;
                lse_s[threadIdx.x] = i < N ? p.lse2[(size_t)bh * N + i] : INFINITY;   // P = 0 beyond the head
                dl_s[threadIdx.x] = i < N ? p.delta[(size_t)bh * N + i] : 0.f;
            }
            __syncthreads();
            {
                float s[MI][NJ], dp[MI][NJ];
                dot_tile<MI, NJ, D>(s, q_s, LDD, k_s, LDD, ty, tx);
                dot_tile<MI, NJ, D>(dp, do_s, LDD, v_s, LDD, ty, tx);
#pragma unroll
                for (int i = 0; i < MI; ++i) {
                    const int r = ty + 16 * i;
                    const float lse = lse_s[r], dl = dl_s[r];
#pragma unroll
                    for (int j = 0; j < NJ; ++j) {
                        const int c = tx + 16 * j;
                        const bool ok = n0 + c < N && (!p.causal || n0 + c <= i0 + r);
                        const float pv = ok ? exp2f(s[i][j] - lse) : 0.f;
                        p_s[r * LDP + c] = pv;
                        ds_s[r * LDP + c] = pv * (dp[i][j] - dl);
                    }
                }
            }
            // the next tile's loads fly during the two products that follow
            if (i0 + BQ < N) fetch(g, i0 + BQ);
            else if (g + 1 < G) fetch(g + 1, i_first);
            __syncthreads();
            // dV += P^T dO, dK~ += dS^T Q~
#pragma unroll 2
            for (int r = 0; r < BQ; ++r) {
                const float2 pv = *reinterpret_cast<const float2*>(p_s + r * LDP + ty * KK), sv = *reinterpret_cast<const float2*>(ds_s + r * LDP + ty * KK);
                const float pa[KK] = {pv.x, pv.y}, sa[KK] = {sv.x, sv.y};
                float b[Cols<D>::kN], c[Cols<D>::kN];
                Cols<D>::load(b, do_s + r * LDD, tx);
                Cols<D>::load(c, q_s + r * LDD, tx);
#pragma unroll
                for (int i = 0; i < KK; ++i)
#pragma unroll
                    for (int n = 0; n < Cols<D>::kN; ++n) {
                        dv[i][n] = fmaf(pa[i], b[n], dv[i][n]);
                        dk[i][n] = fmaf(sa[i], c[n], dk[i][n]);
                    }
            }
        }
    }
    // dV straight from the registers; dK through shared memory, where the two columns of a pair meet (q_s carried sm_scale * log2e:
    // ln2 undoes the log2e)
    float* DK = reinterpret_cast<float*>(p.dk) + row_offset(p.sdk, p.Hkv, kvh, 0);
    float* DV = reinterpret_cast<float*>(p.dv) + row_offset(p.sdv, p.Hkv, kvh, 0);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < KK; ++i) {
        const int j = n0 + KK * ty + i;
#pragma unroll
        for (int n = 0; n < Cols<D>::kN; ++n) {
            const int c = Cols<D>::col(tx, n);
            k_s[(KK * ty + i) * LDD + c] = dk[i][n];
            if (j < N) DV[(int64_t)j * p.sdv.n + c] = dv[i][n];
        }
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < BK * (D / 2); idx += kThreads) {
        const int r = idx / (D / 2), d = idx % (D / 2), pos = n0 + r;
        if (pos >= N) break;
        const float c = rot ? p.cos[pos * p.table_stride + d] : 1.f, s = rot ? p.sin[pos * p.table_stride + d] : 0.f;
        const float a = k_s[r * LDD + d], b = k_s[r * LDD + d + D / 2];
        DK[(int64_t)pos * p.sdk.n + d] = (a * c + b * s) * kLn2;
        DK[(int64_t)pos * p.sdk.n + d + D / 2] = (b * c - a * s) * kLn2;
    }
}

// grid: heads run fastest; then the row blocks, the long ones first and the two kinds in turn
template <int D>
__global__ void __launch_bounds__(kThreads, 2) rope_bwd_fp32_kernel(RopeParams p, Flags f) {
    extern __shared__ __align__(16) float smem[];
    const int blocks = (p.N + kBR - 1) / kBR, G = p.H / p.Hkv, heads = p.B * p.Hkv;
    // outer index = block * (G + 1) + kind: kind 0 is dK / dV of the KV head, kinds 1 .. G are dQ of its G query heads
    const int kvh = blockIdx.x % heads, outer = blockIdx.x / heads, block = outer / (G + 1), kind = outer % (G + 1);
    if (kind == 0)
        dkdv_block<D>(p, f, smem, kvh, block * kBR);
    else
        dq_block<D>(p, f, smem, kvh * G + kind - 1, (blocks - 1 - block) * kBR);
}

// delta = rowsum(O * dO) (fused_rope_attn.py:324-337), one warp per row
__global__ void __launch_bounds__(kThreads) rope_delta_fp32_kernel(const float* __restrict__ o, const float* __restrict__ d_o, float* __restrict__ delta,
                                                                   size_t rows, int D, RowAddr ao, RowAddr ado) {
    const size_t row = (size_t)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (row >= rows) return;
    float s = 0.f;
    const float* orow = o + flat_row_offset(ao, row);
    const float* drow = d_o + flat_row_offset(ado, row);
    for (int d = lane; d < D; d += 32) s = fmaf(orow[d], drow[d], s);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if (lane == 0) delta[row] = s;
}

bool vec_rows(const void* ptr, const Strides& st, size_t elem) {
    return ((uintptr_t)ptr % (4 * elem)) == 0 && st.b % 4 == 0 && st.h % 4 == 0 && st.n % 4 == 0;
}
Flags flags_of(const RopeParams& p, size_t elem) {
    Flags f;
    f.q = vec_rows(p.q, p.sq, elem); f.k = vec_rows(p.k, p.sk, elem); f.v = vec_rows(p.v, p.sv, elem); f.o = vec_rows(p.out_o, p.so, elem);
    f.d_o = vec_rows(p.d_o, p.sdo, elem);
    f.tab = ((uintptr_t)p.cos % 16) == 0 && ((uintptr_t)p.sin % 16) == 0 && p.table_stride % 4 == 0;
    return f;
}

FlatGrid fwd_grid(int B, int H, int N, int BM) { return {(unsigned)(B * H), ceil_div(N, BM)}; }
// 64 rows per CTA load the shared memory least (8 FMAs per 16-byte load of the scores' 4 x 4 tiles against 5.3); below two such CTAs per
// SM, 32-row CTAs balance and hide latency better.  Forward with 32 / 64 rows, in 64-row CTAs per SM: 0.4 (B1 H8 N512 D64) 35 / 50 us,
// 1.7 (B1 H8 N2048 D64) 213 / 236, 1.7 (B4 H8 N512 D128) 113 / 130, 2.6 (B4 H16 N384 D128) 134 / 113, 3.5 (B8 H8 N512 D64) 116 / 87,
// 3.5 (B2 H8 N2048 D128) 810 / 586, 6.9 (B4 H8 N2048 D64) 786 / 560.
bool fwd_64_rows(int B, int H, int N) { return (int64_t)((N + 63) / 64) * B * H >= 2 * sm_count(); }

template <typename T, int D, int BM>
int launch_fwd(const RopeParams& p, cudaStream_t s) {
    constexpr int BN = D == 128 ? 32 : 64;
    constexpr size_t smem = sizeof(float) * (BM * (D + 4) + 2 * BN * (D + 4) + BM * (BN + 4) + BM);
    auto kern = rope_fwd_fp32_kernel<T, D, BM>;
    static std::atomic<uint64_t> smem_ok;
    if (int e = allow_smem(kern, smem, smem_ok)) return e;
    kern<<<fwd_grid(p.B, p.H, p.N, BM).blocks(), kThreads, smem, s>>>(p, flags_of(p, sizeof(T)));
    count_launch();
    return (int)cudaGetLastError();
}
template <typename T, int D>
int launch_fwd_rows(const RopeParams& p, cudaStream_t s) {
    return fwd_64_rows(p.B, p.H, p.N) ? launch_fwd<T, D, 64>(p, s) : launch_fwd<T, D, 32>(p, s);
}
template <int D>
int launch_bwd(const RopeParams& p, cudaStream_t s) {
    const size_t rows = (size_t)p.B * p.H * p.N;
    rope_delta_fp32_kernel<<<(unsigned)((rows + 7) / 8), kThreads, 0, s>>>((const float*)p.o, (const float*)p.d_o, p.delta, rows, p.D,
                                                                          row_addr(p.so, p.H, p.N), row_addr(p.sdo, p.H, p.N));
    count_launch();
    if (cudaError_t e = cudaGetLastError()) return (int)e;
    auto kern = rope_bwd_fp32_kernel<D>;
    static std::atomic<uint64_t> smem_ok;
    if (int e = allow_smem(kern, Bwd<D>::kSmem, smem_ok)) return e;
    kern<<<rope_fp32_bwd_grid(p.B, p.H, p.Hkv, p.N).blocks(), kThreads, Bwd<D>::kSmem, s>>>(p, flags_of(p, 4));
    count_launch();
    return (int)cudaGetLastError();
}
template <typename T>
int fwd_d(const RopeParams& p, cudaStream_t s) {
    switch (p.D) {
        case 32: return launch_fwd_rows<T, 32>(p, s);
        case 64: return launch_fwd_rows<T, 64>(p, s);
        case 128: return launch_fwd_rows<T, 128>(p, s);
        default: return COROPE_ERR_BAD_HEAD_DIM;
    }
}

}  // namespace

FlatGrid rope_fp32_fwd_grid(int B, int H, int N) { return fwd_grid(B, H, N, fwd_64_rows(B, H, N) ? 64 : 32); }
FlatGrid rope_fp32_bwd_grid(int B, int H, int Hkv, int N) { return {(unsigned)(B * Hkv), ceil_div(N, kBR) * (unsigned)(H / Hkv + 1)}; }

int launch_rope_fwd_general(const RopeParams& p, int dtype, cudaStream_t s) {
    switch (dtype) {
        case COROPE_DTYPE_F32: return fwd_d<float>(p, s);
        case COROPE_DTYPE_BF16: return fwd_d<__nv_bfloat16>(p, s);
        case COROPE_DTYPE_F16: return fwd_d<__half>(p, s);
        default: return COROPE_ERR_BAD_DTYPE;
    }
}

// delta and all gradients of fp32 tensors
int launch_rope_bwd_fp32(const RopeParams& p, cudaStream_t s) {
    switch (p.D) {
        case 32: return launch_bwd<32>(p, s);
        case 64: return launch_bwd<64>(p, s);
        case 128: return launch_bwd<128>(p, s);
        default: return COROPE_ERR_BAD_HEAD_DIM;
    }
}

}  // namespace corope
