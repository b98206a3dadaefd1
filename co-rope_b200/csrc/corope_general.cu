// Co-RoPE GQA attention, general kernels: exact per-(i, j, d) phases, fp32 arithmetic on the CUDA cores.
//
// Definition (corope-exp/corope_attn_gqa_pytorch.py:56-124), for one KV head and its G query heads, leader =
// first head of the group:
//     z_ik = sigmoid(s * qL_i . k_k)      a_ij = sum_{k<=j} z_ik      Delta_ij = a_ii - a_ij
//     S_hij = s * sum_d [ (q1 k1 + q2 k2) cos(Delta w_d) - (q2 k1 - q1 k2) sin(Delta w_d) ],  w_d = theta^(-2d/D)
// which is  S_hij = s * sum_d ( q1_hid K'1_ijd + q2_hid K'2_ijd )  with the head-independent rotated key
//     K'1 = k1 cos + k2 sin,   K'2 = k2 cos - k1 sin.
// cos/sin and K' are computed once per (i, j, d) and shared by the G heads of the group.
//
// Tiling: one CTA = 8 consecutive query rows of one (batch, KV head), one warp per row, all G heads of the
// group; K/V stream through shared memory in tiles of 32 keys; lane = key for the score phase, lane = head-dim
// column for the accumulation phase.  The forward sweeps key tiles downward from the diagonal, so
// Delta_ij = sum_{k=j+1..i} z_ik is a running suffix sum and no mileage pre-pass is needed; a_ii falls out at
// the end and is saved for the backward, which sweeps upward (its mileage gradient is a prefix sum in j).
//
// Backward (corope_attn_gqa_pytorch.py:182-298), with g = dS * s and dS = P (dP - delta):
//     dq1_h += g K'1, dq2_h += g K'2;   dk1_j += (sum_h g q1) cos - (sum_h g q2) sin,  dk2_j += (sum_h g q2) cos + (sum_h g q1) sin
//     gD_ij = - sum_h g_hij * sum_d w_d ( q1 (k1 sin - k2 cos) + q2 (k2 sin + k1 cos) )
//     gz_ik = sum_{j<k} gD_ij (k <= i),  graw = gz z (1 - z) s,  dqL_i += graw k,  dk_k += graw qL_i
// dK / dV partial sums of a CTA's 8 rows are combined in registers and added to fp32 global accumulators.
#include "common.cuh"

namespace corope {
namespace {

constexpr int kWarps = 8;      // query rows per CTA
constexpr int kTile = 32;      // keys per step
constexpr int kThreads = kWarps * 32;
constexpr int kPad = 4;        // row padding (floats) of the per-lane K / V tiles: rows stay 16-byte aligned and 16-byte loads of 8
                               // consecutive lanes fall into distinct bank groups

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
// inclusive prefix sum over lanes (lane 0 first)
__device__ __forceinline__ float warp_prefix_incl(float v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        float t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}
// inclusive suffix sum over lanes (lane 31 first)
__device__ __forceinline__ float warp_suffix_incl(float v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        float t = __shfl_down_sync(0xffffffffu, v, o);
        if (lane + o < 32) v += t;
    }
    return v;
}

template <bool ACCURATE>
__device__ __forceinline__ void sincos_phase(float x, float* s, float* c, bool direct) {
    if (ACCURATE) {
        sincosf(x, s, c);
    } else if (direct) {
        // phases up to a few thousand radians (N <= 8192): the hardware approximations alone; their internal range
        // reduction in fp32 costs ~1e-4 rad there, far inside the 16-bit tolerance
        __sincosf(x, s, c);
    } else {
        // 16-bit inputs: two-constant reduction to [-pi, pi] then the fast hardware approximations
        float kf = rintf(x * 0.15915494309189535f);
        float r = fmaf(kf, -6.28318548202514648f, x);
        r = fmaf(kf, 1.7484555e-7f, r);
        __sincosf(r, s, c);
    }
}

template <typename T, int D>
__device__ __forceinline__ void stage_plain(float* dst, int ld, const T* X, int64_t xs, int r0, int rows, int N) {   // xs: row stride of X
    for (int idx = threadIdx.x; idx < rows * D; idx += kThreads) {
        int r = idx / D, d = idx % D;
        int pos = r0 + r;
        dst[r * ld + d] = pos < N ? Elem<T>::to_f32(X[(int64_t)pos * xs + d]) : 0.f;
    }
}

// fp32 tensors: K and V tiles by asynchronous copies into two buffers, the next tile in flight behind the current one.  (Small grids
// put one CTA on an SM, which then waited for every tile's loads: B1 Hq8 Hkv2 N512 D64 forward + backward 287 -> 228 us, with P and
// the leader dot products off the shuffle and multiply-add chains.)  16-bit tensors need a conversion and are staged through
// registers; their grids are large.
template <typename T, int D>
struct Tiles {
    static constexpr bool kAsync = sizeof(T) == 4;
    static constexpr int kBufs = kAsync ? 2 : 1;
};
// kTile rows [r0, r0 + kTile) of X, rows at or beyond N as zeros (one commit group per call of the caller)
template <int D>
__device__ __forceinline__ void copy_tile(float* dst, int ld, const float* X, int64_t xs, int r0, int N, bool vec) {
    if (vec) {
#pragma unroll
        for (int it = 0; it < kTile * D / 4 / kThreads; ++it) {
            const int idx = threadIdx.x + it * kThreads, r = idx / (D / 4), d = idx % (D / 4) * 4;
            const bool have = r0 + r < N;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst + r * ld + d)), "l"(X + (int64_t)(have ? r0 + r : 0) * xs + d),
                         "r"(have ? 16 : 0)
                         : "memory");
        }
    } else {
        for (int idx = threadIdx.x; idx < kTile * D; idx += kThreads) {
            const int r = idx / D, d = idx % D;
            const bool have = r0 + r < N;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(dst + r * ld + d)), "l"(X + (int64_t)(have ? r0 + r : 0) * xs + d),
                         "r"(have ? 4 : 0)
                         : "memory");
        }
    }
}
__device__ __forceinline__ bool vec_rows(const float* X, int64_t xs) { return ((uintptr_t)X % 16) == 0 && xs % 4 == 0; }

// dot product of two rows of D floats in shared memory: four independent chains
template <int D>
__device__ __forceinline__ float row_dot(const float* x, const float* y) {
    float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (int d = 0; d < D; d += 4) {
        const float4 a = *reinterpret_cast<const float4*>(x + d);
        const float4 b = *reinterpret_cast<const float4*>(y + d);
        s[0] = fmaf(a.x, b.x, s[0]);
        s[1] = fmaf(a.y, b.y, s[1]);
        s[2] = fmaf(a.z, b.z, s[2]);
        s[3] = fmaf(a.w, b.w, s[3]);
    }
    return (s[0] + s[1]) + (s[2] + s[3]);
}

// G floats that every lane of the warp reads at one address
template <int G>
__device__ __forceinline__ void load_heads(float (&x)[G], const float* src) {
    if constexpr (G % 4 == 0) {
#pragma unroll
        for (int h = 0; h < G; h += 4) {
            const float4 v = *reinterpret_cast<const float4*>(src + h);
            x[h] = v.x; x[h + 1] = v.y; x[h + 2] = v.z; x[h + 3] = v.w;
        }
    } else {
#pragma unroll
        for (int h = 0; h < G; ++h) x[h] = src[h];
    }
}

// ------------------------------------------------------------------------------------------------
// forward
// ------------------------------------------------------------------------------------------------
template <typename T, int D, int G> constexpr size_t fwd_smem_bytes() {
    return sizeof(float) * ((size_t)G * kWarps * D + Tiles<T, D>::kBufs * (kTile * (D + kPad) + kTile * D) + D / 2 + kWarps * kTile * G);
}
template <typename T, int D, int G, bool ACCURATE>
__global__ void __launch_bounds__(kThreads) corope_fwd_general_kernel(GqaParams p) {
    constexpr int H2 = D / 2;
    constexpr int NC = D / 32;
    extern __shared__ __align__(16) float smem[];
    using L = Tiles<T, D>;
    float* q_s = smem;                                      // [G][8][D]
    float* k_b = q_s + G * kWarps * D;                      // kBufs x [32][D+4]
    float* v_b = k_b + L::kBufs * kTile * (D + kPad);       // kBufs x [32][D]
    float* xp = v_b + L::kBufs * kTile * D;                 // [8][32][G] P
    float* w_s = xp + kWarps * kTile * G;                   // [H2] inverse frequencies

    const int N = p.N;
    const int bg = blockIdx.y;                 // b * Hkv + g
    const int b = bg / p.Hkv, g = bg % p.Hkv;
    const int i0 = (gridDim.x - 1 - blockIdx.x) * kWarps;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int i = i0 + warp;
    const size_t q_head0 = ((size_t)b * p.Hq + (size_t)g * G);
    const T* K = reinterpret_cast<const T*>(p.k) + row_offset(p.sk, p.Hkv, bg, 0);
    const T* V = reinterpret_cast<const T*>(p.v) + row_offset(p.sv, p.Hkv, bg, 0);

    for (int h = 0; h < G; ++h)
        stage_plain<T, D>(q_s + h * kWarps * D, D, reinterpret_cast<const T*>(p.q) + row_offset(p.sq, p.Hq, (int)q_head0 + h, 0), p.sq.n, i0, kWarps, N);
    for (int d = threadIdx.x; d < H2; d += kThreads) w_s[d] = 1.0f / powf(p.theta, (float)(2 * d) / (float)D);

    float m[G], l[G], acc[G][NC];
#pragma unroll
    for (int h = 0; h < G; ++h) {
        m[h] = -INFINITY;
        l[h] = 0.f;
#pragma unroll
        for (int c = 0; c < NC; ++c) acc[h][c] = 0.f;
    }
    float carry = 0.f;  // sum of z_ik over keys already swept (k > current tile), for this warp's row
    const float sc2 = p.sm_scale * kLog2e;
    const bool direct = p.N <= 8192;
    const int i_last = min(N - 1, i0 + kWarps - 1);
    const int j_first = (i_last / kTile) * kTile;
    bool k_vec = false, v_vec = false;
    if constexpr (L::kAsync) {
        k_vec = vec_rows(K, p.sk.n), v_vec = vec_rows(V, p.sv.n);
        copy_tile<D>(k_b, D + kPad, K, p.sk.n, j_first, N, k_vec);
        copy_tile<D>(v_b, D, V, p.sv.n, j_first, N, v_vec);
    }
    int buf = 0;
    for (int j0 = j_first; j0 >= 0; j0 -= kTile, buf ^= L::kBufs - 1) {
        float *k_s = k_b + buf * kTile * (D + kPad), *v_s = v_b + buf * kTile * D;
        if constexpr (L::kAsync) {
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();   // the tile has landed for every thread, and every warp is done with the other buffer
            if (j0 >= kTile) {
                copy_tile<D>(k_b + (buf ^ 1) * kTile * (D + kPad), D + kPad, K, p.sk.n, j0 - kTile, N, k_vec);
                copy_tile<D>(v_b + (buf ^ 1) * kTile * D, D, V, p.sv.n, j0 - kTile, N, v_vec);
            }
        } else {
            __syncthreads();
            stage_plain<T, D>(k_s, D + kPad, K, p.sk.n, j0, kTile, N);
            stage_plain<T, D>(v_s, D, V, p.sv.n, j0, kTile, N);
            __syncthreads();
        }
        if (i >= N) continue;
        const int j = j0 + lane;
        const bool vis = (j <= i);  // implies j < N
        const float* kr = k_s + lane * (D + kPad);
        const float* qL = q_s + warp * D;
        // leader score -> z   (16-byte shared-memory loads throughout: the loop is load-issue bound otherwise)
        const float dot = row_dot<D>(qL, kr);
        float z = vis ? 1.f / (1.f + __expf(-dot * p.sm_scale)) : 0.f;
        // Delta_ij = sum_{k=j+1..i} z_ik = carry + (suffix over lanes above this one)
        float suf = warp_suffix_incl(z, lane);
        float delta = carry + suf - z;
        carry += __shfl_sync(0xffffffffu, suf, 0);
        // scores of the G heads
        float s[G];
#pragma unroll
        for (int h = 0; h < G; ++h) s[h] = 0.f;
#pragma unroll 1
        for (int d = 0; d < H2; d += 4) {
            const float4 w4 = *reinterpret_cast<const float4*>(w_s + d);
            const float4 k1v = *reinterpret_cast<const float4*>(kr + d);
            const float4 k2v = *reinterpret_cast<const float4*>(kr + d + H2);
            const float wv[4] = {w4.x, w4.y, w4.z, w4.w};
            const float k1a[4] = {k1v.x, k1v.y, k1v.z, k1v.w}, k2a[4] = {k2v.x, k2v.y, k2v.z, k2v.w};
            float r1[4], r2[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                float sn, cs;
                sincos_phase<ACCURATE>(delta * wv[e], &sn, &cs, direct);
                r1[e] = fmaf(k1a[e], cs, k2a[e] * sn);
                r2[e] = fmaf(k2a[e], cs, -k1a[e] * sn);
            }
#pragma unroll
            for (int h = 0; h < G; ++h) {
                const float* qh = q_s + (h * kWarps + warp) * D;
                const float4 q1v = *reinterpret_cast<const float4*>(qh + d);
                const float4 q2v = *reinterpret_cast<const float4*>(qh + d + H2);
                float acc = s[h];
                acc = fmaf(q1v.x, r1[0], acc); acc = fmaf(q2v.x, r2[0], acc);
                acc = fmaf(q1v.y, r1[1], acc); acc = fmaf(q2v.y, r2[1], acc);
                acc = fmaf(q1v.z, r1[2], acc); acc = fmaf(q2v.z, r2[2], acc);
                acc = fmaf(q1v.w, r1[3], acc); acc = fmaf(q2v.w, r2[3], acc);
                s[h] = acc;
            }
        }
        // online softmax per head (log2 domain), then P V with lane = column
#pragma unroll
        for (int h = 0; h < G; ++h) {
            float sv = vis ? s[h] * sc2 : -INFINITY;
            float mx = fmaxf(m[h], warp_max(sv));
            float alpha = exp2f(m[h] - mx);   // first tile holds the diagonal, so mx is finite
            float pv = vis ? exp2f(sv - mx) : 0.f;
            l[h] = l[h] * alpha + pv;         // this lane's keys only, added up at the end
            m[h] = mx;
#pragma unroll
            for (int c = 0; c < NC; ++c) acc[h][c] *= alpha;
            xp[(warp * kTile + lane) * G + h] = pv;
        }
        __syncwarp();
#pragma unroll 4
        for (int jj = 0; jj < kTile; ++jj) {
            float vv[NC];
#pragma unroll
            for (int c = 0; c < NC; ++c) vv[c] = v_s[jj * D + lane + 32 * c];
            float pj[G];
            load_heads<G>(pj, xp + (warp * kTile + jj) * G);
#pragma unroll
            for (int h = 0; h < G; ++h)
#pragma unroll
                for (int c = 0; c < NC; ++c) acc[h][c] = fmaf(pj[h], vv[c], acc[h][c]);
        }
        __syncwarp();   // every lane has read P before the next tile's overwrites it
    }
    if (i < N) {
#pragma unroll
        for (int h = 0; h < G; ++h) {
            T* O = reinterpret_cast<T*>(p.out_o) + row_offset(p.so, p.Hq, (int)q_head0 + h, i);
            l[h] = warp_sum(l[h]);
            float inv = 1.f / l[h];
#pragma unroll
            for (int c = 0; c < NC; ++c) O[lane + 32 * c] = Elem<T>::from_f32(acc[h][c] * inv);
            if (lane == 0) p.lse2[(q_head0 + h) * N + i] = m[h] + log2f(l[h]);
        }
        if (lane == 0) p.a_diag[(size_t)bg * N + i] = carry;
    }
}

// ------------------------------------------------------------------------------------------------
// backward
// ------------------------------------------------------------------------------------------------
template <typename T>
__global__ void gqa_delta_kernel(const T* __restrict__ o, const T* __restrict__ d_o, float* __restrict__ delta, size_t rows, int D, RowAddr ao,
                                 RowAddr ado) {
    size_t row = (size_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    int lane = threadIdx.x & 31;
    if (row >= rows) return;
    float s = 0.f;
    const T* orow = o + flat_row_offset(ao, row);
    const T* drow = d_o + flat_row_offset(ado, row);
    for (int d = lane; d < D; d += 32) s += Elem<T>::to_f32(orow[d]) * Elem<T>::to_f32(drow[d]);
    s = warp_sum(s);
    if (lane == 0) delta[row] = s;
}

// fp32 accumulators [rows, D] of dK (y = 0) and dV (y = 1) to the outputs' type and layout
template <typename T>
__global__ void gqa_finalize_kernel(const float* __restrict__ dk_acc, const float* __restrict__ dv_acc, T* __restrict__ dk, T* __restrict__ dv, size_t n,
                                    int D, RowAddr adk, RowAddr adv) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const size_t row = i / (size_t)D;
    const int d = (int)(i % (size_t)D);
    if (blockIdx.y == 0)
        dk[flat_row_offset(adk, row) + d] = Elem<T>::from_f32(dk_acc[i]);
    else
        dv[flat_row_offset(adv, row) + d] = Elem<T>::from_f32(dv_acc[i]);
}

// Shared memory of the backward (floats).  The (cos, sin) of every (row, key, pair) of a tile are kept from the score phase for the
// two gradient phases where they fit and are worth it: sincosf costs some 40 instructions, the hardware approximations two.  Kept /
// formed again: fp32 B1 Hq8 Hkv2 N512 D64 152 / 200 us, D128 288 / 349, B1 Hq4 Hkv4 N600 D128 335 / 490; 16 bits B2 Hq16 Hkv4 N2048 D64
// 2.89 / 3.02 ms, B1 Hq32 Hkv8 N1500 D128 3.78 / 3.29 ms (the table leaves room for one CTA per SM there, where two fit without).
template <typename T, int D, int G, bool ACCURATE> struct BwdSmem {
    static constexpr int kPitch = D + 2;                          // floats per (row, key) of the (cos, sin) table: lane = key writes 8 bytes without conflicts
    static constexpr size_t kTile2 = 2 * kTile * (D + kPad);      // one tile of K and of V
    static constexpr size_t kBase = (size_t)2 * G * kWarps * D + kTile2 + D / 2 + (size_t)kWarps * kTile * (2 * G + 2);
    static constexpr size_t kTable = (size_t)kWarps * kTile * kPitch, kMost = 225 * 1024 / sizeof(float);
    static constexpr bool kStore = (ACCURATE || D <= 64) && kBase + kTable <= kMost;
    // the second buffer of fp32 tiles where the table leaves room for it
    static constexpr bool kAsync = Tiles<T, D>::kAsync && kBase + kTile2 + (kStore ? kTable : 0) <= kMost;
    static constexpr int kBufs = kAsync ? 2 : 1;
    static constexpr size_t kBytes = (kBase + (kAsync ? kTile2 : 0) + (kStore ? kTable : 0)) * sizeof(float);
};

// Three phases per tile of 32 keys.  A: warp = row, lane = key: scores, P, dS, mileage gradient.  B1: warp = row, lane = pair: dq.
// B2: warp = 4 keys, lane = pair / column: dk and dv summed over the CTA's 8 rows in registers, one global reduction per tile.
// (With one phase for dq, dk and dv the rows met in shared-memory atomics, fp32 compare-and-swap loops that all 8 warps aimed at the
// same key: backward of B1 Hq8 Hkv2 N512 D64 fp32 341 against 181 us now, B1 Hq32 Hkv8 N1500 D128 bf16 5.64 against 3.30 ms.)  Bound by
// issue slots and, at small grids, the latency of one CTA's chain of tiles.
template <typename T, int D, int G, bool ACCURATE>
__global__ void __launch_bounds__(kThreads) corope_bwd_general_kernel(GqaParams p) {
    using M = BwdSmem<T, D, G, ACCURATE>;
    constexpr int H2 = D / 2;
    constexpr int NC = D / 32;                    // head-dim columns per lane
    constexpr int NPI = (H2 + 31) / 32;           // (d, d + D/2) pairs per lane
    constexpr int kKeys = kTile / kWarps;         // keys per warp in phase B2
    extern __shared__ __align__(16) float smem[];
    float* q_s = smem;                            // [G][8][D]
    float* do_s = q_s + G * kWarps * D;           // [G][8][D]
    float* k_b = do_s + G * kWarps * D;           // kBufs x [32][D+4]
    float* v_b = k_b + M::kBufs * kTile * (D + kPad);   // kBufs x [32][D+4]
    float* xg = v_b + M::kBufs * kTile * (D + kPad);    // [8][32][G] dS * sm_scale
    float* xp = xg + kWarps * kTile * G;          // [8][32][G] P
    float* xd = xp + kWarps * kTile * G;          // [8][32] Delta
    float* xr = xd + kWarps * kTile;              // [8][32] graw
    float* w_s = xr + kWarps * kTile;             // [H2]
    float* cs_s = w_s + H2;                       // [8][32][D+2] (cos, sin) pairs

    const int N = p.N;
    const int bg = blockIdx.y;
    const int b = bg / p.Hkv, g = bg % p.Hkv;
    const int i0 = (gridDim.x - 1 - blockIdx.x) * kWarps;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int i = i0 + warp;
    const size_t q_head0 = ((size_t)b * p.Hq + (size_t)g * G);
    const T* K = reinterpret_cast<const T*>(p.k) + row_offset(p.sk, p.Hkv, bg, 0);
    const T* V = reinterpret_cast<const T*>(p.v) + row_offset(p.sv, p.Hkv, bg, 0);
    float* dk_acc = p.dk_acc + (size_t)bg * N * D;
    float* dv_acc = p.dv_acc + (size_t)bg * N * D;

    for (int h = 0; h < G; ++h) {
        stage_plain<T, D>(q_s + h * kWarps * D, D, reinterpret_cast<const T*>(p.q) + row_offset(p.sq, p.Hq, (int)q_head0 + h, 0), p.sq.n, i0, kWarps, N);
        stage_plain<T, D>(do_s + h * kWarps * D, D, reinterpret_cast<const T*>(p.d_o) + row_offset(p.sdo, p.Hq, (int)q_head0 + h, 0), p.sdo.n, i0, kWarps, N);
    }
    for (int d = threadIdx.x; d < H2; d += kThreads) w_s[d] = 1.0f / powf(p.theta, (float)(2 * d) / (float)D);

    float lse[G], dl[G], dq1[G][NPI], dq2[G][NPI];
#pragma unroll
    for (int h = 0; h < G; ++h) {
        lse[h] = i < N ? p.lse2[(q_head0 + h) * N + i] : 0.f;
        dl[h] = i < N ? p.delta[(q_head0 + h) * N + i] : 0.f;
#pragma unroll
        for (int pi = 0; pi < NPI; ++pi) dq1[h][pi] = dq2[h][pi] = 0.f;
    }
    const float a_ii = i < N ? p.a_diag[(size_t)bg * N + i] : 0.f;
    float carry_a = 0.f, carry_g = 0.f;
    const float sc2 = p.sm_scale * kLog2e;
    const bool direct = p.N <= 8192;
    const int i_last = min(N - 1, i0 + kWarps - 1);
    // (cos, sin) of row r, key jj, pair pd of the tile
    auto phase = [&](int r, int jj, int pd, float* sn, float* cs) {
        if (M::kStore) {
            const float2 x = *reinterpret_cast<const float2*>(cs_s + (r * kTile + jj) * M::kPitch + 2 * pd);
            *cs = x.x;
            *sn = x.y;
        } else {
            sincos_phase<ACCURATE>(xd[r * kTile + jj] * w_s[pd], sn, cs, direct);
        }
    };
    bool k_vec = false, v_vec = false;
    if constexpr (M::kAsync) {
        k_vec = vec_rows(K, p.sk.n), v_vec = vec_rows(V, p.sv.n);
        copy_tile<D>(k_b, D + kPad, K, p.sk.n, 0, N, k_vec);
        copy_tile<D>(v_b, D + kPad, V, p.sv.n, 0, N, v_vec);
    }
    int buf = 0;
    for (int j0 = 0; j0 <= i_last; j0 += kTile, buf ^= M::kBufs - 1) {
        float *k_s = k_b + buf * kTile * (D + kPad), *v_s = v_b + buf * kTile * (D + kPad);
        if constexpr (M::kAsync) {
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();   // the tile has landed for every thread, and the previous one has been used
            if (j0 + kTile <= i_last) {
                copy_tile<D>(k_b + (buf ^ 1) * kTile * (D + kPad), D + kPad, K, p.sk.n, j0 + kTile, N, k_vec);
                copy_tile<D>(v_b + (buf ^ 1) * kTile * (D + kPad), D + kPad, V, p.sv.n, j0 + kTile, N, v_vec);
            }
        } else {
            __syncthreads();   // the previous tile has been used
            stage_plain<T, D>(k_s, D + kPad, K, p.sk.n, j0, kTile, N);
            stage_plain<T, D>(v_s, D + kPad, V, p.sv.n, j0, kTile, N);
            __syncthreads();
        }
        if (i < N && j0 <= i) {
            // ---------------- phase A: lane = key
            const int j = j0 + lane;
            const bool vis = (j <= i);
            const float* kr = k_s + lane * (D + kPad);
            const float* vr = v_s + lane * (D + kPad);
            const float* qL = q_s + warp * D;
            float* cs_out = cs_s + (warp * kTile + lane) * M::kPitch;
            const float dot = row_dot<D>(qL, kr);
            const float z = vis ? 1.f / (1.f + __expf(-dot * p.sm_scale)) : 0.f;
            const float pre = warp_prefix_incl(z, lane);
            const float delta = a_ii - (carry_a + pre);
            carry_a += __shfl_sync(0xffffffffu, pre, 31);
            float s[G], tq[G], dp[G];
#pragma unroll
            for (int h = 0; h < G; ++h) s[h] = tq[h] = dp[h] = 0.f;
#pragma unroll 1
            for (int d = 0; d < H2; d += 4) {
                const float4 w4 = *reinterpret_cast<const float4*>(w_s + d);
                const float4 k1v = *reinterpret_cast<const float4*>(kr + d);
                const float4 k2v = *reinterpret_cast<const float4*>(kr + d + H2);
                const float wv[4] = {w4.x, w4.y, w4.z, w4.w};
                const float k1a[4] = {k1v.x, k1v.y, k1v.z, k1v.w}, k2a[4] = {k2v.x, k2v.y, k2v.z, k2v.w};
                float r1[4], r2[4], wr1[4], wr2[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    float sn, cs;
                    sincos_phase<ACCURATE>(delta * wv[e], &sn, &cs, direct);
                    if (M::kStore) *reinterpret_cast<float2*>(cs_out + 2 * (d + e)) = make_float2(cs, sn);
                    r1[e] = fmaf(k1a[e], cs, k2a[e] * sn);
                    r2[e] = fmaf(k2a[e], cs, -k1a[e] * sn);
                    wr1[e] = wv[e] * r1[e];
                    wr2[e] = wv[e] * r2[e];
                }
#pragma unroll
                for (int h = 0; h < G; ++h) {
                    const float* qh = q_s + (h * kWarps + warp) * D;
                    const float4 q1v = *reinterpret_cast<const float4*>(qh + d);
                    const float4 q2v = *reinterpret_cast<const float4*>(qh + d + H2);
                    const float q1a[4] = {q1v.x, q1v.y, q1v.z, q1v.w}, q2a[4] = {q2v.x, q2v.y, q2v.z, q2v.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        s[h] = fmaf(q1a[e], r1[e], s[h]);
                        s[h] = fmaf(q2a[e], r2[e], s[h]);
                        tq[h] = fmaf(q2a[e], wr1[e], tq[h]);
                        tq[h] = fmaf(-q1a[e], wr2[e], tq[h]);
                    }
                }
            }
#pragma unroll 2
            for (int d = 0; d < D; d += 4) {
                const float4 vv = *reinterpret_cast<const float4*>(vr + d);
#pragma unroll
                for (int h = 0; h < G; ++h) {
                    const float4 g4 = *reinterpret_cast<const float4*>(do_s + (h * kWarps + warp) * D + d);
                    dp[h] = fmaf(g4.x, vv.x, dp[h]);
                    dp[h] = fmaf(g4.y, vv.y, dp[h]);
                    dp[h] = fmaf(g4.z, vv.z, dp[h]);
                    dp[h] = fmaf(g4.w, vv.w, dp[h]);
                }
            }
            float gD = 0.f;
            const int at = warp * kTile + lane;
#pragma unroll
            for (int h = 0; h < G; ++h) {
                float pv = vis ? exp2f(s[h] * sc2 - lse[h]) : 0.f;
                float gT = pv * (dp[h] - dl[h]) * p.sm_scale;
                gD = fmaf(-gT, tq[h], gD);
                xg[at * G + h] = gT;
                xp[at * G + h] = pv;
            }
            const float gpre = warp_prefix_incl(gD, lane);
            const float gz = carry_g + gpre - gD;
            carry_g += __shfl_sync(0xffffffffu, gpre, 31);
            xd[at] = delta;
            xr[at] = vis ? gz * z * (1.f - z) * p.sm_scale : 0.f;
            __syncwarp();
            // ---------------- phase B1: lane = head-dim pair, the warp's own row
            const int jj_end = min(kTile, i - j0 + 1);
#pragma unroll 2
            for (int jj = 0; jj < jj_end; ++jj) {
                float gT[G];
                load_heads<G>(gT, xg + (warp * kTile + jj) * G);
                const float graw = xr[warp * kTile + jj];
#pragma unroll
                for (int pi = 0; pi < NPI; ++pi) {
                    const int pd = lane + 32 * pi;
                    if (pd < H2) {
                        float sn, cs;
                        phase(warp, jj, pd, &sn, &cs);
                        const float k1 = k_s[jj * (D + kPad) + pd], k2 = k_s[jj * (D + kPad) + pd + H2];
                        const float r1 = fmaf(k1, cs, k2 * sn);
                        const float r2 = fmaf(k2, cs, -k1 * sn);
#pragma unroll
                        for (int h = 0; h < G; ++h) {
                            dq1[h][pi] = fmaf(gT[h], r1, dq1[h][pi]);
                            dq2[h][pi] = fmaf(gT[h], r2, dq2[h][pi]);
                        }
                        dq1[0][pi] = fmaf(graw, k1, dq1[0][pi]);
                        dq2[0][pi] = fmaf(graw, k2, dq2[0][pi]);
                    }
                }
            }
        }
        __syncthreads();
        // ---------------- phase B2: keys kKeys * warp .. of the tile, all rows that reach it
        float dk1[kKeys][NPI], dk2[kKeys][NPI], dv[kKeys][NC];
#pragma unroll
        for (int kk = 0; kk < kKeys; ++kk) {
#pragma unroll
            for (int pi = 0; pi < NPI; ++pi) dk1[kk][pi] = dk2[kk][pi] = 0.f;
#pragma unroll
            for (int c = 0; c < NC; ++c) dv[kk][c] = 0.f;
        }
        const int key0 = j0 + kKeys * warp;
#pragma unroll 1
        for (int r = max(0, key0 - i0); r <= i_last - i0; ++r) {   // rows before the warp's first key do not see any of its keys
            float x[kKeys][G];
#pragma unroll
            for (int kk = 0; kk < kKeys; ++kk) load_heads<G>(x[kk], xg + (r * kTile + kKeys * warp + kk) * G);
#pragma unroll
            for (int pi = 0; pi < NPI; ++pi) {
                const int pd = lane + 32 * pi;
                if (pd < H2) {
                    float a1[kKeys], a2[kKeys];
#pragma unroll
                    for (int kk = 0; kk < kKeys; ++kk) a1[kk] = a2[kk] = 0.f;
#pragma unroll
                    for (int h = 0; h < G; ++h) {
                        const float q1 = q_s[(h * kWarps + r) * D + pd], q2 = q_s[(h * kWarps + r) * D + pd + H2];
#pragma unroll
                        for (int kk = 0; kk < kKeys; ++kk) {
                            a1[kk] = fmaf(x[kk][h], q1, a1[kk]);
                            a2[kk] = fmaf(x[kk][h], q2, a2[kk]);
                        }
                    }
                    const float qL1 = q_s[r * D + pd], qL2 = q_s[r * D + pd + H2];
#pragma unroll
                    for (int kk = 0; kk < kKeys; ++kk) {
                        float sn, cs;
                        phase(r, kKeys * warp + kk, pd, &sn, &cs);
                        const float graw = xr[r * kTile + kKeys * warp + kk];
                        dk1[kk][pi] += a1[kk] * cs - a2[kk] * sn + graw * qL1;
                        dk2[kk][pi] += a2[kk] * cs + a1[kk] * sn + graw * qL2;
                    }
                }
            }
#pragma unroll
            for (int kk = 0; kk < kKeys; ++kk) load_heads<G>(x[kk], xp + (r * kTile + kKeys * warp + kk) * G);
#pragma unroll
            for (int h = 0; h < G; ++h)
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    const float gv = do_s[(h * kWarps + r) * D + lane + 32 * c];
#pragma unroll
                    for (int kk = 0; kk < kKeys; ++kk) dv[kk][c] = fmaf(x[kk][h], gv, dv[kk][c]);
                }
        }
#pragma unroll
        for (int kk = 0; kk < kKeys; ++kk) {
            if (key0 + kk > i_last) continue;
            float *dk_out = dk_acc + (size_t)(key0 + kk) * D + lane, *dv_out = dv_acc + (size_t)(key0 + kk) * D + lane;
#pragma unroll
            for (int pi = 0; pi < NPI; ++pi)
                if (lane + 32 * pi < H2) {
                    atomicAdd(dk_out + 32 * pi, dk1[kk][pi]);
                    atomicAdd(dk_out + 32 * pi + H2, dk2[kk][pi]);
                }
#pragma unroll
            for (int c = 0; c < NC; ++c) atomicAdd(dv_out + 32 * c, dv[kk][c]);
        }
    }
    if (i < N) {
#pragma unroll
        for (int h = 0; h < G; ++h) {
            T* DQ = reinterpret_cast<T*>(p.dq) + row_offset(p.sdq, p.Hq, (int)q_head0 + h, i);
#pragma unroll
            for (int pi = 0; pi < NPI; ++pi) {
                const int pd = lane + 32 * pi;
                if (pd < H2) {
                    DQ[pd] = Elem<T>::from_f32(dq1[h][pi]);
                    DQ[pd + H2] = Elem<T>::from_f32(dq2[h][pi]);
                }
            }
        }
    }
}

template <typename T, int D, int G>
int launch_fwd_g(const GqaParams& p, cudaStream_t s) {
    constexpr bool kAcc = (Elem<T>::kDtype == COROPE_DTYPE_F32);
    constexpr size_t smem = fwd_smem_bytes<T, D, G>();
    auto kern = corope_fwd_general_kernel<T, D, G, kAcc>;
    static std::atomic<uint64_t> smem_ok;
    if (int er = allow_smem(kern, smem, smem_ok)) return er;
    dim3 grid((p.N + kWarps - 1) / kWarps, p.B * p.Hkv);
    kern<<<grid, kThreads, smem, s>>>(p); count_launch();
    return (int)cudaGetLastError();
}

template <typename T, int D, int G>
int launch_bwd_g(const GqaParams& p, cudaStream_t s) {
    constexpr bool kAcc = (Elem<T>::kDtype == COROPE_DTYPE_F32);
    constexpr size_t smem = BwdSmem<T, D, G, kAcc>::kBytes;
    auto kern = corope_bwd_general_kernel<T, D, G, kAcc>;
    static std::atomic<uint64_t> smem_ok;
    if (int er = allow_smem(kern, smem, smem_ok)) return er;
    dim3 grid((p.N + kWarps - 1) / kWarps, p.B * p.Hkv);
    kern<<<grid, kThreads, smem, s>>>(p); count_launch();
    return (int)cudaGetLastError();
}

template <typename T, int D>
int dispatch_g(const GqaParams& p, cudaStream_t s, bool bwd) {
    switch (p.G) {
        case 1: return bwd ? launch_bwd_g<T, D, 1>(p, s) : launch_fwd_g<T, D, 1>(p, s);
        case 2: return bwd ? launch_bwd_g<T, D, 2>(p, s) : launch_fwd_g<T, D, 2>(p, s);
        case 4: return bwd ? launch_bwd_g<T, D, 4>(p, s) : launch_fwd_g<T, D, 4>(p, s);
        case 8: return bwd ? launch_bwd_g<T, D, 8>(p, s) : launch_fwd_g<T, D, 8>(p, s);
        case 3: return bwd ? launch_bwd_g<T, D, 3>(p, s) : launch_fwd_g<T, D, 3>(p, s);
        case 5: return bwd ? launch_bwd_g<T, D, 5>(p, s) : launch_fwd_g<T, D, 5>(p, s);
        case 6: return bwd ? launch_bwd_g<T, D, 6>(p, s) : launch_fwd_g<T, D, 6>(p, s);
        case 7: return bwd ? launch_bwd_g<T, D, 7>(p, s) : launch_fwd_g<T, D, 7>(p, s);
        default: return COROPE_ERR_BAD_GROUP;
    }
}

template <typename T>
int dispatch_gd(const GqaParams& p, cudaStream_t s, bool bwd) {
    switch (p.D) {
        case 32: return dispatch_g<T, 32>(p, s, bwd);
        case 64: return dispatch_g<T, 64>(p, s, bwd);
        case 128: return dispatch_g<T, 128>(p, s, bwd);
        default: return COROPE_ERR_BAD_HEAD_DIM;
    }
}

template <typename T>
int bwd_all(const GqaParams& p, cudaStream_t s) {
    const size_t rows = (size_t)p.B * p.Hq * p.N;
    const size_t kv_elems = (size_t)p.B * p.Hkv * p.N * p.D;
    gqa_delta_kernel<T><<<(unsigned)((rows + 7) / 8), 256, 0, s>>>((const T*)p.o, (const T*)p.d_o, p.delta, rows, p.D, row_addr(p.so, p.Hq, p.N),
                                                                           row_addr(p.sdo, p.Hq, p.N)); count_launch();
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return (int)e;
    // dv_acc follows dk_acc in the workspace
    if ((e = cudaMemsetAsync(p.dk_acc, 0, (size_t)(p.dv_acc + kv_elems - p.dk_acc) * sizeof(float), s)) != cudaSuccess) return (int)e;
    if (int r = p.use_mma ? launch_gqa_bwd_mma(p, Elem<T>::kDtype, s) : dispatch_gd<T>(p, s, true)) return r;
    gqa_finalize_kernel<T><<<dim3((unsigned)((kv_elems + 255) / 256), 2), 256, 0, s>>>(p.dk_acc, p.dv_acc, (T*)p.dk, (T*)p.dv, kv_elems, p.D,
                                                                                      row_addr(p.sdk, p.Hkv, p.N), row_addr(p.sdv, p.Hkv, p.N)); count_launch();
    return (int)cudaGetLastError();
}

}  // namespace

int launch_gqa_fwd_general(const GqaParams& p, int dtype, cudaStream_t s) {
    switch (dtype) {
        case COROPE_DTYPE_F32: return dispatch_gd<float>(p, s, false);
        case COROPE_DTYPE_BF16: return dispatch_gd<__nv_bfloat16>(p, s, false);
        case COROPE_DTYPE_F16: return dispatch_gd<__half>(p, s, false);
        default: return COROPE_ERR_BAD_DTYPE;
    }
}

int launch_gqa_bwd_general(const GqaParams& p, int dtype, cudaStream_t s) {
    switch (dtype) {
        case COROPE_DTYPE_F32: return bwd_all<float>(p, s);
        case COROPE_DTYPE_BF16: return bwd_all<__nv_bfloat16>(p, s);
        case COROPE_DTYPE_F16: return bwd_all<__half>(p, s);
        default: return COROPE_ERR_BAD_DTYPE;
    }
}

}  // namespace corope
