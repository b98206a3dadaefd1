// Co-RoPE GQA attention forward for 16-bit inputs outside the whole tiles of the mma kernels (D = 64, or N no multiple of 64): the
// products on tensor cores (mma.sync), at the fp32 accuracy of the CUDA-core kernel that these shapes ran on.
//
// Same scheme as corope_fwd_mma.cu (one CTA = 8 query rows of one (batch, KV head), one warp per row, key tiles of 64 swept downward,
// S^T = K' Q^T and O^T += V^T P^T with the keys as MMA rows and the group's heads as columns), but the operands stay exact: q, k, v
// enter the MMAs in their own type; the rotation is formed in fp32 and K' and P enter as the sum of several numbers of that type, hi
// + rest.  bf16: three parts, which hold the 24 bits of an fp32 number.  f16: two parts for K' (22 bits; the rows of K are scaled by a
// power of two so that none of it sinks into the subnormals), three for P, times 2^14 for the same reason.  The adder of the MMAs does
// not round to nearest: products of the hi parts go through one MMA each, which fp32 additions join.
//
// Error of O against 64-bit arithmetic, N(0, 1) inputs: the rounding of the result.  Results that are not the exact one rounded, next to
// the CUDA-core kernel (Hq8 Hkv2, inputs times 0.3, where the phases matter least): bf16 N700 D128 0.030 % (0.037 %), f16 N333 D64 0.092 %
// (0.133 %); at scale 1 f16 N512 D64 1.13 % (1.13 %), its LSE 4.9e-7 (4.8e-7).  Two bf16 parts, and f16 parts without the scaling, had
// 0.22 % and 0.21 % at scale 0.3.
// B1 Hq32 Hkv8 N1500 D128 bf16 928 us (CUDA-core kernel 1347; 1160 with conversions in place of permutes and masks), f16 763 (1355; 810 with conversions
// back to fp32 in place of mixed-precision additions), B2 Hq16
// Hkv4 N2048 D64 bf16 899 (1298; 969), B1 Hq16 Hkv2 N300 D64 f16 27.5 (68), B4 Hq4 Hkv4 N100 D64 bf16 21.5 (21.0; 23.3) us, so it takes
// every size.
// What bounds it: issue slots; the rotation costs two special-function operations and some 20 instructions per (query, key, pair)
// triple, shared by the heads, against two per head and pair of the CUDA-core kernel on top of that.
#include "corope_mma.cuh"
#include "rope_split.cuh"

namespace corope {
namespace {

using gqa_mma::kKT;
using gqa_mma::kRows;
using gqa_mma::kThreads;
using gqa_mma::kWStride;
using gqa_mma::lane_pair;
using gqa_mma::movmatrix_trans;
using gqa_mma::perm_slot;

template <int D> struct Geo {
    static constexpr int kPairs = D / 2, kChunks = D / 32;        // 4-pair chunks per lane
    static constexpr int kKRow = kPairs + 16;                     // u32 per K row, padded as in corope_mma.cuh
    static constexpr int kVRowBytes = 2 * D + 16;
    static constexpr int kKTileBytes = kKT * kKRow * 4, kVTileBytes = kKT * kVRowBytes;
    static constexpr int kAqBytes = kThreads * kChunks * 16;
    static constexpr size_t kSmem = 2 * (kKTileBytes + kVTileBytes) + kRows * kPairs * 4 + 2 * kRows * kKT * 4 + 4 * kWStride * 4 + kAqBytes + 2 * kKT * 4;
};

template <typename T> __device__ __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1);
template <> __device__ __forceinline__ void mma<__half>(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) { gqa_mma::mma16816_full(d, a, b0, b1); }
template <> __device__ __forceinline__ void mma<__nv_bfloat16>(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// (a, b) as the sum of PARTS pairs of T, each the rounded rest of those before; three bf16 parts, which hold all 24 bits either way, are cut off
// by byte permutes and masks instead of conversions
template <typename T, int PARTS>
__device__ __forceinline__ void split(float a, float b, uint32_t (&parts)[PARTS]) {
    if constexpr (Elem<T>::kDtype == COROPE_DTYPE_BF16 && PARTS == 3) {
        split3_cut<T>(a, b, parts);
        return;
    }
#pragma unroll
    for (int x = 0; x < PARTS; ++x) {
        parts[x] = pack2<T>(a, b);
        if (x + 1 < PARTS) subtract_pair<T>(parts[x], a, b);
    }
}
// parts of a rotated K: bf16 needs three for the 24 bits of an fp32 number; two of f16 hold 22 where scaled rows keep them out of the
// subnormals.  (Three f16 parts, hi cut to 8 bits: 985 instead of 812 us at B1 Hq32 Hkv8 N1500 D128, results no closer to the exact ones, LSE of
// Hq8 Hkv2 N512 D64 4.89e-7 instead of 4.92e-7: what is left comes from the MMAs' adder, and from the phases.)
template <typename T> constexpr int kParts = Elem<T>::kDtype == COROPE_DTYPE_F16 ? 2 : 3;
// one (k1, k2) pair rotated by `angle` in fp32: (k1 cos + k2 sin, k2 cos - k1 sin), split
template <typename T, bool DIRECT>
__device__ __forceinline__ void rotate_split(uint32_t kpair, float angle, uint32_t (&parts)[kParts<T>]) {
    float sn, cs;
    gqa_mma::sincos_fast<DIRECT>(angle, &sn, &cs);
    const float2 k = unpack2<T>(kpair);
    split<T, kParts<T>>(fmaf(k.x, cs, k.y * sn), fmaf(k.y, cs, -k.x * sn), parts);
}
// hi hi + the smaller products.  An infinity shows in hi hi with the sign it has in fp32; the other parts of such a product are
// meaningless (NaN or either infinity).
__device__ __forceinline__ float join(float main, float small) { return fabsf(main) < INFINITY ? main + small : main; }
template <typename T>
__device__ __forceinline__ uint32_t pair_bits(const T* row, int p, int half) {
    return (uint32_t)*reinterpret_cast<const uint16_t*>(row + p) | (uint32_t)*reinterpret_cast<const uint16_t*>(row + p + half) << 16;
}
__device__ __forceinline__ void cp16(void* dst, const void* src, bool have) {   // zeros when `have` is false (src is then not read)
    const int bytes = have ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes) : "memory");
}

__device__ __forceinline__ uint4 load8_any(const uint16_t* src, bool vec) {   // 8 elements; one by one where rows are not aligned to 16 bytes
    if (vec) return *reinterpret_cast<const uint4*>(src);
    uint32_t w[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) w[e] = (uint32_t)src[2 * e] | (uint32_t)src[2 * e + 1] << 16;
    return make_uint4(w[0], w[1], w[2], w[3]);
}
// K -> (k1, k2) pairs of its own type in the permuted row order; V -> a contiguous copy where the main kernel's 16-byte copies
// could not read it (vc, else null).  One thread per 8 pairs and 16 columns.  f16 rows are multiplied by the power of two that brings
// their largest element into [2^13, 2^14) (K' stays below 2^15), its inverse goes to kscale: two f16 parts of K' then reach down to
// 2^-38 of that element, whatever the magnitude of the row.  (An element that a row loses to the subnormals in being scaled down is
// below 2^-39 of the largest.)
template <typename T, int D>
__global__ void __launch_bounds__(256) gqa_pack_k_kernel(const T* __restrict__ K, uint32_t* __restrict__ kp, float* __restrict__ kscale, const T* __restrict__ V,
                                                         T* __restrict__ vc, size_t rows, RowAddr ak, RowAddr av, bool kvec) {
    constexpr int kPairs = D / 2, kPerRow = kPairs / 8;
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = idx / kPerRow < rows;
    const size_t r = live ? idx / kPerRow : rows - 1;
    const int p0 = (int)(idx % kPerRow) * 8;
    const uint16_t* src = reinterpret_cast<const uint16_t*>(K + flat_row_offset(ak, r) + p0);
    const uint4 x1 = load8_any(src, kvec), x2 = load8_any(src + kPairs, kvec);
    uint32_t a[4] = {x1.x, x1.y, x1.z, x1.w}, b[4] = {x2.x, x2.y, x2.z, x2.w};
    if (Elem<T>::kDtype == COROPE_DTYPE_F16) {
        float mx = 0.f;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float2 fa = unpack2<T>(a[e]), fb = unpack2<T>(b[e]);
            mx = fmaxf(fmaxf(mx, fmaxf(fabsf(fa.x), fabsf(fa.y))), fmaxf(fabsf(fb.x), fabsf(fb.y)));
        }
#pragma unroll
        for (int off = kPerRow / 2; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
        const int e2 = mx > 0.f && mx < INFINITY ? 13 - ilogbf(mx) : 0;
        const float up = ldexpf(1.f, e2);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float2 fa = unpack2<T>(a[e]), fb = unpack2<T>(b[e]);
            a[e] = pack2<T>(fa.x * up, fa.y * up);
            b[e] = pack2<T>(fb.x * up, fb.y * up);
        }
        if (live && p0 == 0) kscale[r] = ldexpf(1.f, -e2);
    }
    if (!live) return;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        kp[r * kPairs + perm_slot(p0 + 2 * e)] = __byte_perm(a[e], b[e], 0x5410);
        kp[r * kPairs + perm_slot(p0 + 2 * e + 1)] = __byte_perm(a[e], b[e], 0x7632);
    }
    if (vc != nullptr) {
        const uint16_t* v = reinterpret_cast<const uint16_t*>(V + flat_row_offset(av, r) + 2 * p0);
        uint4* out = reinterpret_cast<uint4*>(vc + r * D + 2 * p0);
        out[0] = load8_any(v, false);
        out[1] = load8_any(v + 8, false);
    }
}

template <typename T, int D, bool DIRECT>
__global__ void __launch_bounds__(kThreads, 2) corope_fwd_split_kernel(GqaParams p) {
    using M = Geo<D>;
    constexpr int kPairs = M::kPairs, CH = M::kChunks, DB = D / 16;
    constexpr bool kScaled = Elem<T>::kDtype == COROPE_DTYPE_F16;
    extern __shared__ __align__(16) uint8_t smem_dyn[];
    uint8_t* ks_base = smem_dyn;                                              // 2 x K tile, (k1, k2) pairs, permuted rows
    uint8_t* vs_base = ks_base + 2 * M::kKTileBytes;                          // 2 x V tile, row-major
    uint32_t* qls = reinterpret_cast<uint32_t*>(vs_base + 2 * M::kVTileBytes);   // leader rows of the CTA's queries, permuted like K
    float* zs = reinterpret_cast<float*>(qls + kRows * kPairs);
    float* dl = zs + kRows * kKT;
    float* ws = dl + kRows * kKT;                                             // inverse frequencies: those of lane class c from c * kWStride
    const int N = p.N, G = p.G;
    const int bg = blockIdx.y, b = bg / p.Hkv, g = bg % p.Hkv;
    const int i0 = (gridDim.x - 1 - blockIdx.x) * kRows;                      // heavy (late) rows first
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, r = lane >> 2, c = lane & 3;
    const int i = i0 + warp;                                                  // rows at or beyond N compute on zeros and store nothing
    uint4* aqs = reinterpret_cast<uint4*>(ws + 4 * kWStride) + warp * CH * 32;   // the query operand of every lane: chunk s of lane l at [warp][s][l]
    float* kss = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(ws + 4 * kWStride) + M::kAqBytes);   // 2 x kscale of the tile's keys (f16)
    auto key_scale = [&](int buf, int key) { return kScaled ? kss[buf * kKT + key] : 1.f; };
    const size_t q_head0 = (size_t)b * p.Hq + (size_t)g * G;
    const uint32_t* Kp = p.k_pairs + (size_t)bg * N * kPairs;
    const T* V = reinterpret_cast<const T*>(p.v) + row_offset(p.sv, p.Hkv, bg, 0);
    auto load_tile = [&](int j0, int buf) {
        uint8_t *kd = ks_base + buf * M::kKTileBytes, *vd = vs_base + buf * M::kVTileBytes;
        constexpr int kPer = D / 8;   // 16-byte pieces per row, of K pairs and of V alike
#pragma unroll
        for (int it = 0; it < kKT * kPer / kThreads; ++it) {
            const int idx = tid + it * kThreads, row = idx / kPer, ch = idx % kPer;
            const bool have = j0 + row < N;
            const int pos = have ? j0 + row : 0;
            cp16(kd + row * (M::kKRow * 4) + ch * 16, Kp + (size_t)pos * kPairs + ch * 4, have);
            cp16(vd + row * M::kVRowBytes + ch * 16, V + (int64_t)pos * p.sv.n + ch * 8, have);
        }
        if (kScaled && tid < kKT) {
            const bool have = j0 + tid < N;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(kss + buf * kKT + tid)),
                         "l"(p.k_scale + (size_t)bg * N + (have ? j0 + tid : 0)), "r"(have ? 4 : 0)
                         : "memory");
        }
        gqa_mma::cp_async_commit();
    };
    const int i_last = min(N - 1, i0 + kRows - 1), j_first = i_last / kKT * kKT;
    load_tile(j_first, 0);

    const T* Q = reinterpret_cast<const T*>(p.q);
    for (int idx = tid; idx < kRows * kPairs; idx += kThreads) {
        const int row = idx / kPairs, pp = idx % kPairs;
        qls[row * kPairs + perm_slot(pp)] = i0 + row < N ? pair_bits(Q + row_offset(p.sq, p.Hq, (int)q_head0, i0 + row), pp, kPairs) : 0u;
    }
    for (int d = tid; d < kPairs; d += kThreads)
        ws[(d & 3) * kWStride + (d >> 4) * 4 + ((d >> 3) & 1) * 2 + ((d & 7) >> 2)] = 1.0f / powf(p.theta, (float)(2 * d) / (float)D);
    {
        const bool have = r < G && i < N;
        const T* qrow = Q + row_offset(p.sq, p.Hq, (int)q_head0 + (have ? r : 0), have ? i : 0);
#pragma unroll
        for (int s = 0; s < CH; ++s) {
            uint32_t a[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) a[e] = have ? pair_bits(qrow, lane_pair(c, s, e), kPairs) : 0u;
            aqs[s * 32 + lane] = make_uint4(a[0], a[1], a[2], a[3]);
        }
        __syncwarp();
    }

    // lane (r = lane / 4, c = lane % 4): keys r and r + 8 of a 16-key block on the operand side, heads 2c and 2c + 1 on the result side
    float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;
    float o[DB][4];   // O^T: rows d = 16 db + r (+ 8 for entries 2, 3), columns heads 2c, 2c + 1
#pragma unroll
    for (int db = 0; db < DB; ++db) o[db][0] = o[db][1] = o[db][2] = o[db][3] = 0.f;
    float carry = 0.f;   // sum of z_ik over the keys of the tiles already swept
    const float sc2 = p.sm_scale * kLog2e;

    int buf = 0;
    for (int j0 = j_first; j0 >= 0; j0 -= kKT, buf ^= 1) {
        gqa_mma::cp_async_wait_all();
        __syncthreads();   // this tile has landed for every thread, and every warp is done with the previous tile
        if (j0 >= kKT) load_tile(j0 - kKT, buf ^ 1);
        const uint32_t* ks = reinterpret_cast<const uint32_t*>(ks_base + buf * M::kKTileBytes);
        const uint8_t* vs = vs_base + buf * M::kVTileBytes;

        // 1. leader gates: rows of A = the CTA's 8 query rows, warp w takes keys 8w .. 8w + 7 (B = raw K pairs)
        {
            const uint4* kp = reinterpret_cast<const uint4*>(ks + (warp * 8 + r) * M::kKRow) + c;
            const uint4* qp = reinterpret_cast<const uint4*>(qls + r * kPairs) + c;
            float z[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int s = 0; s < CH; ++s) {
                const uint4 kv = kp[4 * s], qv = qp[4 * s];
                const uint32_t a0[4] = {qv.x, 0u, qv.y, 0u}, a1[4] = {qv.z, 0u, qv.w, 0u};
                mma<T>(z, a0, kv.x, kv.y);
                mma<T>(z, a1, kv.z, kv.w);
            }
            const int key = j0 + warp * 8 + 2 * c, qi = i0 + r;
            const float z0 = z[0] * key_scale(buf, warp * 8 + 2 * c), z1 = z[1] * key_scale(buf, warp * 8 + 2 * c + 1);
            zs[r * kKT + warp * 8 + 2 * c] = key <= qi ? 1.f / (1.f + __expf(-z0 * p.sm_scale)) : 0.f;
            zs[r * kKT + warp * 8 + 2 * c + 1] = key + 1 <= qi ? 1.f / (1.f + __expf(-z1 * p.sm_scale)) : 0.f;
        }
        __syncthreads();
        // 2. Delta of this warp's row: carry + sum of z over the keys of the tile above j
        {
            const float za = zs[warp * kKT + 2 * lane], zb = zs[warp * kKT + 2 * lane + 1];
            float suf = za + zb;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const float t = __shfl_down_sync(0xffffffffu, suf, off);
                if (lane + off < 32) suf += t;
            }
            const float above = carry + suf - (za + zb);   // keys beyond this lane's pair
            dl[warp * kKT + 2 * lane + 1] = above;
            dl[warp * kKT + 2 * lane] = above + zb;
            carry += __shfl_sync(0xffffffffu, suf, 0);
        }
        __syncwarp();

        // 3. S^T of the row, 16 keys x 8 heads per block
        float sc[4][4];
#pragma unroll
        for (int kb = 0; kb < 4; ++kb) {
            sc[kb][0] = sc[kb][1] = sc[kb][2] = sc[kb][3] = -INFINITY;
            if (j0 + kb * 16 > i) continue;   // every key of the block is above the diagonal (warp-uniform)
            const float dA = dl[warp * kKT + kb * 16 + r], dB = dl[warp * kKT + kb * 16 + r + 8];
            const uint4* kpA = reinterpret_cast<const uint4*>(ks + (kb * 16 + r) * M::kKRow) + c;
            const uint4* kpB = reinterpret_cast<const uint4*>(ks + (kb * 16 + r + 8) * M::kKRow) + c;
            float acc[4] = {0.f, 0.f, 0.f, 0.f}, acl[4] = {0.f, 0.f, 0.f, 0.f};   // products of the hi parts, and the smaller ones
#pragma unroll
            for (int s = 0; s < CH; ++s) {
                const uint4 kva = kpA[4 * s], kvb = kpB[4 * s], av = aqs[s * 32 + lane];
                const float4 wv = *reinterpret_cast<const float4*>(ws + c * kWStride + s * 4);
                const float w[4] = {wv.x, wv.y, wv.z, wv.w};
                const uint32_t ka[4] = {kva.x, kva.y, kva.z, kva.w}, kk[4] = {kvb.x, kvb.y, kvb.z, kvb.w}, q[4] = {av.x, av.y, av.z, av.w};
#pragma unroll
                for (int t = 0; t < 2; ++t) {
                    uint32_t kr[kParts<T>][4];   // a0 / a2: key r, a1 / a3: key r + 8
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        uint32_t x[kParts<T>], y[kParts<T>];
                        rotate_split<T, DIRECT>(ka[2 * t + e], dA * w[2 * t + e], x);
                        rotate_split<T, DIRECT>(kk[2 * t + e], dB * w[2 * t + e], y);
#pragma unroll
                        for (int part = 0; part < kParts<T>; ++part) kr[part][2 * e] = x[part], kr[part][2 * e + 1] = y[part];
                    }
                    float hi[4] = {0.f, 0.f, 0.f, 0.f};
                    mma<T>(hi, kr[0], q[2 * t], q[2 * t + 1]);
#pragma unroll
                    for (int x = 0; x < 4; ++x) acc[x] += hi[x];
#pragma unroll
                    for (int part = kParts<T> - 1; part > 0; --part) mma<T>(acl, kr[part], q[2 * t], q[2 * t + 1]);
                }
            }
            const int keyA = j0 + kb * 16 + r;
            const float sA = sc2 * key_scale(buf, kb * 16 + r), sB = sc2 * key_scale(buf, kb * 16 + r + 8);
            if (keyA <= i) sc[kb][0] = join(acc[0], acl[0]) * sA, sc[kb][1] = join(acc[1], acl[1]) * sA;
            if (keyA + 8 <= i) sc[kb][2] = join(acc[2], acl[2]) * sB, sc[kb][3] = join(acc[3], acl[3]) * sB;
        }

        // 4. online softmax of heads 2c, 2c + 1 (their 64 scores sit in the 8 lanes of class c), then O^T += V^T P^T
        float mx0 = m0, mx1 = m1;
#pragma unroll
        for (int kb = 0; kb < 4; ++kb) {
            mx0 = fmax3(mx0, sc[kb][0], sc[kb][2]);
            mx1 = fmax3(mx1, sc[kb][1], sc[kb][3]);
        }
#pragma unroll
        for (int off = 4; off < 32; off <<= 1) {
            mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, off));
            mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, off));
        }
        const float alpha0 = exp2f(m0 - mx0), alpha1 = exp2f(m1 - mx1);   // the first tile holds the diagonal: mx is finite
        m0 = mx0, m1 = mx1;
#pragma unroll
        for (int db = 0; db < DB; ++db) {
            o[db][0] *= alpha0, o[db][1] *= alpha1;
            o[db][2] *= alpha0, o[db][3] *= alpha1;
        }
        float ps0 = 0.f, ps1 = 0.f;
#pragma unroll
        for (int kb = 0; kb < 4; ++kb) {
            if (j0 + kb * 16 > i) continue;   // nothing visible in this block (warp-uniform)
            const float pA0 = exp2f(sc[kb][0] - mx0), pA1 = exp2f(sc[kb][1] - mx1);   // key r
            const float pB0 = exp2f(sc[kb][2] - mx0), pB1 = exp2f(sc[kb][3] - mx1);   // key r + 8
            ps0 += pA0 + pB0;
            ps1 += pA1 + pB1;
            // P^T as B operand: (keys 2c, 2c + 1 | head r) is the transpose of what the lane holds (key r | heads 2c, 2c + 1)
            uint32_t pa[3], pb[3];
            split<T, 3>(pA0 * kPScale<T>, pA1 * kPScale<T>, pa);
            split<T, 3>(pB0 * kPScale<T>, pB1 * kPScale<T>, pb);
#pragma unroll
            for (int part = 0; part < 3; ++part) pa[part] = movmatrix_trans(pa[part]), pb[part] = movmatrix_trans(pb[part]);
            // V^T as A operand: four transposed 8x8 blocks (d 0-7 | 8-15) x (keys 0-7 | 8-15) of the block's V rows
            const uint8_t* vrow = vs + (kb * 16 + (lane & 7) + ((lane >> 4) & 1) * 8) * M::kVRowBytes + ((lane >> 3) & 1) * 16;
#pragma unroll
            for (int db = 0; db < DB; ++db) {   // the block's own sum, then one fp32 addition: the adder of the MMAs does not round to nearest
                uint32_t a[4];
                gqa_mma::ldmatrix_x4_trans(a[0], a[1], a[2], a[3], vrow + db * 32);
                float t[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int part = 2; part >= 0; --part) mma<T>(t, a, pa[part], pb[part]);
#pragma unroll
                for (int x = 0; x < 4; ++x) o[db][x] += t[x];
            }
        }
        l0 = l0 * alpha0 + ps0;
        l1 = l1 * alpha1 + ps1;
    }

#pragma unroll
    for (int off = 4; off < 32; off <<= 1) {
        l0 += __shfl_xor_sync(0xffffffffu, l0, off);
        l1 += __shfl_xor_sync(0xffffffffu, l1, off);
    }
    if (i >= N) return;
#pragma unroll
    for (int x = 0; x < 2; ++x) {
        const int head = 2 * c + x;
        if (head >= G) continue;
        const float inv = (1.f / kPScale<T>) / (x ? l1 : l0);
        T* O = reinterpret_cast<T*>(p.out_o) + row_offset(p.so, p.Hq, (int)q_head0 + head, i);
#pragma unroll
        for (int db = 0; db < DB; ++db) {
            O[db * 16 + r] = Elem<T>::from_f32(o[db][x] * inv);
            O[db * 16 + r + 8] = Elem<T>::from_f32(o[db][2 + x] * inv);
        }
        if (r == 0) p.lse2[(q_head0 + head) * N + i] = (x ? m1 : m0) + log2f(x ? l1 : l0);
    }
    if (lane == 0) p.a_diag[(size_t)bg * N + i] = carry;
}

template <typename T, int D>
int launch_t(GqaParams p, bool k_vec, bool v_vec, cudaStream_t s) {
    const size_t rows = (size_t)p.B * p.Hkv * p.N;
    T* vc = v_vec ? nullptr : reinterpret_cast<T*>(p.v_half);
    gqa_pack_k_kernel<T, D><<<(unsigned)((rows * (D / 16) + 255) / 256), 256, 0, s>>>((const T*)p.k, p.k_pairs, p.k_scale, (const T*)p.v, vc, rows,
                                                                                     row_addr(p.sk, p.Hkv, p.N), row_addr(p.sv, p.Hkv, p.N), k_vec);
    if (vc) {
        p.v = vc;
        p.sv = contiguous_strides(p.Hkv, p.N, D);
    }
    count_launch();
    if (cudaError_t e = cudaGetLastError()) return (int)e;
    const bool direct = p.N <= 8192;   // phases up to a few thousand radians go to the hardware sin / cos directly
    auto kern = direct ? corope_fwd_split_kernel<T, D, true> : corope_fwd_split_kernel<T, D, false>;
    static std::atomic<uint64_t> smem_ok[2];
    if (int e = allow_smem(kern, Geo<D>::kSmem, smem_ok[direct])) return e;
    kern<<<dim3((p.N + kRows - 1) / kRows, p.B * p.Hkv), kThreads, Geo<D>::kSmem, s>>>(p);
    count_launch();
    return (int)cudaGetLastError();
}

}  // namespace

bool gqa_split_supported(int D, int dtype) { return (D == 64 || D == 128) && (dtype == COROPE_DTYPE_BF16 || dtype == COROPE_DTYPE_F16); }

int launch_gqa_fwd_split(const GqaParams& p, bool k_vec, bool v_vec, int dtype, cudaStream_t s) {
    if (dtype == COROPE_DTYPE_BF16) return p.D == 64 ? launch_t<__nv_bfloat16, 64>(p, k_vec, v_vec, s) : launch_t<__nv_bfloat16, 128>(p, k_vec, v_vec, s);
    return p.D == 64 ? launch_t<__half, 64>(p, k_vec, v_vec, s) : launch_t<__half, 128>(p, k_vec, v_vec, s);
}

}  // namespace corope
