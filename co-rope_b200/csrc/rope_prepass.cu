// Passes over the inputs that the tensor-core fused-RoPE kernels need before they run: the packed (cos, sin) table, the rotated
// fp16 copy of K (forward) or of Q (backward), and for the backward delta = rowsum(O * dO) and a cleared fp32 dQ accumulator.
//
// Rotating once here instead of once per consumer (a K tile is consumed by up to N/256 forward items, a Q tile by every key
// block at or below its diagonal) takes the rotation out of the main kernels' inner loops.  All of it is bound by HBM.
//
// A block owns a range of positions and walks over a few heads with it: the (cos, sin) entries of a thread's 8 pairs are read
// and packed once and stay in registers for all of those heads, so packing needs no launch of its own and the fp32 tables are
// read heads / heads_per_block times instead of once per head.  (One row per thread group and launch, each reading the fp32
// tables, cost 9 us more at B2 H32 N4096 D128 than a separate packing launch: 512 bytes of table per 256-byte row.)
#include "common.cuh"

namespace corope {
namespace {

constexpr int kThreads = 256;
enum TableMode { kTables, kIdentity, kPacked };

// 8 consecutive (cos, sin) entries of position n from column c on, packed
template <int MODE, int HALF>
__device__ __forceinline__ void table_entries(uint4& t0, uint4& t1, const float* __restrict__ cosT, const float* __restrict__ sinT, int64_t ts,
                                              bool vec, const uint32_t* __restrict__ packed, int n, int c) {
    if (MODE == kPacked) {
        const uint4* tp = reinterpret_cast<const uint4*>(packed + (size_t)n * HALF + c);
        t0 = __ldg(tp);
        t1 = __ldg(tp + 1);
        return;
    }
    uint32_t e[8];
    if (MODE == kIdentity) {
#pragma unroll
        for (int i = 0; i < 8; ++i) e[i] = pack_unorm_pair(1.f, 0.f);
    } else {
        float cv[8], sv[8];
        const float* cp = cosT + n * ts + c;
        const float* sp = sinT + n * ts + c;
        if (vec) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const float4 a = __ldg(reinterpret_cast<const float4*>(cp) + i), b = __ldg(reinterpret_cast<const float4*>(sp) + i);
                cv[4 * i] = a.x; cv[4 * i + 1] = a.y; cv[4 * i + 2] = a.z; cv[4 * i + 3] = a.w;
                sv[4 * i] = b.x; sv[4 * i + 1] = b.y; sv[4 * i + 2] = b.z; sv[4 * i + 3] = b.w;
            }
        } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) cv[i] = __ldg(cp + i), sv[i] = __ldg(sp + i);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) e[i] = pack_unorm_pair(cv[i], sv[i]);
    }
    t0 = make_uint4(e[0], e[1], e[2], e[3]);
    t1 = make_uint4(e[4], e[5], e[6], e[7]);
}

struct PrepassTable {
    const float* cos;
    const float* sin;
    int64_t stride;
    int vec;            // rows of both tables are 16-byte aligned
    uint32_t* packed;   // read (kPacked) or written by the blocks of the first heads; the work counter follows it
};

// Forward: D / 16 threads per row, 8 pairs each.  Position blocks run fastest, then groups of heads.
template <typename T, int D, int MODE>
__global__ void __launch_bounds__(kThreads) rope_fwd_prepass_kernel(const T* __restrict__ k, __half* __restrict__ k_rot, PrepassTable tab, int N,
                                                                    int BH, int heads_per_block, RowAddr ak) {
    constexpr int kPerRow = D / 16, kRows = kThreads / kPerRow, kUnroll = 4;
    pdl_trigger();
    const unsigned pbs = ceil_div(N, kRows), group = blockIdx.x / pbs;
    const int n = (blockIdx.x % pbs) * kRows + threadIdx.x / kPerRow;
    const int c = (threadIdx.x % kPerRow) * 8;
    if (MODE != kPacked && blockIdx.x == 0 && threadIdx.x == 0) tab.packed[(size_t)N * (D / 2)] = 0u;   // work counter
    if (n >= N) return;
    uint4 t0, t1;
    table_entries<MODE, D / 2>(t0, t1, tab.cos, tab.sin, tab.stride, tab.vec, tab.packed, n, c);
    if (MODE != kPacked && group == 0) {
        uint4* out = reinterpret_cast<uint4*>(tab.packed + (size_t)n * (D / 2) + c);
        out[0] = t0;
        out[1] = t1;
    }
    const int h1 = min(BH, (int)(group + 1) * heads_per_block);
    for (int h = group * heads_per_block; h < h1; h += kUnroll) {
        uint4 x1[kUnroll], x2[kUnroll];
#pragma unroll
        for (int u = 0; u < kUnroll; ++u)
            if (h + u < h1) {
                const T* src = k + flat_row_offset(ak, (size_t)(h + u) * N + n) + c;
                x1[u] = __ldg(reinterpret_cast<const uint4*>(src));
                x2[u] = __ldg(reinterpret_cast<const uint4*>(src + D / 2));
            }
#pragma unroll
        for (int u = 0; u < kUnroll; ++u)
            if (h + u < h1) {
                rotate_vec8<T>(x1[u], x2[u], t0, t1, 1.f / 32768.f, -257.f);
                __half* dst = k_rot + ((size_t)(h + u) * N + n) * D + c;
                *reinterpret_cast<uint4*>(dst) = x1[u];
                *reinterpret_cast<uint4*>(dst + D / 2) = x2[u];
            }
    }
}

// Backward: D / 8 threads per row; each takes 8 elements of O . dO and 32 bytes of the accumulator row, the lower half of them
// also 8 pairs of Q.  
template <typename T, int D, int MODE>
__global__ void __launch_bounds__(kThreads) rope_bwd_prepass_kernel(const T* __restrict__ q, const T* __restrict__ o, const T* __restrict__ d_o,
                                                                    PrepassTable tab,
                                                                    __half* __restrict__ q_rot, float* __restrict__ delta, float* __restrict__ dq_acc,
                                                                    int N, int BH, int heads_per_block, float scale, RowAddr aq,
                                                                    RowAddr ao, RowAddr ado) {
    constexpr int kPerRow = D / 8, kRows = kThreads / kPerRow, kUnroll = 2;
    pdl_trigger();
    const unsigned pbs = ceil_div(N, kRows), group = blockIdx.x / pbs;
    const int n = (blockIdx.x % pbs) * kRows + threadIdx.x / kPerRow;
    const int part = threadIdx.x % kPerRow;
    const bool live = n < N, rot = live && part < kPerRow / 2;
    const int c = part * 8;
    if (MODE != kPacked && blockIdx.x == 0 && threadIdx.x == 0) tab.packed[(size_t)N * (D / 2)] = 0u;   // work counter
    uint4 t0 = make_uint4(0u, 0u, 0u, 0u), t1 = t0;
    if (rot) {
        table_entries<MODE, D / 2>(t0, t1, tab.cos, tab.sin, tab.stride, tab.vec, tab.packed, n, c);
        if (MODE != kPacked && group == 0) {
            uint4* out = reinterpret_cast<uint4*>(tab.packed + (size_t)n * (D / 2) + c);
            out[0] = t0;
            out[1] = t1;
        }
    }
    const int h1 = min(BH, (int)(group + 1) * heads_per_block);
    for (int h = group * heads_per_block; h < h1; h += kUnroll) {
        uint4 a[kUnroll], b[kUnroll], x1[kUnroll], x2[kUnroll];
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
            a[u] = b[u] = make_uint4(0u, 0u, 0u, 0u);
            if (live && h + u < h1) {
                const size_t row = (size_t)(h + u) * N + n;
                a[u] = __ldg(reinterpret_cast<const uint4*>(o + flat_row_offset(ao, row) + c));
                b[u] = __ldg(reinterpret_cast<const uint4*>(d_o + flat_row_offset(ado, row) + c));
                if (rot) {
                    const T* src = q + flat_row_offset(aq, row) + c;
                    x1[u] = __ldg(reinterpret_cast<const uint4*>(src));
                    x2[u] = __ldg(reinterpret_cast<const uint4*>(src + D / 2));
                }
            }
        }
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
            const uint32_t aw[4] = {a[u].x, a[u].y, a[u].z, a[u].w}, bw[4] = {b[u].x, b[u].y, b[u].z, b[u].w};
            float s = 0.f;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float2 fa = unpack2<T>(aw[i]), fb = unpack2<T>(bw[i]);
                s = fmaf(fa.x, fb.x, s);
                s = fmaf(fa.y, fb.y, s);
            }
#pragma unroll
            for (int off = kPerRow / 2; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
            if (h + u >= h1) continue;
            const size_t row = (size_t)(h + u) * N + n;
            if (live) {
                if (rot) {
                    rotate_vec8<T>(x1[u], x2[u], t0, t1, scale * (1.f / 32768.f), -257.f * scale);
                    __half* dst = q_rot + row * D + c;
                    *reinterpret_cast<uint4*>(dst) = x1[u];
                    *reinterpret_cast<uint4*>(dst + D / 2) = x2[u];
                }
                uint4* z = reinterpret_cast<uint4*>(dq_acc + row * D) + part * 2;
                z[0] = make_uint4(0u, 0u, 0u, 0u);
                z[1] = make_uint4(0u, 0u, 0u, 0u);
            }
            if (live && part == 0) delta[row] = s;
        }
    }
}

// packed table alone (the kernels that rotate every tile themselves)
__global__ void pack_tables_kernel(const float* __restrict__ cosT, const float* __restrict__ sinT, int64_t ts, uint32_t* __restrict__ out,
                                   int N, int half_d) {
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx == 0) out[(size_t)N * half_d] = 0u;   // work counter of the persistent kernels
    if (idx >= (size_t)N * half_d) return;
    const int n = (int)(idx / half_d), d = (int)(idx % half_d);
    out[idx] = cosT != nullptr ? pack_unorm_pair(cosT[n * ts + d], sinT[n * ts + d]) : pack_unorm_pair(1.f, 0.f);
}

// cos / sin for positions 0 .. N-1 from the per-pair frequencies, as precompute_freqs_cis forms them
// (fused-rope/rope_attn_pytorch.py:29-47): inv_freq[d] = 1 / theta^(2d/D), angle = float(position) * inv_freq[d] in fp32, then
// cos / sin of it.  blockDim.x = half_d: a thread keeps its frequency for kPositions positions.
constexpr int kPositions = 8;
template <bool PACK>
__global__ void synth_tables_kernel(const float* __restrict__ inv_freq, float theta, float* __restrict__ cosT, float* __restrict__ sinT,
                                    uint32_t* __restrict__ packed, int N) {
    const int half_d = blockDim.x, d = threadIdx.x;
    if (PACK && blockIdx.x == 0 && threadIdx.x == 0 && threadIdx.y == 0) packed[(size_t)N * half_d] = 0u;   // work counter
    const float w = inv_freq != nullptr ? inv_freq[d] : 1.0f / powf(theta, (float)(2 * d) / (float)(2 * half_d));
    const int n0 = (blockIdx.x * blockDim.y + threadIdx.y) * kPositions;
    for (int n = n0; n < min(N, n0 + kPositions); ++n) {
        float sn, cs;
        sincosf(__fmul_rn((float)n, w), &sn, &cs);
        const size_t idx = (size_t)n * half_d + d;
        if (PACK) {
            packed[idx] = pack_unorm_pair(cs, sn);
        } else {
            cosT[idx] = cs;
            sinT[idx] = sn;
        }
    }
}

template <bool PACK>
int launch_synth(const float* inv_freq, float theta, float* cos_out, float* sin_out, uint32_t* packed, int N, int half_d, cudaStream_t s) {
    const dim3 block(half_d, 128 / half_d > 0 ? 128 / half_d : 1);
    const int per_block = block.y * kPositions;
    synth_tables_kernel<PACK><<<(unsigned)((N + per_block - 1) / per_block), block, 0, s>>>(inv_freq, theta, cos_out, sin_out, packed, N);
    count_launch();
    return (int)cudaGetLastError();
}

PrepassTable prepass_table(const TableSource& src, uint32_t* packed) {
    PrepassTable t;
    t.cos = src.cos; t.sin = src.sin; t.stride = src.stride; t.packed = packed;
    t.vec = ((uintptr_t)src.cos % 16) == 0 && ((uintptr_t)src.sin % 16) == 0 && src.stride % 4 == 0;
    return t;
}

// Heads per block: as many as still leave about eight blocks per SM, at most eight.
int heads_per_block_for(int position_blocks, int BH) {
    const int64_t want = (int64_t)position_blocks * BH / (sm_count() * 8);
    return want < 1 ? 1 : want > 8 ? 8 : (int)want;
}
int prepass_rows(bool bwd, int D) { return kThreads / (D / (bwd ? 8 : 16)); }   // positions per block

template <typename T, int D, int MODE>
int fwd_prepass_t(const RopeParams& p, const PrepassTable& tab, cudaStream_t s) {
    const int BH = p.B * p.Hkv, hpb = heads_per_block_for(ceil_div(p.N, prepass_rows(false, D)), BH);
    rope_fwd_prepass_kernel<T, D, MODE><<<rope_prepass_grid(false, p.B, p.Hkv, p.N, D).blocks(), kThreads, 0, s>>>((const T*)p.k, (__half*)const_cast<void*>(p.k_rot), tab, p.N, BH, hpb,
                                                                  row_addr(p.sk, p.Hkv, p.N));
    count_launch();
    return (int)cudaGetLastError();
}
template <typename T, int D, int MODE>
int bwd_prepass_t(const RopeParams& p, const PrepassTable& tab, cudaStream_t s) {
    const int BH = p.B * p.H, hpb = heads_per_block_for(ceil_div(p.N, prepass_rows(true, D)), BH);
    rope_bwd_prepass_kernel<T, D, MODE><<<rope_prepass_grid(true, p.B, p.H, p.N, D).blocks(), kThreads, 0, s>>>((const T*)p.q, (const T*)p.o, (const T*)p.d_o, tab,
                                                                  (__half*)const_cast<void*>(p.q_rot), p.delta, p.dq_acc, p.N, BH, hpb,
                                                                  p.sm_scale * kLog2e, row_addr(p.sq, p.H, p.N), row_addr(p.so, p.H, p.N),
                                                                  row_addr(p.sdo, p.H, p.N));
    count_launch();
    return (int)cudaGetLastError();
}

template <typename T, int D>
int prepass_mode(bool bwd, const RopeParams& p, const TableSource& src, uint32_t* packed, cudaStream_t s) {
    const PrepassTable tab = prepass_table(src, packed);
    if (src.packed) return bwd ? bwd_prepass_t<T, D, kPacked>(p, tab, s) : fwd_prepass_t<T, D, kPacked>(p, tab, s);
    if (src.cos) return bwd ? bwd_prepass_t<T, D, kTables>(p, tab, s) : fwd_prepass_t<T, D, kTables>(p, tab, s);
    return bwd ? bwd_prepass_t<T, D, kIdentity>(p, tab, s) : fwd_prepass_t<T, D, kIdentity>(p, tab, s);
}
int prepass(bool bwd, const RopeParams& p, const TableSource& src, uint32_t* packed, int dtype, cudaStream_t s) {
    if (dtype == COROPE_DTYPE_BF16)
        return p.D == 64 ? prepass_mode<__nv_bfloat16, 64>(bwd, p, src, packed, s) : prepass_mode<__nv_bfloat16, 128>(bwd, p, src, packed, s);
    return p.D == 64 ? prepass_mode<__half, 64>(bwd, p, src, packed, s) : prepass_mode<__half, 128>(bwd, p, src, packed, s);
}

}  // namespace

FlatGrid rope_prepass_grid(bool bwd, int B, int H, int N, int D) {
    const unsigned pbs = ceil_div(N, prepass_rows(bwd, D));
    return {pbs, ceil_div(B * H, heads_per_block_for(pbs, B * H))};
}

int launch_rope_fwd_prepass(const RopeParams& p, const TableSource& src, uint32_t* packed, int dtype, cudaStream_t s) {
    return prepass(false, p, src, packed, dtype, s);
}
int launch_rope_bwd_prepass(const RopeParams& p, const TableSource& src, uint32_t* packed, int dtype, cudaStream_t s) {
    return prepass(true, p, src, packed, dtype, s);
}

int launch_pack_tables(const TableSource& src, uint32_t* packed, int N, int half_d, cudaStream_t s) {
    const size_t n = (size_t)N * half_d;
    pack_tables_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(src.cos, src.sin, src.stride, packed, N, half_d);
    count_launch();
    return (int)cudaGetLastError();
}

int launch_synth_tables(const float* inv_freq, float theta, float* cos_out, float* sin_out, int N, int half_d, cudaStream_t s) {
    return launch_synth<false>(inv_freq, theta, cos_out, sin_out, nullptr, N, half_d, s);
}
int launch_synth_packed(const float* inv_freq, float theta, uint32_t* packed, int N, int half_d, cudaStream_t s) {
    return launch_synth<true>(inv_freq, theta, nullptr, nullptr, packed, N, half_d, s);
}

}  // namespace corope
