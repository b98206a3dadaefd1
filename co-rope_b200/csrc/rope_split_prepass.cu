// Pre-pass of the split-operand kernels: K and Q rotated in fp32 and split into three bf16 rows each (of fp32 tensors also V and dO, without
// rotation), for the backward delta = rowsum(O dO), and the work counters of the persistent kernels, in one launch.  Bound by HBM: 8 bytes
// per element of a 16-bit K or Q, 4 more for O and dO; separate launches for K, Q and delta cost a backward of short sequences 8 us more.
#include "rope_split.cuh"

namespace corope {
namespace {

template <typename T> struct Rows {   // rows to split
    const T* x;
    RowAddr at;
    SplitRows out;
    size_t rows;
    float scale;
    int rotate, with_delta, in_lo;   // in_lo: see split3_any
    unsigned end;   // the block behind its last one
};
template <typename T> struct Jobs {
    Rows<T> job[4];
};

// One thread per 8 pairs; the threads of a row are neighbouring lanes.  The blocks of one job follow those of another.
template <typename T, int D>
__global__ void __launch_bounds__(256) split_rows_kernel(const __grid_constant__ Jobs<T> jobs, const float* __restrict__ cosT, const float* __restrict__ sinT,
                                                         int64_t ts, bool vec, const T* __restrict__ o, RowAddr ao, const T* __restrict__ d_o, RowAddr ado,
                                                         float* __restrict__ delta, int* counters) {
    pdl_trigger();
    constexpr int kPerRow = D / 16;
    if (blockIdx.x == 0 && threadIdx.x < 2) counters[threadIdx.x] = 0;
    const int which = (blockIdx.x >= jobs.job[0].end) + (blockIdx.x >= jobs.job[1].end) + (blockIdx.x >= jobs.job[2].end);
    const Rows<T>& in = jobs.job[which];
    const size_t idx = (size_t)(blockIdx.x - (which > 0 ? jobs.job[which - 1].end : 0)) * blockDim.x + threadIdx.x;
    const bool live = idx / kPerRow < in.rows;
    const size_t row = live ? idx / kPerRow : in.rows - 1;   // threads beyond the last row take part in the shuffles with it
    const int d = (int)(idx % kPerRow) * 8, n = (int)(row % (size_t)in.at.N);
    const T* src = in.x + flat_row_offset(in.at, row) + d;
    float2 ra[4], rb[4];
    load8(src, ra);
    load8(src + D / 2, rb);
    if (in.with_delta) {
        const T *po = o + flat_row_offset(ao, row) + d, *pd = d_o + flat_row_offset(ado, row) + d;
        float2 o0[4], o1[4], d0[4], d1[4];
        load8(po, o0);
        load8(po + D / 2, o1);
        load8(pd, d0);
        load8(pd + D / 2, d1);
        float part[8];   // a tree of sums: delta stands against a dP of nearly its size where a row is one-hot
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            part[e] = fmaf(o0[e].x, d0[e].x, o0[e].y * d0[e].y);
            part[4 + e] = fmaf(o1[e].x, d1[e].x, o1[e].y * d1[e].y);
        }
        float sum = ((part[0] + part[1]) + (part[2] + part[3])) + ((part[4] + part[5]) + (part[6] + part[7]));
#pragma unroll
        for (int off = 1; off < kPerRow; off <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
        if (live && d == 0) delta[row] = sum;
    }
    if (in.rotate) {
        float c[8], sn[8];
        load_table8(cosT + (int64_t)n * ts + d, vec, c);
        load_table8(sinT + (int64_t)n * ts + d, vec, sn);
#pragma unroll
        for (int e = 0; e < 4; ++e) rotate(ra[e], rb[e], c + 2 * e, sn + 2 * e);
    }
    if (!live) return;
    uint32_t pa[4][3], pb[4][3];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        split3_any(ra[e].x * in.scale, ra[e].y * in.scale, pa[e], in.in_lo);
        split3_any(rb[e].x * in.scale, rb[e].y * in.scale, pb[e], in.in_lo);
    }
#pragma unroll
    for (int part = 0; part < 3; ++part) {
        __nv_bfloat16* to = in.out.rows + part * in.out.plane + row * D + d;
        *reinterpret_cast<uint4*>(to) = make_uint4(pa[0][part], pa[1][part], pa[2][part], pa[3][part]);
        *reinterpret_cast<uint4*>(to + D / 2) = make_uint4(pb[0][part], pb[1][part], pb[2][part], pb[3][part]);
    }
}

template <typename T, int D>
int launch_t(const RopeParams& p, const SplitCopies& to, bool with_delta, cudaStream_t s) {
    Jobs<T> jobs{};
    unsigned blocks = 0;
    int n = 0;
    auto add = [&](const void* x, const Strides& st, int H, const SplitRows& out, float scale, bool rotated, bool delta, bool in_lo) {
        if (out.rows == nullptr) return;
        Rows<T>& r = jobs.job[n++];
        r = {(const T*)x, row_addr(st, H, p.N), out, (size_t)p.B * H * p.N, scale, rotated && p.cos != nullptr, delta, in_lo, 0};
        r.end = blocks += (unsigned)((r.rows * (D / 16) + 255) / 256);
    };
    add(p.k, p.sk, p.Hkv, to.k, 1.f, true, false, false);
    add(p.q, p.sq, p.H, to.q, p.sm_scale * kLog2e, true, with_delta, false);
    add(p.v, p.sv, p.Hkv, to.v, 1.f, false, false, true);
    add(p.d_o, p.sdo, p.H, to.d_o, 1.f, false, false, true);
    for (; n < 4; ++n) jobs.job[n].end = blocks;
    split_rows_kernel<T, D><<<blocks, 256, 0, s>>>(jobs, p.cos, p.sin, p.table_stride, tables_aligned(p), (const T*)p.o, row_addr(p.so, p.H, p.N), (const T*)p.d_o,
                                                   row_addr(p.sdo, p.H, p.N), p.delta, p.sched_counter);
    count_launch();
    return (int)cudaGetLastError();
}
template <typename T>
int launch_d(const RopeParams& p, const SplitCopies& to, bool with_delta, cudaStream_t s) {
    return p.D == 64 ? launch_t<T, 64>(p, to, with_delta, s) : launch_t<T, 128>(p, to, with_delta, s);
}

}  // namespace

size_t rope_split_workspace_bytes(bool bwd, int B, int Hq, int Hkv, int N, int D, int dtype) {
    size_t heads = (size_t)B * Hkv + (bwd ? (size_t)B * Hq : 0);
    if (dtype == COROPE_DTYPE_F32) heads += (size_t)B * Hkv + (bwd ? (size_t)B * Hq : 0);   // V, dO
    return heads * N * D * 3 * sizeof(__nv_bfloat16);
}
SplitCopies split_copies(const RopeParams& p, void* ws, bool bwd, int dtype) {
    __nv_bfloat16* at = reinterpret_cast<__nv_bfloat16*>(ws);
    auto take = [&](int H) {
        const SplitRows r{at, (size_t)p.B * H * p.N * p.D};
        at += 3 * r.plane;
        return r;
    };
    SplitCopies c{};
    c.k = take(p.Hkv);
    if (bwd) c.q = take(p.H);   // the forward takes Q itself
    if (dtype == COROPE_DTYPE_F32) {
        c.v = take(p.Hkv);
        if (bwd) c.d_o = take(p.H);
    }
    return c;
}

int launch_split_rows(const RopeParams& p, const SplitCopies& to, bool with_delta, int dtype, cudaStream_t s) {
    if (dtype == COROPE_DTYPE_F32) return launch_d<float>(p, to, with_delta, s);
    return dtype == COROPE_DTYPE_BF16 ? launch_d<__nv_bfloat16>(p, to, with_delta, s) : launch_d<__half>(p, to, with_delta, s);
}

}  // namespace corope
