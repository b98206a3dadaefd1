// Shared device/host helpers for the corope_b200 kernels (sm_100a only).
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <utility>

#include "../../include/corope_b200.h"

namespace corope {

constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;

// ---------------------------------------------------------------------------------------------
// element type helpers
// ---------------------------------------------------------------------------------------------
template <typename T> struct Elem;
template <> struct Elem<float> {
    static constexpr int kDtype = COROPE_DTYPE_F32;
    __device__ static float to_f32(float x) { return x; }
    __device__ static float from_f32(float x) { return x; }
};
template <> struct Elem<__nv_bfloat16> {
    static constexpr int kDtype = COROPE_DTYPE_BF16;
    __device__ static float to_f32(__nv_bfloat16 x) { return __bfloat162float(x); }
    __device__ static __nv_bfloat16 from_f32(float x) { return __float2bfloat16_rn(x); }
};
template <> struct Elem<__half> {
    static constexpr int kDtype = COROPE_DTYPE_F16;
    __device__ static float to_f32(__half x) { return __half2float(x); }
    __device__ static __half from_f32(float x) { return __float2half_rn(x); }
};

__host__ __device__ inline size_t dtype_bytes(int dtype) { return dtype == COROPE_DTYPE_F32 ? 4 : 2; }

__host__ __device__ inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

// Strides of a [B, H, N, D] tensor in elements; the head-dim stride is always 1.  Tensor-core paths also need every
// stride to be a multiple of 8 elements (16 bytes, the TMA granularity) -- the entry points check that.
struct Strides {
    int64_t b, h, n;
};
__host__ __device__ inline Strides contiguous_strides(int H, int N, int D) {
    Strides st;
    st.n = D;
    st.h = (int64_t)N * D;
    st.b = (int64_t)H * N * D;
    return st;
}
// rows evenly spaced over heads and batch entries: a 2-D [B H N, D] view with row stride st.n exists
__host__ __device__ inline bool rows_collapse(const Strides& st, int H, int N) { return st.h == (int64_t)N * st.n && st.b == (int64_t)H * st.h; }
// element offset of row n of head-slice bh (= b * H + h) of a tensor with H heads
__host__ __device__ inline int64_t row_offset(const Strides& st, int H, int bh, int n) {
    return (int64_t)(bh / H) * st.b + (int64_t)(bh % H) * st.h + (int64_t)n * st.n;
}

// Addressing of flat row index `row` (= (b * H + h) * N + n) of a strided [B, H, N, D] tensor in the elementwise kernels.  The
// host decides once whether the rows are evenly spaced (every contiguous tensor): then the offset is one multiply; the general
// form costs two integer divisions per thread, which these memory-bound kernels (a few 16-byte accesses per thread) would feel.
struct RowAddr {
    Strides st;
    int H, N;
    int flat;
};
inline RowAddr row_addr(const Strides& st, int H, int N) {
    RowAddr a;
    a.st = st; a.H = H; a.N = N;
    a.flat = rows_collapse(st, H, N) ? 1 : 0;
    return a;
}
__host__ __device__ inline int64_t flat_row_offset(const RowAddr& a, size_t row) {
    if (a.flat) return (int64_t)row * a.st.n;
    const unsigned r = (unsigned)row, bh = r / (unsigned)a.N;   // row counts stay below 2^31 (checked at the entry points)
    return row_offset(a.st, a.H, (int)bh, (int)(r - bh * (unsigned)a.N));
}

// A grid of inner x outer blocks laid out along x alone, inner index fastest: x goes to 2^31 - 1, y and z only to 65 535, which heads
// (up to 2 097 120) and row blocks (N / 16 of them) both exceed.
struct FlatGrid {
    unsigned inner, outer;
    unsigned blocks() const { return inner * outer; }
};
__host__ __device__ inline unsigned ceil_div(unsigned a, unsigned b) { return (a + b - 1) / b; }
// of the kernels that use it (also read by corope_debug_grid)
FlatGrid rope_fp32_fwd_grid(int B, int H, int N);                 // heads x row blocks
FlatGrid rope_fp32_bwd_grid(int B, int H, int Hkv, int N);        // K / V heads x (key block, its query heads' row blocks)
FlatGrid rope_split_fwd_grid(int B, int H, int N);                // heads x row blocks
FlatGrid rope_split_items(int B, int H, int N);                   // heads (of K / V for dK and dV) x 128-row blocks, the items of persistent kernels
FlatGrid rope_prepass_grid(bool bwd, int B, int H, int N, int D); // position blocks x groups of heads

// Launch parameters common to the fused-RoPE kernels.
struct RopeParams {
    const void* q;
    const void* k;
    const void* v;
    const void* o;      // forward output (read by backward)
    const void* d_o;
    void* out_o;        // forward: o
    void* dq;
    void* dk;
    void* dv;
    float* lse2;        // [B,H,N] log2-domain LSE
    float* delta;       // [B,H,N] rowsum(O * dO)
    float* dq_acc;      // [B,H,N,D] fp32 accumulator of rotated-frame dQ (tensor-core backward)
    const float* cos;
    const float* sin;
    int64_t table_stride;
    const uint32_t* packed_tab;  // [N, D/2] (cos, sin) pairs in 16-bit fixed point, built per call in the workspace
    int B, H, N, D;     // H = number of query heads
    int Hkv;            // number of K / V heads (H % Hkv == 0; query head h reads KV head h / (H / Hkv)); equals H for the fused-RoPE ops
    int no_rope;        // 1 = plain attention: no rotation anywhere (cos / sin are null, the packed table holds the identity)
    int causal;
    float sm_scale;
    int* status;
    int* status_mirror; // host memory that a failing kernel copies the status word to, or null
    int* sched_counter; // zeroed word in the workspace: next work item / unit of the persistent tensor-core kernels
    int head_chunk;     // heads per chunk of the persistent kernels' work order (set by their launchers)
    const void* k_rot;  // forward: [B,H,N,D] fp16, K already rotated by the pre-pass; null = the kernel rotates K tiles itself
    const void* q_rot;  // backward: [B,H,N,D] fp16, Q rotated and scaled by the pre-pass; null = the kernel rotates Q tiles itself
    Strides sq, sk, sv, so, sdo, sdq, sdk, sdv;   // strides of q, k, v, o (forward output or backward input), dO, dq, dk, dv
    int flat_q, flat_k, flat_v, flat_do;          // tensor-core kernels: which of their TMA maps are 2-D (set by the launchers)
    int dq_acc_zeroed;  // backward: the pre-pass has already cleared dq_acc (otherwise the launcher of the main kernel does)
};

struct GqaParams {
    const void* q;
    const void* k;
    const void* v;
    const void* o;
    const void* d_o;
    void* out_o;
    void* dq;
    void* dk;
    void* dv;
    float* lse2;     // [B,Hq,N]
    float* a_diag;   // [B,Hkv,N]
    float* delta;    // [B,Hq,N]
    float* dk_acc;   // [B,Hkv,N,D] fp32
    float* dv_acc;   // [B,Hkv,N,D] fp32
    uint32_t* k_pairs;  // tensor-core forward: [B,Hkv,N,D/2] fp16 (k1, k2) pairs in MMA operand order (workspace)
    __half* v_half;     // tensor-core forward: [B,Hkv,N,D] fp16 copy of V (workspace)
    float* k_scale;     // split-operand forward, f16 tensors: [B,Hkv,N] factors that undo the scaling of the rows of k_pairs (workspace)
    int use_mma;        // backward: 1 = tensor-core main kernel (k_pairs / v_half are set), 0 = general kernel
    int B, Hq, Hkv, G, N, D;
    float sm_scale;
    float theta;
    int* status;
    int* status_mirror;   // see RopeParams
    Strides sq, sk, sv, so, sdo, sdq, sdk, sdv;   // strides of q, k, v, o (forward output or backward input), dO, dq, dk, dv
};

#ifdef __CUDACC__
// ---------------------------------------------------------------------------------------------
// mbarrier / TMA / tcgen05 wrappers (inline PTX).  Every wait is bounded.
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void fence_mbar_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0];\n\t}" ::"r"(smem_u32(bar)) : "memory");
}
// One arrival per warp: every lane has finished (and fenced) its part, lane 0 arrives.  Barriers signalled this
// way are initialised with the number of warps, which keeps 128 threads from serialising on one shared word.
__device__ __forceinline__ void mbar_arrive_warp(uint64_t* bar, int lane) {
    __syncwarp();
    if (lane == 0) mbar_arrive(bar);
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Bounded wait.  Returns false (after recording `id` in *status) when the limit is hit; callers
// then leave their loops and fall through to the common exit path.  try_wait itself blocks for
// a hardware-defined slice, so the limit corresponds to well over a second.
constexpr uint32_t kWaitLimit = 1u << 20;
__device__ __forceinline__ bool mbar_wait_limited(uint64_t* bar, uint32_t parity, int* status, int id, volatile int* abort_flag,
                                                  uint32_t limit) {
    for (uint32_t it = 0; it < limit; ++it) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((it & 1023u) == 1023u && *abort_flag) return false;
    }
    *abort_flag = 1;
    if (status) atomicCAS(status, 0, COROPE_DEV_WAIT_EXPIRED | id);
    return false;
}
// A kernel that gave up, or that did not start because an earlier one had, leaves the code in the host mirror too: the host learns of
// every launch that did not compute without a copy or a synchronisation.
__device__ __forceinline__ void report_to_mirror(int code, int* mirror) {
    if (code == 0 || mirror == nullptr) return;
    *reinterpret_cast<volatile int*>(mirror) = code;
    __threadfence_system();
}
__device__ __forceinline__ void report_to_mirror(const int* status, int* mirror) {
    if (status != nullptr) report_to_mirror(*reinterpret_cast<const volatile int*>(status), mirror);
}
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int* status, int id, volatile int* abort_flag) {
    return mbar_wait_limited(bar, parity, status, id, abort_flag, kWaitLimit);
}

// Non-blocking probe of a phase, and a bounded spin on it.  try_wait parks the thread and wakes it some hundreds of
// cycles after the phase completes; the MMA issuer sits on the critical path of every step, so it spins instead
// (one warp; it backs off to try_wait after a while so that a long wait does not burn issue slots).
__device__ __forceinline__ bool mbar_test_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_spin_warp(uint64_t* bar, uint32_t parity, int* status, int id, volatile int* abort_flag) {
    bool done = false;
    for (int it = 0; it < 4096 && !done; ++it) done = mbar_test_wait(bar, parity);
    if (!done) done = mbar_wait(bar, parity, status, id, abort_flag);
    return __all_sync(0xffffffffu, done);
}

// Same, for roles in which all 32 lanes wait: the lanes vote on every poll, so that they leave together and no branch of the loop
// diverges.  A wait whose phase is complete takes 85 cycles; with one vote behind a loop of each lane's own it took 175 (measured on an
// idle SM), which the MMA issuers pay several times per tile.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, int* status, int id, volatile int* abort_flag) {
    if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
    for (uint32_t it = 0; it < kWaitLimit; ++it) {
        if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
        if ((it & 1023u) == 1023u && __any_sync(0xffffffffu, *abort_flag)) return false;
    }
    *abort_flag = 1;
    if (status) atomicCAS(status, 0, COROPE_DEV_WAIT_EXPIRED | id);
    return false;
}

// 2-D tiled TMA load into shared memory, completion on an mbarrier.
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(smem_dst)),
        "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y)
        : "memory");
}
// 4-D tiled TMA load (coordinates: head-dim column, row, head, batch) into shared memory, completion on an mbarrier.
__device__ __forceinline__ void tma_load_4d(void* smem_dst, const CUtensorMap* map, int x, int n, int h, int b, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];" ::"r"(smem_u32(smem_dst)),
        "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(n), "r"(h), "r"(b)
        : "memory");
}
// Row loads of a [B, H, N, D] tensor through either kind of map: `flat` = the tensor's rows are evenly spaced over heads and
// batch entries as well (stride_h = N stride_n, stride_b = H stride_h; every contiguous tensor), so a 2-D map [B H N, D]
// addresses it and one coordinate replaces three; otherwise the 4-D map.  (The 2-D form measured 2 - 10 % faster in the
// backward's Q / dO ring, so it stays the path for the common layout.)
__device__ __forceinline__ void tma_load_rows(void* smem_dst, const CUtensorMap* map, bool flat, int x, int n, int h, int b, int H, int N,
                                              uint64_t* bar) {
    if (flat)
        tma_load_2d(smem_dst, map, x, (b * H + h) * N + n, bar);
    else
        tma_load_4d(smem_dst, map, x, n, h, b, bar);
}
// 1-D bulk copy global -> shared (both 16-byte aligned, size a multiple of 16), completion on an mbarrier.
__device__ __forceinline__ void bulk_load_1d(void* smem_dst, const void* gsrc, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(smem_dst)),
                 "l"(gsrc), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}
// Bulk reduce-add of a dense shared-memory tile into a 2-D tiled global tensor (element type and the add come from the
// tensor map / the instruction: fp32 add).  Completion is tracked with bulk async-groups of the issuing thread.
__device__ __forceinline__ void tma_reduce_add_2d(const CUtensorMap* map, int x, int y, const void* smem_src) {
    asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3}], [%1];" ::"l"(map),
                 "r"(smem_u32(smem_src)), "r"(x), "r"(y)
                 : "memory");
}
__device__ __forceinline__ void bulk_commit_group() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_group_read0() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_group0() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}

// --- tensor memory ---
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_result, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_result)), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() { asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// MMA completion -> mbarrier arrive (implies fence::before_thread_sync).
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// D[tmem] (+)= A[smem desc] * B[smem desc]
__device__ __forceinline__ void umma_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem desc]
__device__ __forceinline__ void umma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
        "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// 128 rows x 32 bytes (one k-step of a 16-bit operand) from a shared-memory tile, described as an A operand, to 8 TMEM columns
__device__ __forceinline__ void tmem_copy_128x256b(uint32_t d_tmem, uint32_t s_lo, uint32_t s_hi) {
    asm volatile(
        "{\n\t.reg .b64 ds;\n\tmov.b64 ds, {%1, %2};\n\t"
        "tcgen05.cp.cta_group::1.128x256b [%0], ds;\n\t}" ::"r"(d_tmem),
        "r"(s_lo), "r"(s_hi)
        : "memory");
}

// Instruction descriptor for kind::f16: fp32 accumulator, A/B formats 0 = f16, 1 = bf16,
// a_mn / b_mn = 1 when the operand's M/N extent (not K) is the contiguous one in memory.
__host__ __device__ constexpr uint32_t make_idesc(int a_fmt, int b_fmt, int a_mn, int b_mn, int M, int N) {
    return (1u << 4) | ((uint32_t)a_fmt << 7) | ((uint32_t)b_fmt << 10) | ((uint32_t)a_mn << 15) | ((uint32_t)b_mn << 16) |
           ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// Shared-memory matrix descriptor, 128-byte swizzle (layout type 2), descriptor version 1.
// lbo / sbo are byte offsets (multiples of 16).
__device__ __forceinline__ uint64_t make_sdesc_sw128(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFFu) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}

// Split form of the same descriptor for the MMA issue loops: a single thread issues every MMA, so the per-MMA
// instruction count is on the critical path (a freshly built 64-bit descriptor per MMA costs ~190 cycles of
// dependent integer work, three times the 64 cycles a 128x128x16 MMA takes to execute).  The high word depends
// only on SBO; the low word is (address >> 4) | (LBO >> 4) << 16, so stepping the start address is one 32-bit add.
__device__ __forceinline__ uint32_t sdesc_lo(uint32_t smem_addr, uint32_t lbo_bytes) {
    return ((smem_addr & 0x3FFFFu) >> 4) | (((lbo_bytes >> 4) & 0x3FFFu) << 16);
}
__host__ __device__ constexpr uint32_t sdesc_hi(uint32_t sbo_bytes) { return ((sbo_bytes >> 4) & 0x3FFFu) | (1u << 14) | (2u << 29); }

__device__ __forceinline__ void umma_ss2(uint32_t d_tmem, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi, uint32_t idesc,
                                         uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\tsetp.ne.b32 p, %6, 0;\n\t"
        "mov.b64 da, {%1, %2};\n\tmov.b64 db, {%3, %4};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p;\n\t}" ::"r"(d_tmem),
        "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void umma_ts2(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t b_hi, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\tsetp.ne.b32 p, %5, 0;\n\t"
        "mov.b64 db, {%2, %3};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t}" ::"r"(d_tmem),
        "r"(a_tmem), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate)
        : "memory");
}

// The same, but only lanes [FROM, TO) of the accumulator are written (the instruction takes one bit per lane that is not).
template <int FROM, int TO>
__device__ __forceinline__ void umma_ts2_lanes(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t b_hi, uint32_t idesc, uint32_t accumulate) {
    auto off = [](int word) {
        uint32_t bits = 0;
        for (int x = 0; x < 32; ++x) bits |= (32 * word + x < FROM || 32 * word + x >= TO ? 1u : 0u) << x;
        return bits;
    };
    constexpr uint32_t m0 = off(0), m1 = off(1), m2 = off(2), m3 = off(3);
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\tsetp.ne.b32 p, %5, 0;\n\t"
        "mov.b64 db, {%2, %3};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, {%6, %7, %8, %9}, p;\n\t}" ::"r"(d_tmem),
        "r"(a_tmem), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate), "r"(m0), "r"(m1), "r"(m2), "r"(m3)
        : "memory");
}

// TMEM <-> registers: 32 lanes x 32-bit, N consecutive columns per thread.
#define COROPE_TMEM_LD32(taddr, r)                                                                                                  \
    asm volatile(                                                                                                                   \
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22," \
        "%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"                                                                              \
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),   \
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),      \
          "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),      \
          "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])                                                                        \
        : "r"(taddr))

#define COROPE_TMEM_ST32(taddr, r)                                                                                                  \
    asm volatile(                                                                                                                   \
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21," \
        "%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),                                                               \
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),   \
        "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]),     \
        "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]),     \
        "r"(r[31])                                                                                                                  \
        : "memory")

#define COROPE_TMEM_LD16(taddr, r)                                                                                                  \
    asm volatile(                                                                                                                   \
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"                     \
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),   \
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])                                              \
        : "r"(taddr))

#define COROPE_TMEM_LD8(taddr, r)                                                                                              \
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"                                      \
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])               \
                 : "r"(taddr))

#define COROPE_TMEM_ST8(taddr, r)                                                                                              \
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]),   \
                 "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])                                              \
                 : "memory")
#define COROPE_TMEM_ST4(taddr, r)                                                                                              \
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]),    \
                 "r"(r[3])                                                                                                     \
                 : "memory")

#define COROPE_TMEM_ST16(taddr, r)                                                                                              \
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr), \
                 "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),       \
                 "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])                                             \
                 : "memory")

__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ void named_bar_sync(int id, int nthreads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory"); }

// Elects one lane of a fully converged warp.  The MMA issuer runs its whole loop warp-uniformly (all 32 lanes wait
// on the barriers and compute the descriptors) and only the issue itself is predicated on the elected lane: the
// same loop inside an `if (lane == 0)` branch issued one MMA every ~210 cycles instead of every 64 (measured).
__device__ __forceinline__ bool elect_one() {
    uint32_t pred;
    asm volatile("{\n\t.reg .b32 rx;\n\t.reg .pred px;\n\telect.sync rx|px, 0xffffffff;\n\tselp.u32 %0, 1, 0, px;\n\t}" : "=r"(pred));
    return pred != 0;
}

// Programmatic dependent launch: a kernel launched by launch_dependent may start once every block of the kernel before it has called
// pdl_trigger (or has ended); what the earlier kernel wrote is there after pdl_wait.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// register re-allocation between warpgroups (all four warps of a warpgroup must execute the same one)
template <int N> __device__ __forceinline__ void reg_alloc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N> __device__ __forceinline__ void reg_dealloc() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }

__device__ __forceinline__ float fmax3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// the same, NaN if one of them is
__device__ __forceinline__ float fmax3_nan(float a, float b, float c) {
    float d;
    asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// Packed pairs of fp32 in one 64-bit register: add / mul / fma on both lanes with one instruction (one issue slot for
// two results; the pipe runs them at half the warp rate of the scalar forms, so the gain is in issue slots).
__device__ __forceinline__ uint64_t f2_pack(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ uint64_t f2_pack_bits(uint32_t lo, uint32_t hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
    return r;
}
__device__ __forceinline__ void f2_unpack(uint64_t v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t f2_sub(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t f2_mul(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// volatile variant: keeps its program order relative to the TMEM loads / stores, which bounds how far the compiler
// can hoist the exponentials of later chunks (and with them the register pressure of the softmax loop)
__device__ __forceinline__ float fast_exp2_ordered(float x) {
    float y;
    asm volatile("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ uint32_t pack_half2(float lo, float hi) {
    __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&h);
}
// two floats -> packed fp16 pair, values beyond the fp16 range saturate to +-65504 instead of becoming inf
__device__ __forceinline__ uint32_t pack_half2_sat(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.satfinite.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}

__device__ __forceinline__ float2 unpack_half2(uint32_t u) {
    __half2 h = *reinterpret_cast<__half2*>(&u);
    return __half22float2(h);
}
__device__ __forceinline__ float2 unpack_bf162(uint32_t u) {
    __nv_bfloat162 h = *reinterpret_cast<__nv_bfloat162*>(&u);
    return __bfloat1622float2(h);
}
__device__ __forceinline__ uint32_t pack_bf162(float lo, float hi) {
    __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&h);
}
// (cos, sin) in [-1, 1] as two 16-bit offset-binary fixed-point numbers u = round((x + 1) * 2^15), clamped to
// 65535 (so +1.0 decodes to 1 - 2^-15; 0 and -1 are exact).  Decoding costs one byte-permute and one FMA per
// value and no conversion instruction: float(0x4B000000 | u) = 2^23 + u exactly.
__device__ __forceinline__ uint32_t pack_unorm_pair(float c, float s) {
    float uc = fminf(fmaxf(rintf((c + 1.f) * 32768.f), 0.f), 65535.f);
    float us = fminf(fmaxf(rintf((s + 1.f) * 32768.f), 0.f), 65535.f);
    return (uint32_t)uc | ((uint32_t)us << 16);
}
__device__ __forceinline__ float2 unpack_unorm_pair(uint32_t u) {
    float lo = __uint_as_float(__byte_perm(u, 0x4B000000u, 0x7410));  // bytes: u.b0, u.b1, 0x00, 0x4B
    float hi = __uint_as_float(__byte_perm(u, 0x4B000000u, 0x7432));  // bytes: u.b2, u.b3, 0x00, 0x4B
    return make_float2(fmaf(lo, 1.f / 32768.f, -257.f), fmaf(hi, 1.f / 32768.f, -257.f));
}
template <typename T> __device__ __forceinline__ float2 unpack2(uint32_t u);
template <> __device__ __forceinline__ float2 unpack2<__nv_bfloat16>(uint32_t u) { return unpack_bf162(u); }
template <> __device__ __forceinline__ float2 unpack2<__half>(uint32_t u) { return unpack_half2(u); }
template <typename T> __device__ __forceinline__ uint32_t pack2(float a, float b);
template <> __device__ __forceinline__ uint32_t pack2<__nv_bfloat16>(float a, float b) { return pack_bf162(a, b); }
template <> __device__ __forceinline__ uint32_t pack2<__half>(float a, float b) { return pack_half2(a, b); }

// In-place half-layout rotation of ROWS rows of a tile held as 128-byte-swizzled boxes of 64 columns; 128 threads, 8 pairs
// (d, d + D/2) per thread and step.  Element (r, c) of a box sits at r*128 + ((c/8) ^ (r%8))*16 + (c%8)*2.
//   D = 128: two boxes, columns [0,64) and [64,128); a pair has the same offset in both; 8 threads per row.
//   D = 64 : one box; the partner of 16-byte chunk u < 4 is chunk u + 4 of the same row, i.e. its swizzled position ^ 4; 4
//            threads per row (two-way bank conflicts, on tiles that are rotated once per work item).
// The result is written as fp16 whatever the input type T.  The packed (cos, sin) rows of the tile (16-bit fixed
// point, see unpack_unorm_pair) are fetched into registers by load_table_regs, which does not depend on the tile
// having landed: callers issue it before waiting for the TMA so that the L2 latency is hidden.
template <int ROWS, int D>
struct TabRegs {
    static constexpr int kRowsPerStep = 128 / (D / 16);
    static constexpr int kSteps = ROWS / kRowsPerStep;
    uint4 t[kSteps * 2];
};

// Table rows row0 .. row0 + ROWS - 1; rows beyond the table (a tile that reaches past the head) repeat its last one.
template <int ROWS, int D>
__device__ __forceinline__ void load_table_regs(TabRegs<ROWS, D>& tr, const uint32_t* __restrict__ tab, int row0, int n_rows, int tid) {
    constexpr int kThreadsPerRow = D / 16;
#pragma unroll
    for (int it = 0; it < TabRegs<ROWS, D>::kSteps; ++it) {
        const int row = it * TabRegs<ROWS, D>::kRowsPerStep + tid / kThreadsPerRow;
        const int u = tid % kThreadsPerRow;
        const int c = D == 128 ? u ^ (row & 7) : u;
        const uint4* tp = reinterpret_cast<const uint4*>(tab + (size_t)min(row0 + row, n_rows - 1) * (D / 2) + c * 8);
        tr.t[2 * it] = __ldg(tp);
        tr.t[2 * it + 1] = __ldg(tp + 1);
    }
}

// Rotation of 8 (x1, x2) pairs held as two 16-byte vectors of T (x1: columns d..d+7, x2: columns d+64..d+71) by the 8
// packed table entries t0, t1; k1 / k0 are the table's decode constants with the output scale folded in.  The result
// is fp16 whatever T.  x1' = x1 c - x2 s,  x2' = x2 c + x1 s  (the reference's rotation, fused_rope_attn.py:96-99).
template <typename T>
__device__ __forceinline__ void rotate_vec8(uint4& x1, uint4& x2, const uint4& t0, const uint4& t1, float k1, float k0) {
    uint32_t a[4] = {x1.x, x1.y, x1.z, x1.w};
    uint32_t b[4] = {x2.x, x2.y, x2.z, x2.w};
    const uint32_t cs[8] = {t0.x, t0.y, t0.z, t0.w, t1.x, t1.y, t1.z, t1.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 fa = unpack2<T>(a[i]), fb = unpack2<T>(b[i]);
        const float c0 = fmaf(__uint_as_float(__byte_perm(cs[2 * i], 0x4B000000u, 0x7410)), k1, k0);
        const float s0 = fmaf(__uint_as_float(__byte_perm(cs[2 * i], 0x4B000000u, 0x7432)), k1, k0);
        const float c1 = fmaf(__uint_as_float(__byte_perm(cs[2 * i + 1], 0x4B000000u, 0x7410)), k1, k0);
        const float s1 = fmaf(__uint_as_float(__byte_perm(cs[2 * i + 1], 0x4B000000u, 0x7432)), k1, k0);
        a[i] = pack_half2_sat(fmaf(fa.x, c0, -fb.x * s0), fmaf(fa.y, c1, -fb.y * s1));
        b[i] = pack_half2_sat(fmaf(fb.x, c0, fa.x * s0), fmaf(fb.y, c1, fa.y * s1));
    }
    x1 = make_uint4(a[0], a[1], a[2], a[3]);
    x2 = make_uint4(b[0], b[1], b[2], b[3]);
}

template <typename T, int ROWS, int D, int BOX_BYTES, int BATCH>
__device__ __forceinline__ void rotate_tile_regs(uint8_t* tile, const TabRegs<ROWS, D>& tr, int tid, float scale) {
    constexpr int kSteps = TabRegs<ROWS, D>::kSteps;
    constexpr int kStepBytes = TabRegs<ROWS, D>::kRowsPerStep * 128;
    constexpr int kBatch = BATCH < kSteps ? BATCH : kSteps;          // rows in flight per thread: loads first, then math, then stores
    const float k1 = scale * (1.f / 32768.f), k0 = -257.f * scale;   // decode constants with the scale folded in
    const int row = tid / (D / 16), u = tid % (D / 16);              // (row & 7) is the same in every step
    uint8_t* p1 = tile + row * 128 + (D == 128 ? u : u ^ (row & 7)) * 16;
    uint8_t* p2 = D == 128 ? p1 + BOX_BYTES : tile + row * 128 + (u ^ (row & 7) ^ 4) * 16;
#pragma unroll
    for (int h = 0; h < kSteps; h += kBatch) {
        uint4 x1[kBatch], x2[kBatch];
#pragma unroll
        for (int v = 0; v < kBatch; ++v) {
            x1[v] = *reinterpret_cast<const uint4*>(p1 + (h + v) * kStepBytes);
            x2[v] = *reinterpret_cast<const uint4*>(p2 + (h + v) * kStepBytes);
        }
#pragma unroll
        for (int v = 0; v < kBatch; ++v) {
            rotate_vec8<T>(x1[v], x2[v], tr.t[2 * (h + v)], tr.t[2 * (h + v) + 1], k1, k0);
        }
#pragma unroll
        for (int v = 0; v < kBatch; ++v) {
            *reinterpret_cast<uint4*>(p1 + (h + v) * kStepBytes) = x1[v];
            *reinterpret_cast<uint4*>(p2 + (h + v) * kStepBytes) = x2[v];
        }
    }
}

#endif  // __CUDACC__

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link-time libcuda dependency); null when unavailable.
typedef CUresult (*TensorMapEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                      const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                      CUtensorMapFloatOOBfill);
inline TensorMapEncodeFn tensor_map_encoder() {
    static const TensorMapEncodeFn fn = [] {
        void* sym = nullptr;
        cudaDriverEntryPointQueryResult qres;
        const cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres);
        return e == cudaSuccess && qres == cudaDriverEntryPointSuccess ? (TensorMapEncodeFn)sym : nullptr;
    }();
    return fn;
}

// A row-major fp32 tensor [rows, cols] without swizzle (box_cols * 4 bytes a multiple of 16, box_cols <= 256): bulk reduce-add of
// dense shared-memory tiles.
inline int encode_tensor_map_f32(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows, uint32_t box_cols) {
    const TensorMapEncodeFn fn = tensor_map_encoder();
    if (!fn) return COROPE_ERR_NO_DEVICE;
    cuuint64_t gdim[2] = {cols, rows};
    cuuint64_t gstride[1] = {cols * 4};
    cuuint32_t box[2] = {box_cols, box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : COROPE_ERR_TENSOR_MAP;
}

int* status_mirror_of(const int* status_word);   // device address of the registered host mirror, or null
// Host costs paid once instead of per launch: the SM count of the current device, and the opt-in to large dynamic shared memory of
// a kernel on it (`done` is a static of the call site, one bit per device).
int sm_count();
template <typename K>
inline int allow_smem(K kernel, size_t bytes, std::atomic<uint64_t>& done) {
    int dev = 0;
    if (cudaError_t e = cudaGetDevice(&dev)) return (int)e;
    const uint64_t bit = 1ull << (dev & 63);
    if (done.load(std::memory_order_relaxed) & bit) return 0;
    if (cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes)) return (int)e;
    done.fetch_or(bit);
    return 0;
}
// Launch whose set-up runs beside the end of the kernel before it in the stream (see pdl_wait).
template <typename... P, typename... A>
inline int launch_dependent(void (*kern)(P...), unsigned grid, unsigned threads, size_t smem, cudaStream_t s, A&&... args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return (int)cudaLaunchKernelEx(&cfg, kern, std::forward<A>(args)...);
}
// Every kernel launch of the library bumps this counter (read through corope_launch_count()).
void count_launch(int n = 1);
// Diagnostics kept by abi.cu (see include/corope_b200_debug.h): which kernel family an op took last, and the policy in force.
void note_kernel_family(int op, int family);
int kernel_policy();

// ---------------------------------------------------------------------------------------------
// host launchers implemented by the kernel translation units (return cudaError_t as int)
// ---------------------------------------------------------------------------------------------
int launch_rope_fwd_general(const RopeParams& p, int dtype, cudaStream_t s);
int launch_rope_bwd_general(const RopeParams& p, int dtype, cudaStream_t s);   // 16-bit types, delta computed before
int launch_rope_bwd_fp32(const RopeParams& p, cudaStream_t s);                 // delta included
int launch_rope_delta(const RopeParams& p, int dtype, cudaStream_t s);
// What the tensor-core kernels need before they run (rope_prepass.cu).
// Where the (cos, sin) pairs of a position come from.
struct TableSource {
    const float* cos = nullptr;      // fp32 tables with row stride `stride`; null (and no packed table) = identity rotation
    const float* sin = nullptr;
    int64_t stride = 0;
    bool packed = false;             // the packed table has already been written (launch_synth_packed)
};
// packed [N, half_d] table alone, + the zeroed work counter behind it
int launch_pack_tables(const TableSource& src, uint32_t* packed, int N, int half_d, cudaStream_t s);
// cos / sin tables [N, half_d] fp32 for positions 0 .. N-1: angle = float(n) * inv_freq[d], inv_freq from the array or, when it
// is null, 1 / theta^(2 d / (2 half_d))
int launch_synth_tables(const float* inv_freq, float theta, float* cos_out, float* sin_out, int N, int half_d, cudaStream_t s);
// the same straight into the packed table, + the zeroed work counter
int launch_synth_packed(const float* inv_freq, float theta, uint32_t* packed, int N, int half_d, cudaStream_t s);
// forward: packed table (unless src.packed) and the rotated fp16 copy of K into p.k_rot
int launch_rope_fwd_prepass(const RopeParams& p, const TableSource& src, uint32_t* packed, int dtype, cudaStream_t s);
// backward: packed table (unless src.packed), delta, the rotated fp16 copy of Q (scaled by sm_scale * log2e) into p.q_rot and a zeroed
// p.dq_acc
int launch_rope_bwd_prepass(const RopeParams& p, const TableSource& src, uint32_t* packed, int dtype, cudaStream_t s);
bool rope_tc_supported(int D, int dtype);   // the tcgen05 kernels: 16-bit types, D = 64 or 128
// 16-byte aligned rows at any N, 16-bit tensors of D = 64 or 128: split operands, `ws` of rope_split_workspace_bytes, two words of workspace
// at p.sched_counter; the backward computes delta
// fp32 tensors on split operands: D = 64, from this length on.  Forward + backward on them / on the CUDA cores: B1 H1 N200 84 / 80 us (as much
// host as GPU time), B2 H4 N300 86 / 94, B4 H8 N512 causal 86 / 261, B1 H8 N1000 100 / 495, B1 H4 N2048 causal 152 / 519.  (D = 128: the
// three parts of K, V and the streamed rows of the backward do not fit a shared memory; those of the forward would, with two stages, which is not
// built.)
inline bool rope_split_fp32(int N, int D, int dtype) { return dtype == COROPE_DTYPE_F32 && D == 64 && N >= 256; }
// Tensors that TMA steps over head by head: a stride of 0 (one head or batch entry shared by all) is none that a tensor map is documented to take.
inline bool no_shared_heads(const Strides& st, int B, int H) { return (B == 1 || st.b > 0) && (H == 1 || st.h > 0); }
size_t rope_split_workspace_bytes(bool bwd, int B, int Hq, int Hkv, int N, int D, int dtype);
int launch_rope_fwd_split(const RopeParams& p, void* ws, int dtype, cudaStream_t s);
int launch_rope_fwd_split_tc(const RopeParams& p, void* ws, int dtype, cudaStream_t s);   // the tcgen05 form of the forward
int launch_rope_bwd_split(const RopeParams& p, void* ws, int dtype, cudaStream_t s);
int launch_rope_fwd_tc(const RopeParams& p, int dtype, cudaStream_t s);
int launch_rope_bwd_tc(const RopeParams& p, int dtype, cudaStream_t s);
bool gqa_fwd_mma_supported(int N, int D, int dtype);
// 16-bit tensors, D = 64 or 128, any N and strides; k_vec / v_vec: rows of k / v are aligned to 16 bytes; p.k_pairs and (without v_vec)
// p.v_half: workspace of 2 B Hkv N D bytes each; f16: p.k_scale, 4 B Hkv N bytes
bool gqa_split_supported(int D, int dtype);
int launch_gqa_fwd_split(const GqaParams& p, bool k_vec, bool v_vec, int dtype, cudaStream_t s);
int launch_gqa_bwd_mma(const GqaParams& p, int dtype, cudaStream_t s);
int launch_gqa_fwd_mma(const GqaParams& p, int dtype, cudaStream_t s);
int launch_gqa_fwd_general(const GqaParams& p, int dtype, cudaStream_t s);
int launch_gqa_bwd_general(const GqaParams& p, int dtype, cudaStream_t s);

// Encodes a 2-D row-major [rows, cols] tensor of 16-bit elements with a [box_rows, box_cols] box and
// 128-byte swizzle (box_cols * 2 bytes must be 128).  Returns 0 on success.
inline int encode_tensor_map_2d_sw128(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows,
                                      uint32_t box_cols, int dtype, uint64_t row_stride_elems = 0) {
    const TensorMapEncodeFn fn = tensor_map_encoder();
    if (!fn) return COROPE_ERR_NO_DEVICE;
    cuuint64_t gdim[2] = {cols, rows};
    cuuint64_t gstride[1] = {(row_stride_elems ? row_stride_elems : cols) * 2};
    cuuint32_t box[2] = {box_cols, box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUtensorMapDataType dt = dtype == COROPE_DTYPE_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    CUresult r = fn(out, dt, 2, const_cast<void*>(base), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : COROPE_ERR_TENSOR_MAP;
}

// The same for a [B, H, N, D] tensor of 16-bit elements with arbitrary batch / head / row strides (multiples of 8 elements):
// a 4-D map with dimensions (D, N, H, B) and a [box_rows, box_cols] box inside one head.  Rows beyond N read as zeros.
inline int encode_tensor_map_4d_sw128(CUtensorMap* out, const void* base, uint64_t B, uint64_t H, uint64_t N, uint64_t D, const Strides& st,
                                      uint32_t box_rows, uint32_t box_cols, int dtype) {
    const TensorMapEncodeFn fn = tensor_map_encoder();
    if (!fn) return COROPE_ERR_NO_DEVICE;
    cuuint64_t gdim[4] = {D, N, H, B};
    // a dimension of extent 1 is never stepped over, but its stride still has to be a valid one
    cuuint64_t gstride[3] = {(cuuint64_t)st.n * 2, (cuuint64_t)(H > 1 ? st.h : st.n * (int64_t)N) * 2, (cuuint64_t)(B > 1 ? st.b : st.n * (int64_t)N) * 2};
    cuuint32_t box[4] = {box_cols, box_rows, 1, 1};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    CUtensorMapDataType dt = dtype == COROPE_DTYPE_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    CUresult r = fn(out, dt, 4, const_cast<void*>(base), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : COROPE_ERR_TENSOR_MAP;
}

// 2-D map when the rows collapse, else 4-D; `flat` tells the kernel which coordinates to use.
inline int encode_rows_map(CUtensorMap* out, bool* flat, const void* base, int B, int H, int N, int D, const Strides& st, uint32_t box_rows,
                           uint32_t box_cols, int dtype) {
    *flat = rows_collapse(st, H, N);
    if (*flat) return encode_tensor_map_2d_sw128(out, base, (uint64_t)B * H * N, D, box_rows, box_cols, dtype, (uint64_t)st.n);
    return encode_tensor_map_4d_sw128(out, base, B, H, N, D, st, box_rows, box_cols, dtype);
}

}  // namespace corope
