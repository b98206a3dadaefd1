// Fused-RoPE / plain attention backward for 16-bit tensors at lengths that are not whole 128-row tiles, D = 64 or 128, at the accuracy of
// fp32 operands: tcgen05 MMAs on operands split into 16-bit parts (rope_split.cuh, rope_split_fwd_sm100.cu).
//
// Two kernels of one form, each sum with one owner and one order (the same bits every time, no fp32 accumulator of dQ in memory):
//     KV = true    owns 128 keys of a K / V head, sweeps 64-row blocks of the queries of its group's heads: dK, dV
//     KV = false   owns 128 queries, sweeps 64-row blocks of the keys: dQ
// Owned rows are the A operands and the TMEM lanes, streamed rows the B operands:
//     S  = own~ str~^T                 5 products of a smaller part into one accumulator, hi hi into another (join_products)
//     dP = V dO^T  (dO V^T)            inputs as they are (fp32 tensors, D = 64: split too, 6 products, as of P dO)
//     dV += P dO                       P in three parts of the inputs' type (f16: times 2^14)
//     dK += dS Q~, (dQ += dS K~)       dS in three bf16 parts: 6 products
// dV and dK / dQ of a block are their own sums in TMEM, which fp32 registers collect.  On the diagonal the MMAs leave out the owned rows that a
// k-step of 16 streamed rows is hidden from (block_product), so that a row with infinities or NaNs only reaches its own group of 16.
//
// Persistent CTAs (one per SM) take items (owned blocks, most work first) from a counter.  640 threads:
//   warp 0      TMA producer: items; the owned rows; ring of stages, each the parts of 64 streamed rotated rows and their plain rows
//   warp 1      MMA issuer and TMEM owner; copies owned operands from a ring stage to TMEM (tcgen05.cp);  warps 2, 3 idle
//   warps 4-19  four groups of 128 threads, thread = owned row; group w has columns [16 w, 16 w + 16) of a block, reads S, writes P over
//               columns of S that it alone reads, reads dP, writes dS likewise; D / 4 columns of dK / dQ and of dV in registers
//
// What bounds it: D = 128, dK and dV: 96 MMAs per block of 64 queries (4750 cycles at a shared-memory port shared with the tiles' arrival) and
// the chain of waits, exponentials and splits between them, which nothing overlaps in the 512 columns: 4.15 us (8160 cycles of 1965
// MHz) per block, 17 us per launch besides.  D = 64: score products overlap the softmax of the block before, 2.06 us per block.  GPU time of forward and
// backward of B1 H32 N1777 D128 bf16 causal 1720 -> 541 us (two mma.sync kernels that form the scores at three parts before), B4 H16 N1000 D64
// bf16 full 1032 -> 353 us, B1 H2 N5999 D128 1826 -> 570 us, B1 H8 N4001 D64 f16 1230 -> 312 us; of the backward of B1 H1 N65 D64 28.5 -> 14.8 us.
// Share of results off the exact rounding before and now (f16, N(0, 1) inputs, B1 H4 N1777 D128 causal): dQ 0.19 / 0.20, dK 0.22 / 0.22, dV 0.22 / 0.22 %; bf16
// dQ 0.057 / 0.044, dK 0.041 / 0.041, dV 0.040 / 0.040 %.  fp32 (B1 H4 N512 D64 causal), CUDA cores / here: dQ 3.6e-7 / 2.5e-7, dK 5.7e-7 /
// 2.7e-7, dV 5.5e-7 / 2.3e-7.
//
// Math: fused-rope/rope_attn_pytorch.py:187-222.
#include "rope_split.cuh"

namespace corope {
namespace {

constexpr int kBM = 128, kBN = 64;
constexpr int kThreads = 640, kComputeWarp0 = 4, kComputeWarps = 16;
constexpr int kLaunchRegs = 96, kRegsCtl = 64, kRegsCompute = 104;
static_assert(128 * (kRegsCtl + 4 * kRegsCompute) <= kThreads * kLaunchRegs, "register budget");
constexpr int kItemSlots = 2, kItemReaders = 1 + kComputeWarps;
constexpr uint32_t kHi = sdesc_hi(1024);

// KP: parts of K~; XP: of V and dO
template <int D, int KP, int XP, bool KV> struct Bwd {
    static constexpr int kOwnParts = KV ? KP : 3, kStrParts = KV ? 3 : KP;
    static constexpr int kTile = kBN * D * 2, kStage = (kStrParts + XP) * kTile;   // 64 streamed rows: parts, then the plain rows
    static constexpr int kOwnTile = kBM * D * 2;
    // S twice where TMEM has room (D = 64): the score products of the next block run beside the softmax of this one
    static constexpr int kBufs = D == 64 ? 2 : 1;
    // owned tiles (parts, then the plain rows): the first kTmemTiles in TMEM, the others in shared memory (where a set for the next item fits)
    static constexpr int kOwnTiles = kOwnParts + XP, kTmemTiles = D == 64 ? (KV ? 0 : 2) : KV ? 1 : 3, kSmemTiles = kOwnTiles - kTmemTiles;
    static constexpr int kOwnSets = D == 64 && XP == 1 ? 2 : 1, kOwnSet = kSmemTiles * kOwnTile;
    static constexpr int kPerStage = kStage / kOwnTile;                            // owned tiles that pass through one stage of the ring
    // dP is summed in two (D = 64), three (dQ) or four (dK, dV) pieces of the head dimension that meet in registers, because the adder of the
    // MMAs truncates: with one sum the share of dQ off the exact rounding grew from 0.19 to 0.21 % (D = 128, f16).  The further pieces have
    // their own columns (D = 64), or those of dK / dQ and dV between the collection of the block before and the products of this one.
    // Parts of V and dO (XP = 3): hi hi is one piece, the smaller products are the other.
    static constexpr bool kOwnPieces = D == 64;
    static constexpr int kPieces = D == 64 ? 2 : KV ? 4 : 3;
    static_assert(XP == 1 || D == 64, "pieces of dP");
    __host__ __device__ static constexpr int piece_end(int i) { return D == 64 || KV ? 2 * (i + 1) : i < 2 ? 3 * (i + 1) : 8; }   // k-steps
    __host__ __device__ static constexpr int piece_col(int i) { return i == 0 ? kDP : (kOwnPieces ? kDP + 64 * i : kAcc + 64 * (i - 1)); }   // dV follows dK
    enum Bar { ITEM_FULL = 0, ITEM_EMPTY = ITEM_FULL + kItemSlots, S_FULL = ITEM_EMPTY + kItemSlots, DP_FULL = S_FULL + 2, P_READY, DS_READY, ACC_FULL, ACC_READ, OWN_FULL, OWN_EMPTY = OWN_FULL + 2, FULL = OWN_EMPTY + 2 };
    static constexpr size_t kSlots = kComputeWarps * 32 * sizeof(float), kSlack = 512, kFixed = kSlots + 256 + 32 + kSlack;
    static constexpr int kFit = (int)((232448 - kFixed - (size_t)kOwnSets * kOwnSet) / kStage), kStages = kFit < 5 ? kFit : 5;
    static constexpr int EMPTY = FULL + kStages, NUM_BARS = EMPTY + kStages;
    static_assert(NUM_BARS * 8 <= 256 && kStages >= 2, "shared memory budget");
    static constexpr size_t kSmem = (size_t)kStages * kStage + (size_t)kOwnSets * kOwnSet + kFixed;
    // TMEM columns: per buffer S (hi hi | the rest); dP; dK or dQ, dV, owned operands
    static constexpr int kBuf = 128, kDP = kBufs * kBuf, kAcc = kDP + (kOwnPieces ? 128 : 64), kDV = kAcc + D, kOwn = kAcc + (KV ? 2 : 1) * D;
    static_assert(kOwn + kTmemTiles * (D / 2) <= 512, "TMEM columns");
    // 8-column operands of k-step w (16 streamed rows) over the columns of S and dP that group w reads
    __host__ __device__ static constexpr int p_col(int buf, int part, int w) { return buf * kBuf + (part == 2 ? 64 : part * 8) + 16 * w; }
    __host__ __device__ static constexpr int ds_col(int buf, int part, int w) { return (part == 0 ? buf * kBuf + 72 : kDP + (part - 1) * 8) + 16 * w; }
};

struct WorkItem {
    int t, head;
};
__device__ __forceinline__ WorkItem work_item(int w, int n_blocks, int heads, int head_chunk, bool last_first) {
    const int chunk_items = head_chunk * n_blocks, chunk = w / chunk_items, within = w % chunk_items;
    const int heads_here = min(head_chunk, heads - chunk * head_chunk), t = within / heads_here;
    return {last_first ? n_blocks - 1 - t : t, chunk * head_chunk + within % heads_here};
}

template <typename T, int D, int KP, bool KV>
__global__ void __launch_bounds__(kThreads, 1)
rope_bwd_split_sm100_kernel(const __grid_constant__ CUtensorMap mapOwn, const __grid_constant__ CUtensorMap mapOwnX, const __grid_constant__ CUtensorMap mapStr,
                            const __grid_constant__ CUtensorMap mapStrX, const __grid_constant__ RopeParams p) {
    constexpr int XP = Plain<T>::kParts;
    using W = Bwd<D, KP, XP, KV>;
    constexpr int ST = W::kStages, OP = W::kOwnParts, SP = W::kStrParts;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* sOwn = sm + ST * W::kStage;
    float* slots = reinterpret_cast<float*>(sOwn + W::kOwnSets * W::kOwnSet);   // [warp][lse of 16 streamed rows | delta]
    uint64_t* bars = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(slots) + W::kSlots);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 32);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    volatile int* item_ring = reinterpret_cast<volatile int*>(tmem_slot + 2);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int N = p.N, G = p.H / p.Hkv, heads = p.B * (KV ? p.Hkv : p.H);
    const int n_own = (N - 1) / kBM + 1, n_items = n_own * heads, nb_all = (N - 1) / kBN + 1;
    const bool causal = p.causal != 0;
    auto item_of = [&](int w) { return work_item(w, n_own, heads, p.head_chunk, !KV); };
    auto first_of = [&](int t) { return KV && causal ? 2 * t : 0; };                               // first streamed block
    auto steps_of = [&](int t) { return KV ? nb_all - first_of(t) : causal ? min(nb_all, 2 * t + 2) : nb_all; };   // streamed blocks (KV: of each query head)

    if (reinterpret_cast<uintptr_t>(sm) - reinterpret_cast<uintptr_t>(smem_raw) > W::kSlack) {   // base less aligned than assumed
        if (threadIdx.x == 0 && p.status) {
            atomicCAS(p.status, 0, COROPE_DEV_WAIT_EXPIRED | 0xfff);
            report_to_mirror(COROPE_DEV_WAIT_EXPIRED | 0xfff, p.status_mirror);
        }
        pdl_wait();
        return;
    }
    if (p.status != nullptr) {   // an earlier launch gave up on a wait: see rope_fwd_sm100_kernel
        // one answer for the whole block: a launch beside this one may set the word while its threads read it
        if (__syncthreads_or(*reinterpret_cast<volatile int*>(p.status))) {
            if (threadIdx.x == 0) report_to_mirror(p.status, p.status_mirror);
            pdl_wait();
            return;
        }
    }
    if (threadIdx.x == 0) {
        *abort_flag = 0;
        for (int i = 0; i < ST; ++i) {
            mbar_init(&bars[W::FULL + i], 1);
            mbar_init(&bars[W::EMPTY + i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&bars[W::S_FULL + i], 1);
            mbar_init(&bars[W::OWN_FULL + i], 1);
            mbar_init(&bars[W::OWN_EMPTY + i], 1);
        }
        mbar_init(&bars[W::DP_FULL], 1);
        mbar_init(&bars[W::P_READY], kComputeWarps);
        mbar_init(&bars[W::DS_READY], kComputeWarps);
        mbar_init(&bars[W::ACC_FULL], 1);
        mbar_init(&bars[W::ACC_READ], kComputeWarps);
        for (int i = 0; i < kItemSlots; ++i) {
            mbar_init(&bars[W::ITEM_FULL + i], 1);
            mbar_init(&bars[W::ITEM_EMPTY + i], kItemReaders);
        }
        fence_mbar_init();
        tma_prefetch_desc(&mapOwn);
        tma_prefetch_desc(&mapOwnX);
        tma_prefetch_desc(&mapStr);
        tma_prefetch_desc(&mapStrX);
    }
    __syncthreads();
    if (warp == 1) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    // KV: split rows, delta, counters.  The other kernel reads nothing of the KV one, which has waited for all of that before its blocks
    // made way for this launch: it fills the SMs that the KV kernel leaves idle, and only ends after it.
    if (KV) {
        pdl_wait();
        pdl_trigger();
    }
    // the n-th item of this CTA, or -1 when there is none left (or a wait gave up); one arrival per warp
    auto fetch_item = [&](int n) {
        const int slot = n % kItemSlots;
        if (!mbar_wait_warp(&bars[W::ITEM_FULL + slot], (n / kItemSlots) & 1, p.status, W::ITEM_FULL, abort_flag)) return -1;
        const int w = item_ring[slot];
        mbar_arrive_warp(&bars[W::ITEM_EMPTY + slot], lane);
        return w;
    };

    if (warp < kComputeWarp0) {
        reg_dealloc<kRegsCtl>();
        if (warp == 0) {
            // -------------------------------------------------------------- TMA producer
            if (lane == 0) {
                int g = 0;   // stages filled
                bool ok = true;
                auto stage_free = [&]() { return g < ST || (ok = mbar_wait(&bars[W::EMPTY + g % ST], ((g / ST) - 1) & 1, p.status, W::EMPTY, abort_flag)); };
                // 128 owned rows: tile `i` (parts, then the plain rows)
                auto load_own = [&](uint8_t* dst, int i, int row, int head, int b, int h, uint64_t* bar) {
#pragma unroll
                    for (int c = 0; c < D / 64; ++c)
#pragma unroll
                        for (int half = 0; half < 2; ++half) {
                            uint8_t* to = dst + c * (kBM * 128) + half * (kBN * 128);
                            if (i < OP)
                                tma_load_4d(to, &mapOwn, c * 64, row + half * kBN, head, i, bar);
                            else   // the copies of fp32 rows are laid out as the rotated ones
                                tma_load_4d(to, &mapOwnX, c * 64, row + half * kBN, XP > 1 ? head : h, XP > 1 ? i - OP : b, bar);
                        }
                };
                for (int n = 0; ok; ++n) {
                    const int slot = n % kItemSlots;
                    if (n >= kItemSlots && !(ok = mbar_wait(&bars[W::ITEM_EMPTY + slot], ((n / kItemSlots) - 1) & 1, p.status, W::ITEM_EMPTY, abort_flag))) break;
                    int w = n == 0 ? (int)blockIdx.x : (int)gridDim.x + atomicAdd(p.sched_counter, 1);
                    if (w >= n_items) w = -1;
                    item_ring[slot] = w;
                    mbar_arrive(&bars[W::ITEM_FULL + slot]);
                    if (w < 0) break;
                    const WorkItem wi = item_of(w);
                    const int own0 = wi.t * kBM, H_own = KV ? p.Hkv : p.H, ob = wi.head / H_own, oh = wi.head % H_own;
                    // owned tiles for TMEM pass through the ring
                    for (int i = 0; i < W::kTmemTiles; i += W::kPerStage, ++g) {
                        if (!stage_free()) break;
                        const int count = min(W::kPerStage, W::kTmemTiles - i);
                        uint64_t* bar = &bars[W::FULL + g % ST];
                        mbar_arrive_expect_tx(bar, count * W::kOwnTile);
                        for (int x = 0; x < count; ++x) load_own(sm + (g % ST) * W::kStage + x * W::kOwnTile, i + x, own0, wi.head, ob, oh, bar);
                    }
                    if (!ok) break;
                    if (W::kSmemTiles > 0) {
                        const int set = n % W::kOwnSets, use = n / W::kOwnSets;
                        if (use > 0 && !(ok = mbar_wait(&bars[W::OWN_EMPTY + set], (use - 1) & 1, p.status, W::OWN_EMPTY, abort_flag))) break;
                        mbar_arrive_expect_tx(&bars[W::OWN_FULL + set], W::kOwnSet);
                        for (int x = 0; x < W::kSmemTiles; ++x)
                            load_own(sOwn + set * W::kOwnSet + x * W::kOwnTile, W::kTmemTiles + x, own0, wi.head, ob, oh, &bars[W::OWN_FULL + set]);
                    }
                    const int first = first_of(wi.t), steps = steps_of(wi.t);
                    for (int hq = 0; hq < (KV ? G : 1) && ok; ++hq) {
                        const int head = KV ? wi.head * G + hq : wi.head / G, H_str = KV ? p.H : p.Hkv, sb = head / H_str, sh = head % H_str;
                        for (int j = 0; j < steps; ++j, ++g) {
                            if (!stage_free()) break;
                            uint8_t* dst = sm + (g % ST) * W::kStage;
                            uint64_t* bar = &bars[W::FULL + g % ST];
                            const int r = (first + j) * kBN;
                            mbar_arrive_expect_tx(bar, W::kStage);
#pragma unroll
                            for (int c = 0; c < D / 64; ++c) {
#pragma unroll
                                for (int part = 0; part < SP; ++part) tma_load_4d(dst + part * W::kTile + c * (kBN * 128), &mapStr, c * 64, r, head, part, bar);
#pragma unroll
                                for (int part = 0; part < XP; ++part)
                                    tma_load_4d(dst + (SP + part) * W::kTile + c * (kBN * 128), &mapStrX, c * 64, r, XP > 1 ? head : sh, XP > 1 ? part : sb, bar);
                            }
                        }
                    }
                }
            }
            __syncwarp();
        } else if (warp == 1) {
            // -------------------------------------------------------------- MMA issuer
            const bool leader = elect_one();
            constexpr int kFmt = Plain<T>::kDtype == COROPE_DTYPE_F16 ? 0 : 1;
            const uint32_t idesc_s = make_idesc(1, 1, 0, 0, kBM, kBN), idesc_dp = make_idesc(kFmt, kFmt, 0, 0, kBM, kBN);
            const uint32_t idesc_acc = make_idesc(1, 1, 0, 1, kBM, D), idesc_dv = make_idesc(kFmt, kFmt, 0, 1, kBM, D);
            const uint32_t stage_lo = sdesc_lo(smem_u32(sm), 0), own_lo = sdesc_lo(smem_u32(sOwn), 0);
            constexpr uint32_t kLbo = (uint32_t)(kBN * 128 >> 4) << 16;   // streamed rows as the K dimension: next 64 columns of the head dimension
            int gs = 0, gb = 0, g = 0;   // stages, blocks whose scores / whose gradients have been issued so far
            bool ok = true;
            // owned tile `op` times streamed tile `sp` (both with the head dimension as K), k-steps [k0, k1)
            auto scores = [&](int op, int sp, uint32_t d, uint32_t st_lo, uint32_t set_lo, uint32_t idesc, bool first, int k0, int k1) {
#pragma unroll
                for (int kk = k0; kk < k1; ++kk) {
                    const uint32_t b = st_lo + ((sp * W::kTile + (kk >> 2) * (kBN * 128) + (kk & 3) * 32) >> 4), acc = (first && kk == k0) ? 0u : 1u;
                    if (op < W::kTmemTiles) {
                        if (leader) umma_ts2(d, tmem + W::kOwn + op * (D / 2) + kk * 8, b, kHi, idesc, acc);
                    } else {
                        const uint32_t a = set_lo + (((op - W::kTmemTiles) * W::kOwnTile + (kk >> 2) * (kBM * 128) + (kk & 3) * 32) >> 4);
                        if (leader) umma_ss2(d, a, kHi, b, kHi, idesc, acc);
                    }
                }
            };
            constexpr int KS = D / 16;
            auto issue_s = [&](uint32_t set_lo) {
                const int st = gs % ST, buf = gb % W::kBufs;
                if (!(ok = mbar_wait_warp(&bars[W::FULL + st], (gs / ST) & 1, p.status, W::FULL, abort_flag))) return;
                tc_fence_after();
                const uint32_t st_lo = stage_lo + st * (W::kStage >> 4), s0 = tmem + buf * W::kBuf;
                scores(1, 1, s0 + 64, st_lo, set_lo, idesc_s, true, 0, KS);
                if (SP > 2) scores(0, 2, s0 + 64, st_lo, set_lo, idesc_s, false, 0, KS);
                if (OP > 2) scores(2, 0, s0 + 64, st_lo, set_lo, idesc_s, false, 0, KS);
                scores(0, 1, s0 + 64, st_lo, set_lo, idesc_s, false, 0, KS);
                scores(1, 0, s0 + 64, st_lo, set_lo, idesc_s, false, 0, KS);
                scores(0, 0, s0, st_lo, set_lo, idesc_s, true, 0, KS);
                if (leader) umma_commit(&bars[W::S_FULL + buf]);
            };
            auto issue_dp = [&](uint32_t set_lo) {   // of the block of the last issue_s
                const uint32_t st_lo = stage_lo + (gs % ST) * (W::kStage >> 4);
                if constexpr (XP > 1) {
#pragma unroll
                    for (int i = 0; i + 1 < kProducts; ++i)
                        scores(OP + product_a(i), SP + product_b(i), tmem + W::piece_col(1), st_lo, set_lo, idesc_dp, i == 0, 0, KS);
                    scores(OP, SP, tmem + W::piece_col(0), st_lo, set_lo, idesc_dp, true, 0, KS);
                } else {
                    scores(OP, SP, tmem + W::piece_col(0), st_lo, set_lo, idesc_dp, true, 0, W::piece_end(0));
                    if (!W::kOwnPieces && gb > 0) {
                        if (!(ok = mbar_wait_warp(&bars[W::ACC_READ], (gb - 1) & 1, p.status, W::ACC_READ, abort_flag))) return;
                        tc_fence_after();
                    }
#pragma unroll
                    for (int i = 1; i < W::kPieces; ++i) scores(OP, SP, tmem + W::piece_col(i), st_lo, set_lo, idesc_dp, true, W::piece_end(i - 1), W::piece_end(i));
                }
                if (leader) umma_commit(&bars[W::DP_FULL]);
                ++gs;
                ++gb;
            };
            for (int n = 0; ok; ++n) {
                const int w = fetch_item(n);
                if (w < 0) break;
                const int t = item_of(w).t, steps = steps_of(t), nb = steps * (KV ? G : 1), set = n % W::kOwnSets;
                const uint32_t set_lo = own_lo + set * (W::kOwnSet >> 4);
                if (W::kTmemTiles > 0 && g > 0 && !(ok = mbar_wait_warp(&bars[W::ACC_FULL], (g - 1) & 1, p.status, W::ACC_FULL, abort_flag))) break;   // the owned operands in TMEM are free
                for (int i = 0; i < W::kTmemTiles; i += W::kPerStage, ++gs) {
                    const int st = gs % ST;
                    if (!(ok = mbar_wait_warp(&bars[W::FULL + st], (gs / ST) & 1, p.status, W::FULL, abort_flag))) break;
                    tc_fence_after();
                    for (int x = 0; x < min(W::kPerStage, W::kTmemTiles - i); ++x)
#pragma unroll
                        for (int kk = 0; kk < D / 16; ++kk)
                            if (leader)
                                tmem_copy_128x256b(tmem + W::kOwn + (i + x) * (D / 2) + kk * 8,
                                                   stage_lo + ((st * W::kStage + x * W::kOwnTile + (kk >> 2) * (kBM * 128) + (kk & 3) * 32) >> 4), kHi);
                    if (leader) umma_commit(&bars[W::EMPTY + st]);
                }
                if (!ok) break;
                if (W::kSmemTiles > 0 && !(ok = mbar_wait_warp(&bars[W::OWN_FULL + set], (n / W::kOwnSets) & 1, p.status, W::OWN_FULL, abort_flag))) break;
                int grad_stage = gs % ST;
                issue_s(set_lo);
                if (ok) issue_dp(set_lo);
                int left = nb;
                auto block = [&](auto where) {
                    const bool more = --left > 0;
                    if (W::kBufs == 2 && more) {
                        issue_s(set_lo);
                        if (!ok) return;
                    }
                    const uint32_t t_lo = stage_lo + grad_stage * (W::kStage >> 4) + kLbo;
                    const int buf = g % W::kBufs;
                    auto product = [&](uint32_t d, auto a_col, int sp, uint32_t idesc, bool start) {
                        block_product<KV>(where, leader, d, [&](int kk) { return tmem + a_col(kk); }, [&](int kk) { return t_lo + ((sp * W::kTile + kk * 2048) >> 4); }, kHi, idesc, start);
                    };
                    if (KV) {
                        if (!(ok = mbar_wait_warp(&bars[W::P_READY], g & 1, p.status, W::P_READY, abort_flag))) return;
                        tc_fence_after();
#pragma unroll
                        for (int i = 0; i < (XP > 1 ? kProducts : 3); ++i)   // small parts first
                            product(tmem + W::kDV, [&](int kk) { return W::p_col(buf, XP > 1 ? product_a(i) : 2 - i, kk); }, SP + (XP > 1 ? product_b(i) : 0), idesc_dv, i == 0);
                    }
                    if (!(ok = mbar_wait_warp(&bars[W::DS_READY], g & 1, p.status, W::DS_READY, abort_flag))) return;
                    tc_fence_after();
                    auto gradient = [&](int dp, int sp, bool start) { product(tmem + W::kAcc, [&](int kk) { return W::ds_col(buf, dp, kk); }, sp, idesc_acc, start); };
                    gradient(1, 1, true);
                    if (SP > 2) gradient(0, 2, false);
                    gradient(2, 0, false);
                    gradient(0, 1, false);
                    gradient(1, 0, false);
                    gradient(0, 0, false);
                    if (leader) umma_commit(&bars[W::ACC_FULL]);
                    if (leader) umma_commit(&bars[W::EMPTY + grad_stage]);
                    grad_stage = grad_stage + 1 == ST ? 0 : grad_stage + 1;
                    ++g;
                    if (W::kBufs == 1 && more) issue_s(set_lo);
                    if (ok && more) issue_dp(set_lo);
                };
                // the blocks on the diagonal, a sweep's first two (keys) or last two (queries), stand outside the loop: see the forward
                for (int sweep = 0; sweep < (KV ? G : 1) && ok; ++sweep) {
                    const int whole = !causal ? steps : KV ? max(steps - 2, 0) : 2 * t, diagonal = steps - whole;
                    if (KV && diagonal > 0) block(FirstOnDiagonal{});
                    if (KV && diagonal > 1 && ok) block(SecondOnDiagonal{});
                    for (int x = 0; x < whole && ok; ++x) block(WholeBlock{});
                    if (!KV && diagonal > 0 && ok) block(FirstOnDiagonal{});
                    if (!KV && diagonal > 1 && ok) block(SecondOnDiagonal{});
                }
                if (W::kSmemTiles > 0 && leader) umma_commit(&bars[W::OWN_EMPTY + set]);
            }
            __syncwarp();
        }
    } else {
        // ------------------------------------------------------------------ P, dS, sums of the gradients
        reg_alloc<kRegsCompute>();
        const int wg = (warp - kComputeWarp0) >> 2, quad = warp & 3;   // the TMEM lane quadrant a warp may touch is warp_id % 4
        const int row = quad * 32 + lane;
        const uint32_t lanes = tmem + ((uint32_t)(quad * 32) << 16);
        constexpr int E = D / 8;                                       // columns [wg E, wg E + E) and the same of the other half: rotation pairs
        float* slot = slots + (warp - kComputeWarp0) * 32;
        const bool table_vec = tables_aligned(p);
        int g = 0;                                                     // blocks so far
        bool ok = true;
        uint64_t acc[2][E / 2], dv[2][KV ? E / 2 : 1];
        // words of an operand chunk (two columns of S or dP each) that are formed at a time: half of them where dV and dK take 64 registers
        constexpr int kPasses = D == 128 && KV ? 2 : 1, kWords = 8 / kPasses;
        auto store_words = [&](uint32_t col, const uint32_t (&r)[kWords]) {
            if constexpr (kPasses == 2)
                COROPE_TMEM_ST4(col, r);
            else
                COROPE_TMEM_ST8(col, r);
        };
        auto add_columns = [&](uint32_t col, uint64_t (&to)[E / 2]) {
            uint32_t r[E];
            if constexpr (D == 128)
                COROPE_TMEM_LD16(lanes + col, r);
            else
                COROPE_TMEM_LD8(lanes + col, r);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < E / 2; ++i) to[i] = f2_add(to[i], f2_pack_bits(r[2 * i], r[2 * i + 1]));
        };
        // Nothing is added where none of the warp's owned rows has a part in the block (`seen`): their products have not been formed.  Keys: in the
        // first block of a sweep; queries: in the last one.
        auto collect = [&](int block, bool seen) {
            if (!(ok = mbar_wait_warp(&bars[W::ACC_FULL], block & 1, p.status, W::ACC_FULL, abort_flag))) return;
            tc_fence_after();
            if (seen) {
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    add_columns(W::kAcc + half * (D / 2) + wg * E, acc[half]);
                    if constexpr (KV) add_columns(W::kDV + half * (D / 2) + wg * E, dv[half]);
                }
            }
            tc_fence_before();
            if (!W::kOwnPieces) mbar_arrive_warp(&bars[W::ACC_READ], lane);
        };
        for (int n = 0; ok; ++n) {
            const int w = fetch_item(n);
            if (w < 0) break;
            const WorkItem wi = item_of(w);
            const int own0 = wi.t * kBM, pos = own0 + row, steps = steps_of(wi.t), nb = steps * (KV ? G : 1), r_first = first_of(wi.t) * kBN;
            float lse = 0.f, delta = 0.f;   // of the owned query
            if (!KV) {
                lse = pos < N ? p.lse2[(size_t)wi.head * N + pos] : INFINITY;   // P = 0 beyond the head
                delta = pos < N ? p.delta[(size_t)wi.head * N + pos] : 0.f;
            }
            // lse (lanes 0-15) and delta (16-31) of this group's 16 streamed queries of step j, one step ahead
            auto stream_stat = [&](int j) {
                const int q = r_first + (j % steps) * kBN + wg * 16 + (lane & 15);
                const size_t at = (size_t)(wi.head * G + j / steps) * N + q;
                return lane < 16 ? (q < N ? p.lse2[at] : INFINITY) : (q < N ? p.delta[at] : 0.f);
            };
            bool seen = true;   // the block before
            float stat = KV ? stream_stat(0) : 0.f;
#pragma unroll
            for (int half = 0; half < 2; ++half)
#pragma unroll
                for (int i = 0; i < E / 2; ++i) {
                    acc[half][i] = 0;
                    if constexpr (KV) dv[half][i] = 0;
                }
            for (int j = 0; j < nb; ++j, ++g) {
                const int buf = g % W::kBufs;
                const uint32_t tS = lanes + buf * W::kBuf;
                if (W::kBufs == 1 && j > 0) {
                    collect(g - 1, seen);
                    if (!ok) break;
                }
                if (KV) {
                    __syncwarp();
                    slot[lane] = stat;
                    __syncwarp();
                    if (j + 1 < nb) stat = stream_stat(j + 1);
                }
                if (!(ok = mbar_wait_warp(&bars[W::S_FULL + buf], (g / W::kBufs) & 1, p.status, W::S_FULL, abort_flag))) break;
                tc_fence_after();
                const int str0 = r_first + (KV ? j % steps : j) * kBN + wg * 16;   // this group's first streamed row
                float s[16];
                {
                    uint32_t main[16], small[16];
                    COROPE_TMEM_LD16(tS + wg * 16, main);
                    COROPE_TMEM_LD16(tS + 64 + wg * 16, small);
                    tmem_wait_ld();
#pragma unroll
                    for (int i = 0; i < 8; ++i) f2_unpack(join_products<D>(f2_pack_bits(main[2 * i], main[2 * i + 1]), f2_pack_bits(small[2 * i], small[2 * i + 1])), s[2 * i], s[2 * i + 1]);
                }
                float nan0 = 0.f, nan1 = 0.f;
#pragma unroll
                for (int i = 0; i < 16; i += 4) nan0 = fmax3_nan(nan0, s[i], s[i + 1]), nan1 = fmax3_nan(nan1, s[i + 2], s[i + 3]);
                if (__any_sync(0xffffffffu, nan0 != nan0 || nan1 != nan1)) infinite_scores(tS + wg * 16, s);   // infinities or NaNs among the operands
#pragma unroll
                for (int i = 0; i < 16; i += 4) {
                    const float4 l = KV ? *reinterpret_cast<const float4*>(slot + i) : make_float4(lse, lse, lse, lse);
                    s[i] = fast_exp2(s[i] - l.x), s[i + 1] = fast_exp2(s[i + 1] - l.y), s[i + 2] = fast_exp2(s[i + 2] - l.z), s[i + 3] = fast_exp2(s[i + 3] - l.w);
                }
                // pairs that are not seen, rows beyond the head
                const int block0 = str0 - wg * 16;
                if (block0 > N - kBN || (causal && (KV ? block0 < own0 + quad * 32 + 31 : block0 + kBN - 1 > own0 + quad * 32))) {
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const int str = str0 + i;
                        if (str >= N || (causal && (KV ? str < pos : str > pos))) s[i] = 0.f;
                    }
                }
                if (KV) {
#pragma unroll
                    for (int h = 0; h < kPasses; ++h) {
                        uint32_t parts[3][kWords];
#pragma unroll
                        for (int i = 0; i < kWords; ++i) {
                            uint32_t y[3];
                            const int c = 2 * (h * kWords + i);
                            split3_cut<typename Plain<T>::Mma>(s[c] * kPScale<T>, s[c + 1] * kPScale<T>, y);
                            parts[0][i] = y[0], parts[1][i] = y[1], parts[2][i] = y[2];
                        }
#pragma unroll
                        for (int part = 0; part < 3; ++part) store_words(lanes + W::p_col(buf, part, wg) + h * kWords, parts[part]);
                    }
                    tmem_wait_st();
                }
                if (!(ok = mbar_wait_warp(&bars[W::DP_FULL], g & 1, p.status, W::DP_FULL, abort_flag))) break;
                tc_fence_after();
                float dp[16];   // pieces of it may sit in columns of dV: P is handed over behind these reads
#pragma unroll
                for (int h = 0; h < kPasses; ++h) {
                    constexpr int kCols = 16 / kPasses;
#pragma unroll
                    for (int c = 0; c < W::kPieces; ++c) {
                        uint32_t r[kCols];
                        if constexpr (kPasses == 2)
                            COROPE_TMEM_LD8(lanes + W::piece_col(c) + wg * 16 + h * kCols, r);
                        else
                            COROPE_TMEM_LD16(lanes + W::piece_col(c) + wg * 16 + h * kCols, r);
                        tmem_wait_ld();
#pragma unroll
                        for (int i = 0; i < kCols; i += 2) {
                            float &d0 = dp[h * kCols + i], &d1 = dp[h * kCols + i + 1];
                            const uint64_t x = f2_pack_bits(r[i], r[i + 1]);
                            f2_unpack(c == 0 ? x : XP > 1 ? join_products<D>(f2_pack(d0, d1), x) : f2_add(f2_pack(d0, d1), x), d0, d1);
                        }
                    }
                }
                if (KV) {
                    if (W::kBufs == 2 && j > 0) {   // dV and dK of the block before leave TMEM to this one
                        collect(g - 1, seen);
                        if (!ok) break;
                    }
                    tc_fence_before();
                    mbar_arrive_warp(&bars[W::P_READY], lane);
                }
#pragma unroll
                for (int h = 0; h < kPasses; ++h) {
                    uint32_t parts[3][kWords];
#pragma unroll
                    for (int i = 0; i < kWords; i += 2) {
                        const int c = 2 * (h * kWords + i);
                        const float4 d = KV ? *reinterpret_cast<const float4*>(slot + 16 + c) : make_float4(delta, delta, delta, delta);
                        uint32_t y[3];
                        split3_cut<__nv_bfloat16>(s[c] * (dp[c] - d.x), s[c + 1] * (dp[c + 1] - d.y), y);
                        parts[0][i] = y[0], parts[1][i] = y[1], parts[2][i] = y[2];
                        split3_cut<__nv_bfloat16>(s[c + 2] * (dp[c + 2] - d.z), s[c + 3] * (dp[c + 3] - d.w), y);
                        parts[0][i + 1] = y[0], parts[1][i + 1] = y[1], parts[2][i + 1] = y[2];
                    }
#pragma unroll
                    for (int part = 0; part < 3; ++part) store_words(lanes + W::ds_col(buf, part, wg) + h * kWords, parts[part]);
                }
                tmem_wait_st();
                if (!KV && W::kBufs == 2 && j > 0) {   // dQ of the block before leaves TMEM to this one
                    collect(g - 1, true);
                    if (!ok) break;
                }
                tc_fence_before();
                mbar_arrive_warp(&bars[W::DS_READY], lane);
                if (KV) seen = !(causal && quad >= 2 && j % steps == 0);
            }
            if (!ok) break;
            if (!KV) seen = !causal || (nb - 1) * kBN <= own0 + quad * 32 + 31;
            collect(g - 1, seen);
            if (!ok) break;
            // gradients of the rotated rows turned back; Q~ carries sm_scale * log2e, so dK only takes the log2e off again
            if (pos < N) {
                const float scale = KV ? kLn2 : p.sm_scale;
                T* out = reinterpret_cast<T*>(KV ? p.dk : p.dq) + (KV ? row_offset(p.sdk, p.Hkv, wi.head, pos) : row_offset(p.sdq, p.H, wi.head, pos)) + wg * E;
#pragma unroll
                for (int v = 0; v < E / 8; ++v) {
                    float c[8], sn[8];
                    if (p.cos != nullptr) {
                        load_table8(p.cos + (int64_t)pos * p.table_stride + wg * E + 8 * v, table_vec, c);
                        load_table8(p.sin + (int64_t)pos * p.table_stride + wg * E + 8 * v, table_vec, sn);
                    }
                    float2 lo[4], hi[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        float a0, a1, b0, b1;
                        f2_unpack(acc[0][4 * v + e], a0, a1);
                        f2_unpack(acc[1][4 * v + e], b0, b1);
                        if (p.cos != nullptr) {
                            const float x0 = a0 * c[2 * e] + b0 * sn[2 * e], x1 = a1 * c[2 * e + 1] + b1 * sn[2 * e + 1];
                            b0 = b0 * c[2 * e] - a0 * sn[2 * e], b1 = b1 * c[2 * e + 1] - a1 * sn[2 * e + 1];
                            a0 = x0, a1 = x1;
                        }
                        lo[e] = make_float2(a0 * scale, a1 * scale);
                        hi[e] = make_float2(b0 * scale, b1 * scale);
                    }
                    store8(out + 8 * v, lo);
                    store8(out + D / 2 + 8 * v, hi);
                }
                if constexpr (KV) {
                    constexpr float kUnscale = 1.f / kPScale<T>;
                    T* o2 = reinterpret_cast<T*>(p.dv) + row_offset(p.sdv, p.Hkv, wi.head, pos) + wg * E;
#pragma unroll
                    for (int half = 0; half < 2; ++half)
#pragma unroll
                        for (int v = 0; v < E / 8; ++v) {
                            float2 o[4];
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                f2_unpack(dv[half][4 * v + e], o[e].x, o[e].y);
                                o[e].x *= kUnscale, o[e].y *= kUnscale;
                            }
                            store8(o2 + half * (D / 2) + 8 * v, o);
                        }
                }
            }
        }
        tc_fence_before();
    }
    __syncthreads();
    if (threadIdx.x == 0 && *abort_flag) report_to_mirror(p.status, p.status_mirror);
    if (!KV) pdl_wait();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

template <typename T, int D, int KP, bool KV>
int launch_t(const RopeParams& p, const SplitCopies& x, int* counter, cudaStream_t s) {
    constexpr int XP = Plain<T>::kParts;
    using W = Bwd<D, KP, XP, KV>;
    CUtensorMap mq, mk, mv, mdo;
    Strides sq = contiguous_strides(p.B * p.H, p.N, D), sk = contiguous_strides(p.B * p.Hkv, p.N, D);
    sq.b = (int64_t)x.q.plane, sk.b = (int64_t)x.k.plane;   // the parts take the place of the batch dimension
    if (int e = encode_tensor_map_4d_sw128(&mq, x.q.rows, 3, p.B * p.H, p.N, D, sq, kBN, 64, COROPE_DTYPE_BF16)) return e;
    if (int e = encode_tensor_map_4d_sw128(&mk, x.k.rows, KP, p.B * p.Hkv, p.N, D, sk, kBN, 64, COROPE_DTYPE_BF16)) return e;
    if (XP > 1) {
        if (int e = encode_tensor_map_4d_sw128(&mv, x.v.rows, XP, p.B * p.Hkv, p.N, D, sk, kBN, 64, COROPE_DTYPE_BF16)) return e;
        if (int e = encode_tensor_map_4d_sw128(&mdo, x.d_o.rows, XP, p.B * p.H, p.N, D, sq, kBN, 64, COROPE_DTYPE_BF16)) return e;
    } else {
        if (int e = encode_tensor_map_4d_sw128(&mv, p.v, p.B, p.Hkv, p.N, D, p.sv, kBN, 64, Elem<T>::kDtype)) return e;
        if (int e = encode_tensor_map_4d_sw128(&mdo, p.d_o, p.B, p.H, p.N, D, p.sdo, kBN, 64, Elem<T>::kDtype)) return e;
    }
    RopeParams pp = p;
    pp.sched_counter = counter;
    pp.head_chunk = p.N >= 4096 ? 8 : 8 * (4096 / (p.N < 128 ? 128 : p.N));
    auto kern = rope_bwd_split_sm100_kernel<T, D, KP, KV>;
    static std::atomic<uint64_t> smem_ok;
    if (int e = allow_smem(kern, W::kSmem, smem_ok)) return e;
    const unsigned items = rope_split_items(p.B, KV ? p.Hkv : p.H, p.N).blocks(), sms = (unsigned)sm_count();
    count_launch();
    return launch_dependent(kern, items < sms ? items : sms, kThreads, W::kSmem, s, KV ? mk : mq, KV ? mv : mdo, KV ? mq : mk, KV ? mdo : mv, pp);
}
template <typename T, int D, int KP>
int launch_both(const RopeParams& p, const SplitCopies& x, cudaStream_t s) {
    if (int e = launch_t<T, D, KP, true>(p, x, p.sched_counter, s)) return e;
    return launch_t<T, D, KP, false>(p, x, p.sched_counter + 1, s);
}
template <typename T, int KP>
int launch_d(const RopeParams& p, const SplitCopies& x, cudaStream_t s) {
    return p.D == 64 ? launch_both<T, 64, KP>(p, x, s) : launch_both<T, 128, KP>(p, x, s);
}

}  // namespace

int launch_rope_bwd_split(const RopeParams& p, void* ws, int dtype, cudaStream_t s) {
    const SplitCopies x = split_copies(p, ws, true, dtype);
    if (int e = launch_split_rows(p, x, true, dtype, s)) return e;
    if (dtype == COROPE_DTYPE_F32) return launch_both<float, 64, 3>(p, x, s);
    if (dtype == COROPE_DTYPE_F16) return launch_d<__half, 3>(p, x, s);
    // bf16 keys without rotation have 8 bits: hi and mid hold all of them
    return p.cos == nullptr ? launch_d<__nv_bfloat16, 2>(p, x, s) : launch_d<__nv_bfloat16, 3>(p, x, s);
}

}  // namespace corope
