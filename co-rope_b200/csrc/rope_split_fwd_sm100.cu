// Fused-RoPE / plain attention forward for 16-bit tensors at lengths that are not whole 128-row tiles, D = 64 or 128, at the accuracy of
// fp32 operands: tcgen05 MMAs on operands split into 16-bit parts (rope_split.cuh).
//     S  = Q~ K~^T   both rotated in fp32 and split into three bf16 parts: hi hi in one accumulator, the five products of a smaller
//                    part in a second one; join_products adds them (without mid lo, lo mid, lo lo: about 2^-25)
//     O += P V       P split into three numbers of the inputs' type, V as it is; the product of each 64-key block is its own sum in
//                    TMEM (small parts first), which fp32 registers collect; on the diagonal the MMAs leave out the rows that a k-step of 16 keys is
//                    hidden from (block_product), so that a key with infinities or NaNs only reaches the rows of its own group of 16
// P <= 1 of f16 tensors enters its products times 2^14.  fp32 tensors of D = 64 run here at every length from rope_split_fp32 on: V is split too,
// P V are 6 products.
//
// A work item is 128 query rows of one head; persistent CTAs (one per SM) take items from a counter, heaviest first.  640 threads:
//   warp 0      TMA producer: fetches items; ring of stages, each the parts of 64 rows of K~ and the rows of V (zeros beyond the head)
//   warp 1      MMA issuer and TMEM owner;  warps 2, 3 idle
//   warps 4-19  four groups of 128 threads, thread = query row; group w has keys [16 w, 16 w + 16) of a block (one k-step of P V) and D / 4
//               columns of O.  Per item they rotate and split Q; per block: S -> max over the four groups -> P, split, over S in TMEM;
//               then the product of the block before is added to O in registers
// TMEM: parts of Q~ (A operands read from TMEM leave the shared-memory port to the B operands: 33 instead of 49 cycles per N = 64
// MMA; D = 128: lo has no room and sits in shared memory) | two S buffers of 64 + 64 columns, so that Q K^T of the next block runs beside
// the softmax of this one | O of a block.
//
// What bounds it: 48 + 12 MMAs per block of 64 keys (D = 128; 2520 cycles), measured at 1.52 us (2990 cycles of 1965 MHz) per block, D = 64 at
// 1.17 us; a launch with one item per SM takes 8 us besides (launch, rotation and split of Q, output).  GPU time: B1 H32 N1777 D128 bf16 causal
// 397 -> 112 us (mma.sync kernel before), B4 H16 N1000 D64 bf16 full 243 -> 104 us, B1 H2 N5999 D128 538 -> 153 us.  Error against 64-bit arithmetic next to that kernel (N(0, 1) inputs, B1 H4 N1777 D128 causal f16): LSE
// 3.6e-7 (3.8e-7), results that are not the exact one rounded 0.119 % (0.123 %); q and k times 4: LSE 4.7e-6 (4.5e-6; CUDA cores 6.9e-6),
// 0.31 % (0.30 %; 0.47 %).  fp32 (B1 H4 N512 D64 causal): O 1.3e-7 (CUDA cores 2.3e-7), also where channels differ in scale by 1000.
//
// Replaces _attn_fwd of the reference (fused-rope/fused_rope_attn.py:219-320) for these lengths; math: rope_attn_pytorch.py:108-155.
#include "rope_split.cuh"

namespace corope {
namespace {

constexpr int kBM = 128, kBN = 64;
constexpr int kThreads = 640, kComputeWarp0 = 4, kComputeWarps = 16;
// launch registers 65536 / 640 rounded down to a multiple of 8; what the control warps give up the others may take.  The issue loop is scheduled by what
// it may keep: 40 / 48 / 64 registers, B4 H16 N1000 D64 102.8 / 108.0 / 103.8 us, B1 H32 N1777 D128 113.4 / 111.6 / 113.1 us.
constexpr int kLaunchRegs = 96, kRegsCompute = 104;
template <int D> constexpr int kRegsCtl = D == 64 ? 40 : 48;
static_assert(128 * (kRegsCtl<128> + 4 * kRegsCompute) <= kThreads * kLaunchRegs && kRegsCtl<64> <= kRegsCtl<128>, "register budget");
constexpr int kItemSlots = 2, kItemReaders = 1 + kComputeWarps;
constexpr uint32_t kHi = sdesc_hi(1024);

// KP, VP: parts of K~ and V
template <int D, int KP, int VP> struct Fwd {
    static constexpr int kTile = kBN * D * 2, kStage = (KP + VP) * kTile;   // 64 rows; parts of K~, then V
    static constexpr int kStages = VP == 3 ? 4 : D == 64 ? 5 : KP == 3 ? 3 : 4;
    static constexpr int kQTile = kBM * D * 2;   // one part of Q~ on its way to TMEM; D = 128: lo stays here
    enum Bar { FULL = 0, EMPTY = FULL + kStages, S_FULL = EMPTY + kStages, P_FULL = S_FULL + 2, O_FULL = P_FULL + 2, Q_READY, ITEM_FULL, ITEM_EMPTY = ITEM_FULL + kItemSlots, NUM_BARS = ITEM_EMPTY + kItemSlots };
    static constexpr size_t kXch = 4 * kBM * sizeof(float) + 4 * sizeof(int), kSlack = 512;
    static constexpr size_t kSmem = (size_t)kStages * kStage + kQTile + kXch + NUM_BARS * 8 + 32 + kSlack;
    static_assert(kSmem <= 232448, "shared memory budget");
    // TMEM columns
    static constexpr int kQPart = D / 2, kS = 128, kO = 384;
};

struct WorkItem {
    int t, bh;
};
// heads in chunks, so that the K~ and V in use stay in L2; the longest causal rows of a chunk first
__device__ __forceinline__ WorkItem work_item(int w, int n_qt, int BH, int head_chunk) {
    const int chunk_items = head_chunk * n_qt, chunk = w / chunk_items, within = w % chunk_items;
    const int heads_here = min(head_chunk, BH - chunk * head_chunk);
    return {n_qt - 1 - within / heads_here, chunk * head_chunk + within % heads_here};
}

template <typename T, int D, int KP>
__global__ void __launch_bounds__(kThreads, 1)
rope_fwd_split_sm100_kernel(const __grid_constant__ CUtensorMap mapK, const __grid_constant__ CUtensorMap mapV, const __grid_constant__ RopeParams p) {
    constexpr int VP = Plain<T>::kParts;
    using F = Fwd<D, KP, VP>;
    constexpr int ST = F::kStages;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* sQ = sm + ST * F::kStage;
    float* xch = reinterpret_cast<float*>(sQ + F::kQTile);   // [group][row]
    volatile int* left = reinterpret_cast<volatile int*>(xch + 4 * kBM);   // per four warps with the same rows: they leave together
    uint64_t* bars = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(xch) + F::kXch);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + F::NUM_BARS);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    volatile int* item_ring = reinterpret_cast<volatile int*>(tmem_slot + 2);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int N = p.N, BH = p.B * p.H, G = p.H / p.Hkv;
    const int n_qt = (N - 1) / kBM + 1, n_items = n_qt * BH, nb_all = (N - 1) / kBN + 1;
    const bool causal = p.causal != 0;
    auto blocks_of = [&](int t) { return causal ? min(nb_all, 2 * t + 2) : nb_all; };

    if (reinterpret_cast<uintptr_t>(sm) - reinterpret_cast<uintptr_t>(smem_raw) > F::kSlack) {   // base less aligned than assumed
        if (threadIdx.x == 0 && p.status) {
            atomicCAS(p.status, 0, COROPE_DEV_WAIT_EXPIRED | 0xfff);
            report_to_mirror(COROPE_DEV_WAIT_EXPIRED | 0xfff, p.status_mirror);
        }
        pdl_wait();   // no launch ends before the one in front of it
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
        for (int i = 0; i < 4; ++i) left[i] = 0;
        for (int i = 0; i < ST; ++i) {
            mbar_init(&bars[F::FULL + i], 1);
            mbar_init(&bars[F::EMPTY + i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&bars[F::S_FULL + i], 1);
            mbar_init(&bars[F::P_FULL + i], kComputeWarps);
        }
        mbar_init(&bars[F::O_FULL], 1);
        mbar_init(&bars[F::Q_READY], kComputeWarps);
        for (int i = 0; i < kItemSlots; ++i) {
            mbar_init(&bars[F::ITEM_FULL + i], 1);
            mbar_init(&bars[F::ITEM_EMPTY + i], kItemReaders);
        }
        fence_mbar_init();
        tma_prefetch_desc(&mapK);
        tma_prefetch_desc(&mapV);
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
    // the n-th item of this CTA, -1 when there is none left, -2 where the wait gave up; one arrival per warp
    auto fetch_item = [&](int n) {
        const int slot = n % kItemSlots;
        if (!mbar_wait_warp(&bars[F::ITEM_FULL + slot], (n / kItemSlots) & 1, p.status, F::ITEM_FULL, abort_flag)) return -2;
        const int w = item_ring[slot];
        mbar_arrive_warp(&bars[F::ITEM_EMPTY + slot], lane);
        return w;
    };

    if (warp < kComputeWarp0) {
        reg_dealloc<kRegsCtl<D>>();
        if (warp == 0) {
            // -------------------------------------------------------------- TMA producer
            if (lane == 0) {
                pdl_wait();   // the parts of K~ and the zeroed counter; nothing else is read from the pre-pass
                int g = 0;
                bool ok = true;
                for (int n = 0; ok; ++n) {
                    const int slot = n % kItemSlots;
                    if (n >= kItemSlots && !(ok = mbar_wait(&bars[F::ITEM_EMPTY + slot], ((n / kItemSlots) - 1) & 1, p.status, F::ITEM_EMPTY, abort_flag))) break;
                    int w = n == 0 ? (int)blockIdx.x : (int)gridDim.x + atomicAdd(p.sched_counter, 1);
                    if (w >= n_items) w = -1;
                    item_ring[slot] = w;
                    mbar_arrive(&bars[F::ITEM_FULL + slot]);
                    if (w < 0) break;
                    const WorkItem wi = work_item(w, n_qt, BH, p.head_chunk);
                    const int nb = blocks_of(wi.t), kvh = wi.bh / G, vb = kvh / p.Hkv, vh = kvh % p.Hkv;
                    for (int j = 0; j < nb; ++j, ++g) {
                        const int st = g % ST;
                        if (g >= ST && !(ok = mbar_wait(&bars[F::EMPTY + st], ((g / ST) - 1) & 1, p.status, F::EMPTY, abort_flag))) break;
                        uint8_t* dst = sm + st * F::kStage;
                        uint64_t* bar = &bars[F::FULL + st];
                        mbar_arrive_expect_tx(bar, F::kStage);
#pragma unroll
                        for (int c = 0; c < D / 64; ++c) {
#pragma unroll
                            for (int part = 0; part < KP; ++part) tma_load_4d(dst + part * F::kTile + c * (kBN * 128), &mapK, c * 64, j * kBN, kvh, part, bar);
                            if constexpr (VP > 1) {   // the copies of fp32 V are laid out as those of K
#pragma unroll
                                for (int part = 0; part < VP; ++part) tma_load_4d(dst + (KP + part) * F::kTile + c * (kBN * 128), &mapV, c * 64, j * kBN, kvh, part, bar);
                            } else {
                                tma_load_4d(dst + KP * F::kTile + c * (kBN * 128), &mapV, c * 64, j * kBN, vh, vb, bar);
                            }
                        }
                    }
                }
            }
            __syncwarp();
        } else if (warp == 1) {
            // -------------------------------------------------------------- MMA issuer
            const bool leader = elect_one();
            constexpr int kVFmt = Plain<T>::kDtype == COROPE_DTYPE_F16 ? 0 : 1;
            const uint32_t idesc_qk = make_idesc(1, 1, 0, 0, kBM, kBN), idesc_pv = make_idesc(kVFmt, kVFmt, 0, 1, kBM, D);
            const uint32_t stage_lo = sdesc_lo(smem_u32(sm), 0), qlo_lo = sdesc_lo(smem_u32(sQ), 0), v_lo = sdesc_lo(smem_u32(sm) + KP * F::kTile, kBN * 128);
            // one product of a part of Q~ and a part of K~
            auto product = [&](int qp, int kp, uint32_t d, uint32_t k_lo, bool first) {
#pragma unroll
                for (int kk = 0; kk < D / 16; ++kk) {
                    const uint32_t b = k_lo + ((kp * F::kTile + (kk >> 2) * (kBN * 128) + (kk & 3) * 32) >> 4);
                    if (D == 128 && qp == 2) {
                        if (leader) umma_ss2(d, qlo_lo + (((kk >> 2) * (kBM * 128) + (kk & 3) * 32) >> 4), kHi, b, kHi, idesc_qk, (first && kk == 0) ? 0u : 1u);
                    } else {
                        if (leader) umma_ts2(d, tmem + qp * F::kQPart + kk * 8, b, kHi, idesc_qk, (first && kk == 0) ? 0u : 1u);
                    }
                }
            };
            int gq = 0, gp = 0;   // blocks so far: Q K^T, P V
            bool ok = true;
            // Q K^T in two pieces, so that MMAs are still queued while the warp waits: the wait for P (85 cycles even where its phase is
            // complete, and the fences around it) stands between the pieces, the one for the K~ stage behind P V
            auto qk_head = [&]() {
                const int st = gq % ST;
                if (!(ok = mbar_wait_warp(&bars[F::FULL + st], (gq / ST) & 1, p.status, F::FULL, abort_flag))) return;
                tc_fence_after();
                const uint32_t k_lo = stage_lo + st * (F::kStage >> 4), d = tmem + F::kS + (gq & 1) * 128;
                product(1, 1, d + 64, k_lo, true);
                if (KP > 2) product(0, 2, d + 64, k_lo, false);
                product(0, 1, d + 64, k_lo, false);
                product(1, 0, d + 64, k_lo, false);
                product(2, 0, d + 64, k_lo, false);
            };
            auto qk_tail = [&]() {
                product(0, 0, tmem + F::kS + (gq & 1) * 128, stage_lo + (gq % ST) * (F::kStage >> 4), true);
                if (leader) umma_commit(&bars[F::S_FULL + (gq & 1)]);
                ++gq;
            };
            for (int n = 0; ok; ++n) {
                const int w = fetch_item(n);
                if (w < 0) break;
                const int t = work_item(w, n_qt, BH, p.head_chunk).t, nb = blocks_of(t);
                if (!(ok = mbar_wait_warp(&bars[F::Q_READY], n & 1, p.status, F::Q_READY, abort_flag))) break;
                tc_fence_after();
                // P V of block j; Q K^T of block j + 2, and at j = -2 alone all of block 0's
                auto turn = [&](int j, auto where) {
                    if (j >= 0) {
                        const int buf = gp & 1, st = gp % ST;
                        if (!(ok = mbar_wait_warp(&bars[F::P_FULL + buf], (gp >> 1) & 1, p.status, F::P_FULL, abort_flag))) return;
                        tc_fence_after();
                        if (j + 1 < nb) qk_tail();
                        const uint32_t b0 = v_lo + st * (F::kStage >> 4), a0 = tmem + F::kS + buf * 128;
#pragma unroll
                        for (int i = 0; i < (VP > 1 ? kProducts : 3); ++i)   // small parts first
                            block_product<false>(where, leader, tmem + F::kO, [&](int kk) { return a0 + (VP > 1 ? product_a(i) : 2 - i) * 32 + kk * 8; },
                                                 [&](int kk) { return b0 + (((VP > 1 ? product_b(i) : 0) * F::kTile + kk * 2048) >> 4); }, kHi, idesc_pv, i == 0);
                        if (leader) umma_commit(&bars[F::O_FULL]);
                        if (leader) umma_commit(&bars[F::EMPTY + st]);
                        ++gp;
                    }
                    if (j == -1) qk_tail();
                    if (j + 2 < nb) qk_head();
                };
                // the blocks on the diagonal stand behind the loop: within it their forms cost 4 % (B1 H2 N5999 D128 153.8 -> 160.2 us)
                const int whole = causal ? 2 * t : nb;
                for (int j = -2; j < whole && ok; ++j) turn(j, WholeBlock{});
                if (ok && whole < nb) turn(whole, FirstOnDiagonal{});
                if (ok && whole + 1 < nb) turn(whole + 1, SecondOnDiagonal{});
            }
            __syncwarp();
        }
    } else {
        // ------------------------------------------------------------------ rotation and split of Q, softmax, sums of O
        reg_alloc<kRegsCompute>();
        const int wg = (warp - kComputeWarp0) >> 2, quad = warp & 3;   // the TMEM lane quadrant a warp may touch is warp_id % 4
        const int row = quad * 32 + lane, quad_bar = 1 + quad;         // named barrier of the four warps that hold the same rows
        const uint32_t lanes = tmem + ((uint32_t)(quad * 32) << 16);
        constexpr int OC = D / 4;                                      // columns of O
        const bool table_vec = tables_aligned(p);
        int g = 0;                                                     // blocks so far
        bool ok = true;
        uint64_t acc[OC / 2];
        // O += product of the block before, alpha = what the reference max moved by at that block; nothing where the warp's rows all lie in front
        // of the block (`seen`; an item's last block alone can be such a one): their product has not been formed
        auto collect = [&](int block, float alpha, bool seen, bool last) {
            if (!(ok = mbar_wait_warp(&bars[F::O_FULL], block & 1, p.status, F::O_FULL, abort_flag))) return;
            tc_fence_after();
            uint32_t r[OC];
            if constexpr (D == 128)
                COROPE_TMEM_LD32(lanes + F::kO + wg * OC, r);
            else
                COROPE_TMEM_LD16(lanes + F::kO + wg * OC, r);
            tmem_wait_ld();
            tc_fence_before();
            if (!last) mbar_arrive_warp(&bars[F::P_FULL + ((block + 1) & 1)], lane);   // P of the next block, and O is free
            if (!seen) return;
            const uint64_t a2 = f2_pack(alpha, alpha);
#pragma unroll
            for (int i = 0; i < OC / 2; ++i) acc[i] = f2_fma(acc[i], a2, f2_pack_bits(r[2 * i], r[2 * i + 1]));
        };
        // A warp whose wait gave up must not leave the three that meet it at quad_bar alone: it goes on to the next of two places where they
        // look for it, the start of an item (`left`) and the exchange of a block's maxima (NaN, which no maximum is), and all four leave behind it.
        // tests/test_give_up_cpu.py goes through every order of this.
        for (int n = 0;; ++n) {
            const int w = ok ? fetch_item(n) : -2;
            if (w == -2) left[quad] = 1;
            named_bar_sync(quad_bar, 128);
            if (w < 0 || left[quad] != 0) break;
            const WorkItem wi = work_item(w, n_qt, BH, p.head_chunk);
            const int nb = blocks_of(wi.t), pos = wi.t * kBM + row;
            {   // Q~: 8 rotation pairs of a row per lane (whole rows are read at a time), the parts by way of shared memory to the threads
                // that own the rows in TMEM.  Every MMA of the item before has completed (its last O_FULL).
                constexpr int LPR = D / 16, RPS = 32 / LPR, STEPS = 8 / RPS;   // lanes per row, rows per step, steps of a warp's 8 rows
                const int u = lane % LPR;
                uint32_t pa[STEPS][3][4], pb[STEPS][3][4];
                auto at = [&](int r, int chunk) {   // 16-byte chunk of row r of a tile of 64-column boxes, 128-byte swizzle
                    return reinterpret_cast<uint4*>(sQ + (chunk >> 3) * (kBM * 128) + r * 128 + (((chunk & 7) ^ (r & 7)) * 16));
                };
#pragma unroll
                for (int st = 0; st < STEPS; ++st) {
                    const int r = quad * 32 + wg * 8 + st * RPS + lane / LPR, n = min(wi.t * kBM + r, N - 1);   // rows beyond the head repeat its last one
                    const T* src = reinterpret_cast<const T*>(p.q) + row_offset(p.sq, p.H, wi.bh, n) + u * 8;
                    float2 a[4], b[4];
                    load8(src, a);
                    load8(src + D / 2, b);
                    if (p.cos != nullptr) {
                        float c[8], sn[8];
                        load_table8(p.cos + (int64_t)n * p.table_stride + u * 8, table_vec, c);
                        load_table8(p.sin + (int64_t)n * p.table_stride + u * 8, table_vec, sn);
#pragma unroll
                        for (int e = 0; e < 4; ++e) rotate(a[e], b[e], c + 2 * e, sn + 2 * e);
                    }
                    const float scale = p.sm_scale * kLog2e;
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        uint32_t x[3], y[3];
                        split3_any(a[e].x * scale, a[e].y * scale, x);
                        split3_any(b[e].x * scale, b[e].y * scale, y);
#pragma unroll
                        for (int part = 0; part < 3; ++part) pa[st][part][e] = x[part], pb[st][part][e] = y[part];
                    }
                }
#pragma unroll
                for (int part = 0; part < 3; ++part) {
#pragma unroll
                    for (int st = 0; st < STEPS; ++st) {
                        const int r = quad * 32 + wg * 8 + st * RPS + lane / LPR;
                        *at(r, u) = make_uint4(pa[st][part][0], pa[st][part][1], pa[st][part][2], pa[st][part][3]);
                        *at(r, u + D / 16) = make_uint4(pb[st][part][0], pb[st][part][1], pb[st][part][2], pb[st][part][3]);
                    }
                    if (D == 128 && part == 2) {   // stays where it is
                        fence_proxy_async();
                        break;
                    }
                    named_bar_sync(quad_bar, 128);
                    uint32_t w4[D / 8];
#pragma unroll
                    for (int v = 0; v < D / 32; ++v) {
                        const uint4 x = *at(row, wg * (D / 32) + v);
                        w4[4 * v] = x.x, w4[4 * v + 1] = x.y, w4[4 * v + 2] = x.z, w4[4 * v + 3] = x.w;
                    }
                    if constexpr (D == 128)
                        COROPE_TMEM_ST16(lanes + part * F::kQPart + wg * (D / 8), w4);
                    else
                        COROPE_TMEM_ST8(lanes + part * F::kQPart + wg * (D / 8), w4);
                    if (part < 2) named_bar_sync(quad_bar, 128);
                }
                tmem_wait_st();
                tc_fence_before();
                mbar_arrive_warp(&bars[F::Q_READY], lane);
            }
            float m = -INFINITY, l = 0.f, alpha_before = 0.f;
            bool all_here = false;
#pragma unroll
            for (int i = 0; i < OC / 2; ++i) acc[i] = 0;
            for (int j = 0; j < nb; ++j, ++g) {
                const int buf = g & 1;
                if (ok) ok = mbar_wait_warp(&bars[F::S_FULL + buf], (g >> 1) & 1, p.status, F::S_FULL, abort_flag);
                if (!ok) {
                    xch[wg * kBM + row] = __int_as_float(0x7fffffff);
                    named_bar_sync(quad_bar, 128);
                    named_bar_sync(quad_bar, 128);
                    break;
                }
                tc_fence_after();
                const uint32_t tS = lanes + F::kS + buf * 128;
                uint32_t main[16], small[16];
                COROPE_TMEM_LD16(tS + wg * 16, main);
                COROPE_TMEM_LD16(tS + 64 + wg * 16, small);
                tmem_wait_ld();
                const int key0 = j * kBN + wg * 16;
                float s[16];
#pragma unroll
                for (int i = 0; i < 8; ++i) f2_unpack(join_products<D>(f2_pack_bits(main[2 * i], main[2 * i + 1]), f2_pack_bits(small[2 * i], small[2 * i + 1])), s[2 * i], s[2 * i + 1]);
                float mx = -INFINITY;
#pragma unroll
                for (int i = 0; i < 16; i += 2) mx = fmax3_nan(mx, s[i], s[i + 1]);
                if (__any_sync(0xffffffffu, mx != mx)) {   // infinities or NaNs among the operands
                    infinite_scores(tS + wg * 16, s);
                    mx = -INFINITY;
#pragma unroll
                    for (int i = 0; i < 16; i += 2) mx = fmax3(mx, s[i], s[i + 1]);
                }
                if (j * kBN > N - kBN || (causal && j * kBN + kBN - 1 > wi.t * kBM + quad * 32)) {   // keys that rows of the warp do not see
                    const int last = (causal ? min(pos, N - 1) : N - 1) - key0;
                    mx = -INFINITY;
#pragma unroll
                    for (int i = 0; i < 16; ++i) s[i] = i > last ? -INFINITY : s[i];
#pragma unroll
                    for (int i = 0; i < 16; i += 2) mx = fmax3(mx, s[i], s[i + 1]);
                }
                xch[wg * kBM + row] = mx;
                named_bar_sync(quad_bar, 128);   // also: all four have read their S, so P may be written anywhere over it
                const float others = fmax3_nan(xch[(wg ^ 1) * kBM + row], xch[(wg ^ 2) * kBM + row], xch[(wg ^ 3) * kBM + row]);
                const float m_new = fmax3(m, mx, others);
                const float ref = m_new == -INFINITY ? 0.f : m_new;   // a row that has seen no key yet
                const float alpha = fast_exp2(m - ref);
                m = m_new;
                const uint64_t neg_ref = f2_pack(-ref, -ref);
                uint64_t sum = 0;
                uint32_t parts[3][8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    float x0, x1;
                    f2_unpack(f2_add(f2_pack(s[2 * i], s[2 * i + 1]), neg_ref), x0, x1);
                    x0 = fast_exp2(x0), x1 = fast_exp2(x1);
                    sum = f2_add(sum, f2_pack(x0, x1));
                    uint32_t y[3];
                    split3_cut<typename Plain<T>::Mma>(x0 * kPScale<T>, x1 * kPScale<T>, y);
                    parts[0][i] = y[0], parts[1][i] = y[1], parts[2][i] = y[2];
                }
#pragma unroll
                for (int part = 0; part < 3; ++part) COROPE_TMEM_ST8(tS + part * 32 + wg * 8, parts[part]);
                float s0, s1;
                f2_unpack(sum, s0, s1);
                l = l * alpha + (s0 + s1);   // this group's keys only
                tmem_wait_st();
                if (j > 0) {
                    collect(g - 1, alpha_before, true, false);
                } else {
                    tc_fence_before();
                    mbar_arrive_warp(&bars[F::P_FULL + buf], lane);
                }
                alpha_before = alpha;
                named_bar_sync(quad_bar, 128);   // all four have read the exchanged maxima
                if (others != others) break;     // one of them gave up; in all lanes alike
                all_here = j + 1 == nb;
            }
            if (!all_here) break;
            if (ok) collect(g - 1, alpha_before, !causal || (nb - 1) * kBN <= wi.t * kBM + quad * 32 + 31, true);
            xch[wg * kBM + row] = l;
            named_bar_sync(quad_bar, 128);
            const float total = (xch[row] + xch[kBM + row]) + (xch[2 * kBM + row] + xch[3 * kBM + row]);
            named_bar_sync(quad_bar, 128);
            if (ok && pos < N) {
                const float inv = total > 0.f ? (1.f / kPScale<T>) / total : 0.f;
                T* dst = reinterpret_cast<T*>(p.out_o) + row_offset(p.so, p.H, wi.bh, pos) + wg * OC;
#pragma unroll
                for (int v = 0; v < OC / 8; ++v) {
                    float2 o[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        f2_unpack(acc[4 * v + e], o[e].x, o[e].y);
                        o[e].x *= inv, o[e].y *= inv;
                    }
                    store8(dst + 8 * v, o);
                }
                if (wg == 0) p.lse2[(size_t)wi.bh * N + pos] = m + log2f(total);
            }
        }
        tc_fence_before();
    }
    __syncthreads();
    if (threadIdx.x == 0 && *abort_flag) report_to_mirror(p.status, p.status_mirror);
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

template <typename T, int D, int KP>
int launch_t(const RopeParams& p, const SplitCopies& x, cudaStream_t s) {
    constexpr int VP = Plain<T>::kParts;
    using F = Fwd<D, KP, VP>;
    CUtensorMap mk, mv;
    Strides sk = contiguous_strides(p.B * p.Hkv, p.N, D);
    sk.b = (int64_t)x.k.plane;   // the parts take the place of the batch dimension
    if (int e = encode_tensor_map_4d_sw128(&mk, x.k.rows, KP, p.B * p.Hkv, p.N, D, sk, kBN, 64, COROPE_DTYPE_BF16)) return e;
    if (int e = VP > 1 ? encode_tensor_map_4d_sw128(&mv, x.v.rows, VP, p.B * p.Hkv, p.N, D, sk, kBN, 64, COROPE_DTYPE_BF16)
                       : encode_tensor_map_4d_sw128(&mv, p.v, p.B, p.Hkv, p.N, D, p.sv, kBN, 64, Elem<T>::kDtype))
        return e;
    RopeParams pp = p;
    pp.head_chunk = p.N >= 4096 ? 8 : 8 * (4096 / (p.N < 128 ? 128 : p.N));
    auto kern = rope_fwd_split_sm100_kernel<T, D, KP>;
    static std::atomic<uint64_t> smem_ok;
    if (int e = allow_smem(kern, F::kSmem, smem_ok)) return e;
    const unsigned items = rope_split_items(p.B, p.H, p.N).blocks(), sms = (unsigned)sm_count();
    count_launch();
    return launch_dependent(kern, items < sms ? items : sms, kThreads, F::kSmem, s, mk, mv, pp);
}
template <typename T, int KP>
int launch_d(const RopeParams& p, const SplitCopies& x, cudaStream_t s) {
    return p.D == 64 ? launch_t<T, 64, KP>(p, x, s) : launch_t<T, 128, KP>(p, x, s);
}

}  // namespace

FlatGrid rope_split_items(int B, int H, int N) { return {(unsigned)(B * H), ceil_div(N, kBM)}; }

int launch_rope_fwd_split_tc(const RopeParams& p, void* ws, int dtype, cudaStream_t s) {
    const SplitCopies x = split_copies(p, ws, false, dtype);
    if (int e = launch_split_rows(p, x, false, dtype, s)) return e;
    if (dtype == COROPE_DTYPE_F32) return launch_t<float, 64, 3>(p, x, s);
    if (dtype == COROPE_DTYPE_F16) return launch_d<__half, 3>(p, x, s);
    // bf16 keys without rotation have 8 bits: hi and mid hold all of them
    return p.cos == nullptr ? launch_d<__nv_bfloat16, 2>(p, x, s) : launch_d<__nv_bfloat16, 3>(p, x, s);
}

}  // namespace corope
