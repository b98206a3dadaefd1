// extern "C" entry points of libcorope_b200.so: argument validation, workspace carving, kernel selection.
#include <atomic>
#include <mutex>

#include "common.cuh"

namespace corope {
namespace {

std::atomic<int> g_policy{0};
std::atomic<unsigned long long> g_launches{0};
std::atomic<int> g_last_family[4] = {{0}, {0}, {0}, {0}};
std::atomic<int> g_last_split[4] = {{0}, {0}, {0}, {0}};
// what the call in hand of an op takes: 1 tensor-core kernels at whole tiles, 0 the others, of those `split` with split operands
void note_kernels(int op, int family, bool split) {
    g_last_family[op] = family;
    g_last_split[op] = split ? 1 : 0;
}

constexpr size_t kAlign = 256;

bool head_dim_ok(int D) { return D == 32 || D == 64 || D == 128; }

struct RopeWorkspace {
    size_t packed_tab, synth_cos, synth_sin, rot, delta, dq_acc, total;
    bool tc;      // room for the tcgen05 kernels
    bool split;   // room for the split-operand kernels
};

// Hq query heads, Hkv K / V heads (equal for the fused-RoPE ops).  `synth`: room for fp32 cos / sin tables [N, D/2] that the
// entry points taking frequencies instead of tables fill in.  `any_n`: room for tensor-core kernels whatever N is, not only
// for multiples of 128.
RopeWorkspace rope_workspace_layout(bool bwd, int B, int Hq, int Hkv, int N, int D, int dtype, bool synth, bool any_n) {
    RopeWorkspace w{};
    w.tc = rope_tc_supported(D, dtype) && N % 128 == 0;
    w.split = any_n && (rope_tc_supported(D, dtype) ? N % 128 != 0 : rope_split_fp32(N, D, dtype));
    const size_t q_elems = (size_t)B * Hq * N * D, kv_elems = (size_t)B * Hkv * N * D;
    size_t off = 0;
    w.packed_tab = off;
    off += align_up((size_t)N * (D / 2) * sizeof(uint32_t) + 64, kAlign);   // + the work counter behind the table
    if (synth) {
        w.synth_cos = off;
        off += align_up((size_t)N * (D / 2) * sizeof(float), kAlign);
        w.synth_sin = off;
        off += align_up((size_t)N * (D / 2) * sizeof(float), kAlign);
    }
    w.rot = off;   // tcgen05 kernels: fp16 copy of the rotated K (forward) / rotated and scaled Q (backward); the split-operand kernels: parts of K and Q
    if (w.tc) off += align_up((bwd ? q_elems : kv_elems) * 2, kAlign);
    if (w.split) off += align_up(rope_split_workspace_bytes(bwd, B, Hq, Hkv, N, D, dtype), kAlign);
    if (bwd) {
        w.delta = off;
        off += align_up((size_t)B * Hq * N * sizeof(float), kAlign);
        w.dq_acc = off;
        if (w.tc) off += align_up(q_elems * sizeof(float), kAlign);
    }
    w.total = off < kAlign ? kAlign : off;
    return w;
}

// What corope_workspace_bytes answers for the fused-RoPE and plain ops.  16-bit D = 64 problems with N % 128 == 0 once ran
// zero-padded to D = 128 and callers were told 16 (forward) / 32 (backward) bytes per element of q; that bound stays in force.
size_t rope_workspace_bytes(bool bwd, int B, int Hq, int Hkv, int N, int D, int dtype, bool synth) {
    const size_t need = rope_workspace_layout(bwd, B, Hq, Hkv, N, D, dtype, synth, false).total;
    if (D != 64 || dtype == COROPE_DTYPE_F32 || N % 128 != 0) return need;
    const size_t told = align_up((size_t)B * Hq * N * D * (bwd ? 32 : 16), kAlign);
    return need > told ? need : told;
}

struct GqaWorkspace {
    size_t delta, dk_acc, dv_acc, k_pairs, v_half, k_scale, total;
};

// `any_n`: room for the split-operand forward where the mma kernels do not apply.
GqaWorkspace gqa_workspace_layout(bool bwd, int B, int Hq, int Hkv, int N, int D, int dtype, bool any_n) {
    GqaWorkspace w{};
    size_t off = 0;
    const bool split = any_n && !bwd && gqa_split_supported(D, dtype);
    // fp16 operand copies of K (pair order) and V for the mma kernels; K in pair order, its own type, and a copy of V if its rows are
    // not aligned for the split-operand forward
    if (gqa_fwd_mma_supported(N, D, dtype) || split) {
        w.k_pairs = off;
        off += align_up((size_t)B * Hkv * N * D * 2, kAlign);
        w.v_half = off;
        off += align_up((size_t)B * Hkv * N * D * 2, kAlign);
    }
    if (split && dtype == COROPE_DTYPE_F16) {
        w.k_scale = off;
        off += align_up((size_t)B * Hkv * N * sizeof(float), kAlign);
    }
    if (bwd) {
        w.delta = off;
        off += align_up((size_t)B * Hq * N * sizeof(float), kAlign);
        w.dk_acc = off;
        off += align_up((size_t)B * Hkv * N * D * sizeof(float), kAlign);
        w.dv_acc = off;
        off += align_up((size_t)B * Hkv * N * D * sizeof(float), kAlign);
    }
    w.total = off < kAlign ? kAlign : off;
    return w;
}

int check_common(int B, int H, int N, int D, int dtype) {
    if (B <= 0 || H <= 0 || N <= 0 || D <= 0) return COROPE_ERR_BAD_SHAPE;
    if (!head_dim_ok(D)) return COROPE_ERR_BAD_HEAD_DIM;
    if (dtype != COROPE_DTYPE_F32 && dtype != COROPE_DTYPE_BF16 && dtype != COROPE_DTYPE_F16) return COROPE_ERR_BAD_DTYPE;
    if ((size_t)B * H > 65535u * 32u) return COROPE_ERR_TOO_LARGE;
    if ((size_t)B * H * N >= (1ull << 31)) return COROPE_ERR_TOO_LARGE;   // row indices are 32-bit in the kernels
    return COROPE_OK;
}

int check_workspace(const void* ws, size_t have, size_t need) {
    if (!ws || have < need || ((uintptr_t)ws % kAlign) != 0) return COROPE_ERR_WORKSPACE;
    return COROPE_OK;
}

}  // namespace

int sm_count() {
    static std::atomic<int> known[64];
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 148;
    if (dev >= 0 && dev < 64 && (sms = known[dev].load(std::memory_order_relaxed)) > 0) return sms;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) return 148;
    if (dev >= 0 && dev < 64) known[dev].store(sms, std::memory_order_relaxed);
    return sms;
}
void count_launch(int n) { g_launches.fetch_add((unsigned long long)n); }
void note_kernel_family(int op, int family) {
    if (op >= 0 && op < 4) note_kernels(op, family, false);
}
int kernel_policy() { return g_policy.load(); }

int* status_mirror_of(const int* status_word);   // below, beside the registration

}  // namespace corope

using namespace corope;

extern "C" {

int corope_abi_version(void) { return 1; }

// ---- host mirror of the status word -----------------------------------------------------------------------------------
// A side stream per device copies the word to a pinned host location whenever the caller's stream reaches the point of the
// call; the caller's stream is not delayed (it only records an event) and the host never synchronises.
namespace {
struct MirrorState {
    cudaStream_t side = nullptr;
    cudaEvent_t reached = nullptr;
};
MirrorState g_mirror[64];
std::mutex g_mirror_mutex;
int mirror_state(MirrorState** out) {
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    if (dev < 0 || dev >= 64) return COROPE_ERR_TOO_LARGE;
    std::lock_guard<std::mutex> lock(g_mirror_mutex);
    MirrorState& m = g_mirror[dev];
    if (!m.side) {
        if ((e = cudaStreamCreateWithFlags(&m.side, cudaStreamNonBlocking)) != cudaSuccess) return (int)e;
        if ((e = cudaEventCreateWithFlags(&m.reached, cudaEventDisableTiming)) != cudaSuccess) return (int)e;
    }
    *out = &m;
    return COROPE_OK;
}
}  // namespace

int corope_status_mirror_refresh(const int* status_word, int* host_mirror, void* stream) {
    if (!status_word || !host_mirror) return COROPE_ERR_NULL_POINTER;
    MirrorState* m = nullptr;
    if (int e = mirror_state(&m)) return e;
    cudaError_t e = cudaEventRecord(m->reached, (cudaStream_t)stream);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(m->side, m->reached, 0);
    if (e == cudaSuccess) e = cudaMemcpyAsync(host_mirror, status_word, sizeof(int), cudaMemcpyDeviceToHost, m->side);
    return (int)e;
}

int corope_status_mirror_clear(int* status_word, int* host_mirror, void* stream) {
    if (!status_word || !host_mirror) return COROPE_ERR_NULL_POINTER;
    MirrorState* m = nullptr;
    if (int e = mirror_state(&m)) return e;
    cudaError_t e = cudaStreamSynchronize(m->side);   // no copy of the old value may land after the mirror is reset
    if (e == cudaSuccess) e = cudaMemsetAsync(status_word, 0, sizeof(int), (cudaStream_t)stream);
    *host_mirror = 0;
    return (int)e;
}

// Registered (word, mirror) pairs: a handful per process, looked up by every launch.
namespace {
struct MirrorPair {
    std::atomic<const int*> word{nullptr};
    std::atomic<int*> mirror{nullptr};
};
MirrorPair g_pairs[128];
}  // namespace

int corope_status_mirror_register(const int* status_word, int* host_mirror) {
    if (!status_word || !host_mirror) return COROPE_ERR_NULL_POINTER;
    void* dev = nullptr;
    if (cudaError_t e = cudaHostGetDevicePointer(&dev, host_mirror, 0)) return (int)e;
    std::lock_guard<std::mutex> lock(g_mirror_mutex);
    for (MirrorPair& p : g_pairs)
        if (p.word.load() == nullptr || p.word.load() == status_word) {
            p.mirror.store(static_cast<int*>(dev));
            p.word.store(status_word);
            return COROPE_OK;
        }
    return COROPE_ERR_TOO_LARGE;
}

const char* corope_status_string(int status) {
    switch (status) {
        case COROPE_OK: return "ok";
        case COROPE_ERR_NULL_POINTER: return "null pointer argument";
        case COROPE_ERR_BAD_SHAPE: return "non-positive tensor extent";
        case COROPE_ERR_BAD_HEAD_DIM: return "unsupported head dimension (supported: 32, 64, 128)";
        case COROPE_ERR_BAD_DTYPE: return "unsupported element type";
        case COROPE_ERR_WORKSPACE: return "workspace missing, too small or not 256-byte aligned";
        case COROPE_ERR_BAD_GROUP: return "query heads must be a multiple of KV heads with group size <= 8";
        case COROPE_ERR_SEQ_NOT_128: return "sequence length must be a multiple of 128";
        case COROPE_ERR_TENSOR_MAP: return "TMA tensor map could not be encoded";
        case COROPE_ERR_NO_DEVICE: return "no usable CUDA device or driver entry point";
        case COROPE_ERR_TOO_LARGE: return "size beyond the supported maximum";
        case COROPE_ERR_BAD_STRIDE: return "row stride smaller than the head dimension, or a negative stride";
        default: break;
    }
    if (status > 0) return cudaGetErrorString((cudaError_t)status);
    return "unknown status";
}

size_t corope_workspace_bytes(int op, int B, int Hq, int Hkv, int N, int D, int dtype) {
    if (B <= 0 || Hq <= 0 || Hkv <= 0 || N <= 0 || D <= 0) return 0;
    switch (op) {
        case COROPE_OP_ROPE_FWD: return rope_workspace_bytes(false, B, Hq, Hq, N, D, dtype, false);
        case COROPE_OP_ROPE_BWD: return rope_workspace_bytes(true, B, Hq, Hq, N, D, dtype, false);
        case COROPE_OP_ROPE_FWD_FREQS: return rope_workspace_bytes(false, B, Hq, Hq, N, D, dtype, true);
        case COROPE_OP_ROPE_BWD_FREQS: return rope_workspace_bytes(true, B, Hq, Hq, N, D, dtype, true);
        case COROPE_OP_FLASH_FWD: return Hq % Hkv ? 0 : rope_workspace_bytes(false, B, Hq, Hkv, N, D, dtype, false);
        case COROPE_OP_FLASH_BWD: return Hq % Hkv ? 0 : rope_workspace_bytes(true, B, Hq, Hkv, N, D, dtype, false);
        case COROPE_OP_GQA_FWD: return gqa_workspace_layout(false, B, Hq, Hkv, N, D, dtype, false).total;
        case COROPE_OP_GQA_BWD: return gqa_workspace_layout(true, B, Hq, Hkv, N, D, dtype, false).total;
        default: return 0;
    }
}

size_t corope_workspace_bytes_any_n(int op, int B, int Hq, int Hkv, int N, int D, int dtype) {
    if (B <= 0 || Hq <= 0 || Hkv <= 0 || N <= 0 || D <= 0) return 0;
    switch (op) {
        case COROPE_OP_ROPE_FWD: return rope_workspace_layout(false, B, Hq, Hq, N, D, dtype, false, true).total;
        case COROPE_OP_ROPE_BWD: return rope_workspace_layout(true, B, Hq, Hq, N, D, dtype, false, true).total;
        case COROPE_OP_ROPE_FWD_FREQS: return rope_workspace_layout(false, B, Hq, Hq, N, D, dtype, true, true).total;
        case COROPE_OP_ROPE_BWD_FREQS: return rope_workspace_layout(true, B, Hq, Hq, N, D, dtype, true, true).total;
        case COROPE_OP_FLASH_FWD: return Hq % Hkv ? 0 : rope_workspace_layout(false, B, Hq, Hkv, N, D, dtype, false, true).total;
        case COROPE_OP_FLASH_BWD: return Hq % Hkv ? 0 : rope_workspace_layout(true, B, Hq, Hkv, N, D, dtype, false, true).total;
        case COROPE_OP_GQA_FWD: return gqa_workspace_layout(false, B, Hq, Hkv, N, D, dtype, true).total;
        default: return corope_workspace_bytes(op, B, Hq, Hkv, N, D, dtype);
    }
}

uint64_t corope_launch_count(void) { return (uint64_t)g_launches.load(); }

int corope_set_kernel_policy(int policy) { return g_policy.exchange(policy); }

int corope_last_kernel_family(int op) { return (op >= 0 && op < 4) ? g_last_family[op].load() : -1; }

int corope_last_kernel_split(int op) { return (op >= 0 && op < 4) ? g_last_split[op].load() : -1; }

}  // extern "C"

namespace {

// Where the rotation comes from: caller tables (cos / sin + row stride), per-pair frequencies (given, or those of a base theta),
// or nothing at all (plain attention).
struct Rotation {
    const float* cos = nullptr;
    const float* sin = nullptr;
    int64_t stride = 0;
    const float* inv_freq = nullptr;
    float theta = 0.f;
    bool freqs = false;   // tables are synthesized from inv_freq (or theta when it is null)
    bool none = false;
};

// Fills the kernels' stride fields from the ABI struct (null = contiguous [B, H, N, D]).
void set_strides(RopeParams& p, const corope_strides_t* st, int Hq, int Hkv, int N, int D) {
    auto conv = [](const int64_t (&a)[3]) {
        Strides r;
        r.b = a[0]; r.h = a[1]; r.n = a[2];
        return r;
    };
    const Strides cq = contiguous_strides(Hq, N, D), ckv = contiguous_strides(Hkv, N, D);
    p.sq = st ? conv(st->q) : cq;
    p.sk = st ? conv(st->k) : ckv;
    p.sv = st ? conv(st->v) : ckv;
    p.so = st ? conv(st->o) : cq;
    p.sdo = st ? conv(st->d_o) : cq;
    p.sdq = st ? conv(st->dq) : cq;
    p.sdk = st ? conv(st->dk) : ckv;
    p.sdv = st ? conv(st->dv) : ckv;
}
void set_gqa_strides(GqaParams& p, const corope_strides_t* st) {
    auto conv = [](const int64_t (&a)[3]) {
        Strides r;
        r.b = a[0]; r.h = a[1]; r.n = a[2];
        return r;
    };
    const Strides cq = contiguous_strides(p.Hq, p.N, p.D), ckv = contiguous_strides(p.Hkv, p.N, p.D);
    p.sq = st ? conv(st->q) : cq;
    p.sk = st ? conv(st->k) : ckv;
    p.sv = st ? conv(st->v) : ckv;
    p.so = st ? conv(st->o) : cq;
    p.sdo = st ? conv(st->d_o) : cq;
    p.sdq = st ? conv(st->dq) : cq;
    p.sdk = st ? conv(st->dk) : ckv;
    p.sdv = st ? conv(st->dv) : ckv;
}
// The tensor-core paths move rows with TMA and 16-byte vector accesses: base pointers and all strides must be multiples of 16 bytes.
bool vec_ok(const void* ptr, const Strides& st) {
    return ((uintptr_t)ptr % 16) == 0 && st.b % 8 == 0 && st.h % 8 == 0 && st.n % 8 == 0 && st.n > 0;
}
bool strides_positive(const Strides& st, int D) { return st.n >= D && st.b >= 0 && st.h >= 0; }

// ops whose kernel family is recorded: the fused-RoPE pair also stands for its variants
constexpr int kFamFwd = COROPE_OP_ROPE_FWD, kFamBwd = COROPE_OP_ROPE_BWD;

// The workspace layout a call runs with: the one with room for the split-operand kernels when the caller's workspace has
// it (corope_workspace_bytes_any_n), else the one of corope_workspace_bytes.
int pick_workspace(RopeWorkspace& w, bool bwd, int B, int Hq, int Hkv, int N, int D, int dtype, bool synth, const void* ws, size_t have) {
    w = rope_workspace_layout(bwd, B, Hq, Hkv, N, D, dtype, synth, true);
    if (have >= w.total) return check_workspace(ws, have, w.total);
    w = rope_workspace_layout(bwd, B, Hq, Hkv, N, D, dtype, synth, false);
    return check_workspace(ws, have, w.total);
}

// Tensor-core kernels: packed table in the workspace, or where the pre-pass gets it from.
int table_source(TableSource& src, const Rotation& rot, uint32_t* tab, int N, int D, cudaStream_t s) {
    if (rot.freqs) {
        src.packed = true;
        return launch_synth_packed(rot.inv_freq, rot.theta, tab, N, D / 2, s);
    }
    if (!rot.none) src.cos = rot.cos, src.sin = rot.sin, src.stride = rot.stride;
    return COROPE_OK;
}
// General kernels: fp32 tables.
int fp32_tables(RopeParams& p, const Rotation& rot, void* workspace, const RopeWorkspace& w, cudaStream_t s) {
    p.cos = rot.none ? nullptr : rot.cos; p.sin = rot.none ? nullptr : rot.sin; p.table_stride = rot.stride;
    if (!rot.freqs) return COROPE_OK;
    float* c = reinterpret_cast<float*>((char*)workspace + w.synth_cos);
    float* sn = reinterpret_cast<float*>((char*)workspace + w.synth_sin);
    p.cos = c; p.sin = sn; p.table_stride = p.D / 2;
    return launch_synth_tables(rot.inv_freq, rot.theta, c, sn, p.N, p.D / 2, s);
}

int rope_fwd_impl(const void* q, const void* k, const void* v, Rotation rot, void* o, float* lse2, int B, int Hq, int Hkv, int N, int D,
                  int dtype, int causal, float sm_scale, void* workspace, size_t workspace_bytes, int* status_word, void* stream,
                  const corope_strides_t* strides = nullptr) {
    if (!q || !k || !v || !o || !lse2) return COROPE_ERR_NULL_POINTER;
    if (!rot.none && !rot.freqs && (!rot.cos || !rot.sin)) return COROPE_ERR_NULL_POINTER;
    if (int e = check_common(B, Hq, N, D, dtype)) return e;
    if (Hkv <= 0 || Hq % Hkv != 0) return COROPE_ERR_BAD_GROUP;
    RopeWorkspace w;
    if (int e = pick_workspace(w, false, B, Hq, Hkv, N, D, dtype, rot.freqs, workspace, workspace_bytes)) return e;
    cudaStream_t s = (cudaStream_t)stream;
    RopeParams p{};
    p.q = q; p.k = k; p.v = v; p.out_o = o; p.lse2 = lse2;
    p.B = B; p.H = Hq; p.Hkv = Hkv; p.no_rope = rot.none ? 1 : 0;
    p.N = N; p.D = D; p.causal = causal ? 1 : 0; p.sm_scale = sm_scale; p.status = status_word; p.status_mirror = status_mirror_of(status_word);
    set_strides(p, strides, Hq, Hkv, N, D);
    if (!strides_positive(p.sq, D) || !strides_positive(p.sk, D) || !strides_positive(p.sv, D) || !strides_positive(p.so, D)) return COROPE_ERR_BAD_STRIDE;
    // rows are moved with TMA / 16-byte vectors on the tensor-core paths; otherwise the CUDA-core kernels take over
    const bool vec = vec_ok(q, p.sq) && vec_ok(k, p.sk) && vec_ok(v, p.sv) && vec_ok(o, p.so);
    const int policy = vec ? g_policy.load() : 1;
    if (w.tc && policy != 1) {
        uint32_t* tab = reinterpret_cast<uint32_t*>((char*)workspace + w.packed_tab);
        TableSource src;
        if (int e = table_source(src, rot, tab, N, D, s)) return e;
        p.packed_tab = tab;
        p.sched_counter = reinterpret_cast<int*>(tab + (size_t)N * (D / 2));
        // policy 2: every K tile is rotated in shared memory by the main kernel, nothing rotated is written to HBM (for plain
        // attention the "rotation" by the identity table is what brings K to fp16, the format Q is written in)
        if (policy == 0) {
            p.k_rot = (char*)workspace + w.rot;
            if (int e = launch_rope_fwd_prepass(p, src, tab, dtype, s)) return e;
        } else if (!src.packed) {
            if (int e = launch_pack_tables(src, tab, N, D / 2, s)) return e;
        }
        note_kernels(kFamFwd, 1, false);
        return launch_rope_fwd_tc(p, dtype, s);
    }
    if (int e = fp32_tables(p, rot, workspace, w, s)) return e;
    // rows that can be moved in 16-byte vectors, ragged N or fp32 of D = 64: split operands at fp32 accuracy (rope_split*.cu have both
    // sides' figures)
    const bool split = w.split && policy == 0;
    note_kernels(kFamFwd, 0, split);
    p.sched_counter = reinterpret_cast<int*>((char*)workspace + w.packed_tab) + (size_t)N * (D / 2);   // the table itself is not used
    if (split) return launch_rope_fwd_split(p, (char*)workspace + w.rot, dtype, s);
    return launch_rope_fwd_general(p, dtype, s);
}

int rope_bwd_impl(const void* q, const void* k, const void* v, const void* o, const void* d_o, const float* lse2, Rotation rot, void* dq,
                  void* dk, void* dv, int B, int Hq, int Hkv, int N, int D, int dtype, int causal, float sm_scale, void* workspace,
                  size_t workspace_bytes, int* status_word, void* stream, const corope_strides_t* strides = nullptr) {
    if (!q || !k || !v || !o || !d_o || !lse2 || !dq || !dk || !dv) return COROPE_ERR_NULL_POINTER;
    if (!rot.none && !rot.freqs && (!rot.cos || !rot.sin)) return COROPE_ERR_NULL_POINTER;
    if (int e = check_common(B, Hq, N, D, dtype)) return e;
    if (Hkv <= 0 || Hq % Hkv != 0) return COROPE_ERR_BAD_GROUP;
    RopeWorkspace w;
    if (int e = pick_workspace(w, true, B, Hq, Hkv, N, D, dtype, rot.freqs, workspace, workspace_bytes)) return e;
    cudaStream_t s = (cudaStream_t)stream;
    RopeParams p{};
    p.q = q; p.k = k; p.v = v; p.o = o; p.d_o = d_o; p.dq = dq; p.dk = dk; p.dv = dv;
    p.lse2 = const_cast<float*>(lse2);
    p.delta = reinterpret_cast<float*>((char*)workspace + w.delta);
    p.B = B; p.H = Hq; p.Hkv = Hkv; p.no_rope = rot.none ? 1 : 0;
    p.N = N; p.D = D; p.causal = causal ? 1 : 0; p.sm_scale = sm_scale; p.status = status_word; p.status_mirror = status_mirror_of(status_word);
    set_strides(p, strides, Hq, Hkv, N, D);
    for (const Strides* st : {&p.sq, &p.sk, &p.sv, &p.so, &p.sdo, &p.sdq, &p.sdk, &p.sdv})
        if (!strides_positive(*st, D)) return COROPE_ERR_BAD_STRIDE;
    const bool vec = vec_ok(q, p.sq) && vec_ok(k, p.sk) && vec_ok(v, p.sv) && vec_ok(o, p.so) && vec_ok(d_o, p.sdo) && vec_ok(dq, p.sdq) &&
                     vec_ok(dk, p.sdk) && vec_ok(dv, p.sdv);
    const int policy = vec ? g_policy.load() : 1;
    if (w.tc && policy != 1) {
        uint32_t* tab = reinterpret_cast<uint32_t*>((char*)workspace + w.packed_tab);
        TableSource src;
        if (int e = table_source(src, rot, tab, N, D, s)) return e;
        p.packed_tab = tab;
        p.sched_counter = reinterpret_cast<int*>(tab + (size_t)N * (D / 2));   // zeroed with the table
        p.dq_acc = reinterpret_cast<float*>((char*)workspace + w.dq_acc);
        if (policy == 0) {
            p.q_rot = (char*)workspace + w.rot;
            if (int e = launch_rope_bwd_prepass(p, src, tab, dtype, s)) return e;   // table, delta, rotated Q, cleared dQ accumulator
            p.dq_acc_zeroed = 1;
        } else {   // policy 2: every Q tile is rotated in shared memory by the main kernel, nothing rotated is written to HBM
            if (int e = launch_rope_delta(p, dtype, s)) return e;
            if (!src.packed)
                if (int e = launch_pack_tables(src, tab, N, D / 2, s)) return e;
        }
        note_kernels(kFamBwd, 1, false);
        return launch_rope_bwd_tc(p, dtype, s);
    }
    if (int e = fp32_tables(p, rot, workspace, w, s)) return e;
    const bool split = w.split && policy == 0 && (dtype == COROPE_DTYPE_F32 || (no_shared_heads(p.sv, B, Hkv) && no_shared_heads(p.sdo, B, Hq)));
    note_kernels(kFamBwd, 0, split);
    p.sched_counter = reinterpret_cast<int*>((char*)workspace + w.packed_tab) + (size_t)N * (D / 2);   // the table itself is not used
    if (split) return launch_rope_bwd_split(p, (char*)workspace + w.rot, dtype, s);
    if (dtype == COROPE_DTYPE_F32) return launch_rope_bwd_fp32(p, s);
    if (int e = launch_rope_delta(p, dtype, s)) return e;
    return launch_rope_bwd_general(p, dtype, s);
}

Rotation from_tables(const float* cos, const float* sin, int64_t stride) {
    Rotation r;
    r.cos = cos; r.sin = sin; r.stride = stride;
    return r;
}
Rotation from_freqs(const float* inv_freq) {
    Rotation r;
    r.inv_freq = inv_freq;
    r.freqs = true;
    return r;
}
Rotation from_theta(float theta) {
    Rotation r;
    r.theta = theta;
    r.freqs = true;
    return r;
}
Rotation no_rotation() {
    Rotation r;
    r.none = true;
    return r;
}

}  // namespace

int* corope::status_mirror_of(const int* status_word) {
    if (status_word)
        for (const MirrorPair& p : g_pairs) {
            const int* w = p.word.load();
            if (w == status_word) return p.mirror.load();
            if (w == nullptr) break;
        }
    return nullptr;
}

extern "C" {

int corope_rope_attn_fwd(const void* q, const void* k, const void* v, const float* cos, const float* sin, int64_t table_row_stride, void* o,
                         float* lse2, int B, int H, int N, int D, int dtype, int causal, float sm_scale, void* workspace,
                         size_t workspace_bytes, int* status_word, void* stream) {
    return rope_fwd_impl(q, k, v, from_tables(cos, sin, table_row_stride), o, lse2, B, H, H, N, D, dtype, causal, sm_scale, workspace,
                         workspace_bytes, status_word, stream);
}

int corope_rope_attn_bwd(const void* q, const void* k, const void* v, const void* o, const void* d_o, const float* lse2, const float* cos,
                         const float* sin, int64_t table_row_stride, void* dq, void* dk, void* dv, int B, int H, int N, int D, int dtype,
                         int causal, float sm_scale, void* workspace, size_t workspace_bytes, int* status_word, void* stream) {
    return rope_bwd_impl(q, k, v, o, d_o, lse2, from_tables(cos, sin, table_row_stride), dq, dk, dv, B, H, H, N, D, dtype, causal, sm_scale,
                         workspace, workspace_bytes, status_word, stream);
}

int corope_rope_attn_fwd_strided(const void* q, const void* k, const void* v, const float* cos, const float* sin, int64_t table_row_stride,
                                 void* o, float* lse2, int B, int H, int N, int D, int dtype, int causal, float sm_scale, void* workspace,
                                 size_t workspace_bytes, int* status_word, void* stream, const corope_strides_t* strides) {
    return rope_fwd_impl(q, k, v, from_tables(cos, sin, table_row_stride), o, lse2, B, H, H, N, D, dtype, causal, sm_scale, workspace,
                         workspace_bytes, status_word, stream, strides);
}

int corope_rope_attn_bwd_strided(const void* q, const void* k, const void* v, const void* o, const void* d_o, const float* lse2,
                                 const float* cos, const float* sin, int64_t table_row_stride, void* dq, void* dk, void* dv, int B, int H,
                                 int N, int D, int dtype, int causal, float sm_scale, void* workspace, size_t workspace_bytes,
                                 int* status_word, void* stream, const corope_strides_t* strides) {
    return rope_bwd_impl(q, k, v, o, d_o, lse2, from_tables(cos, sin, table_row_stride), dq, dk, dv, B, H, H, N, D, dtype, causal, sm_scale,
                         workspace, workspace_bytes, status_word, stream, strides);
}

int corope_flash_attn_fwd_strided(const void* q, const void* k, const void* v, void* o, float* lse2, int B, int Hq, int Hkv, int N, int D,
                                  int dtype, int causal, float sm_scale, void* workspace, size_t workspace_bytes, int* status_word,
                                  void* stream, const corope_strides_t* strides) {
    return rope_fwd_impl(q, k, v, no_rotation(), o, lse2, B, Hq, Hkv, N, D, dtype, causal, sm_scale, workspace, workspace_bytes, status_word,
                         stream, strides);
}

int corope_flash_attn_bwd_strided(const void* q, const void* k, const void* v, const void* o, const void* d_o, const float* lse2, void* dq,
                                  void* dk, void* dv, int B, int Hq, int Hkv, int N, int D, int dtype, int causal, float sm_scale,
                                  void* workspace, size_t workspace_bytes, int* status_word, void* stream,
                                  const corope_strides_t* strides) {
    return rope_bwd_impl(q, k, v, o, d_o, lse2, no_rotation(), dq, dk, dv, B, Hq, Hkv, N, D, dtype, causal, sm_scale, workspace,
                         workspace_bytes, status_word, stream, strides);
}

int corope_rope_attn_fwd_freqs(const void* q, const void* k, const void* v, const float* inv_freq, void* o, float* lse2, int B, int H, int N,
                               int D, int dtype, int causal, float sm_scale, void* workspace, size_t workspace_bytes, int* status_word,
                               void* stream) {
    if (!inv_freq) return COROPE_ERR_NULL_POINTER;
    return rope_fwd_impl(q, k, v, from_freqs(inv_freq), o, lse2, B, H, H, N, D, dtype, causal, sm_scale, workspace, workspace_bytes,
                         status_word, stream);
}

int corope_rope_attn_bwd_freqs(const void* q, const void* k, const void* v, const void* o, const void* d_o, const float* lse2,
                               const float* inv_freq, void* dq, void* dk, void* dv, int B, int H, int N, int D, int dtype, int causal,
                               float sm_scale, void* workspace, size_t workspace_bytes, int* status_word, void* stream) {
    if (!inv_freq) return COROPE_ERR_NULL_POINTER;
    return rope_bwd_impl(q, k, v, o, d_o, lse2, from_freqs(inv_freq), dq, dk, dv, B, H, H, N, D, dtype, causal, sm_scale, workspace,
                         workspace_bytes, status_word, stream);
}

int corope_rope_attn_fwd_theta(const void* q, const void* k, const void* v, float theta, void* o, float* lse2, int B, int H, int N, int D,
                               int dtype, int causal, float sm_scale, void* workspace, size_t workspace_bytes, int* status_word, void* stream,
                               const corope_strides_t* strides) {
    return rope_fwd_impl(q, k, v, from_theta(theta), o, lse2, B, H, H, N, D, dtype, causal, sm_scale, workspace, workspace_bytes, status_word,
                         stream, strides);
}

int corope_rope_attn_bwd_theta(const void* q, const void* k, const void* v, const void* o, const void* d_o, const float* lse2, float theta,
                               void* dq, void* dk, void* dv, int B, int H, int N, int D, int dtype, int causal, float sm_scale,
                               void* workspace, size_t workspace_bytes, int* status_word, void* stream, const corope_strides_t* strides) {
    return rope_bwd_impl(q, k, v, o, d_o, lse2, from_theta(theta), dq, dk, dv, B, H, H, N, D, dtype, causal, sm_scale, workspace,
                         workspace_bytes, status_word, stream, strides);
}

int corope_flash_attn_fwd(const void* q, const void* k, const void* v, void* o, float* lse2, int B, int Hq, int Hkv, int N, int D, int dtype,
                          int causal, float sm_scale, void* workspace, size_t workspace_bytes, int* status_word, void* stream) {
    return rope_fwd_impl(q, k, v, no_rotation(), o, lse2, B, Hq, Hkv, N, D, dtype, causal, sm_scale, workspace, workspace_bytes, status_word,
                         stream);
}

int corope_flash_attn_bwd(const void* q, const void* k, const void* v, const void* o, const void* d_o, const float* lse2, void* dq, void* dk,
                          void* dv, int B, int Hq, int Hkv, int N, int D, int dtype, int causal, float sm_scale, void* workspace,
                          size_t workspace_bytes, int* status_word, void* stream) {
    return rope_bwd_impl(q, k, v, o, d_o, lse2, no_rotation(), dq, dk, dv, B, Hq, Hkv, N, D, dtype, causal, sm_scale, workspace,
                         workspace_bytes, status_word, stream);
}

static int check_gqa(int B, int Hq, int Hkv, int N, int D, int dtype) {
    if (B <= 0 || Hq <= 0 || Hkv <= 0 || N <= 0 || D <= 0) return COROPE_ERR_BAD_SHAPE;
    if (Hq % Hkv != 0 || Hq / Hkv > 8) return COROPE_ERR_BAD_GROUP;
    return check_common(B, Hq, N, D, dtype);
}

int corope_gqa_fwd(const void* q, const void* k, const void* v, void* o, float* lse2, float* a_diag, int B, int Hq, int Hkv, int N, int D,
                   int dtype, float sm_scale, float theta, void* workspace, size_t workspace_bytes, int* status_word, void* stream) {
    return corope_gqa_fwd_strided(q, k, v, o, lse2, a_diag, B, Hq, Hkv, N, D, dtype, sm_scale, theta, workspace, workspace_bytes, status_word,
                                  stream, nullptr);
}

int corope_gqa_fwd_strided(const void* q, const void* k, const void* v, void* o, float* lse2, float* a_diag, int B, int Hq, int Hkv, int N,
                           int D, int dtype, float sm_scale, float theta, void* workspace, size_t workspace_bytes, int* status_word,
                           void* stream, const corope_strides_t* strides) {
    if (!q || !k || !v || !o || !lse2 || !a_diag) return COROPE_ERR_NULL_POINTER;
    if (int e = check_gqa(B, Hq, Hkv, N, D, dtype)) return e;
    GqaWorkspace w = gqa_workspace_layout(false, B, Hq, Hkv, N, D, dtype, false);
    if (int e = check_workspace(workspace, workspace_bytes, w.total)) return e;
    GqaParams p{};
    p.q = q; p.k = k; p.v = v; p.out_o = o; p.lse2 = lse2; p.a_diag = a_diag;
    p.B = B; p.Hq = Hq; p.Hkv = Hkv; p.G = Hq / Hkv; p.N = N; p.D = D; p.sm_scale = sm_scale; p.theta = theta; p.status = status_word; p.status_mirror = status_mirror_of(status_word);
    set_gqa_strides(p, strides);
    if (!strides_positive(p.sq, D) || !strides_positive(p.sk, D) || !strides_positive(p.sv, D) || !strides_positive(p.so, D)) return COROPE_ERR_BAD_STRIDE;
    // the tensor-core kernels read K and V in 16-byte vectors and store O in element pairs
    if (g_policy.load() == 0 && gqa_fwd_mma_supported(N, D, dtype) && vec_ok(q, p.sq) && vec_ok(k, p.sk) && vec_ok(v, p.sv) && vec_ok(o, p.so)) {
        p.k_pairs = reinterpret_cast<uint32_t*>((char*)workspace + w.k_pairs);
        p.v_half = reinterpret_cast<__half*>((char*)workspace + w.v_half);
        note_kernels(COROPE_OP_GQA_FWD, 1, false);
        return launch_gqa_fwd_mma(p, dtype, (cudaStream_t)stream);
    }
    // D = 64, a ragged N, or rows that the mma kernels cannot read: fp32 accuracy on tensor cores where the workspace has room
    const GqaWorkspace any = gqa_workspace_layout(false, B, Hq, Hkv, N, D, dtype, true);
    const bool split = g_policy.load() == 0 && gqa_split_supported(D, dtype) && workspace_bytes >= any.total;
    note_kernels(COROPE_OP_GQA_FWD, 0, split);
    if (split) {
        p.k_pairs = reinterpret_cast<uint32_t*>((char*)workspace + any.k_pairs);
        p.v_half = reinterpret_cast<__half*>((char*)workspace + any.v_half);
        p.k_scale = reinterpret_cast<float*>((char*)workspace + any.k_scale);
        return launch_gqa_fwd_split(p, vec_ok(k, p.sk), vec_ok(v, p.sv), dtype, (cudaStream_t)stream);
    }
    return launch_gqa_fwd_general(p, dtype, (cudaStream_t)stream);
}

int corope_gqa_bwd(const void* q, const void* k, const void* v, const void* o, const void* d_o, const float* lse2, const float* a_diag,
                   void* dq, void* dk, void* dv, int B, int Hq, int Hkv, int N, int D, int dtype, float sm_scale, float theta,
                   void* workspace, size_t workspace_bytes, int* status_word, void* stream) {
    return corope_gqa_bwd_strided(q, k, v, o, d_o, lse2, a_diag, dq, dk, dv, B, Hq, Hkv, N, D, dtype, sm_scale, theta, workspace,
                                  workspace_bytes, status_word, stream, nullptr);
}

int corope_gqa_bwd_strided(const void* q, const void* k, const void* v, const void* o, const void* d_o, const float* lse2,
                           const float* a_diag, void* dq, void* dk, void* dv, int B, int Hq, int Hkv, int N, int D, int dtype,
                           float sm_scale, float theta, void* workspace, size_t workspace_bytes, int* status_word, void* stream,
                           const corope_strides_t* strides) {
    if (!q || !k || !v || !o || !d_o || !lse2 || !a_diag || !dq || !dk || !dv) return COROPE_ERR_NULL_POINTER;
    if (int e = check_gqa(B, Hq, Hkv, N, D, dtype)) return e;
    GqaWorkspace w = gqa_workspace_layout(true, B, Hq, Hkv, N, D, dtype, false);
    if (int e = check_workspace(workspace, workspace_bytes, w.total)) return e;
    GqaParams p{};
    p.q = q; p.k = k; p.v = v; p.o = o; p.d_o = d_o; p.dq = dq; p.dk = dk; p.dv = dv;
    p.lse2 = const_cast<float*>(lse2); p.a_diag = const_cast<float*>(a_diag);
    p.delta = reinterpret_cast<float*>((char*)workspace + w.delta);
    p.dk_acc = reinterpret_cast<float*>((char*)workspace + w.dk_acc);
    p.dv_acc = reinterpret_cast<float*>((char*)workspace + w.dv_acc);
    p.B = B; p.Hq = Hq; p.Hkv = Hkv; p.G = Hq / Hkv; p.N = N; p.D = D; p.sm_scale = sm_scale; p.theta = theta; p.status = status_word; p.status_mirror = status_mirror_of(status_word);
    set_gqa_strides(p, strides);
    for (const Strides* st : {&p.sq, &p.sk, &p.sv, &p.so, &p.sdo, &p.sdq, &p.sdk, &p.sdv})
        if (!strides_positive(*st, D)) return COROPE_ERR_BAD_STRIDE;
    const bool vec = vec_ok(q, p.sq) && vec_ok(k, p.sk) && vec_ok(v, p.sv) && vec_ok(o, p.so) && vec_ok(d_o, p.sdo) && vec_ok(dq, p.sdq) &&
                     vec_ok(dk, p.sdk) && vec_ok(dv, p.sdv);
    if (g_policy.load() == 0 && gqa_fwd_mma_supported(N, D, dtype) && vec) {
        p.k_pairs = reinterpret_cast<uint32_t*>((char*)workspace + w.k_pairs);
        p.v_half = reinterpret_cast<__half*>((char*)workspace + w.v_half);
        p.use_mma = 1;
    }
    note_kernels(COROPE_OP_GQA_BWD, p.use_mma, false);
    return launch_gqa_bwd_general(p, dtype, (cudaStream_t)stream);
}

}  // extern "C"
