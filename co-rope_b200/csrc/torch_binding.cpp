// Host path of the Python entry points: argument checks, layouts, workspaces and autograd nodes in C++, calling the C ABI of
// include/corope_b200.h.  A forward + backward through Python (ctypes calls, torch.autograd.Function) cost 210 us of host time per
// step, more than the kernels of every small shape take; this path costs a fraction of it.
//
// The checks and their exceptions are those of the reference's entry points: fused-rope/fused_rope_attn.py:657-661,
// fused-rope/flash_attn_v2_triton.py:517-521, corope-exp/flash_attn_co_rope_gqa_triton.py:407-425.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/extension.h>

#include <mutex>
#include <stdexcept>

#include "../../include/corope_b200.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

struct AssertError : std::runtime_error {   // surfaces as AssertionError
    using std::runtime_error::runtime_error;
};
struct ValueError : std::runtime_error {    // surfaces as ValueError
    using std::runtime_error::runtime_error;
};
void require(bool ok, const char* what) {
    if (!ok) throw AssertError(what);
}
void require_value(bool ok, const std::string& what) {
    if (!ok) throw ValueError(what);
}

// ------------------------------------------------------------------------------------------------ device status
// The status word of one GPU and its pinned host mirror.  The kernels write the mirror themselves when they fail, so looking at
// it before a call costs one host load and no copy is enqueued behind the call.
struct DeviceStatus {
    Tensor word, mirror;
    int* word_ptr = nullptr;
    volatile int* mirror_ptr = nullptr;
};
constexpr int kMaxDevices = 64;
DeviceStatus g_status[kMaxDevices];
std::once_flag g_status_once[kMaxDevices];

DeviceStatus& device_status(int index) {
    TORCH_CHECK(index >= 0 && index < kMaxDevices, "corope_b200: device index out of range");
    std::call_once(g_status_once[index], [index] {
        DeviceStatus& st = g_status[index];
        st.word = at::zeros({1}, at::TensorOptions().dtype(at::kInt).device(at::kCUDA, index));
        st.mirror = at::zeros({1}, at::TensorOptions().dtype(at::kInt)).pin_memory();
        st.word_ptr = st.word.data_ptr<int>();
        st.mirror_ptr = st.mirror.data_ptr<int>();
        const int rc = corope_status_mirror_register(st.word_ptr, const_cast<int*>(st.mirror_ptr));
        TORCH_CHECK(rc == 0, "corope_b200: the status mirror could not be registered (", rc, ")");
    });
    return g_status[index];
}

std::string status_message(int v) {
    if (v & 0x2000)
        return "a gradient term left the value range of the 16-bit Co-RoPE backward and was clamped (results of that call are inaccurate)";
    return "a bounded device-side wait expired (results of that call and of later calls are undefined)";
}

// Raises if an earlier call on this device left the status word set; clears it first.
void look_at_status(DeviceStatus& st, cudaStream_t stream) {
    const int v = *st.mirror_ptr;
    if (v == 0) return;
    corope_status_mirror_clear(st.word_ptr, const_cast<int*>(st.mirror_ptr), stream);
    char text[64];
    snprintf(text, sizeof text, "corope_b200: an earlier kernel reported device status 0x%x: ", v);
    throw std::runtime_error(text + status_message(v));
}

void raise_for_status(int rc, const char* what) {
    if (rc == 0) return;
    const std::string msg = corope_status_string(rc);
    if (rc == COROPE_ERR_BAD_HEAD_DIM) throw AssertError(std::string(what) + ": " + msg);
    if (rc == COROPE_ERR_BAD_GROUP) throw ValueError(std::string(what) + ": " + msg);
    throw std::runtime_error(std::string(what) + " failed with status " + std::to_string(rc) + ": " + msg);
}

// ------------------------------------------------------------------------------------------------ tensors
int dtype_code(const Tensor& t) {
    switch (t.scalar_type()) {
        case at::kFloat: return COROPE_DTYPE_F32;
        case at::kBFloat16: return COROPE_DTYPE_BF16;
        case at::kHalf: return COROPE_DTYPE_F16;
        default: return -1;
    }
}
void require_cuda(const Tensor& t) {
    if (!t.is_cuda())
        throw std::runtime_error("corope_b200 runs on CUDA tensors only (got a " + c10::DeviceTypeName(t.device().type(), true) +
                                 " tensor); there is no CPU path.");
}
// `t` itself when the kernels can take its layout (unit stride along the head dimension, no overlapping or broadcast strides),
// else a contiguous copy.
Tensor kernel_layout(const Tensor& t) {
    const auto st = t.strides();
    if (st[3] == 1 && st[0] > 0 && st[1] > 0 && st[2] >= t.size(3)) return t;
    return t.contiguous();
}
// Outputs and gradients: laid out like the input, or contiguous (the entry point that takes theta)
Tensor new_like(const Tensor& t, bool contiguous) { return contiguous ? at::empty(t.sizes(), t.options()) : at::empty_like(t); }
void set_strides(int64_t (&dst)[3], const Tensor& t) {
    const auto st = t.strides();
    dst[0] = st[0]; dst[1] = st[1]; dst[2] = st[2];
}

// Everything one library call needs besides its tensors.
struct Call {
    c10::cuda::CUDAGuard guard;
    cudaStream_t stream;
    DeviceStatus& status;
    explicit Call(const Tensor& t) : guard(t.device()), stream(at::cuda::getCurrentCUDAStream(t.device().index())), status(device_status(t.device().index())) {
        look_at_status(status, stream);
    }
};
struct Workspace {
    Tensor buf;
    size_t bytes;
    Workspace(int op, int64_t B, int64_t Hq, int64_t Hkv, int64_t N, int64_t D, int dtype, const Tensor& like) {
        bytes = corope_workspace_bytes_any_n(op, (int)B, (int)Hq, (int)Hkv, (int)N, (int)D, dtype);
        auto allocate = [&] { buf = at::empty({(int64_t)std::max<size_t>(bytes, 256)}, like.options().dtype(at::kByte)); };
        try {
            allocate();
        } catch (const c10::OutOfMemoryError&) {   // the split copies are for speed: without them a call runs on the CUDA cores
            const size_t least = corope_workspace_bytes(op, (int)B, (int)Hq, (int)Hkv, (int)N, (int)D, dtype);
            if (least >= bytes) throw;
            bytes = least;
            allocate();
        }
    }
    void* ptr() const { return buf.data_ptr(); }
};
Tensor new_rows(const Tensor& like, int64_t B, int64_t H, int64_t N) { return at::empty({B, H, N}, like.options().dtype(at::kFloat)); }

// RoPE tables: fp32, unit column stride, one row stride for both
struct Tables {
    Tensor cos, sin;
    int64_t stride;
};
Tables tables(const Tensor& freqs_cos, const Tensor& freqs_sin, int64_t N, int64_t D) {
    require_value(freqs_cos.dim() == 2 && freqs_cos.sizes() == freqs_sin.sizes(), "freqs_cos and freqs_sin must be 2-D tensors of the same shape");
    if (freqs_cos.size(0) < N || freqs_cos.size(1) < D / 2) {
        std::ostringstream os;
        os << "RoPE tables must cover [N, D/2] = [" << N << ", " << D / 2 << "], got (" << freqs_cos.size(0) << ", " << freqs_cos.size(1) << ")";
        throw ValueError(os.str());
    }
    auto fix = [](const Tensor& t) {
        require_cuda(t);
        return t.scalar_type() == at::kFloat && t.stride(1) == 1 ? t : t.to(at::kFloat).contiguous();
    };
    Tables r{fix(freqs_cos), fix(freqs_sin), 0};
    if (r.cos.stride(0) != r.sin.stride(0)) r.cos = r.cos.contiguous(), r.sin = r.sin.contiguous();
    r.stride = r.cos.stride(0);
    return r;
}

// checks shared by the fused-RoPE and the plain entry points
void check_mha(const Tensor& q, const Tensor& k, const Tensor& v, bool grouped) {
    require(q.dim() >= 1 && k.dim() >= 1 && v.dim() >= 1, "q, k, v must be 4-D tensors");
    const int64_t D = k.size(-1);
    require(q.size(-1) == D && D == v.size(-1), "q, k and v must share one head dimension");
    require(D == 32 || D == 64 || D == 128, "corope_b200 supports head dims (32, 64, 128)");
    require(q.dim() == 4 && k.sizes() == v.sizes(), "q, k, v must be [B, H, N, D] tensors, k and v of one shape");
    if (grouped) {
        require(k.dim() == 4 && q.size(0) == k.size(0) && q.size(2) == k.size(2), "q and k must agree in batch and sequence length");
    } else {
        require(q.sizes() == k.sizes(), "q, k and v must share one shape");
    }
    require(q.scalar_type() == k.scalar_type() && q.scalar_type() == v.scalar_type() && dtype_code(q) >= 0,
            "q, k, v must share one dtype out of float32, bfloat16, float16");
    if (grouped) require(k.size(1) > 0 && q.size(1) % k.size(1) == 0, "number of query heads must be a multiple of the number of K / V heads");
    for (const Tensor* t : {&q, &k, &v}) require_cuda(*t);
}

// ------------------------------------------------------------------------------------------------ attention with rotation or without
enum Kind { kRope, kTheta, kFlash };

struct Saved {
    Tensor q, k, v, o, m;
    Tables tab;   // kRope only
};

Saved mha_forward(Kind kind, const Tensor& q_in, const Tensor& k_in, const Tensor& v_in, bool causal, double sm_scale, const Tensor& freqs_cos,
                  const Tensor& freqs_sin, double theta) {
    check_mha(q_in, k_in, v_in, kind == kFlash);
    const int64_t B = q_in.size(0), Hq = q_in.size(1), N = q_in.size(2), D = q_in.size(3), Hkv = k_in.size(1);
    const int dt = dtype_code(q_in);
    Saved s;
    if (kind == kRope) s.tab = tables(freqs_cos, freqs_sin, N, D);
    Call call(q_in);
    s.q = kernel_layout(q_in);
    s.k = kernel_layout(k_in);
    s.v = kernel_layout(v_in);
    s.o = new_like(s.q, kind == kTheta);
    s.m = new_rows(s.q, B, Hq, N);
    const int op = kind == kRope ? COROPE_OP_ROPE_FWD : kind == kTheta ? COROPE_OP_ROPE_FWD_FREQS : COROPE_OP_FLASH_FWD;
    Workspace ws(op, B, Hq, Hkv, N, D, dt, s.q);
    corope_strides_t st{};
    set_strides(st.q, s.q);
    set_strides(st.k, s.k);
    set_strides(st.v, s.v);
    set_strides(st.o, s.o);
    float* m = s.m.data_ptr<float>();
    const int Bi = (int)B, Hi = (int)Hq, Ni = (int)N, Di = (int)D, ca = causal ? 1 : 0;
    const float sc = (float)sm_scale;
    if (kind == kRope) {
        raise_for_status(corope_rope_attn_fwd_strided(s.q.data_ptr(), s.k.data_ptr(), s.v.data_ptr(), s.tab.cos.data_ptr<float>(),
                                                      s.tab.sin.data_ptr<float>(), s.tab.stride, s.o.data_ptr(), m, Bi, Hi, Ni, Di, dt, ca, sc, ws.ptr(),
                                                      ws.bytes, call.status.word_ptr, call.stream, &st),
                         "corope_rope_attn_fwd");
    } else if (kind == kTheta) {
        raise_for_status(corope_rope_attn_fwd_theta(s.q.data_ptr(), s.k.data_ptr(), s.v.data_ptr(), (float)theta, s.o.data_ptr(), m, Bi, Hi, Ni, Di, dt, ca,
                                                    sc, ws.ptr(), ws.bytes, call.status.word_ptr, call.stream, &st),
                         "corope_rope_attn_fwd_theta");
    } else {
        raise_for_status(corope_flash_attn_fwd_strided(s.q.data_ptr(), s.k.data_ptr(), s.v.data_ptr(), s.o.data_ptr(), m, Bi, Hi, (int)Hkv, Ni, Di, dt, ca,
                                                       sc, ws.ptr(), ws.bytes, call.status.word_ptr, call.stream, &st),
                         "corope_flash_attn_fwd");
    }
    return s;
}

struct Grads {
    Tensor dq, dk, dv;
};

// The reference asserts a contiguous dO, equal strides and N % 128 == 0 (fused_rope_attn.py:727-728, 750); these kernels take any N
// and every tensor's own strides.
Grads mha_backward(Kind kind, const Saved& s, const Tensor& d_out, bool causal, double sm_scale, double theta) {
    const int64_t B = s.q.size(0), Hq = s.q.size(1), N = s.q.size(2), D = s.q.size(3), Hkv = s.k.size(1);
    const int dt = dtype_code(s.q);
    Call call(s.q);
    const Tensor d_o = kernel_layout(d_out);
    TORCH_CHECK(d_o.is_cuda() && d_o.scalar_type() == s.q.scalar_type() && d_o.sizes() == s.o.sizes(), "dO must match o");
    Grads g{new_like(s.q, kind == kTheta), new_like(s.k, kind == kTheta), new_like(s.v, kind == kTheta)};
    const int op = kind == kRope ? COROPE_OP_ROPE_BWD : kind == kTheta ? COROPE_OP_ROPE_BWD_FREQS : COROPE_OP_FLASH_BWD;
    Workspace ws(op, B, Hq, Hkv, N, D, dt, s.q);
    corope_strides_t st;
    set_strides(st.q, s.q);
    set_strides(st.k, s.k);
    set_strides(st.v, s.v);
    set_strides(st.o, s.o);
    set_strides(st.d_o, d_o);
    set_strides(st.dq, g.dq);
    set_strides(st.dk, g.dk);
    set_strides(st.dv, g.dv);
    const float* m = s.m.data_ptr<float>();
    const int Bi = (int)B, Hi = (int)Hq, Ni = (int)N, Di = (int)D, ca = causal ? 1 : 0;
    const float sc = (float)sm_scale;
    if (kind == kRope) {
        raise_for_status(corope_rope_attn_bwd_strided(s.q.data_ptr(), s.k.data_ptr(), s.v.data_ptr(), s.o.data_ptr(), d_o.data_ptr(), m,
                                                      s.tab.cos.data_ptr<float>(), s.tab.sin.data_ptr<float>(), s.tab.stride, g.dq.data_ptr(), g.dk.data_ptr(),
                                                      g.dv.data_ptr(), Bi, Hi, Ni, Di, dt, ca, sc, ws.ptr(), ws.bytes, call.status.word_ptr, call.stream, &st),
                         "corope_rope_attn_bwd");
    } else if (kind == kTheta) {
        raise_for_status(corope_rope_attn_bwd_theta(s.q.data_ptr(), s.k.data_ptr(), s.v.data_ptr(), s.o.data_ptr(), d_o.data_ptr(), m, (float)theta,
                                                    g.dq.data_ptr(), g.dk.data_ptr(), g.dv.data_ptr(), Bi, Hi, Ni, Di, dt, ca, sc, ws.ptr(), ws.bytes,
                                                    call.status.word_ptr, call.stream, &st),
                         "corope_rope_attn_bwd_theta");
    } else {
        raise_for_status(corope_flash_attn_bwd_strided(s.q.data_ptr(), s.k.data_ptr(), s.v.data_ptr(), s.o.data_ptr(), d_o.data_ptr(), m, g.dq.data_ptr(),
                                                       g.dk.data_ptr(), g.dv.data_ptr(), Bi, Hi, (int)Hkv, Ni, Di, dt, ca, sc, ws.ptr(), ws.bytes,
                                                       call.status.word_ptr, call.stream, &st),
                         "corope_flash_attn_bwd");
    }
    return g;
}

// ------------------------------------------------------------------------------------------------ Co-RoPE
struct GqaSaved {
    Tensor q, k, v, o, lse2, a_diag;
};

GqaSaved gqa_forward(const Tensor& q_in, const Tensor& k_in, const Tensor& v_in, bool causal, double sm_scale, double theta) {
    require_value(causal, "CoRoPE fused kernel supports causal=True only.");
    require_value(q_in.dim() == 4 && k_in.dim() == 4 && v_in.dim() == 4, "Expected q, k, v to have shape (batch, heads, seqlen, dim).");
    require_value(k_in.sizes() == v_in.sizes(), "k and v must share the same shape in GQA.");
    require_value(q_in.size(0) == k_in.size(0) && q_in.size(2) == k_in.size(2) && q_in.size(3) == k_in.size(3),
                  "k must align with q along batch/sequence/head_dim.");
    const int64_t B = q_in.size(0), Hq = q_in.size(1), N = q_in.size(2), D = q_in.size(3), Hkv = k_in.size(1);
    require_value(Hkv > 0 && Hq % Hkv == 0, "Number of query heads must be divisible by KV heads.");
    require_value(Hq / Hkv <= 8, "CoRoPE backbone currently limits group_size <= 8 (got " + std::to_string(Hq / Hkv) + ").");
    require_value(q_in.scalar_type() == k_in.scalar_type() && q_in.scalar_type() == v_in.scalar_type() && dtype_code(q_in) >= 0,
                  "q, k, v must share one dtype out of float32, bfloat16, float16.");
    for (const Tensor* t : {&q_in, &k_in, &v_in}) require_cuda(*t);
    const int dt = dtype_code(q_in);
    Call call(q_in);
    GqaSaved s;
    s.q = kernel_layout(q_in);
    s.k = kernel_layout(k_in);
    s.v = kernel_layout(v_in);
    s.o = at::empty_like(s.q);
    s.lse2 = new_rows(s.q, B, Hq, N);
    s.a_diag = new_rows(s.q, B, Hkv, N);
    Workspace ws(COROPE_OP_GQA_FWD, B, Hq, Hkv, N, D, dt, s.q);
    corope_strides_t st{};
    set_strides(st.q, s.q);
    set_strides(st.k, s.k);
    set_strides(st.v, s.v);
    set_strides(st.o, s.o);
    raise_for_status(corope_gqa_fwd_strided(s.q.data_ptr(), s.k.data_ptr(), s.v.data_ptr(), s.o.data_ptr(), s.lse2.data_ptr<float>(),
                                            s.a_diag.data_ptr<float>(), (int)B, (int)Hq, (int)Hkv, (int)N, (int)D, dt, (float)sm_scale, (float)theta, ws.ptr(),
                                            ws.bytes, call.status.word_ptr, call.stream, &st),
                     "corope_gqa_fwd");
    return s;
}

// dk / dv are summed over each group
Grads gqa_backward(const GqaSaved& s, const Tensor& d_out, double sm_scale, double theta) {
    const int64_t B = s.q.size(0), Hq = s.q.size(1), N = s.q.size(2), D = s.q.size(3), Hkv = s.k.size(1);
    const int dt = dtype_code(s.q);
    Call call(s.q);
    const Tensor d_o = kernel_layout(d_out);
    TORCH_CHECK(d_o.is_cuda() && d_o.scalar_type() == s.q.scalar_type() && d_o.sizes() == s.o.sizes(), "dO must match o");
    Grads g{at::empty_like(s.q), at::empty_like(s.k), at::empty_like(s.v)};
    Workspace ws(COROPE_OP_GQA_BWD, B, Hq, Hkv, N, D, dt, s.q);
    corope_strides_t st;
    set_strides(st.q, s.q);
    set_strides(st.k, s.k);
    set_strides(st.v, s.v);
    set_strides(st.o, s.o);
    set_strides(st.d_o, d_o);
    set_strides(st.dq, g.dq);
    set_strides(st.dk, g.dk);
    set_strides(st.dv, g.dv);
    raise_for_status(corope_gqa_bwd_strided(s.q.data_ptr(), s.k.data_ptr(), s.v.data_ptr(), s.o.data_ptr(), d_o.data_ptr(), s.lse2.data_ptr<float>(),
                                            s.a_diag.data_ptr<float>(), g.dq.data_ptr(), g.dk.data_ptr(), g.dv.data_ptr(), (int)B, (int)Hq, (int)Hkv, (int)N,
                                            (int)D, dt, (float)sm_scale, (float)theta, ws.ptr(), ws.bytes, call.status.word_ptr, call.stream, &st),
                     "corope_gqa_bwd");
    return g;
}

// ------------------------------------------------------------------------------------------------ autograd nodes
Tensor save(AutogradContext* ctx, Kind kind, const Saved& s, bool causal, double sm_scale, double theta) {
    variable_list t{s.q, s.k, s.v, s.o, s.m};
    if (kind == kRope) t.insert(t.end(), {s.tab.cos, s.tab.sin});
    ctx->save_for_backward(std::move(t));
    ctx->saved_data["kind"] = (int64_t)kind;
    ctx->saved_data["causal"] = causal;
    ctx->saved_data["sm_scale"] = sm_scale;
    ctx->saved_data["theta"] = theta;
    return s.o;
}
Grads saved_backward(AutogradContext* ctx, const Tensor& d_out) {
    const variable_list t = ctx->get_saved_variables();
    const Kind kind = (Kind)ctx->saved_data["kind"].toInt();
    Saved s{t[0], t[1], t[2], t[3], t[4], {}};
    if (kind == kRope) s.tab = Tables{t[5], t[6], t[5].stride(0)};
    return mha_backward(kind, s, d_out, ctx->saved_data["causal"].toBool(), ctx->saved_data["sm_scale"].toDouble(), ctx->saved_data["theta"].toDouble());
}

struct RopeFunction : torch::autograd::Function<RopeFunction> {
    static Tensor forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, bool causal, double sm_scale, const Tensor& cos,
                          const Tensor& sin) {
        return save(ctx, kRope, mha_forward(kRope, q, k, v, causal, sm_scale, cos, sin, 0.0), causal, sm_scale, 0.0);
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        Grads g = saved_backward(ctx, grads[0]);
        return {g.dq, g.dk, g.dv, Tensor(), Tensor(), Tensor(), Tensor()};
    }
};

struct MhaFunction : torch::autograd::Function<MhaFunction> {   // without table arguments
    static Tensor forward(AutogradContext* ctx, int64_t kind, const Tensor& q, const Tensor& k, const Tensor& v, bool causal, double sm_scale, double theta) {
        return save(ctx, (Kind)kind, mha_forward((Kind)kind, q, k, v, causal, sm_scale, Tensor(), Tensor(), theta), causal, sm_scale, theta);
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        Grads g = saved_backward(ctx, grads[0]);
        return {Tensor(), g.dq, g.dk, g.dv, Tensor(), Tensor(), Tensor()};
    }
};

struct GqaFunction : torch::autograd::Function<GqaFunction> {
    static Tensor forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, bool causal, double sm_scale, double theta) {
        GqaSaved s = gqa_forward(q, k, v, causal, sm_scale, theta);
        ctx->save_for_backward({s.q, s.k, s.v, s.o, s.lse2, s.a_diag});
        ctx->saved_data["sm_scale"] = sm_scale;
        ctx->saved_data["theta"] = theta;
        return s.o;
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const variable_list t = ctx->get_saved_variables();
        Grads g = gqa_backward(GqaSaved{t[0], t[1], t[2], t[3], t[4], t[5]}, grads[0], ctx->saved_data["sm_scale"].toDouble(),
                               ctx->saved_data["theta"].toDouble());
        return {g.dq, g.dk, g.dv, Tensor(), Tensor(), Tensor()};
    }
};

}  // namespace

PYBIND11_MODULE(_corope_torch, m) {
    py::register_exception_translator([](std::exception_ptr p) {
        try {
            if (p) std::rethrow_exception(p);
        } catch (const AssertError& e) {
            PyErr_SetString(PyExc_AssertionError, e.what());
        } catch (const ValueError& e) {
            PyErr_SetString(PyExc_ValueError, e.what());
        }
    });
    // The GIL is released for every call: a launch blocks once the launch queue is full, and other Python threads go on meanwhile.
    // autograd entry points
    using NoGil = py::call_guard<py::gil_scoped_release>;
    m.def("rope_attention", [](const Tensor& q, const Tensor& k, const Tensor& v, bool causal, double sm_scale, const Tensor& cos, const Tensor& sin) {
        return RopeFunction::apply(q, k, v, causal, sm_scale, cos, sin);
    }, NoGil());
    m.def("theta_attention", [](const Tensor& q, const Tensor& k, const Tensor& v, bool causal, double sm_scale, double theta) {
        return MhaFunction::apply((int64_t)kTheta, q, k, v, causal, sm_scale, theta);
    }, NoGil());
    m.def("flash_attention", [](const Tensor& q, const Tensor& k, const Tensor& v, bool causal, double sm_scale) {
        return MhaFunction::apply((int64_t)kFlash, q, k, v, causal, sm_scale, 0.0);
    }, NoGil());
    m.def("gqa_attention", [](const Tensor& q, const Tensor& k, const Tensor& v, bool causal, double sm_scale, double theta) {
        return GqaFunction::apply(q, k, v, causal, sm_scale, theta);
    }, NoGil());
    // the library calls alone, without autograd
    m.def("rope_forward", [](const Tensor& q, const Tensor& k, const Tensor& v, bool causal, double sm_scale, const Tensor& cos, const Tensor& sin) {
        Saved s = mha_forward(kRope, q, k, v, causal, sm_scale, cos, sin, 0.0);
        return std::make_tuple(s.q, s.k, s.v, s.o, s.m, s.tab.cos, s.tab.sin, s.tab.stride);
    }, NoGil());
    m.def("rope_backward", [](const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o, const Tensor& lse, const Tensor& cos, const Tensor& sin,
                              int64_t stride, const Tensor& d_o, bool causal, double sm_scale) {
        Grads g = mha_backward(kRope, Saved{q, k, v, o, lse, Tables{cos, sin, stride}}, d_o, causal, sm_scale, 0.0);
        return std::make_tuple(g.dq, g.dk, g.dv);
    }, NoGil());
    m.def("gqa_forward", [](const Tensor& q, const Tensor& k, const Tensor& v, bool causal, double sm_scale, double theta) {
        GqaSaved s = gqa_forward(q, k, v, causal, sm_scale, theta);
        return std::make_tuple(s.q, s.k, s.v, s.o, s.lse2, s.a_diag);
    }, NoGil());
    m.def("gqa_backward", [](const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o, const Tensor& lse2, const Tensor& a_diag, const Tensor& d_o,
                             double sm_scale, double theta) {
        Grads g = gqa_backward(GqaSaved{q, k, v, o, lse2, a_diag}, d_o, sm_scale, theta);
        return std::make_tuple(g.dq, g.dk, g.dv);
    }, NoGil());
    // (status word tensor, pinned mirror tensor) of a device, created on first use
    m.def("device_status", [](int index) {
        c10::cuda::CUDAGuard guard((c10::DeviceIndex)index);
        DeviceStatus& st = device_status(index);
        return std::make_tuple(st.word, st.mirror);
    }, NoGil());
}
