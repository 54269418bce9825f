// The operator's host path in native code: one call per forward, one autograd node for the
// backward, over the C ABI of libevoattn.so (include/evoattn.h).
//
// What it replaces is the Python body of TKEvoAttention.forward / backward for the plain case --
// CUDA tensors, a head dim the library takes as it is, no process group (tk_evo_attention_layer.py
// keeps that body for everything else).  At small sizes the step is host work: through Python,
// ctypes and torch's Python autograd node a forward + backward took 200 us of host time around
// 35 us of kernels.
//
// `apply` returns None for a call it does not handle (the Python body then runs, or raises the
// reference's own assertion); it never falls back to another implementation of the math.
#include <torch/extension.h>

#include <ATen/core/CachingHostAllocator.h>
#include <ATen/cuda/CUDAEvent.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>

#include "../../include/evoattn.h"

namespace {

using at::Tensor;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

bool supported_dim(int64_t d) { return d == 16 || d == 32 || d == 64 || d == 96 || d == 128; }

bool aligned(const Tensor& t) { return (reinterpret_cast<uintptr_t>(t.const_data_ptr()) & 15u) == 0; }

void check(int rc, const char* what) {
    if (rc == EVO_OK) return;
    std::string detail = evo_strerror(rc);
    if (rc == EVO_ERR_CUDA) detail += " (cudaError " + std::to_string(evo_last_cuda_error()) + ")";
    if (rc == EVO_ERR_TENSOR_MAP) detail += std::string(" (") + evo_last_error_detail() + ")";
    TORCH_CHECK(false, "libevoattn: ", what, " failed with ", rc, ": ", detail);
}

// Where q, k and v lie, and where the tensors this call allocates go.
struct Layout {
    bool in_view = false;      // q, k, v are read through `in`; otherwise contiguous
    bool out_view = false;     // o and the gradients carry the strides of q; otherwise contiguous
    EvoStrides in{};
    int64_t strides[5]{};      // of q
};

// q, k, v bf16 views with the same strides, contiguous head dim, steps of 16 bytes and (B, N_SEQ)
// flattenable can be read in place.  If the strides tile the storage without holes (a permutation of a
// contiguous tensor), outputs take them as well; a view with holes (sliced out of a fused projection)
// or with overlap does not qualify for that, one with overlap for neither.
Layout classify(const Tensor& q, const Tensor& k, const Tensor& v) {
    Layout l;
    if (q.is_contiguous()) return l;
    if (q.scalar_type() != at::kBFloat16 || k.scalar_type() != at::kBFloat16 || v.scalar_type() != at::kBFloat16) return l;
    const auto st = q.strides();
    if (k.strides() != st || v.strides() != st || st[4] != 1) return l;
    const auto sz = q.sizes();
    for (int i = 0; i < 4; ++i)
        if (sz[i] > 1 && (st[i] <= 0 || st[i] % 8 != 0)) return l;
    if (sz[0] > 1 && sz[1] > 1 && st[0] != sz[1] * st[1]) return l;
    int order[5] = {0, 1, 2, 3, 4};
    std::sort(order, order + 5, [&](int a, int b) { return st[a] != st[b] ? st[a] < st[b] : sz[a] < sz[b]; });
    bool dense = true;
    int64_t span = 1;
    for (int a : order) {
        if (sz[a] <= 1) continue;
        if (st[a] < span) return l;      // overlap
        if (st[a] != span) dense = false;
        span = st[a] * sz[a];
    }
    if (!aligned(q) || !aligned(k) || !aligned(v)) return l;
    l.in_view = true;
    l.out_view = dense;
    l.in = EvoStrides{st[0], st[1], st[2], st[3]};
    for (int i = 0; i < 5; ++i) l.strides[i] = st[i];
    return l;
}

Tensor bf16_contiguous(const Tensor& t) {
    return (t.scalar_type() == at::kBFloat16 ? t : t.to(at::kBFloat16)).contiguous();
}

Tensor empty_like_act(const Tensor& q, const Layout& l) {
    if (l.out_view)
        return at::detail::empty_strided_cuda(q.sizes(), at::IntArrayRef(l.strides, 5), at::kBFloat16, q.device());
    return at::detail::empty_cuda(q.sizes(), at::kBFloat16, q.device(), std::nullopt);
}

// `t` in the layout of the outputs, copied only if it is not there already.
Tensor as_output(const Tensor& t, const Tensor& q, const Layout& l) {
    if (l.out_view) {
        if (t.scalar_type() == at::kBFloat16 && t.strides() == at::IntArrayRef(l.strides, 5) && aligned(t)) return t;
        Tensor c = empty_like_act(q, l);
        c.copy_(t);
        return c;
    }
    Tensor c = bf16_contiguous(t);
    if (!aligned(c)) c = c.clone();
    return c;
}

// `t` contiguous, 16-byte aligned and of the given type, copied only if it is not.
Tensor plain(const Tensor& t, at::ScalarType type) {
    Tensor c = (t.scalar_type() == type ? t : t.to(type)).contiguous();
    return aligned(c) ? c : c.clone();
}

// Can q, k or v be read through the strides of `l`?
bool lies_as_input(const Tensor& t, const Layout& l) {
    return t.scalar_type() == at::kBFloat16 && t.strides() == at::IntArrayRef(l.strides, 5) && aligned(t);
}

struct Call {
    Tensor q, k, v, bias, mask, gate;      // gate: undefined without one
    Layout lay;
    EvoDims dims;
    float scale;
    at::ScalarType bias_type;
};

struct Forward {
    Tensor out, o, o_resid, lse;           // out: o, or the gated output
};

Forward run_forward(const Call& c, bool need_grad) {
    const c10::cuda::CUDAGuard guard(c.q.device());
    Forward f;
    f.o = empty_like_act(c.q, c.lay);
    Tensor gated;
    if (c.gate.defined()) gated = empty_like_act(c.q, c.lay);
    // rounding residual of O, kept for the backward only (accurate delta -> accurate dBias)
    if (need_grad) f.o_resid = empty_like_act(c.q, c.lay);
    f.lse = at::detail::empty_cuda({c.dims.B, c.dims.S, c.dims.H, c.dims.N}, at::kFloat, c.q.device(), std::nullopt);
    check(evo_fwd_views(&c.dims, c.lay.in_view ? &c.lay.in : nullptr, c.lay.out_view ? &c.lay.in : nullptr, c.q.const_data_ptr(),
                        c.k.const_data_ptr(), c.v.const_data_ptr(), c.bias.const_data_ptr(), c.mask.const_data_ptr(),
                        c.gate.defined() ? c.gate.const_data_ptr() : nullptr, f.o.data_ptr(),
                        gated.defined() ? gated.data_ptr() : nullptr, need_grad ? f.o_resid.data_ptr() : nullptr,
                        static_cast<float*>(f.lse.data_ptr()), c.scale, c10::cuda::getCurrentCUDAStream().stream()),
          "evo_fwd_views");
    f.out = gated.defined() ? gated : f.o;
    return f;
}

// The backward's autograd node.  Its edges are the operator's arguments in their order: q, k, v, res_mask (which gets no
// gradient), pair_bias and, with a gate, the place of process_group and the gate.  What is saved are the bf16, laid-out
// forms that the kernels read.
struct EvoBackward : public torch::autograd::Node {
    SavedVariable q, k, v, bias, mask, gate, o, o_resid, lse;
    bool gated = false;
    Layout lay;
    EvoDims dims{};
    c10::Device device = c10::Device(c10::DeviceType::CUDA, 0);
    float scale = 0.f;
    at::ScalarType bias_type = at::kBFloat16;

    std::string name() const override { return "TKEvoAttentionBackward"; }

    void release_variables() override {
        const std::lock_guard<std::mutex> lock(mutex_);
        for (SavedVariable* x : {&q, &k, &v, &bias, &mask, &gate, &o, &o_resid, &lse}) x->reset_data();
    }

    variable_list apply(variable_list&& grads) override {
        const std::lock_guard<std::mutex> lock(mutex_);
        const at::NoGradGuard no_grad;
        const auto self = getptr();
        // What a saved-tensor hook hands back has the values that were saved, but need not lie where they lay: a view may
        // come back contiguous, or off its alignment.
        auto whole = [&](const Tensor& t, int64_t numel) -> const Tensor& {
            TORCH_CHECK(t.device() == device && t.numel() == numel,
                        "TKEvoAttention: a saved tensor came back on another device or with another size than it had");
            return t;
        };
        const int64_t rows = int64_t{dims.B} * dims.S * dims.N, acts = rows * dims.H * dims.D;
        const c10::cuda::CUDAGuard guard(device);
        Tensor q_ = whole(q.unpack(), acts), k_ = whole(k.unpack(), acts), v_ = whole(v.unpack(), acts);
        const bool in_view = lay.in_view && lies_as_input(q_, lay) && lies_as_input(k_, lay) && lies_as_input(v_, lay);
        if (!in_view) {
            q_ = plain(q_, at::kBFloat16);
            k_ = plain(k_, at::kBFloat16);
            v_ = plain(v_, at::kBFloat16);
        }
        const Tensor bias_ = plain(whole(bias.unpack(), int64_t{dims.B} * dims.H * dims.N * dims.N), at::kBFloat16);
        const Tensor mask_ = plain(whole(mask.unpack(), rows), at::kBFloat16);
        const Tensor lse_ = plain(whole(lse.unpack(), rows * dims.H), at::kFloat);
        const Tensor o_ = as_output(whole(o.unpack(self), acts), q_, lay), resid_ = as_output(whole(o_resid.unpack(), acts), q_, lay);
        const Tensor gate_ = gated ? as_output(whole(gate.unpack(), acts), q_, lay) : Tensor();
        const Tensor d_out = grads[0].defined() ? as_output(grads[0], q_, lay) : empty_like_act(q_, lay).zero_();
        Tensor dq = empty_like_act(q_, lay), dk = empty_like_act(q_, lay), dv = empty_like_act(q_, lay), d_gate;
        if (gated) d_gate = empty_like_act(q_, lay);
        const bool bf = bias_type == at::kBFloat16;
        Tensor dbias = at::detail::empty_cuda({dims.B, 1, dims.H, dims.N, dims.N}, bf ? at::kBFloat16 : at::kFloat, q_.device(),
                                              std::nullopt);
        EvoBwdArgs a{};
        a.dims = dims;
        a.s_qkv = in_view ? &lay.in : nullptr;
        a.s_out = a.s_grad = lay.out_view ? &lay.in : nullptr;
        a.q = q_.const_data_ptr();
        a.k = k_.const_data_ptr();
        a.v = v_.const_data_ptr();
        a.pair_bias = bias_.const_data_ptr();
        a.res_mask = mask_.const_data_ptr();
        a.gate = gated ? gate_.const_data_ptr() : nullptr;
        a.o = o_.const_data_ptr();
        a.o_resid = resid_.const_data_ptr();
        a.lse = static_cast<const float*>(lse_.const_data_ptr());
        a.d_out = d_out.const_data_ptr();
        a.dq = dq.data_ptr();
        a.dk = dk.data_ptr();
        a.dv = dv.data_ptr();
        a.d_gate = gated ? d_gate.data_ptr() : nullptr;
        a.dbias = dbias.data_ptr();
        a.dbias_bf16 = bf;
        a.workspace_bytes = evo_bwd_ex_workspace_bytes(&dims, gated, bf);
        const Tensor ws = at::detail::empty_cuda({static_cast<int64_t>(a.workspace_bytes)}, at::kByte, q_.device(), std::nullopt);
        a.workspace = ws.data_ptr();
        a.scale = scale;
        a.phases = EVO_BWD_PHASE_DBIAS | EVO_BWD_PHASE_DQKV;
        a.stream = c10::cuda::getCurrentCUDAStream().stream();
        check(evo_bwd_ex(&a), "evo_bwd_ex");
        if (!bf && bias_type != at::kFloat) dbias = dbias.to(bias_type);
        if (gated) return {dq, dk, dv, Tensor(), dbias, Tensor(), d_gate};
        return {dq, dk, dv, Tensor(), dbias};
    }
};

std::optional<Tensor> apply(const Tensor& Q, const Tensor& K, const Tensor& V, const Tensor& res_mask, const Tensor& pair_bias,
                            const std::optional<Tensor>& gate) {
    // A trace has to record the operator, and function transforms have to refuse it: both as the Python one does.
    if (torch::jit::tracer::isTracing() ||
        c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode)) return std::nullopt;
    if (Q.dim() != 5 || !Q.is_cuda()) return std::nullopt;
    const auto sz = Q.sizes();
    const int64_t B = sz[0], S = sz[1], N = sz[2], H = sz[3], D = sz[4];
    if (K.sizes() != sz || V.sizes() != sz || !supported_dim(D) || N % 8 != 0 || N <= 0 || B <= 0 || S <= 0 || H <= 0) return std::nullopt;
    if (res_mask.sizes() != at::IntArrayRef({B, S, 1, 1, N}) || pair_bias.sizes() != at::IntArrayRef({B, 1, H, N, N})) return std::nullopt;
    if (gate && gate->sizes() != sz) return std::nullopt;
    const auto dev = Q.device();
    if (K.device() != dev || V.device() != dev || res_mask.device() != dev || pair_bias.device() != dev) return std::nullopt;
    if (gate && gate->device() != dev) return std::nullopt;
    // no forward-mode derivative: the Python operator says so
    for (const Tensor* t : {&Q, &K, &V, &res_mask, &pair_bias, gate ? &*gate : &Q})
        if (t->_fw_grad(0).defined()) return std::nullopt;
    if (B > INT32_MAX || S > INT32_MAX || N > INT32_MAX || H > INT32_MAX) return std::nullopt;

    const bool need_grad = at::GradMode::is_enabled() &&
                           (Q.requires_grad() || K.requires_grad() || V.requires_grad() || res_mask.requires_grad() ||
                            pair_bias.requires_grad() || (gate && gate->requires_grad()));
    Call c;
    {
        const at::NoGradGuard no_grad;
        c.lay = classify(Q, K, V);
        if (c.lay.in_view) {
            c.q = Q; c.k = K; c.v = V;
        } else {
            c.q = bf16_contiguous(Q);
            c.k = bf16_contiguous(K);
            c.v = bf16_contiguous(V);
        }
        c.bias = bf16_contiguous(pair_bias);
        c.mask = bf16_contiguous(res_mask);
        if (!aligned(c.q) || !aligned(c.k) || !aligned(c.v) || !aligned(c.bias) || !aligned(c.mask)) return std::nullopt;
        if (gate) c.gate = as_output(*gate, c.q, c.lay);
        c.dims = EvoDims{static_cast<int32_t>(B), static_cast<int32_t>(S), static_cast<int32_t>(N), static_cast<int32_t>(H),
                         static_cast<int32_t>(D)};
        c.scale = static_cast<float>(1.0 / std::sqrt(static_cast<double>(D)));
        c.bias_type = pair_bias.scalar_type();
        if (!need_grad) return run_forward(c, false).out;
    }
    Forward f;
    {
        const at::NoGradGuard no_grad;
        f = run_forward(c, true);
    }
    const std::shared_ptr<EvoBackward> node(new EvoBackward(), torch::autograd::deleteNode);
    variable_list inputs{Q, K, V, res_mask, pair_bias};
    if (gate) inputs.insert(inputs.end(), {Tensor(), *gate});
    node->set_next_edges(torch::autograd::collect_next_edges(inputs));
    node->q = SavedVariable(c.q, false);
    node->k = SavedVariable(c.k, false);
    node->v = SavedVariable(c.v, false);
    node->bias = SavedVariable(c.bias, false);
    node->mask = SavedVariable(c.mask, false);
    node->gated = c.gate.defined();
    if (node->gated) node->gate = SavedVariable(c.gate, false);
    node->o_resid = SavedVariable(f.o_resid, false);
    node->lse = SavedVariable(f.lse, false);
    node->lay = c.lay;
    node->dims = c.dims;
    node->device = dev;
    node->scale = c.scale;
    node->bias_type = c.bias_type;
    torch::autograd::set_history(f.out, node);
    node->o = SavedVariable(f.o, /*is_output=*/!node->gated);
    return f.out;
}

// The chunks of HostStreamedEvoAttention.run (tk_evo_attention_layer.py has what they are): rows [s0, s0 + r) of batch b in,
// through the kernels and out, on three streams and three sets of device buffers.  ins: q, k, v, dO, mask and outs: o, dq,
// dk, dv in host memory, contiguous; a set: q, k, v, do, mask, o, ores, dq, dk, dv, lse, dbias, ws for at least the rows
// of a chunk.  Through torch's Python operators a chunk was about 200 us of host time, and small steps
// were bound by it.  What the library refuses comes back as its error code and the name of the call, EVO_OK otherwise.
std::pair<int, std::string> host_chunks(const std::vector<std::tuple<int64_t, int64_t, int64_t>>& chunks, const std::vector<Tensor>& ins, const Tensor& bias,
                 const Tensor& dbias, const std::vector<Tensor>& outs, const std::vector<std::vector<Tensor>>& sets,
                 const std::vector<std::tuple<int64_t, int64_t, int64_t>>& streams) {
    TORCH_CHECK(ins.size() == 5 && outs.size() == 4 && sets.size() == 3 && streams.size() == 3, "host_chunks: wrong number of arguments");
    const int64_t S = ins[0].size(1), N = ins[0].size(2), H = ins[0].size(3), D = ins[0].size(4);
    auto stream_of = [&](int i) {
        const auto& [id, index, type] = streams[i];
        return c10::cuda::CUDAStream::unpack3(id, static_cast<c10::DeviceIndex>(index), static_cast<c10::DeviceType>(type));
    };
    const c10::cuda::CUDAStream s_in = stream_of(0), s_cmp = stream_of(1), s_out = stream_of(2);
    const c10::cuda::CUDAGuard guard(bias.device());
    const size_t act = static_cast<size_t>(2 * N * H * D), mask_row = static_cast<size_t>(2 * N);     // bytes of a row
    auto copy = [](void* dst, const void* src, size_t bytes, cudaMemcpyKind kind, const c10::cuda::CUDAStream& s) {
        const cudaError_t e = cudaMemcpyAsync(dst, src, bytes, kind, s.stream());
        TORCH_CHECK(e == cudaSuccess, "HostStreamedEvoAttention: a copy failed: ", cudaGetErrorString(e));
    };
    // whatever happens, pinned memory is not handed out again before the copies queued so far are done
    struct Hold {
        const std::vector<Tensor>*ins, *outs;
        c10::Stream in, out;
        ~Hold() {
            for (const Tensor& t : *ins) at::getHostAllocator(at::kCUDA)->record_event(t.data_ptr(), t.storage().data_ptr().get_context(), in);
            for (const Tensor& t : *outs) at::getHostAllocator(at::kCUDA)->record_event(t.data_ptr(), t.storage().data_ptr().get_context(), out);
        }
    } const hold{&ins, &outs, s_in.unwrap(), s_out.unwrap()};
    for (const Tensor& t : outs) t.unsafeGetTensorImpl()->bump_version();
    at::cuda::CUDAEvent ev_in[3], ev_cmp[3], ev_out[3];
    for (size_t c = 0; c < chunks.size(); ++c) {
        const auto [b, s0, r] = chunks[c];
        const std::vector<Tensor>& st = sets[c % 3];
        const size_t row = static_cast<size_t>(b * S + s0);
        if (c >= 3) ev_out[c % 3].block(s_in);               // this set's previous results are out
        for (int i = 0; i < 5; ++i) {
            const size_t bytes = i < 4 ? act : mask_row;
            copy(st[i].data_ptr(), static_cast<const char*>(ins[i].const_data_ptr()) + row * bytes, r * bytes, cudaMemcpyHostToDevice, s_in);
        }
        ev_in[c % 3].record(s_in);
        ev_in[c % 3].block(s_cmp);
        // a chunk with fewer rows than its set uses the leading rows of the (contiguous) buffers
        const EvoDims dims{1, static_cast<int32_t>(r), static_cast<int32_t>(N), static_cast<int32_t>(H), static_cast<int32_t>(D)};
        const void* bias_b = static_cast<const char*>(bias.const_data_ptr()) + b * 2 * H * N * N;
        float* lse = static_cast<float*>(st[10].data_ptr());
        int rc = evo_fwd(&dims, st[0].data_ptr(), st[1].data_ptr(), st[2].data_ptr(), bias_b, st[4].data_ptr(), st[5].data_ptr(),
                         st[6].data_ptr(), lse, 0.f, s_cmp.stream());
        if (rc != EVO_OK) return {rc, "evo_fwd"};
        rc = evo_bwd_phased(&dims, nullptr, st[0].data_ptr(), st[1].data_ptr(), st[2].data_ptr(), bias_b, st[4].data_ptr(), st[5].data_ptr(),
                            st[6].data_ptr(), lse, st[3].data_ptr(), st[7].data_ptr(), st[8].data_ptr(), st[9].data_ptr(),
                            static_cast<float*>(st[11].data_ptr()), st[12].data_ptr(), static_cast<size_t>(st[12].numel()), 0.f,
                            EVO_BWD_PHASE_DBIAS | EVO_BWD_PHASE_DQKV | EVO_BWD_BESIDE_COPIES, 0, s_cmp.stream());
        if (rc != EVO_OK) return {rc, "evo_bwd_phased"};
        {
            const c10::cuda::CUDAStreamGuard on(s_cmp);
            dbias.select(0, b).add_(st[11].select(0, 0));
        }
        ev_cmp[c % 3].record(s_cmp);
        ev_cmp[c % 3].block(s_out);
        for (int i = 0; i < 4; ++i)
            copy(static_cast<char*>(outs[i].data_ptr()) + row * act, st[i == 0 ? 5 : 6 + i].data_ptr(), r * act, cudaMemcpyDeviceToHost, s_out);
        ev_out[c % 3].record(s_out);
    }
    return {EVO_OK, ""};
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
    m.def("apply", &apply, "EvoAttention with its autograd node; None if the call is not one of the plain kind");
    m.def("host_chunks", &host_chunks, "The chunks of HostStreamedEvoAttention.run", pybind11::call_guard<pybind11::gil_scoped_release>());
}
