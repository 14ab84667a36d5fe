// PyTorch front end of the C ABI (include/simnets_b200.h): the Similarity and MEX operators on torch CUDA tensors, with
// their gradients wired into autograd natively, as _torch_ops.so.
//
// What bounds a small layer is not its kernels (3-10 us) but what the host does between them: with the descriptors, checks,
// allocations and autograd wiring in Python a MEX layer of the 1x28x28 example network took about 110 us of host time per
// forward call, against about 10 us here.  A plan holds the descriptor and geometry of one (shape, type, attributes)
// combination, the backward pass runs in autograd's own threads without the interpreter lock, and scratch comes from the
// caching allocator on the current stream, so that concurrent streams and threads never share it.
#include <torch/extension.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <algorithm>
#include <atomic>
#include <cstring>
#include <memory>
#include <mutex>
#include <string>
#include <vector>
#include "simnets_b200.h"

namespace py = pybind11;
using at::Tensor;
using OptTensor = std::optional<Tensor>;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

namespace {

struct StatusError : std::runtime_error {
    int status;
    explicit StatusError(int s) : std::runtime_error(std::string("simnets_b200: ") + simnets_status_string(s) + " (status " + std::to_string(s) + ")"), status(s) {}
};
inline void check(int status) { if (status != 0) throw StatusError(status); }

// ------------------------------------------------------------------------------------------ optional per-op device timing
struct ProfileRow { std::string key; cudaEvent_t begin, end; double bytes, terms; };
std::atomic<bool> g_profiling{false};
std::mutex g_profile_mu;
std::vector<ProfileRow> g_profile;

template <class Plan>
struct Timed {
    cudaEvent_t begin = nullptr;
    cudaStream_t stream;
    const Plan& plan;
    const char* op;
    const char* kind;
    double saved_bytes;
    Timed(const Plan& p, const char* op_, const char* kind_, cudaStream_t s, double saved = 0) : stream(s), plan(p), op(op_), kind(kind_), saved_bytes(saved) {
        if (!g_profiling.load(std::memory_order_relaxed)) return;
        cudaEventCreate(&begin);
        cudaEventRecord(begin, stream);
    }
    void done() {
        if (!begin) return;
        ProfileRow row;
        row.begin = begin;
        cudaEventCreate(&row.end);
        cudaEventRecord(row.end, stream);
        plan.cost(kind, &row.bytes, &row.terms);
        row.bytes -= saved_bytes;
        row.key = std::string(op) + "[" + plan.signature() + (saved_bytes > 0 ? " dy/4]" : "]");
        std::lock_guard<std::mutex> lock(g_profile_mu);
        g_profile.push_back(std::move(row));
        begin = nullptr;
    }
    ~Timed() { if (begin) cudaEventDestroy(begin); }
};

py::list profile_take() {
    std::vector<ProfileRow> rows;
    { std::lock_guard<std::mutex> lock(g_profile_mu); rows.swap(g_profile); }
    py::list out;
    for (auto& r : rows) {
        float ms = 0.f;
        cudaEventElapsedTime(&ms, r.begin, r.end);
        cudaEventDestroy(r.begin);
        cudaEventDestroy(r.end);
        out.append(py::make_tuple(r.key, ms, r.bytes, r.terms));
    }
    return out;
}

// ------------------------------------------------------------------------------------------------------------ tensor checks
void require_cuda(const Tensor& first, const Tensor& t) {
    if (!t.is_cuda()) throw std::runtime_error("simnets_b200 has no CPU kernels: every tensor must live on a CUDA device");
    if (t.device() != first.device()) throw std::runtime_error("all tensors of one op call must be on the same device");
    if (t.scalar_type() != first.scalar_type()) throw py::type_error("all tensors of one op call must share a dtype");
}
template <class... Ts>
void require_cuda_all(const Tensor& first, const Ts&... rest) {
    require_cuda(first, first);
    (require_cuda(first, rest), ...);
}
std::string shape_text(at::IntArrayRef s) {
    std::string out = "(";
    for (size_t i = 0; i < s.size(); ++i) out += (i ? ", " : "") + std::to_string(s[i]);
    return out + ")";
}
Tensor scratch(const Tensor& like, size_t bytes) {
    return at::empty({int64_t(bytes)}, at::TensorOptions().dtype(at::kByte).device(like.device()));
}
// The operators have no forward-mode derivative: a tangent is refused, as a torch.autograd.Function without a jvp refuses it,
// instead of being dropped (the kernels see values only).
void refuse_tangents(std::initializer_list<const Tensor*> inputs) {
    for (const Tensor* t : inputs)
        if (t->_fw_grad(0).defined()) {
            PyErr_SetString(PyExc_NotImplementedError, "simnets_b200 operators have no forward-mode derivative (jvp)");
            throw py::error_already_set();
        }
}
inline cudaStream_t stream_of(const Tensor& t) { return at::cuda::getCurrentCUDAStream(t.device().index()).stream(); }
inline void* ptr(const Tensor& t) { return t.data_ptr(); }

// ------------------------------------------------------------------------------------------------------------------- plans
// The descriptor of one (shape, type, attributes) combination, checked once.
struct MexPlan {
    simnets_mex_desc d;
    simnets_mex_geometry g;
    explicit MexPlan(const std::string& desc) {
        if (desc.size() != sizeof(d)) throw std::invalid_argument("MexPlan: wrong descriptor size");
        std::memcpy(&d, desc.data(), sizeof(d));
        check(simnets_mex_dims(&d, &g));
    }
    simnets_mex_desc with(uint32_t flags) const { simnets_mex_desc q = d; q.flags |= flags; return q; }
    bool overlapping() const { return g.stride_c < g.block_c || g.stride_h < g.block_h || g.stride_w < g.block_w; }
    size_t workspace_bytes(uint32_t flags) const { const simnets_mex_desc q = with(flags); return simnets_mex_forward_workspace_bytes(&q); }
    // room for the forward call and, if wanted, the gradient calls with a pooled dy
    size_t layer_bytes(uint32_t flags, bool pooled) const {
        return std::max<size_t>(256, std::max(workspace_bytes(flags), pooled ? workspace_bytes(flags | SIMNETS_FLAG_MEX_DY_POOLED2) : size_t(0)));
    }
    std::string signature() const {
        char buf[160];
        snprintf(buf, sizeof(buf), "B%d C%d %dx%d M%d K%d N%d R%d", d.batch, d.channels, d.height, d.width, g.M, g.K, g.N, g.num_regions);
        return buf;
    }
    // algorithmic bytes (every input read once, every output written once) and terms of one call
    void cost(const char* kind, double* bytes, double* terms) const {
        const double x = double(d.batch) * d.channels * d.height * d.width, o = double(g.num_regions) * g.M * g.K, y = double(d.batch) * g.M * g.N;
        const double e = d.dtype == SIMNETS_F64 ? 8 : 4;
        const std::string k(kind);
        *bytes = e * (k == "fwd" ? x + o + y : k == "dx" ? 2 * x + o + 2 * y : k == "doff" ? x + 2 * o + 2 * y : 2 * x + 2 * o + 2 * y);
        *terms = y * g.K * (k == "bwd" ? 2 : 1);
    }
    std::vector<int64_t> out_shape(int k = 1) const { return {d.batch, g.channels_out_total, g.height_out / k, g.width_out / k}; }
    void check_input(const Tensor& x) const {
        if (x.dim() != 4 || x.size(0) != d.batch || x.size(1) != d.channels || x.size(2) != d.height || x.size(3) != d.width)
            throw std::invalid_argument("input does not have the planned shape");
        if ((x.scalar_type() == at::kDouble) != (d.dtype == SIMNETS_F64)) throw py::type_error("input does not have the planned dtype");
    }
    void check_offsets(const Tensor& off) const {
        const int64_t want[5] = {g.num_regions, g.M, g.block_c, g.block_h, g.block_w};
        if (off.sizes() != at::IntArrayRef(want, 5))
            throw std::invalid_argument("offsets must have shape " + shape_text(at::IntArrayRef(want, 5)) + ", got " + shape_text(off.sizes()));
    }
    void check_dy(const Tensor& dy, bool pooled) const {
        const auto want = out_shape(pooled ? 2 : 1);
        if (dy.sizes() != at::IntArrayRef(want))
            throw std::invalid_argument("output_grad must have shape " + shape_text(want) + ", got " + shape_text(dy.sizes()));
    }
};

struct SimPlan {
    simnets_sim_desc d;
    int32_t oh = 0, ow = 0;
    explicit SimPlan(const std::string& desc) {
        if (desc.size() != sizeof(d)) throw std::invalid_argument("SimPlan: wrong descriptor size");
        std::memcpy(&d, desc.data(), sizeof(d));
        check(simnets_similarity_output_dims(&d, &oh, &ow));
    }
    simnets_sim_desc with(uint32_t flags) const { simnets_sim_desc q = d; q.flags |= flags; return q; }
    std::string signature() const {
        char buf[128];
        snprintf(buf, sizeof(buf), "B%d C%d %dx%d M%d K%d", d.batch, d.channels, d.height, d.width, d.num_instances, d.channels * d.block_h * d.block_w);
        return buf;
    }
    void cost(const char* kind, double* bytes, double* terms) const {
        const double k = double(d.channels) * d.block_h * d.block_w, y = double(d.batch) * d.num_instances * oh * ow;
        const double x = double(d.batch) * d.channels * d.height * d.width, p = d.num_instances * k;
        const std::string q(kind);
        *bytes = (d.dtype == SIMNETS_F64 ? 8 : 4) * (q == "fwd" ? x + 2 * p + y : q == "dx" ? 2 * x + 2 * p + y : x + y + 4 * p);
        *terms = y * k;
    }
    void check_tensors(const Tensor& x, const Tensor& t, const Tensor& w) const {
        if (x.dim() != 4 || x.size(0) != d.batch || x.size(1) != d.channels || x.size(2) != d.height || x.size(3) != d.width)
            throw std::invalid_argument("input does not have the planned shape");
        if ((x.scalar_type() == at::kDouble) != (d.dtype == SIMNETS_F64)) throw py::type_error("input does not have the planned dtype");
        if (t.dim() != 4 || t.size(0) != d.num_instances || t.size(1) != d.channels || t.size(2) != d.block_h || t.size(3) != d.block_w || t.sizes() != w.sizes())
            throw std::invalid_argument("templates and weights must have the planned shape");
    }
    void check_dy(const Tensor& dy) const {
        if (dy.dim() != 4 || dy.size(0) != d.batch || dy.size(1) != d.num_instances || dy.size(2) != oh || dy.size(3) != ow)
            throw std::invalid_argument("output_grad must have shape " + shape_text({d.batch, d.num_instances, oh, ow}) + ", got " + shape_text(dy.sizes()));
    }
};
using MexPlanPtr = std::shared_ptr<MexPlan>;
using SimPlanPtr = std::shared_ptr<SimPlan>;

// --------------------------------------------------------------------------------------------------------------------- MEX
Tensor mex_workspace(const MexPlan& p, const Tensor& x, uint32_t flags, const OptTensor& own) {
    const size_t n = p.workspace_bytes(flags);
    if (!own) return scratch(x, std::max<size_t>(n, 256));
    if (own->scalar_type() != at::kByte || own->device() != x.device() || !own->is_contiguous() || size_t(own->numel()) < n)
        throw std::invalid_argument("workspace: need a contiguous uint8 tensor of at least " + std::to_string(n) + " bytes on " + x.device().str());
    return *own;
}

// (y, pooled y or an undefined tensor).  keep_y = false: only the pooled output is wanted; y shares one allocation with the scratch of
// the call (an allocation is 1.7 us of host time, a tenth of what a small layer takes) and is not returned.
std::pair<Tensor, Tensor> mex_forward_impl(const MexPlan& p, const Tensor& x_in, const Tensor& off_in, uint32_t flags, const OptTensor& own, bool pool,
                                           bool keep_y = true) {
    require_cuda_all(x_in, off_in);
    p.check_input(x_in);
    p.check_offsets(off_in);
    const Tensor x = x_in.contiguous(), off = off_in.contiguous();
    const c10::cuda::CUDAGuard guard(x.device());
    const cudaStream_t s = stream_of(x);
    const simnets_mex_desc d = p.with(flags);
    if (!pool || own) keep_y = true;
    Tensor y, yp, ws;
    void* y_at;
    size_t ws_bytes;
    if (keep_y) {
        y = at::empty(p.out_shape(), x.options());
        if (pool) yp = at::empty(p.out_shape(2), x.options());
        ws = mex_workspace(p, x, flags, own);
        y_at = ptr(y);
        ws_bytes = ws.numel();
    } else {
        yp = at::empty(p.out_shape(2), x.options());
        const size_t values = size_t(d.batch) * p.g.channels_out_total * p.g.height_out * p.g.width_out;
        ws_bytes = (std::max<size_t>(p.workspace_bytes(flags), 256) + 511) & ~size_t(511);          // (the allocator's own alignment, for y behind it)
        ws = scratch(x, ws_bytes + values * x.element_size());
        y_at = static_cast<char*>(ptr(ws)) + ws_bytes;
    }
    Timed<MexPlan> timed(p, "mex_forward", "fwd", s);
    check(pool ? simnets_mex_forward_pool2x2(&d, ptr(x), ptr(off), y_at, ptr(yp), ptr(ws), ws_bytes, s)
               : simnets_mex_forward(&d, ptr(x), ptr(off), y_at, ptr(ws), ws_bytes, s));
    timed.done();
    return {y, yp};
}

Tensor mex_forward(const MexPlanPtr& p, const Tensor& x, const Tensor& off, uint32_t flags, const OptTensor& ws) {
    return mex_forward_impl(*p, x, off, flags, ws, false).first;
}
std::pair<Tensor, Tensor> mex_forward_pool2(const MexPlanPtr& p, const Tensor& x, const Tensor& off, uint32_t flags, const OptTensor& ws) {
    return mex_forward_impl(*p, x, off, flags, ws, true);
}

Tensor grad_target(const Tensor& like, const OptTensor& out) {
    if (!out) return at::empty(like.sizes(), like.options());
    TORCH_CHECK(out->is_contiguous() && out->numel() == like.numel() && out->scalar_type() == like.scalar_type(), "out: need a contiguous tensor of the gradient's size and dtype");
    return *out;
}

// Which of the two gradients to compute; `primed`: the workspace the forward call of the same input and offsets ran in.
std::pair<Tensor, Tensor> mex_grads(const MexPlan& p, const Tensor& x_in, const Tensor& off_in, const Tensor& y_in, const Tensor& dy_in, uint32_t flags,
                                    const OptTensor& primed, bool pooled, bool want_dx, bool want_doff, const OptTensor& out) {
    require_cuda_all(x_in, off_in, y_in, dy_in);
    p.check_input(x_in);
    p.check_offsets(off_in);
    p.check_dy(dy_in, pooled);
    flags |= (pooled ? SIMNETS_FLAG_MEX_DY_POOLED2 : 0u) | (primed ? SIMNETS_FLAG_MEX_WORKSPACE_PRIMED : 0u);
    const Tensor x = x_in.contiguous(), off = off_in.contiguous(), y = y_in.contiguous(), dy = dy_in.contiguous();
    const c10::cuda::CUDAGuard guard(x.device());
    const cudaStream_t s = stream_of(x);
    const simnets_mex_desc d = p.with(flags);
    Tensor dx, doff;
    if (want_dx) dx = at::empty(x.sizes(), x.options());
    if (want_doff) doff = grad_target(off, out);
    const Tensor ws = mex_workspace(p, x, flags, primed);
    Tensor products;            // (overlapping blocks: not part of a workspace that a layer keeps between its passes)
    if (const size_t n = want_dx && p.overlapping() ? simnets_mex_products_bytes(&d) : 0) products = scratch(x, n);
    const char* op = want_dx && want_doff ? "mex_backward" : want_dx ? "mex_input_grad" : "mex_offsets_grad";
    const char* kind = want_dx && want_doff ? "bwd" : want_dx ? "dx" : "doff";
    Timed<MexPlan> timed(p, op, kind, s, pooled && want_dx && want_doff ? 3.0 * dy.numel() * dy.element_size() : 0.0);
    check(simnets_mex_gradients(&d, ptr(x), ptr(off), ptr(y), ptr(dy), want_dx ? ptr(dx) : nullptr, want_doff ? ptr(doff) : nullptr, ptr(ws), ws.numel(),
                                products.defined() ? ptr(products) : nullptr, products.defined() ? products.numel() : 0, s));
    timed.done();
    return {dx, doff};
}

Tensor mex_input_grad(const MexPlanPtr& p, const Tensor& x, const Tensor& off, const Tensor& y, const Tensor& dy, uint32_t flags, const OptTensor& primed, bool pooled) {
    return mex_grads(*p, x, off, y, dy, flags, primed, pooled, true, false, std::nullopt).first;
}
Tensor mex_offsets_grad(const MexPlanPtr& p, const Tensor& x, const Tensor& off, const Tensor& y, const Tensor& dy, uint32_t flags, const OptTensor& primed, bool pooled, const OptTensor& out) {
    return mex_grads(*p, x, off, y, dy, flags, primed, pooled, false, true, out).second;
}
std::pair<Tensor, Tensor> mex_backward(const MexPlanPtr& p, const Tensor& x, const Tensor& off, const Tensor& y, const Tensor& dy, uint32_t flags, const OptTensor& primed, bool pooled, const OptTensor& out) {
    return mex_grads(*p, x, off, y, dy, flags, primed, pooled, true, true, out);
}

// Gradient node of one MEX layer.  The forward pass of a differentiated layer runs in a workspace of its own, which this
// node keeps and finds primed (per-position extrema, offset tables, operand tiles).
struct MexNode : torch::autograd::Node {
    MexPlanPtr plan;
    SavedVariable x, off, y;    // (y of a pooled layer is not an output of the node)
    OptTensor ws, sink;
    uint32_t flags = 0;
    bool pooled = false;
    std::string name() const override { return pooled ? "MexSumPool2Backward" : "MexBackward"; }
    variable_list apply(variable_list&& grads) override {
        std::lock_guard<std::mutex> lock(mutex_);
        variable_list out(2);
        if (!grads[0].defined()) return out;
        const bool want_dx = task_should_compute_output(0), want_doff = task_should_compute_output(1);
        if (!want_dx && !want_doff) return out;
        const Tensor xv = x.unpack(), ov = off.unpack(), yv = y.unpack(pooled ? nullptr : shared_from_this());
        // (with a sink the offsets gradient is added straight into the caller's tensor, a gradient bucket; nothing is left to accumulate)
        const auto g = mex_grads(*plan, xv, ov, yv, grads[0], flags | (sink ? SIMNETS_FLAG_ACCUMULATE : 0u), ws, pooled, want_dx, want_doff, sink);
        if (want_dx) out[0] = g.first;
        if (want_doff && !sink) out[1] = g.second;
        return out;
    }
    void release_variables() override {
        std::lock_guard<std::mutex> lock(mutex_);
        x.reset_data(); off.reset_data(); y.reset_data();
        ws.reset();
    }
};

// The differentiable op; `pooled` returns the 2x2 sum pooling of the output.  See ops/mex.py for the extras.
Tensor mex_apply(const MexPlanPtr& p, const Tensor& x, const Tensor& off, OptTensor ws, uint32_t fwd_flags, uint32_t op_flags, bool pooled, const OptTensor& sink) {
    refuse_tangents({&x, &off});
    const bool track = at::GradMode::is_enabled() && (x.requires_grad() || off.requires_grad());
    Tensor y, out;
    {
        at::AutoDispatchBelowADInplaceOrView below;
        if (track && !ws && x.is_cuda() && p->d.batch > 0) ws = scratch(x, p->layer_bytes(op_flags, pooled));
        if (pooled && p->d.dtype == SIMNETS_F32 && p->d.batch > 0) {
            std::tie(y, out) = mex_forward_impl(*p, x, off, fwd_flags | op_flags, ws, true, track);
        } else {
            y = out = mex_forward_impl(*p, x, off, fwd_flags | op_flags, ws, false).first;
            if (pooled) out = at::avg_pool2d(y, {2, 2}, {2, 2}, 0, false, true, 1);        // (the sum of each window)
        }
    }
    if (!track) return out;
    auto node = std::shared_ptr<MexNode>(new MexNode(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(x, off));
    node->plan = p;
    node->x = SavedVariable(x, false);
    node->off = SavedVariable(off, false);
    node->ws = std::move(ws);
    node->sink = sink;
    node->flags = op_flags;
    node->pooled = pooled;
    torch::autograd::set_history(out, node);
    node->y = pooled ? SavedVariable(y, false) : SavedVariable(out, true);
    return out;
}

// -------------------------------------------------------------------------------------------------------------- Similarity
Tensor sim_workspace(const simnets_sim_desc& d, const Tensor& x) { return scratch(x, std::max<size_t>(simnets_similarity_workspace_bytes(&d), 256)); }

Tensor sim_forward(const SimPlanPtr& p, const Tensor& x_in, const Tensor& t_in, const Tensor& w_in, uint32_t flags, uint64_t ch_max, uint64_t ch_min) {
    require_cuda_all(x_in, t_in, w_in);
    p->check_tensors(x_in, t_in, w_in);
    const Tensor x = x_in.contiguous(), t = t_in.contiguous(), w = w_in.contiguous();
    const c10::cuda::CUDAGuard guard(x.device());
    const cudaStream_t s = stream_of(x);
    const simnets_sim_desc d = p->with(flags);
    Tensor y = at::empty({d.batch, d.num_instances, p->oh, p->ow}, x.options());
    const Tensor ws = sim_workspace(d, x);
    Timed<SimPlan> timed(*p, "similarity_forward", "fwd", s);
    if (ch_max || ch_min)
        check(simnets_similarity_forward_extrema(&d, ptr(x), ptr(t), ptr(w), ptr(y), reinterpret_cast<void*>(ch_max), reinterpret_cast<void*>(ch_min), ptr(ws), ws.numel(), s));
    else
        check(simnets_similarity_forward(&d, ptr(x), ptr(t), ptr(w), ptr(y), ptr(ws), ws.numel(), s));
    timed.done();
    return y;
}

Tensor sim_input_grad(const SimPlanPtr& p, const Tensor& x_in, const Tensor& t_in, const Tensor& w_in, const Tensor& dy_in, uint32_t flags) {
    require_cuda_all(x_in, t_in, w_in, dy_in);
    p->check_tensors(x_in, t_in, w_in);
    p->check_dy(dy_in);
    const Tensor x = x_in.contiguous(), t = t_in.contiguous(), w = w_in.contiguous(), dy = dy_in.contiguous();
    const c10::cuda::CUDAGuard guard(x.device());
    const cudaStream_t s = stream_of(x);
    const simnets_sim_desc d = p->with(flags);
    Tensor dx = at::empty(x.sizes(), x.options());
    const Tensor ws = sim_workspace(d, x);
    Timed<SimPlan> timed(*p, "similarity_input_grad", "dx", s);
    check(simnets_similarity_input_grad(&d, ptr(x), ptr(t), ptr(w), ptr(dy), ptr(dx), ptr(ws), ws.numel(), s));
    timed.done();
    return dx;
}

std::pair<Tensor, Tensor> sim_params_grad(const SimPlanPtr& p, const Tensor& x_in, const Tensor& t_in, const Tensor& w_in, const Tensor& dy_in, uint32_t flags,
                                          const OptTensor& dt_out, const OptTensor& dw_out) {
    require_cuda_all(x_in, t_in, w_in, dy_in);
    p->check_tensors(x_in, t_in, w_in);
    p->check_dy(dy_in);
    const Tensor x = x_in.contiguous(), t = t_in.contiguous(), w = w_in.contiguous(), dy = dy_in.contiguous();
    const c10::cuda::CUDAGuard guard(x.device());
    const cudaStream_t s = stream_of(x);
    const simnets_sim_desc d = p->with(flags);
    const Tensor dt = grad_target(t, dt_out), dw = grad_target(w, dw_out), ws = sim_workspace(d, x);
    Timed<SimPlan> timed(*p, "similarity_params_grad", "dp", s);
    check(simnets_similarity_params_grad(&d, ptr(x), ptr(t), ptr(w), ptr(dy), ptr(dt), ptr(dw), ptr(ws), ws.numel(), s));
    timed.done();
    return {dt, dw};
}

struct SimNode : torch::autograd::Node {
    SimPlanPtr plan;
    SavedVariable x, t, w;
    OptTensor dt_sink, dw_sink;
    uint32_t flags = 0;
    std::string name() const override { return "SimilarityBackward"; }
    variable_list apply(variable_list&& grads) override {
        std::lock_guard<std::mutex> lock(mutex_);
        variable_list out(3);
        if (!grads[0].defined()) return out;
        const Tensor xv = x.unpack(), tv = t.unpack(), wv = w.unpack();
        if (task_should_compute_output(0)) out[0] = sim_input_grad(plan, xv, tv, wv, grads[0], flags);
        if (task_should_compute_output(1) || task_should_compute_output(2)) {
            const bool add = dt_sink && dw_sink;        // both parameter gradients are added straight into the caller's tensors
            auto g = sim_params_grad(plan, xv, tv, wv, grads[0], flags | (add ? SIMNETS_FLAG_ACCUMULATE : 0u), add ? dt_sink : std::nullopt, add ? dw_sink : std::nullopt);
            if (!add) { out[1] = g.first; out[2] = g.second; }
        }
        return out;
    }
    void release_variables() override {
        std::lock_guard<std::mutex> lock(mutex_);
        x.reset_data(); t.reset_data(); w.reset_data();
    }
};

Tensor sim_apply(const SimPlanPtr& p, const Tensor& x, const Tensor& t, const Tensor& w, uint32_t flags, uint64_t ch_max, uint64_t ch_min,
                 const OptTensor& dt_sink, const OptTensor& dw_sink) {
    refuse_tangents({&x, &t, &w});
    const bool track = at::GradMode::is_enabled() && (x.requires_grad() || t.requires_grad() || w.requires_grad());
    Tensor y;
    {
        at::AutoDispatchBelowADInplaceOrView below;
        y = sim_forward(p, x, t, w, flags, ch_max, ch_min);
    }
    if (!track) return y;
    auto node = std::shared_ptr<SimNode>(new SimNode(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(x, t, w));
    node->plan = p;
    node->x = SavedVariable(x, false);
    node->t = SavedVariable(t, false);
    node->w = SavedVariable(w, false);
    node->flags = flags;
    node->dt_sink = dt_sink;
    node->dw_sink = dw_sink;
    torch::autograd::set_history(y, node);
    return y;
}

// ----------------------------------------------------------------------------------------------------------------- mixture
// Flat statistics of one EM step, or nothing where the library has no kernels for the shape.
OptTensor mixture_statistics(const SimPlanPtr& p, const Tensor& x_in, const Tensor& means_in, const Tensor& covs_in) {
    require_cuda_all(x_in, means_in, covs_in);
    p->check_tensors(x_in, means_in, covs_in);
    const size_t n = simnets_mixture_workspace_bytes(&p->d);
    if (n == 0) return std::nullopt;
    const Tensor x = x_in.contiguous(), means = means_in.contiguous(), covs = covs_in.contiguous();
    const c10::cuda::CUDAGuard guard(x.device());
    Tensor stats = at::empty({2 * means.numel() + means.size(0)}, means.options());
    const Tensor ws = scratch(x, n);
    check(simnets_mixture_statistics(&p->d, ptr(x), ptr(means), ptr(covs), ptr(stats), ptr(ws), ws.numel(), stream_of(x)));
    return stats;
}

std::pair<Tensor, Tensor> mixture_parameters(const Tensor& stats, const Tensor& means_in, double min_var) {
    require_cuda_all(stats, means_in);
    const Tensor means = means_in.contiguous();
    TORCH_CHECK(stats.scalar_type() == at::kFloat && stats.is_contiguous() && stats.numel() == 2 * means.numel() + means.size(0), "stats do not belong to these means");
    const c10::cuda::CUDAGuard guard(means.device());
    Tensor new_means = at::empty(means.sizes(), means.options()), new_covs = at::empty(means.sizes(), means.options());
    check(simnets_mixture_parameters(int32_t(means.size(0)), int32_t(means.numel() / means.size(0)), float(min_var), stats.data_ptr<float>(), means.data_ptr<float>(),
                                     new_means.data_ptr<float>(), new_covs.data_ptr<float>(), stream_of(means)));
    return {new_means, new_covs};
}

// ---------------------------------------------------------------------------------------------------- softmax cross-entropy
std::pair<Tensor, Tensor> xent_with_grad(const Tensor& logits_in, const Tensor& labels_in, double scale) {
    require_cuda_all(logits_in);
    if (!labels_in.is_cuda() || labels_in.device() != logits_in.device()) throw std::runtime_error("labels must live on the device of the logits");
    if (logits_in.scalar_type() != at::kFloat || labels_in.scalar_type() != at::kLong || logits_in.dim() != 2 || labels_in.dim() != 1 || labels_in.size(0) != logits_in.size(0))
        throw std::invalid_argument("logits must be float32 [batch, classes] and labels int64 [batch]");
    const Tensor logits = logits_in.contiguous(), labels = labels_in.contiguous();
    const c10::cuda::CUDAGuard guard(logits.device());
    Tensor loss = at::empty({}, logits.options()), dlogits = at::empty(logits.sizes(), logits.options());
    const Tensor ws = scratch(logits, std::max<size_t>(simnets_softmax_cross_entropy_workspace_bytes(int32_t(logits.size(0))), 256));
    check(simnets_softmax_cross_entropy(int32_t(logits.size(0)), int32_t(logits.size(1)), float(scale), logits.data_ptr<float>(), labels.data_ptr<int64_t>(),
                                        loss.data_ptr<float>(), dlogits.data_ptr<float>(), ptr(ws), ws.numel(), stream_of(logits)));
    return {loss, dlogits};
}

struct XentNode : torch::autograd::Node {
    SavedVariable dlogits;
    std::string name() const override { return "SoftmaxCrossEntropyBackward"; }
    variable_list apply(variable_list&& grads) override {
        std::lock_guard<std::mutex> lock(mutex_);
        if (!grads[0].defined()) return variable_list(1);
        return {dlogits.unpack() * grads[0]};
    }
    void release_variables() override {
        std::lock_guard<std::mutex> lock(mutex_);
        dlogits.reset_data();
    }
};

Tensor xent_apply(const Tensor& logits, const Tensor& labels, double scale) {
    refuse_tangents({&logits});
    const bool track = at::GradMode::is_enabled() && logits.requires_grad();
    Tensor loss, dlogits;
    {
        at::AutoDispatchBelowADInplaceOrView below;
        std::tie(loss, dlogits) = xent_with_grad(logits, labels, scale);
    }
    if (!track) return loss;
    auto node = std::shared_ptr<XentNode>(new XentNode(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(logits));
    node->dlogits = SavedVariable(dlogits, false);
    torch::autograd::set_history(loss, node);
    return loss;
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
    // a status becomes the exception that the ctypes layer raises for it (ValueError or SimnetsError)
    py::register_exception_translator([](std::exception_ptr p) {
        try {
            if (p) std::rethrow_exception(p);
        } catch (const StatusError& e) {
            try {
                py::module_::import("simnets_tf_b200._lib").attr("check")(e.status);
            } catch (py::error_already_set& raised) {
                raised.restore();
            }
        }
    });
    py::class_<MexPlan, MexPlanPtr>(m, "MexPlan")
        .def(py::init([](const py::bytes& desc) { return std::make_shared<MexPlan>(std::string(desc)); }))
        .def_property_readonly("height_out", [](const MexPlan& p) { return p.g.height_out; })
        .def_property_readonly("width_out", [](const MexPlan& p) { return p.g.width_out; })
        .def("layer_bytes", &MexPlan::layer_bytes, py::arg("flags"), py::arg("pooled"))
        .def("layer_workspace", [](const MexPlan& p, uint32_t flags, bool pooled, at::Device device) {
            return at::empty({int64_t(p.layer_bytes(flags, pooled))}, at::TensorOptions().dtype(at::kByte).device(device));
        })
        .def("maxima", [](const MexPlan& p, uint32_t flags, const Tensor& ws) {
            const simnets_mex_desc d = p.with(flags);
            return reinterpret_cast<uint64_t>(simnets_mex_workspace_maxima(&d, ws.data_ptr()));
        });
    py::class_<SimPlan, SimPlanPtr>(m, "SimPlan")
        .def(py::init([](const py::bytes& desc) { return std::make_shared<SimPlan>(std::string(desc)); }))
        .def_property_readonly("out_shape", [](const SimPlan& p) { return py::make_tuple(p.d.batch, p.d.num_instances, p.oh, p.ow); });
    m.def("mex_forward", &mex_forward);
    m.def("mex_forward_pool2", &mex_forward_pool2);
    m.def("mex_input_grad", &mex_input_grad);
    m.def("mex_offsets_grad", &mex_offsets_grad);
    m.def("mex_backward", &mex_backward);
    m.def("mex_apply", &mex_apply);
    m.def("sim_forward", &sim_forward);
    m.def("sim_input_grad", &sim_input_grad);
    m.def("sim_params_grad", &sim_params_grad);
    m.def("sim_apply", &sim_apply);
    m.def("mixture_statistics", &mixture_statistics);
    m.def("mixture_parameters", &mixture_parameters);
    m.def("xent_with_grad", &xent_with_grad);
    m.def("xent_apply", &xent_apply);
    m.def("profile_start", [] { py::list dropped = profile_take(); g_profiling = true; });
    m.def("profile_stop", [] { g_profiling = false; return profile_take(); });
}
