// Autograd nodes of the quantized operators, in C++: the backward of a node runs in the engine's thread without the
// Python interpreter.  Each operator is a forward function and a node whose backward() returns one gradient per tensor
// input.  int8 operands and scales of the forward pass are kept by the node itself (they are not differentiable);
// forward results that the backward reads are kept as SavedVariables, so that a write to them in between is noticed.
#include "torch_autograd.h"

#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/autograd/variable.h>

namespace tango_host {

using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

// Below the autograd and view-tracking layers: forward and backward bodies only produce fresh, non-differentiable tensors.
using Raw = at::AutoDispatchBelowADInplaceOrView;

struct OnceNode : Node {
    virtual variable_list backward(const variable_list &grads) = 0;

    variable_list apply(variable_list &&grads) override {
        variable_list out;
        {
            const c10::AutoGradMode no_grad(false);
            const Raw raw;
            out = backward(grads);
        }
        if (!c10::GradMode::is_enabled()) return out;
        bool differentiable = false;
        for (const Tensor &g : grads) differentiable |= g.defined() && g.requires_grad();
        if (!differentiable) return out;
        // a graph of the gradients was asked for: results that raise when they are differentiated again
        for (Tensor &t : out)
            if (t.defined()) {
                t = t.detach();
                t.set_requires_grad(true);
            }
        return torch::autograd::DelayedError("trying to differentiate twice a function that was marked with "
                                             "@once_differentiable", (int)out.size())(std::move(out));
    }
    bool needs(size_t input) const { return task_should_compute_output(input); }
};

// A node whose operands pass through the saved-tensor hooks and are given back after the backward pass.
struct SavingNode : OnceNode {
    std::vector<SavedVariable> saved;
    bool released = false;
    // call it after set_history; the first `outputs` of them are outputs of the node
    void keep(std::initializer_list<Tensor> tensors, size_t outputs = 0) {
        saved.reserve(tensors.size());
        for (const Tensor &t : tensors) {
            saved.emplace_back(t, outputs > 0);
            if (outputs > 0) --outputs;
        }
    }
    std::vector<Tensor> kept() {
        TORCH_CHECK(!released, torch::autograd::ERR_BACKWARD_TWICE);
        std::vector<Tensor> t;
        t.reserve(saved.size());
        for (SavedVariable &s : saved) t.push_back(s.unpack(shared_from_this()));
        return t;
    }
    void release_variables() override {
        for (SavedVariable &s : saved) s.reset_data();
        released = true;
    }
};

// An int8 GEMM operand whose rows are padded to 16 bytes, as alloc_int8 lays it out: a saved-tensor hook may have given it back
// packed.
static Tensor padded(const Tensor &t) {
    if (t.dim() < 2 || t.size(0) == 0 || t.stride(0) % 16 == 0) return t;
    const Tensor p = alloc_int8(t.sizes(), t.device(), 16);
    p.as_strided({t.size(0), p.stride(0)}, {p.stride(0), 1}).zero_();
    return p.copy_(t);
}

// The node of an operation on `inputs`, or null when no gradient is recorded.
template <class N, class... T>
static std::shared_ptr<N> make_node(const T &...inputs) {
    if (!torch::autograd::compute_requires_grad(inputs...)) return nullptr;
    auto node = std::shared_ptr<N>(new N(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(inputs...));
    return node;
}

static int64_t row_width(const Tensor &t) { return t.dim() > 1 && t.size(0) ? t.numel() / t.size(0) : t.numel(); }
// the scratch of an aggregation of t's rows
static Tensor aggregation_scratch(const Graph &g, bool reverse, const Tensor &t) {
    return spmm_scratch(g, reverse, row_width(t), t);
}
static Tensor zeros1(const Tensor &like) { return at::zeros({1}, like.options().dtype(at::kFloat)); }
static uint64_t call_if(int mode) { return mode == TANGO_ROUND_STOCHASTIC ? next_call() : 0; }

// ------------------------------------------------------------------------------------------------ QLinear
struct QLinearBackward : OnceNode {
    std::string name() const override { return "QLinearBackward"; }
    Quantized x, w;
    bool has_bias = false;
    variable_list backward(const variable_list &grads) override {
        const Tensor &dy = grads[0];
        if (!dy.defined()) return variable_list(3);
        QuantJob job = quant_job(dy);
        job.colsum = has_bias && needs(2);          // the bias gradient comes out of the quantizer's first sweep
        if (needs(1)) job.clear = dw_scratch(dy.size(0), dy.size(1), x.q.size(1), dy);
        const Quantized q = quantize(job);
        Tensor dx = needs(0) ? gemm_dx(q, w) : Tensor();
        Tensor dw = needs(1) ? gemm_dw(q, x, job.clear) : Tensor();
        return {dx, dw, q.colsum};
    }
};

// The GEMM's epilogue reads the bias by its address: one contiguous fp32 value per row of w.
static Tensor checked_bias(const Tensor &x, const Tensor &w, const Tensor &b) {
    require(x.size(1) == w.size(1), "x and w must have the same number of columns");
    require(!b.defined() || b.numel() == w.size(0), "one bias per row of w expected");
    require(!b.defined() || b.scalar_type() == at::kFloat, "fp32 bias expected");
    require(x.is_cuda() && w.device() == x.device() && (!b.defined() || b.device() == x.device()),
            "x, w and b must be on the same GPU");
    return b.defined() ? b.detach().contiguous() : b;
}

std::tuple<Tensor, Tensor, Tensor, Tensor> qlinear(const Tensor &x, const Tensor &w, const Tensor &b, bool want_scale,
                                                   const Tensor &xq_, const Tensor &sx_) {
    const Tensor bias = checked_bias(x, w, b);
    Tensor y, sy;
    Quantized xq, wq;
    {
        const Raw raw;
        const int mode = settings().mode_gemm;
        const uint64_t seed = settings().seed, call = call_if(mode);
        if (mode == TANGO_ROUND_STOCHASTIC) next_call();       // the weight draws from call + 1
        QuantJob jw{w, mode, seed, call + 1};
        if (want_scale) jw.clear = sy = floats({1}, x);
        if (xq_.defined()) {
            xq.q = xq_; xq.scale = sx_;
            wq = quantize(jw);
        } else {
            const auto q = quantize_all({jw, {x, mode, seed, call}});
            wq = q[0]; xq = q[1];
        }
        y = gemm_nt(xq, wq, bias, sy);
    }
    if (auto node = make_node<QLinearBackward>(x, w, b)) {
        node->x = xq; node->w = wq; node->has_bias = b.defined();
        torch::autograd::set_history(y, node);
    }
    return {y, sy, xq.q, xq.scale};
}

std::vector<Tensor> qlinear_group(const Tensor &x, const std::vector<Tensor> &w, const std::vector<Tensor> &b) {
    const int mode = settings().mode_gemm;
    const uint64_t seed = settings().seed;
    require(w.size() >= 1 && w.size() <= 3 && w.size() == b.size(), "one to three layers");
    require(mode != TANGO_ROUND_STOCHASTIC, "stochastic rounding draws anew for every layer");
    std::vector<Tensor> y, bias;
    std::vector<Quantized> q;
    for (size_t k = 0; k < w.size(); ++k) bias.push_back(checked_bias(x, w[k], b[k]));
    {
        const Raw raw;
        std::vector<QuantJob> jobs;
        for (const Tensor &t : w) jobs.push_back({t, mode, seed, 0});
        jobs.push_back({x, mode, seed, 0});
        q = quantize_all(jobs);
        for (size_t k = 0; k < w.size(); ++k) y.push_back(gemm_nt(q.back(), q[k], bias[k]));
    }
    for (size_t k = 0; k < w.size(); ++k)
        if (auto node = make_node<QLinearBackward>(x, w[k], b[k])) {
            node->x = q.back(); node->w = q[k]; node->has_bias = b[k].defined();
            torch::autograd::set_history(y[k], node);
        }
    return y;
}

// ------------------------------------------------------------------------------------------------ aggregation
struct SpmmCopyUBackward : OnceNode {
    std::string name() const override { return "SpmmCopyUBackward"; }
    GraphPtr g;
    variable_list backward(const variable_list &grads) override {
        if (!grads[0].defined() || !needs(0)) return variable_list(1);
        QuantJob job = quant_job(grads[0]);
        job.clear = aggregation_scratch(*g, true, grads[0]);
        return {spmm_copy_u(*g, true, quantize(job), job.clear)};
    }
};

Tensor spmm_copy_u_fn(const GraphPtr &g, const Tensor &n, const Tensor &scale) {
    Tensor out;
    {
        const Raw raw;
        QuantJob job = quant_job(n);
        job.scale = scale;
        job.clear = aggregation_scratch(*g, false, n);
        out = spmm_copy_u(*g, false, quantize(job), job.clear);
    }
    if (auto node = make_node<SpmmCopyUBackward>(n)) {
        node->g = g;
        torch::autograd::set_history(out, node);
    }
    return out;
}

// True when the edge feature broadcasts over the node feature's last dimension, so that dE is a per-head dot product
// (cuda/SPMM.py:26-34 of the reference).
static bool reduces_last_dim(const Tensor &n, const Tensor &e) {
    if (e.dim() < 2 || n.dim() != e.dim() || e.size(-1) != 1 || n.size(-1) <= 1) return false;
    for (int64_t d = 1; d < n.dim() - 1; ++d)
        if (n.size(d) != e.size(d)) return false;
    return true;
}

struct SpmmUMulEBackward : OnceNode {
    std::string name() const override { return "SpmmUMulEBackward"; }
    GraphPtr g;
    Tensor nq, sn, eq, se, scale;
    bool reduce_last = false;
    std::vector<int64_t> e_shape;
    variable_list backward(const variable_list &grads) override {
        if (!grads[0].defined()) return variable_list(2);
        const bool compat = settings().compat_dn_scale;
        QuantJob job = quant_job(grads[0]);
        if (!compat) job.times[0] = se;
        if (needs(0)) job.clear = aggregation_scratch(*g, true, grads[0]);
        const Quantized z = quantize(job);
        Tensor dn, de;
        if (needs(0)) dn = spmm_u_mul_e(*g, true, z.q, eq, compat ? scale : z.product[0], job.clear);
        if (needs(1)) de = sddmm(*g, reduce_last ? "dot" : "mul", nq, z.q, sn, z.scale, {}, false).reshape(e_shape);
        return {dn, de};
    }
};

Tensor spmm_u_mul_e_fn(const GraphPtr &g, const Tensor &n, const Tensor &e, const Tensor &scale_e) {
    Tensor out, sn, se, scale;
    Quantized eq, nq;
    {
        const Raw raw;
        QuantJob je = quant_job(e.reshape({e.size(0), -1}), 1);    // [E, H] int8, edge-id order (no transposed copy)
        je.scale = scale_e;                                        // the producer may already know max|E| / 127
        QuantJob jn = quant_job(n);
        jn.times_job = 0;
        jn.clear = aggregation_scratch(*g, false, n);
        const auto q = quantize_all({je, jn});
        eq = q[0]; nq = q[1];
        sn = nq.scale; se = eq.scale; scale = nq.product[0];
        out = spmm_u_mul_e(*g, false, nq.q, eq.q, scale, jn.clear);
    }
    if (auto node = make_node<SpmmUMulEBackward>(n, e)) {
        node->g = g; node->nq = nq.q; node->sn = sn; node->eq = eq.q; node->se = se; node->scale = scale;
        node->reduce_last = reduces_last_dim(n, e);
        node->e_shape = e.sizes().vec();
        torch::autograd::set_history(out, node);
    }
    return out;
}

// ------------------------------------------------------------------------------------------------ edge scores
// Per-edge and per-node tensors narrower than 16 bytes stay packed; wider rows are padded for 128-bit accesses.
static int64_t row_align(const Tensor &t) {
    const int64_t rows = t.size(0);
    return (rows ? t.numel() / rows : 0) < 16 ? 1 : 16;
}

struct SddmmUAddVBackward : OnceNode {
    std::string name() const override { return "SddmmUAddVBackward"; }
    GraphPtr g;
    variable_list backward(const variable_list &grads) override {
        if (!grads[0].defined()) return variable_list(2);
        QuantJob job = quant_job(grads[0], row_align(grads[0]));
        if (needs(0)) job.clear = aggregation_scratch(*g, true, grads[0]);
        if (needs(1)) job.clear2 = aggregation_scratch(*g, false, grads[0]);
        const Quantized z = quantize(job);
        Tensor du = needs(0) ? incidence_sum(*g, true, z, job.clear) : Tensor();
        Tensor dv = needs(1) ? incidence_sum(*g, false, z, job.clear2) : Tensor();
        return {du, dv};
    }
};

Tensor sddmm_u_add_v_fn(const GraphPtr &g, const Tensor &u, const Tensor &v, const Tensor &su, const Tensor &sv) {
    Tensor out;
    {
        const Raw raw;
        const int64_t align = row_align(u);
        std::vector<QuantJob> jobs{quant_job(u, align)};
        jobs[0].scale = su;
        if (!u.is_same(v)) {
            jobs.push_back(quant_job(v, align));
            jobs[1].scale = sv;
        }
        const auto q = quantize_all(jobs);
        const Quantized &uq = q.front(), &vq = q.back();
        out = sddmm(*g, "add", uq.q, vq.q, uq.scale, vq.scale, {}, false);
    }
    if (auto node = make_node<SddmmUAddVBackward>(u, v)) {
        node->g = g;
        torch::autograd::set_history(out, node);
    }
    return out;
}

struct SddmmUDotVBackward : OnceNode {
    std::string name() const override { return "SddmmUDotVBackward"; }
    GraphPtr g;
    Tensor uq, su, vq, sv;
    variable_list backward(const variable_list &grads) override {
        const Tensor &dz = grads[0];
        if (!dz.defined()) return variable_list(2);
        QuantJob job = quant_job(dz.reshape({dz.size(0), -1}), 1);
        job.times[0] = sv; job.times[1] = su;
        if (needs(0)) job.clear = aggregation_scratch(*g, true, vq);
        if (needs(1)) job.clear2 = aggregation_scratch(*g, false, uq);
        const Quantized z = quantize(job);
        const bool flat = uq.dim() != 3;
        auto side = [&](bool reverse, const Tensor &xq, const Tensor &scale, const Tensor &scratch) {
            const Tensor d = spmm_u_mul_e(*g, reverse, flat ? xq.unsqueeze(1) : xq, z.q, scale, scratch);
            return flat ? d.squeeze(1) : d;
        };
        Tensor du, dv;
        if (needs(0)) du = side(true, vq, z.product[0], job.clear);
        if (needs(1)) dv = side(false, uq, z.product[1], job.clear2);
        return {du, dv};
    }
};

Tensor sddmm_u_dot_v_fn(const GraphPtr &g, const Tensor &u, const Tensor &v) {
    Tensor out;
    Quantized uq, vq;
    {
        const Raw raw;
        std::vector<QuantJob> jobs{quant_job(u)};
        if (!u.is_same(v)) jobs.push_back(quant_job(v));
        const auto q = quantize_all(jobs);
        uq = q.front(); vq = q.back();
        out = sddmm(*g, "dot", uq.q, vq.q, uq.scale, vq.scale, {}, false);
    }
    if (auto node = make_node<SddmmUDotVBackward>(u, v)) {
        node->g = g; node->uq = uq.q; node->su = uq.scale; node->vq = vq.q; node->sv = vq.scale;
        torch::autograd::set_history(out, node);
    }
    return out;
}

// ------------------------------------------------------------------------------------------------ graph convolution
// act((A . X') W^T ...) with the norms of both sides, bias and ReLU.  `first` says which product runs first: the linear
// layer where it narrows the features (its int8 output is aggregated), else the aggregation (its fp32 output is quantized for
// the linear layer).  Either way the element-wise steps sit in the kernels next to them, and every tensor that a kernel here
// produces for a quantizer brings its scale along (epilogue maximum), so only the inputs of the layer are swept for theirs.
enum class First { linear, aggregate };

struct GcnConvBackward : SavingNode {
    std::string name() const override { return "GcnConvBackward"; }
    GraphPtr g;
    First first = First::linear;
    bool relu = false, has_bias = false;

    variable_list backward(const variable_list &grads) override {
        const Tensor &d = grads[0];
        const std::vector<Tensor> k = kept();      // out (undefined without ReLU), the linear layer's operands, the norms
        if (!d.defined()) return variable_list(3);
        Quantized x, w;
        x.q = padded(k[1]); x.scale = k[2]; w.q = padded(k[3]); w.scale = k[4];
        const Tensor &out = k[0], &out_norm = k[5], &in_norm = k[6];
        // ReLU mask, bias gradient, right norm, absmax and quantisation: two sweeps of one launch over (grad, out)
        QuantJob job = quant_job(d);
        job.row_scale = in_norm;
        job.colsum = has_bias && needs(2);
        if (relu) job.gate = out;
        const Tensor dw_tmp = needs(1) ? dw_scratch(d.size(0), w.q.size(0), x.q.size(1), d) : Tensor();
        const Tensor scale = floats({1}, d);
        Tensor dx, dw;
        if (first == First::linear) {
            job.clear = scale;
            job.clear2 = aggregation_scratch(*g, true, d);
            const Quantized z = quantize(job);
            const Tensor dh = spmm_copy_u(*g, true, z, job.clear2, {}, {}, false, scale);
            QuantJob jh = quant_job(dh);
            jh.scale = scale;
            jh.clear = dw_tmp;
            const Quantized h = quantize(jh);
            // the backward of the left norm is the row factor in dX's epilogue
            if (needs(0)) dx = gemm_dx(h, w, out_norm);
            if (needs(1)) dw = gemm_dw(h, x, dw_tmp);
            return {dx, dw, z.colsum};
        }
        job.clear = dw_tmp;
        job.clear2 = scale;
        const Quantized z = quantize(job);
        if (needs(1)) dw = gemm_dw(z, x, dw_tmp);
        if (needs(0)) {
            const Tensor da = gemm_dx(z, w, {}, scale);
            QuantJob ja = quant_job(da);
            ja.scale = scale;
            ja.clear = aggregation_scratch(*g, true, da);
            dx = spmm_copy_u(*g, true, quantize(ja), ja.clear, out_norm);
        }
        return {dx, dw, z.colsum};
    }
};

Tensor gcn_conv_fn(const GraphPtr &g, const Tensor &x_, const Tensor &w, const Tensor &b, const Tensor &out_norm,
                   const Tensor &in_norm, bool relu, bool linear_first) {
    require(x_.dim() == 2 && w.dim() == 2 && x_.size(1) == w.size(1), "features and weight must have the same number of columns");
    require(x_.size(0) == g->n_nodes, "one feature row per node expected");
    require(out_norm.numel() == g->n_nodes && in_norm.numel() == g->n_nodes, "one norm per node expected");
    require(!b.defined() || b.numel() == w.size(0), "one bias per output feature expected");
    for (const Tensor *t : {&x_, &w, &out_norm, &in_norm, &b})
        require(!t->defined() || (t->is_cuda() && t->scalar_type() == at::kFloat && t->device() == x_.device()),
                "fp32 tensors on one CUDA device expected");
    const Tensor bias = b.defined() ? b.detach().contiguous() : b, out_n = out_norm.contiguous(), in_n = in_norm.contiguous();
    Tensor out;
    Quantized x, wq;
    {
        const Raw raw;
        const int mode = settings().mode_gemm;
        const uint64_t seed = settings().seed;
        const Tensor scale = floats({1}, x_);
        if (linear_first) {
            const uint64_t call = call_if(mode);
            if (mode == TANGO_ROUND_STOCHASTIC) next_call();
            QuantJob jx{x_, mode, seed, call};
            jx.row_scale = out_n;
            jx.clear = scale;
            const auto q = quantize_all({{w, mode, seed, call + 1}, jx});
            wq = q[0]; x = q[1];
            const Tensor h = gemm_nt(x, wq, {}, scale);
            QuantJob jh = quant_job(h);
            jh.scale = scale;
            jh.clear = aggregation_scratch(*g, false, h);
            out = spmm_copy_u(*g, false, quantize(jh), jh.clear, in_n, bias, relu);
        } else {
            QuantJob jx = quant_job(x_);
            jx.row_scale = out_n;
            jx.clear = scale;
            jx.clear2 = aggregation_scratch(*g, false, x_);
            const Tensor a = spmm_copy_u(*g, false, quantize(jx), jx.clear2, {}, {}, false, scale);
            const uint64_t call = call_if(mode);
            if (mode == TANGO_ROUND_STOCHASTIC) next_call();
            QuantJob ja{a, mode, seed, call};
            ja.scale = scale;
            const auto q = quantize_all({{w, mode, seed, call + 1}, ja});
            wq = q[0]; x = q[1];
            out = gemm_nt(x, wq, bias, {}, in_n, relu);
        }
    }
    if (auto node = make_node<GcnConvBackward>(x_, w, b)) {
        node->g = g; node->first = linear_first ? First::linear : First::aggregate;
        node->relu = relu; node->has_bias = b.defined();
        torch::autograd::set_history(out, node);
        node->keep({relu ? out : Tensor(), x.q, x.scale, wq.q, wq.scale, out_n, in_n}, 1);
    }
    return out;
}

// ------------------------------------------------------------------------------------------------ edge softmax
static const int32_t *row_order(const Direction &d) { return d.sched.present ? ptr<int32_t>(d.sched.row_order) : nullptr; }

struct EdgeSoftmaxBackward : SavingNode {
    std::string name() const override { return "EdgeSoftmaxBackward"; }
    GraphPtr g;
    float factor = 1.f;
    variable_list backward(const variable_list &grads) override {
        const std::vector<Tensor> k = kept();
        if (!grads[0].defined()) return variable_list(1);
        const Tensor &at = k[0], a2 = at.reshape({at.size(0), -1}).contiguous();
        const c10::cuda::CUDAGuard guard(a2.device());
        const Tensor da = grads[0].reshape(a2.sizes()).contiguous(), dz = at::empty_like(a2);
        const Direction &d = g->dir(false);
        check(tango_edge_softmax_bwd(ptr<int32_t>(d.indptr), ptr<int32_t>(d.edge_ids), row_order(d), d.sched.n_block_rows,
                                     g->n_nodes, (int)a2.size(1), factor, ptr<float>(a2), ptr<float>(da), ptr<float>(dz),
                                     nullptr, cuda_stream()), "edge_softmax_bwd");
        count(1);
        return {dz.view(at.sizes())};
    }
};

std::tuple<Tensor, Tensor> edge_softmax_fn(const GraphPtr &g, const Tensor &z, double factor) {
    require(z.is_cuda() && z.scalar_type() == at::kFloat, "fp32 CUDA scores expected");
    Tensor a, sa;
    {
        const Raw raw;
        const c10::cuda::CUDAGuard guard(z.device());
        const Tensor z2 = z.reshape({z.size(0), -1}).contiguous();
        require(z2.size(0) == g->n_edges(), "one score row per edge");
        if (z2.size(1) > 8) throw std::invalid_argument("edge_softmax: at most 8 heads");
        const Tensor a2 = at::empty_like(z2);
        sa = zeros1(z);
        const Direction &d = g->dir(false);
        check(tango_edge_softmax(ptr<int32_t>(d.indptr), ptr<int32_t>(d.edge_ids), row_order(d), d.sched.n_block_rows,
                                 g->n_nodes, ptr<float>(z2), (int)z2.size(1), (float)factor, ptr<float>(a2), ptr<float>(sa),
                                 cuda_stream()), "edge_softmax");
        count(1);
        a = a2.view(z.sizes());
    }
    if (auto node = make_node<EdgeSoftmaxBackward>(z)) {
        node->g = g; node->factor = (float)factor;
        torch::autograd::set_history(a, node);
        node->keep({a}, 1);
    }
    return {a, sa};
}

// ------------------------------------------------------------------------------------------------ graph attention
constexpr int64_t kMaxHeads = 8;       // of the softmax kernels

// The two softmax flavours share everything but where the weights live; g, el, er as int8 [N, H] with their scales.
struct GatLogits {
    GraphPtr g;
    Quantized el, er;
    float slope;
    int h;
    const Direction &d() const { return g->dir(false); }
    int64_t n_block() const { return d().sched.n_block_rows; }
};

// `clear`: set to zero by the same launch.
static GatLogits gat_logits(const GraphPtr &g, const Tensor &el, const Tensor &er, double slope, const Tensor &clear) {
    const int64_t n = el.size(0), h = el.size(1);
    if (h < 1 || h > kMaxHeads) throw Failure("gat_attention: 1 to 8 heads");
    QuantJob jl = quant_job(el.reshape({n, h}), 1);
    const QuantJob jr = quant_job(er.reshape({n, h}), 1);
    jl.clear = clear;
    const auto q = quantize_all({jl, jr});
    return {g, q[0], q[1], (float)slope, (int)h};
}

// d_el / d_er from the gradient of the logits: int8, then summed over out-edges and in-edges.
static std::pair<Tensor, Tensor> gat_logit_grads(const GatLogits &a, const Tensor &dz, const Tensor &sdz, bool want_l,
                                                 bool want_r, at::IntArrayRef shape_l, at::IntArrayRef shape_r) {
    QuantJob job = quant_job(dz, 1);
    job.scale = sdz;
    if (want_l) job.clear = aggregation_scratch(*a.g, true, dz);
    if (want_r) job.clear2 = aggregation_scratch(*a.g, false, dz);
    const Quantized q = quantize(job);
    Tensor dl = want_l ? incidence_sum(*a.g, true, q, job.clear).view(shape_l) : Tensor();
    Tensor dr = want_r ? incidence_sum(*a.g, false, q, job.clear2).view(shape_r) : Tensor();
    return {dl, dr};
}

// fp32 weights [E, H]; `sa` holds 0 and receives their scale.
static Tensor gat_softmax(const GatLogits &l, const Tensor &sa) {
    const Tensor a = floats({l.g->n_edges(), l.h}, sa);
    const Direction &d = l.d();
    check(tango_gat_edge_softmax(ptr<int32_t>(d.indptr), ptr<int32_t>(d.indices), ptr<int32_t>(d.edge_ids), row_order(d),
                                 l.n_block(), l.g->n_nodes, ptr<int8_t>(l.el.q), ptr<int8_t>(l.er.q), l.h,
                                 ptr<float>(l.el.scale), ptr<float>(l.er.scale), l.slope, ptr<float>(a), ptr<float>(sa),
                                 cuda_stream()), "gat_edge_softmax");
    count(1);
    return a;
}

// Gradient of the logits from the weights `a` and their gradient, both [E, H]; `sdz` holds 0 and receives its scale.
static Tensor gat_softmax_bwd(const GatLogits &l, const Tensor &a, const Tensor &da, const Tensor &sdz) {
    const Tensor dz = at::empty_like(a);
    const Direction &d = l.d();
    check(tango_gat_edge_softmax_bwd(ptr<int32_t>(d.indptr), ptr<int32_t>(d.indices), ptr<int32_t>(d.edge_ids), row_order(d),
                                     l.n_block(), l.g->n_nodes, ptr<int8_t>(l.el.q), ptr<int8_t>(l.er.q), l.h,
                                     ptr<float>(l.el.scale), ptr<float>(l.er.scale), l.slope, ptr<float>(a),
                                     ptr<float>(da), ptr<float>(dz), ptr<float>(sdz), cuda_stream()), "gat_edge_softmax_bwd");
    count(1);
    return dz;
}

struct GatAttentionBackward : SavingNode {
    std::string name() const override { return "GatAttentionBackward"; }
    GatLogits l;                               // without el and er, which are saved
    std::vector<int64_t> shape_l, shape_r;
    variable_list backward(const variable_list &grads) override {
        const std::vector<Tensor> k = kept();
        if (!grads[0].defined()) return variable_list(2);
        const Tensor &at = k[0];
        GatLogits l = this->l;
        l.el.q = k[1]; l.el.scale = k[2]; l.er.q = k[3]; l.er.scale = k[4];
        const c10::cuda::CUDAGuard guard(at.device());
        const Tensor sdz = zeros1(at);
        const Tensor dz = gat_softmax_bwd(l, at.reshape({-1, l.h}), grads[0].reshape({-1, l.h}).contiguous(), sdz);
        const auto [dl, dr] = gat_logit_grads(l, dz, sdz, needs(0), needs(1), shape_l, shape_r);
        return {dl, dr};
    }
};

std::tuple<Tensor, Tensor> gat_attention_fn(const GraphPtr &g, const Tensor &el, const Tensor &er, double slope) {
    Tensor a, sa;
    GatLogits l;
    {
        const Raw raw;
        const c10::cuda::CUDAGuard guard(el.device());
        sa = floats({1}, el);
        l = gat_logits(g, el, er, slope, sa);
        a = gat_softmax(l, sa).view({-1, l.h, 1});
    }
    if (auto node = make_node<GatAttentionBackward>(el, er)) {
        node->l = l; node->l.el = node->l.er = {};
        node->shape_l = el.sizes().vec(); node->shape_r = er.sizes().vec();
        torch::autograd::set_history(a, node);
        node->keep({a, l.el.q, l.el.scale, l.er.q, l.er.scale}, 1);
    }
    return {a, sa};
}

// The layer behind the linear projection, in two forms that differ in where the attention weights live.
struct GatLayerBackward : SavingNode {
    std::string name() const override { return "GatLayerBackward"; }
    GatLogits l;                               // without el and er, which are saved
    bool int8_weights = false, has_bias = false;
    variable_list backward(const variable_list &grads) override {
        const std::vector<Tensor> k = kept();
        if (!grads[0].defined()) return variable_list(4);
        const c10::cuda::CUDAGuard guard(grads[0].device());
        GatLogits l = this->l;
        l.el.q = k[0]; l.el.scale = k[1]; l.er.q = k[2]; l.er.scale = k[3];
        const Tensor &eq = k[4], &se = k[5], nq = padded(k[6]), &sn = k[7], &ft = k[8], &al = k[9], &ar = k[10];
        const int64_t n = l.g->n_nodes, dim = nq.size(2);
        const bool logits = needs(0) || needs(1) || needs(2), project = needs(1) || needs(2);
        const bool compat = !int8_weights && settings().compat_dn_scale;

        QuantJob job = quant_job(grads[0]);
        job.colsum = has_bias && needs(3);
        if (!compat) job.times[0] = se;
        if (needs(0)) job.clear = aggregation_scratch(*l.g, true, grads[0]);
        const Tensor sdz = job.clear2 = floats({1}, grads[0]);
        const Quantized z = quantize(job);
        Tensor d_ft, dal, dar;
        if (needs(0)) d_ft = spmm_u_mul_e(*l.g, true, z.q, eq, compat ? k[12] : z.product[0], job.clear);
        if (logits) {
            const Tensor da = sddmm(*l.g, int8_weights || dim > 1 ? "dot" : "mul", nq, z.q, sn, z.scale, {}, false)
                                  .reshape({l.g->n_edges(), l.h});
            Tensor dz;
            if (int8_weights) {
                dz = at::empty_like(da);
                const Direction &d = l.d();
                check(tango_gat_edge_softmax_bwd_stats(ptr<int32_t>(d.indptr), ptr<int32_t>(d.indices), ptr<int32_t>(d.edge_ids),
                                                       row_order(d), l.n_block(), n, ptr<int8_t>(l.el.q), ptr<int8_t>(l.er.q),
                                                       l.h, ptr<float>(l.el.scale), ptr<float>(l.er.scale), l.slope,
                                                       ptr<float>(k[11]), ptr<float>(k[12]), ptr<float>(da), ptr<float>(dz),
                                                       ptr<float>(sdz), cuda_stream()), "gat_edge_softmax_bwd_stats");
                count(1);
            } else {
                dz = gat_softmax_bwd(l, k[11], da, sdz);
            }
            const auto [dl, dr] = gat_logit_grads(l, dz, sdz, true, true, {n, l.h}, {n, l.h});
            if (project) { dal = at::empty_like(al); dar = at::empty_like(ar); }
            const Matrix x = matrix(ft);
            const int64_t bytes = project ? tango_gat_project_bwd_scratch_bytes(n, l.h, (int)dim) : 0;
            const Tensor scratch = at::empty({std::max<int64_t>(bytes, 16)}, dl.options().dtype(at::kByte));
            check(tango_gat_project_bwd(ptr<float>(x.t), n, l.h, (int)dim, ptr<float>(al), ptr<float>(ar), ptr<float>(dl),
                                        ptr<float>(dr), ptr<float>(d_ft), ptr<float>(dal), ptr<float>(dar), ptr(scratch), bytes,
                                        cuda_stream()), "gat_project_bwd");
            count(1 + project);
        }
        return {d_ft, needs(1) ? dal : Tensor(), needs(2) ? dar : Tensor(), z.colsum};
    }
};

Tensor gat_layer_fn(const GraphPtr &g, const Tensor &ft_, const Tensor &al_, const Tensor &ar_, const Tensor &bias, double slope,
                    bool int8_weights) {
    require(ft_.dim() == 3, "features [N, H, D] expected");
    const int64_t n = ft_.size(0), h = ft_.size(1), dim = ft_.size(2);
    require(n == g->n_nodes, "one feature row per node expected");
    if (h < 1 || h > kMaxHeads) throw Failure("gat_layer: 1 to 8 heads");      // before the first launch
    for (const Tensor *t : {&al_, &ar_, &bias})
        require(!t->defined() || t->numel() == h * dim, "parameters of H * D elements expected");
    for (const Tensor *t : {&ft_, &al_, &ar_, &bias})
        require(!t->defined() || (t->is_cuda() && t->scalar_type() == at::kFloat && t->device() == ft_.device()),
                "fp32 tensors on one CUDA device expected");
    Tensor out, ft, al, ar, weights, inv, scale;
    GatLogits l;
    Quantized eq, nq;
    {
        const Raw raw;
        const c10::cuda::CUDAGuard guard(ft_.device());
        ft = ft_.contiguous(); al = al_.contiguous(); ar = ar_.contiguous();
        // the sums of the operator chain: the codes of el and er, and with them every gradient, hang on their last bit
        const Tensor el = at::mul(ft, al.view({1, h, dim})).sum(-1), er = at::mul(ft, ar.view({1, h, dim})).sum(-1);
        const Tensor sa = floats({1}, ft);
        l = gat_logits(g, el, er, slope, sa);
        QuantJob jn;
        if (int8_weights) {
            const Direction &d = l.d();
            weights = floats({n, h}, ft);
            inv = at::empty_like(weights);
            eq.scale = sa;
            check(tango_gat_edge_softmax_stats(ptr<int32_t>(d.indptr), ptr<int32_t>(d.indices), row_order(d), l.n_block(), n,
                                               ptr<int8_t>(l.el.q), ptr<int8_t>(l.er.q), l.h, ptr<float>(l.el.scale),
                                               ptr<float>(l.er.scale), l.slope, ptr<float>(weights), ptr<float>(inv),
                                               ptr<float>(eq.scale), cuda_stream()), "gat_edge_softmax_stats");
            const int mode = settings().mode_quantize;
            const uint64_t call = call_if(mode);
            eq.q = at::empty({g->n_edges(), h}, ft.options().dtype(at::kChar));
            check(tango_gat_edge_softmax_quantized(ptr<int32_t>(d.indptr), ptr<int32_t>(d.indices), ptr<int32_t>(d.edge_ids),
                                                   row_order(d), l.n_block(), n, ptr<int8_t>(l.el.q), ptr<int8_t>(l.er.q), l.h,
                                                   ptr<float>(l.el.scale), ptr<float>(l.er.scale), l.slope, ptr<float>(weights),
                                                   ptr<float>(inv), ptr<float>(eq.scale), ptr<int8_t>(eq.q), mode,
                                                   settings().seed, call, settings().step, cuda_stream()),
                  "gat_edge_softmax_quantized");
            count(2);
            jn = quant_job(ft);
            jn.times[0] = eq.scale;
            jn.clear = aggregation_scratch(*g, false, ft);
            nq = quantize(jn);
        } else {
            weights = gat_softmax(l, sa);
            QuantJob je = quant_job(weights, 1);
            je.scale = sa;
            jn = quant_job(ft);
            jn.times_job = 0;
            jn.clear = aggregation_scratch(*g, false, ft);
            const auto q = quantize_all({je, jn});
            eq = q[0]; nq = q[1];
        }
        scale = nq.product[0];
        out = spmm_u_mul_e(*g, false, nq.q, eq.q, scale, jn.clear, bias.defined() ? bias.contiguous() : bias);
    }
    if (auto node = make_node<GatLayerBackward>(ft_, al_, ar_, bias)) {
        node->l = l; node->l.el = node->l.er = {};
        node->int8_weights = int8_weights; node->has_bias = bias.defined();
        torch::autograd::set_history(out, node);
        node->keep({l.el.q, l.el.scale, l.er.q, l.er.scale, eq.q, eq.scale, nq.q, nq.scale, ft, al, ar, weights,
                    int8_weights ? inv : scale});
    }
    return out;
}

}  // namespace tango_host
