// The operators of this package over at::Tensor: shapes, allocation of outputs and scratch, and the C ABI calls.
#include "torch_ops.h"

#include <map>
#include <mutex>

namespace tango_host {

void check(int rc, const char *what) {
    if (rc == TANGO_OK) return;
    std::string msg = std::string(what) + ": " + tango_strerror(rc);
    if (rc == TANGO_ECUDA) msg += " (cudaError " + std::to_string(tango_last_cuda_error()) + ")";
    throw Failure(msg);
}

Settings &settings() {
    static Settings s;
    return s;
}

Matrix matrix(const Tensor &t) {
    if (t.dim() <= 1) {
        Tensor c = t.contiguous();
        const int64_t n = c.numel();
        return {c, 1, n, std::max<int64_t>(n, 1)};
    }
    const int64_t rows = t.size(0), cols = rows ? t.numel() / rows : 0;
    // the row stride comes first: a single row of a padded tensor counts as contiguous, but its pitch is the padded one
    if (rows > 0 && t.stride(0) >= cols) {
        int64_t want = 1;
        bool packed = true;
        for (int64_t d = t.dim() - 1; d >= 1 && packed; --d) {
            packed = t.size(d) == 1 || t.stride(d) == want;
            want *= t.size(d);
        }
        if (packed) return {t, rows, cols, std::max<int64_t>(t.stride(0), 1)};
    }
    if (t.is_contiguous()) return {t, rows, cols, std::max<int64_t>(cols, 1)};
    return {t.contiguous(), rows, cols, std::max<int64_t>(cols, 1)};
}

Tensor alloc_int8(at::IntArrayRef shape, const at::Device &device, int64_t align) {
    const auto opt = at::TensorOptions().dtype(at::kChar).device(device);
    if (shape.size() < 2) return at::empty(shape, opt);
    int64_t cols = 1;
    for (size_t d = 1; d < shape.size(); ++d) cols *= shape[d];
    const int64_t ld = (std::max<int64_t>(cols, 1) + align - 1) / align * align;
    if (ld == cols) return at::empty(shape, opt);
    std::vector<int64_t> stride(shape.size(), 1);
    for (size_t d = shape.size() - 1; d-- > 1;) stride[d] = stride[d + 1] * shape[d + 1];
    stride[0] = ld;
    return at::empty({shape[0] * ld}, opt).as_strided(shape, stride);
}

Tensor status_word(const at::Device &device) {
    static std::mutex mutex;
    static std::map<int, Tensor> words;      // one per device, for the life of the process
    std::lock_guard<std::mutex> lock(mutex);
    Tensor &w = words[device.index()];
    if (!w.defined()) w = at::zeros({1}, at::TensorOptions().dtype(at::kInt).device(device));
    return w;
}

// ------------------------------------------------------------------------------------------------ quantisation
static void require_float(const Tensor &t) { require(t.is_cuda() && t.scalar_type() == at::kFloat, "fp32 CUDA tensor expected"); }

Tensor absmax_scale(const Tensor &t, const Tensor &row_scale) {
    require_float(t);
    const c10::cuda::CUDAGuard guard(t.device());
    const Matrix x = matrix(t);
    Tensor scale = floats({1}, t);
    check(tango_absmax_scale(ptr<float>(x.t), x.rows, x.cols, x.ld, ptr<float>(row_scale), ptr<float>(scale), cuda_stream()),
          "get_scale");
    count(1);
    return scale;
}

QuantJob quant_job(const Tensor &t, int64_t align) {
    QuantJob j;
    j.t = t;
    j.mode = settings().mode_quantize;
    j.seed = settings().seed;
    j.call = j.mode == TANGO_ROUND_STOCHASTIC ? next_call() : 0;
    j.align = align;
    return j;
}

// A matrix too large for the fused kernel (32-bit indices, scratch of column sums): scale, then quantize, then column sums, one after the other.
static void quantize_large(const QuantJob &j, const tango_quant_job &c, Quantized &o) {
    if (c.gate) {
        require(!c.fixed_scale, "a gated matrix of this size finds its own scale");
        const int64_t bytes = tango_relu_grad_stats_scratch_bytes(c.rows, c.cols);
        const Tensor scratch = at::empty({std::max<int64_t>(bytes, 16)}, j.t.options().dtype(at::kByte));
        check(tango_relu_grad_stats(c.x, c.ldx, c.gate, c.ldgate, c.rows, c.cols, c.row_scale, c.scale, c.colsum, ptr(scratch),
                                    bytes, cuda_stream()), "relu_grad_stats");
        check(tango_quantize_relu_grad(c.x, c.ldx, c.gate, c.ldgate, c.rows, c.cols, c.row_scale, c.scale, c.q, c.ldq, c.mode,
                                       c.seed, c.call, settings().step, cuda_stream()), "quantize_relu_grad");
    } else {
        if (!c.fixed_scale)
            check(tango_absmax_scale(c.x, c.rows, c.cols, c.ldx, c.row_scale, c.scale, cuda_stream()), "get_scale");
        check(tango_quantize(c.x, c.rows, c.cols, c.ldx, c.row_scale, c.scale, c.q, c.ldq, c.mode, c.seed, c.call,
                             settings().step, cuda_stream()), "quantize");
        if (c.colsum) at::sum_out(o.colsum, j.t.reshape({c.rows, c.cols}), at::IntArrayRef{0});
    }
    count(3);
}

std::vector<Quantized> quantize_all(const std::vector<QuantJob> &jobs) {
    const c10::cuda::CUDAGuard guard(jobs[0].t.device());
    const size_t n = jobs.size();
    std::vector<Quantized> out(n);
    tango_quant_job c[4];
    Matrix x[4], gate[4];
    const auto fp = jobs[0].t.options().dtype(at::kFloat);
    for (size_t k = 0; k < n; ++k) {
        const QuantJob &j = jobs[k];
        Quantized &o = out[k];
        require_float(j.t);
        x[k] = matrix(j.t);
        o.q = alloc_int8(j.t.sizes(), j.t.device(), j.align);
        o.scale = j.scale.defined() ? j.scale : at::empty({1}, fp);
        if (j.gate.defined()) gate[k] = matrix(j.gate);
        if (j.colsum) o.colsum = at::empty({x[k].cols}, fp);
        const Matrix q = matrix(o.q);
        c[k] = tango_quant_job{};
        c[k].x = ptr<float>(x[k].t); c[k].rows = x[k].rows; c[k].cols = x[k].cols; c[k].ldx = x[k].ld;
        c[k].gate = ptr<float>(gate[k].t); c[k].ldgate = gate[k].ld;
        c[k].row_scale = ptr<float>(j.row_scale);
        c[k].scale = ptr<float>(o.scale);
        c[k].fixed_scale = j.scale.defined();
        c[k].times_job = j.times_job;
        for (int i = 0; i < 2; ++i)
            if (j.times[i].defined() || (i == 0 && j.times_job >= 0)) {
                o.product[i] = at::empty({1}, fp);
                c[k].times[i] = ptr<float>(j.times[i]);
                c[k].product[i] = ptr<float>(o.product[i]);
            }
        c[k].colsum = ptr<float>(o.colsum);
        const Tensor *clear[2] = {&j.clear, &j.clear2};
        for (int i = 0; i < 2; ++i)
            if (clear[i]->defined()) { c[k].clear[i] = ptr(*clear[i]); c[k].clear_words[i] = clear[i]->numel(); }
        c[k].q = ptr<int8_t>(o.q); c[k].ldq = q.ld;
        c[k].mode = j.mode; c[k].seed = j.seed; c[k].call = j.call;
    }
    const int64_t bytes = tango_quantize_fused_scratch_bytes(c, (int)n);
    if (bytes < 0 && bytes != TANGO_ESIZE) check((int)bytes, "quantize");
    if (bytes < 0) {
        for (size_t k = 0; k < n; ++k) {
            for (const Tensor &t : {jobs[k].clear, jobs[k].clear2})
                if (t.defined()) t.zero_();
            quantize_large(jobs[k], c[k], out[k]);
        }
        for (size_t k = 0; k < n; ++k)
            for (int i = 0; i < 2; ++i)
                if (c[k].product[i])
                    at::mul_out(out[k].product[i], out[k].scale, jobs[k].times[i].defined() ? jobs[k].times[i] : out[jobs[k].times_job].scale);
        return out;
    }
    const Tensor scratch = at::empty({std::max<int64_t>(bytes, 16)}, fp.dtype(at::kByte));
    check(tango_quantize_fused(c, (int)n, settings().step, ptr(scratch), bytes, cuda_stream()), "quantize");
    count(1);
    return out;
}

Quantized quantize(const QuantJob &job) { return quantize_all({job})[0]; }

// ------------------------------------------------------------------------------------------------ GEMMs
Tensor gemm_nt(const Quantized &xq, const Quantized &wq, const Tensor &bias, const Tensor &scale_out, const Tensor &row_scale,
               bool relu) {
    const c10::cuda::CUDAGuard guard(xq.q.device());
    const Matrix x = matrix(xq.q), w = matrix(wq.q);
    Tensor y = floats({x.rows, w.rows}, xq.scale);
    check(tango_qgemm_layer(ptr<int8_t>(x.t), x.ld, ptr<int8_t>(w.t), w.ld, x.rows, w.rows, x.cols, ptr<float>(xq.scale),
                            ptr<float>(wq.scale), ptr<float>(row_scale), ptr<float>(bias), relu, ptr<float>(y), w.rows,
                            ptr<float>(scale_out), nullptr, ptr<int>(status_word(y.device())), cuda_stream()), "qgemm_nt");
    count(1);
    return y;
}

Tensor gemm_dx(const Quantized &dyq, const Quantized &wq, const Tensor &row_scale, const Tensor &scale_out) {
    const c10::cuda::CUDAGuard guard(dyq.q.device());
    const Matrix dy = matrix(dyq.q), w = matrix(wq.q);
    Tensor dx = floats({dy.rows, w.cols}, dyq.scale);
    check(tango_qgemm_dx_layer(ptr<int8_t>(dy.t), dy.ld, ptr<int8_t>(w.t), w.ld, dy.rows, dy.cols, w.cols,
                               ptr<float>(dyq.scale), ptr<float>(wq.scale), ptr<float>(row_scale), ptr<float>(dx), w.cols,
                               ptr<float>(scale_out), ptr<int>(status_word(dx.device())), cuda_stream()),
          "QGEMM_backward_gradX");
    count(1);
    return dx;
}

Tensor dw_scratch(int64_t m, int64_t n, int64_t k, const Tensor &like) {
    return at::empty({tango_qgemm_dw_scratch_bytes(m, n, k) / 4}, like.options().dtype(at::kInt));
}

Tensor gemm_dw(const Quantized &dyq, const Quantized &xq, const Tensor &scratch) {
    const c10::cuda::CUDAGuard guard(dyq.q.device());
    const Matrix dy = matrix(dyq.q), x = matrix(xq.q);
    Tensor dw = floats({dy.cols, x.cols}, dyq.scale);
    check(tango_qgemm_dw_cleared(ptr<int8_t>(dy.t), dy.ld, ptr<int8_t>(x.t), x.ld, dy.rows, dy.cols, x.cols,
                                 ptr<float>(dyq.scale), ptr<float>(xq.scale), ptr<float>(dw), x.cols, ptr(scratch),
                                 scratch.numel() * 4, ptr<int>(status_word(dw.device())), cuda_stream()), "QGEMM_backward_gradW");
    count(1);
    return dw;
}

// ------------------------------------------------------------------------------------------------ graph operators
// The C ABI's view of a schedule, and the scratch that has to live until the call returns (the allocator orders its
// reuse behind the launches on this stream).
struct Plan {
    tango_spmm_plan p{};
    Tensor ws, packed;
    const tango_spmm_plan *get(const Schedule &s) const { return s.present ? &p : nullptr; }
};

static Plan make_plan(const Schedule &s, int64_t f, const Tensor &like, const Tensor &scratch) {
    Plan plan;
    if (!s.present) return plan;
    tango_spmm_plan &p = plan.p;
    p.split_threshold = s.threshold;
    p.row_order = ptr<int32_t>(s.row_order);
    p.n_long_rows = p.row_order ? s.n_long : -1;
    p.row_info = p.row_order ? ptr<int32_t>(s.row_info) : nullptr;
    p.n_over_few = s.n_over_few;
    p.n_over_one = s.n_over_one;
    if (s.n_heavy == 0) return plan;
    const int64_t ld = (f + 15) / 16 * 16;
    if (scratch.defined()) {
        plan.ws = scratch;
        p.arrivals = ptr<int32_t>(scratch) + s.n_heavy * ld;
        p.unit_slots = s.unit;
    } else {
        plan.ws = at::empty({s.n_heavy, ld}, like.options().dtype(at::kInt));
    }
    p.units = ptr<int32_t>(s.units);
    p.n_units = s.n_units;
    p.heavy_rows = ptr<int32_t>(s.heavy_rows);
    p.n_heavy = s.n_heavy;
    p.ws = ptr<int32_t>(plan.ws);
    p.ws_ld = ld;
    if (s.has_hub) {
        plan.packed = at::empty({s.dense_cols.numel(), ld}, like.options().dtype(at::kChar));
        p.dense_a = ptr<int8_t>(s.dense);
        p.dense_n_tiles = s.n_tiles;
        p.dense_rows = s.dense_rows;
        p.dense_units = ptr<int32_t>(s.dense_units);
        p.dense_n_units = s.dense_units.size(0);
        p.dense_cols = ptr<int32_t>(s.dense_cols);
        p.dense_n_cols = s.dense_cols.numel();
        p.dense_b = ptr<int8_t>(plan.packed);
        p.dense_status = ptr<int>(status_word(like.device()));
        p.n_skip_rows = s.n_skip;
    }
    return plan;
}

// Pointer of a mandatory index array; an empty one (graph without edges) still needs a valid address, and the row
// pointers in front of it are one.
static const int32_t *index_ptr(const Tensor &t, const Tensor &indptr) {
    return t.numel() > 0 ? ptr<int32_t>(t) : ptr<int32_t>(indptr);
}

static const Schedule &schedule_for(const Direction &d, bool hub) { return hub ? d.hub_sched : d.sched; }
// the dense hub region takes feature rows at exactly their padded width, the layout every quantizer here writes
static bool takes_hub(const Direction &d, const Tensor &nq, int64_t cols) {
    return d.has_hub && nq.dim() >= 2 && nq.stride(0) == (cols + 15) / 16 * 16;
}

Tensor spmm_scratch(const Graph &g, bool reverse, int64_t f, const Tensor &like) {
    const Schedule &s = g.dir(reverse).sched;
    if (!s.present || s.n_units == 0) return {};
    return at::empty({s.n_heavy * ((f + 15) / 16 * 16 + 1)}, like.options().dtype(at::kInt));
}

Tensor spmm_copy_u(const Graph &g, bool reverse, const Quantized &nq, const Tensor &scratch, const Tensor &row_scale,
                   const Tensor &bias, bool relu, const Tensor &scale_out) {
    const c10::cuda::CUDAGuard guard(nq.q.device());
    const Direction &d = g.dir(reverse);
    const Matrix n = matrix(nq.q);
    const bool hub = takes_hub(d, nq.q, n.cols);
    const Schedule &s = schedule_for(d, hub);
    std::vector<int64_t> shape(nq.q.sizes().begin(), nq.q.sizes().end());
    shape[0] = g.n_nodes;
    Tensor out = floats(shape, nq.scale);
    const Plan plan = make_plan(s, n.cols, nq.q, hub ? Tensor() : scratch);
    const Tensor &indptr = hub ? d.hub_indptr : d.indptr;
    check(tango_spmm_copy_u(ptr<int32_t>(indptr), index_ptr(hub ? d.hub_indices : d.indices, indptr), g.n_nodes, 1,
                            ptr<int8_t>(n.t), n.ld, n.cols, ptr<float>(nq.scale), ptr<float>(row_scale), ptr<float>(bias),
                            relu, ptr<float>(out), n.cols, ptr<float>(scale_out), plan.get(s), cuda_stream()), "csr_SPMM");
    count(1 + (s.n_heavy > 0 && !plan.p.arrivals) + (hub ? 2 : 0));
    return out;
}

Tensor spmm_u_mul_e(const Graph &g, bool reverse, const Tensor &nq, const Tensor &eq, const Tensor &scale,
                    const Tensor &scratch, const Tensor &bias) {
    require(nq.dim() == 3, "node features must be [N, H, D]");
    const c10::cuda::CUDAGuard guard(nq.device());
    const Direction &d = g.dir(reverse);
    const Matrix n = matrix(nq);
    const Tensor e = eq.numel() ? eq.contiguous() : at::zeros({1}, nq.options());
    Tensor out = floats({d.n_rows(), nq.size(1), nq.size(2)}, scale);
    const Plan plan = make_plan(d.sched, n.cols, nq, scratch);
    check(tango_spmm_u_mul_e_bias(ptr<int32_t>(d.indptr), index_ptr(d.indices, d.indptr), ptr<int32_t>(d.edge_ids), d.n_rows(),
                                  ptr<int8_t>(n.t), n.ld, (int)nq.size(1), (int)nq.size(2), ptr<int8_t>(e), ptr<float>(scale),
                                  ptr<float>(bias), ptr<float>(out), n.cols, plan.get(d.sched), cuda_stream()),
          "multi_cusparse_SPMM");
    count(1 + (d.sched.n_units > 0 && !plan.p.arrivals));
    return out;
}

Tensor incidence_sum(const Graph &g, bool reverse, const Quantized &zq, const Tensor &scratch) {
    const c10::cuda::CUDAGuard guard(zq.q.device());
    const Direction &d = g.dir(reverse);
    const Matrix z = matrix(zq.q);
    std::vector<int64_t> shape(zq.q.sizes().begin(), zq.q.sizes().end());
    shape[0] = g.n_nodes;
    Tensor out = floats(shape, zq.scale);
    const int64_t f = z.cols;
    const Plan plan = make_plan(d.sched, f, zq.q, scratch);
    check(tango_spmm_incidence(ptr<int32_t>(d.indptr), ptr<int32_t>(d.edge_ids), d.n_rows(), ptr<int8_t>(z.t), z.ld, f,
                               ptr<float>(zq.scale), ptr<float>(out), f, plan.get(d.sched), cuda_stream()), "incidence_SPMM");
    count(1 + (d.sched.n_units > 0 && !plan.p.arrivals));
    return out;
}

// Average edges per row from which the dot product walks rows (the fixed operand stays in registers).  With a handful
// of edges per row the endpoint-list kernel (32 edges per warp, whatever their rows) measured faster: 169,343 nodes /
// 1.3 M edges, 4 heads x 32: 0.060 ms against 0.069 ms.
constexpr int64_t kRowwiseDotMinDegree = 32;

static bool sddmm_dot_rows(const Graph &g, bool reverse, const Matrix &u, const Matrix &v, int h, int dim, const Tensor &su,
                           const Tensor &sv, const Tensor &out, const Tensor &scale) {
    const Direction &d = g.dir(reverse);
    const Schedule &s = d.sched;
    tango_spmm_plan p{};
    p.units = ptr<int32_t>(s.units); p.n_units = s.n_units; p.split_threshold = s.threshold;
    p.row_order = ptr<int32_t>(s.row_order); p.n_long_rows = p.row_order ? s.n_long : -1;
    const int rc = tango_sddmm_dot_rows(ptr<int32_t>(d.indptr), index_ptr(d.indices, d.indptr), ptr<int32_t>(d.edge_ids),
                                        d.n_rows(), ptr<int8_t>(u.t), u.ld, ptr<int8_t>(v.t), v.ld, h, dim, ptr<float>(su),
                                        ptr<float>(sv), ptr<float>(out), ptr<float>(scale), s.present ? &p : nullptr,
                                        cuda_stream());
    if (rc == TANGO_EALIGN) return false;      // an operand layout that only the endpoint-list kernel takes
    check(rc, "mySDDMM_int8(dot, rows)");
    count(1 + (s.present && s.n_long < s.row_order.numel()));
    return true;
}

Tensor sddmm(const Graph &g, const std::string &op, const Tensor &u_, const Tensor &v_, const Tensor &su, const Tensor &sv,
             const Tensor &scale, bool reverse) {
    require(g.src.is_cuda() && g.dst.is_cuda() && u_.is_cuda() && v_.is_cuda() && su.is_cuda() && sv.is_cuda(),
            "CUDA tensors expected");
    const c10::cuda::CUDAGuard guard(u_.device());
    const bool flat = u_.dim() == 2 && v_.dim() == 2;
    const Tensor u = flat ? u_.unsqueeze(1) : u_, v = flat ? v_.unsqueeze(1) : v_;
    const Tensor &src = reverse ? g.dst : g.src, &dst = reverse ? g.src : g.dst;
    const int64_t n_edges = src.numel();
    const bool dot = op == "dot";
    // trailing-shape broadcast (dgl.sparse.infer_broadcast_shape in the reference); "dot" collapses the last dimension
    if (dot && u.size(-1) != v.size(-1)) throw std::invalid_argument("dot needs equal feature sizes");
    const int64_t nd = std::max(u.dim(), v.dim());
    std::vector<int64_t> shape{n_edges};
    for (int64_t k = 1; k < nd; ++k) {
        const int64_t a = k - (nd - u.dim()) >= 1 ? u.size(k - (nd - u.dim())) : 1;
        const int64_t b = k - (nd - v.dim()) >= 1 ? v.size(k - (nd - v.dim())) : 1;
        if (a != b && a != 1 && b != 1) throw std::invalid_argument("cannot broadcast the feature shapes");
        shape.push_back(std::max(a, b));
    }
    if (dot) shape.back() = 1;
    Tensor out = floats(shape, su);
    const Matrix um = matrix(u), vm = matrix(v);
    if (dot) {
        const int h = (int)u.size(-2), dim = (int)u.size(-1);
        const bool rows = n_edges > 0 && n_edges >= kRowwiseDotMinDegree * g.n_nodes && u.dim() == 3 &&
                          u.sizes().slice(1) == v.sizes().slice(1) && u.size(0) == g.n_nodes && v.size(0) == g.n_nodes;
        if (!rows || !sddmm_dot_rows(g, reverse, um, vm, h, dim, su, sv, out, scale)) {
            check(tango_sddmm_dot(ptr<int32_t>(src), ptr<int32_t>(dst), n_edges, ptr<int8_t>(um.t), um.ld, ptr<int8_t>(vm.t),
                                  vm.ld, h, dim, ptr<float>(su), ptr<float>(sv), ptr<float>(out), ptr<float>(scale),
                                  cuda_stream()), "mySDDMM_int8(dot)");
            count(1);
        }
    } else {
        const int code = op == "add" ? TANGO_OP_ADD : op == "sub" ? TANGO_OP_SUB : op == "mul" ? TANGO_OP_MUL
                       : op == "div" ? TANGO_OP_DIV : -1;
        if (code < 0) throw std::invalid_argument(op + " op not supported");
        require(um.cols == vm.cols, "element-wise SDDMM needs equal feature shapes");
        check(tango_sddmm_elementwise(code, ptr<int32_t>(src), ptr<int32_t>(dst), n_edges, ptr<int8_t>(um.t), um.ld,
                                      ptr<int8_t>(vm.t), vm.ld, um.cols, ptr<float>(su), ptr<float>(sv), ptr<float>(out),
                                      ptr<float>(scale), cuda_stream()), "mySDDMM_int8");
        count(1);
    }
    return flat ? out.squeeze(1) : out;
}

}  // namespace tango_host
