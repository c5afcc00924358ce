// Python bindings of the host layer: module `_torch_ops`, loaded by tango_b200/_native.py.
#include <torch/csrc/utils/pybind.h>

#include "torch_autograd.h"

namespace py = pybind11;
using namespace tango_host;

static Tensor tensor_attr(const py::handle &o, const char *name) { return o.attr(name).cast<Tensor>(); }
static Tensor optional(const py::object &o) { return o.is_none() ? Tensor() : o.cast<Tensor>(); }

static Schedule schedule(const py::object &s, bool with_hub) {
    Schedule out;
    if (s.is_none()) return out;
    out.present = true;
    out.units = tensor_attr(s, "units");
    out.heavy_rows = tensor_attr(s, "heavy_rows");
    out.row_order = tensor_attr(s, "row_order");
    if (const py::object info = s.attr("row_info"); !info.is_none()) out.row_info = info.cast<Tensor>();
    out.n_over_few = s.attr("n_over_few").cast<int64_t>();
    out.n_over_one = s.attr("n_over_one").cast<int64_t>();
    out.unit = s.attr("unit").cast<int>();
    out.n_units = s.attr("n_units").cast<int64_t>();
    out.n_heavy = s.attr("n_heavy").cast<int64_t>();
    out.n_long = s.attr("n_long").cast<int64_t>();
    out.n_block_rows = s.attr("n_block_rows").cast<int64_t>();
    out.n_skip = s.attr("n_skip").cast<int64_t>();
    out.threshold = s.attr("threshold").cast<int>();
    if (with_hub) {
        const py::object hub = s.attr("hub");
        out.dense = tensor_attr(hub, "dense");
        out.dense_units = tensor_attr(hub, "units");
        out.dense_cols = tensor_attr(hub, "cols");
        out.n_tiles = hub.attr("n_tiles").cast<int64_t>();
        out.dense_rows = tensor_attr(hub, "rows").numel();
        out.has_hub = true;
    }
    return out;
}

// bundle: (indptr, indices, edge_ids or None); hub: tango_b200.graph.HubBlock or None
static std::shared_ptr<Direction> direction(const py::tuple &bundle, const py::object &sched, const py::object &hub) {
    auto d = std::make_shared<Direction>();
    d->indptr = bundle[0].cast<Tensor>();
    d->indices = bundle[1].cast<Tensor>();
    d->edge_ids = optional(bundle[2]);
    d->sched = schedule(sched, false);
    if (!hub.is_none()) {
        d->has_hub = true;
        d->hub_indptr = tensor_attr(hub, "indptr");
        d->hub_indices = tensor_attr(hub, "indices");
        d->hub_sched = schedule(hub.attr("schedule"), true);
    }
    return d;
}

static py::object wrap(const Tensor &t) { return t.defined() ? py::cast(t) : py::none(); }

PYBIND11_MODULE(_torch_ops, m) {
    py::object error = py::module_::import("tango_b200._lib").attr("TangoError");
    static py::handle tango_error = error.release();      // lives as long as the module
    py::register_exception_translator([](std::exception_ptr p) {
        try {
            if (p) std::rethrow_exception(p);
        } catch (const Failure &e) {
            PyErr_SetString(tango_error.ptr(), e.what());
        } catch (const Violation &e) {
            PyErr_SetString(PyExc_AssertionError, e.what());
        }
    });

    py::class_<Direction, std::shared_ptr<Direction>>(m, "Direction").def(py::init(&direction));
    py::class_<Graph, GraphPtr>(m, "Graph")
        .def(py::init([](std::shared_ptr<Direction> csc, std::shared_ptr<Direction> csr, Tensor src, Tensor dst, int64_t n) {
            auto g = std::make_shared<Graph>();
            g->csc = std::move(csc); g->csr = std::move(csr); g->src = std::move(src); g->dst = std::move(dst); g->n_nodes = n;
            return g;
        }));

    m.def("set_rounding", [](int gemm, int quantize, uint64_t seed) {
        settings().mode_gemm = gemm; settings().mode_quantize = quantize; settings().seed = seed;
    });
    m.def("set_step_counter", [](const py::object &t) {   // the Python side keeps the tensor alive
        settings().step = t.is_none() ? nullptr : reinterpret_cast<const uint64_t *>(t.cast<Tensor>().data_ptr());
    });
    m.def("set_compat_dn_scale", [](bool on) { settings().compat_dn_scale = on; });
    m.def("next_call", [] { return next_call(); });
    m.def("set_call_counter", [](uint64_t v) { settings().calls = v; });
    m.def("launches", [] { return settings().launches.load(); });
    m.def("set_launches", [](int64_t v) { settings().launches = v; });
    m.def("status_word", [](const Tensor &like) { return status_word(like.device()); });

    m.def("get_scale", [](const Tensor &t, const py::object &row_scale) { return absmax_scale(t, optional(row_scale)); },
          py::arg("t"), py::arg("row_scale") = py::none());
    m.def("quantize", [](const Tensor &t, const py::object &scale, int mode, uint64_t seed, uint64_t call, int64_t align) {
        require(t.is_cuda(), "tensor must be on GPU");
        QuantJob job{t, mode, seed, call, align};
        job.scale = optional(scale);
        const Quantized q = quantize(job);
        return py::make_tuple(q.q, q.scale);
    });

    m.def("qlinear", [](const Tensor &x, const Tensor &w, const py::object &b, bool want_scale, const py::object &xq,
                        const py::object &sx) {
        auto [y, sy, xq2, sx2] = qlinear(x, w, optional(b), want_scale, optional(xq), optional(sx));
        return py::make_tuple(y, wrap(sy), xq2, sx2);
    });
    m.def("qlinear_group", [](const Tensor &x, const std::vector<Tensor> &w, const std::vector<py::object> &b) {
        std::vector<Tensor> bias;
        for (const py::object &o : b) bias.push_back(optional(o));
        return qlinear_group(x, w, bias);
    });
    m.def("spmm_copy_u", [](const GraphPtr &g, const Tensor &n, const py::object &s) { return spmm_copy_u_fn(g, n, optional(s)); });
    m.def("spmm_u_mul_e", [](const GraphPtr &g, const Tensor &n, const Tensor &e, const py::object &s) {
        return spmm_u_mul_e_fn(g, n, e, optional(s));
    });
    m.def("sddmm_u_add_v", [](const GraphPtr &g, const Tensor &u, const Tensor &v, const py::object &su, const py::object &sv) {
        return sddmm_u_add_v_fn(g, u, v, optional(su), optional(sv));
    });
    m.def("sddmm_u_dot_v", &sddmm_u_dot_v_fn);
    m.def("gcn_conv", [](const GraphPtr &g, const Tensor &x, const Tensor &w, const py::object &b, const Tensor &out_norm,
                         const Tensor &in_norm, bool relu, bool linear_first) {
        return gcn_conv_fn(g, x, w, optional(b), out_norm, in_norm, relu, linear_first);
    });
    m.def("edge_softmax", &edge_softmax_fn);
    m.def("gat_attention", &gat_attention_fn);
    m.def("gat_layer", [](const GraphPtr &g, const Tensor &ft, const Tensor &al, const Tensor &ar, const py::object &bias,
                          double slope, bool int8_weights) {
        return gat_layer_fn(g, ft, al, ar, optional(bias), slope, int8_weights);
    });
}
