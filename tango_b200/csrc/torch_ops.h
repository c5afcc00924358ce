// Shared by the host layer (torch_*.cpp): the operators of this package over at::Tensor, without Python.
//
// Why a native host layer: one training pass of a small model is a few dozen kernels of 2-10 microseconds each, and
// the same calls issued operator by operator from Python cost 15-30 microseconds apiece (tensor wrappers, ctypes
// marshalling, autograd nodes that take the interpreter lock in the engine's thread).  Here an autograd node is a C++
// object whose backward runs without the interpreter, and a kernel call is a plain function call into the C ABI.
#pragma once
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>

#include <atomic>
#include <memory>
#include <string>
#include <vector>

#include "tango_b200.h"

namespace tango_host {

using at::Tensor;

// A failed C ABI call (TangoError in Python) and a violated precondition (AssertionError).
struct Failure : std::runtime_error {
    using std::runtime_error::runtime_error;
};
struct Violation : std::runtime_error {
    using std::runtime_error::runtime_error;
};
void check(int rc, const char *what);
inline void require(bool ok, const char *what) {
    if (!ok) throw Violation(what);
}

// Process-wide settings, written by tango_b200.config (see there for their meaning).
struct Settings {
    std::atomic<int> mode_gemm{TANGO_ROUND_TRUNC}, mode_quantize{TANGO_ROUND_NEAREST};
    std::atomic<uint64_t> seed{0};
    std::atomic<const uint64_t *> step{nullptr};
    std::atomic<bool> compat_dn_scale{false};      // read by the backward passes
    std::atomic<uint64_t> calls{0};      // keys the stochastic-rounding stream of successive calls
    std::atomic<int64_t> launches{0};    // kernels launched so far
};
Settings &settings();
inline uint64_t next_call() { return settings().calls.fetch_add(1) + 1; }
inline void count(int64_t n) { settings().launches.fetch_add(n, std::memory_order_relaxed); }

// The row schedule of one index bundle (tango_b200.graph.SpmmSchedule) and its dense hub region, if any.
struct Schedule {
    Tensor units, heavy_rows, row_order, row_info;
    int64_t n_units = 0, n_heavy = 0, n_long = 0, n_block_rows = 0, n_skip = 0, n_over_few = 0, n_over_one = 0;
    int threshold = 0, unit = 0;
    bool present = false;
    // hub region (tango_b200.graph.HubBlock)
    Tensor dense, dense_units, dense_cols;
    int64_t n_tiles = 0, dense_rows = 0;
    bool has_hub = false;
};

// One direction of a graph: CSC rows are destinations, CSR rows are sources.
struct Direction {
    Tensor indptr, indices, edge_ids;    // edge_ids undefined: slot k holds edge k
    Schedule sched;
    bool has_hub = false;
    Tensor hub_indptr, hub_indices;      // the edges outside the hub region
    Schedule hub_sched;
    int64_t n_rows() const { return indptr.numel() - 1; }
};

struct Graph {
    std::shared_ptr<Direction> csc, csr;
    Tensor src, dst;
    int64_t n_nodes = 0;
    const Direction &dir(bool reverse) const { return reverse ? *csr : *csc; }
    int64_t n_edges() const { return src.numel(); }
};
using GraphPtr = std::shared_ptr<Graph>;

// `t` seen as a row-major [rows, cols] matrix with leading dimension ld (elements); `t` may be a contiguous copy.
struct Matrix {
    Tensor t;
    int64_t rows = 0, cols = 0, ld = 0;
};
Matrix matrix(const Tensor &t);

template <class T = void>
inline T *ptr(const Tensor &t) {
    return t.defined() && t.numel() > 0 ? static_cast<T *>(t.data_ptr()) : nullptr;
}
inline tango_stream_t cuda_stream() { return at::cuda::getCurrentCUDAStream().stream(); }

Tensor alloc_int8(at::IntArrayRef shape, const at::Device &device, int64_t align);
inline Tensor floats(at::IntArrayRef shape, const Tensor &like) { return at::empty(shape, like.options().dtype(at::kFloat)); }
Tensor status_word(const at::Device &device);

// ---- quantisation
struct Quantized {
    Tensor q, scale;
    Tensor colsum;        // when asked for: column sums of the (gated) input
    Tensor product[2];    // when asked for: scale * times[i]
};
// What to quantize, with every option of the fused kernel (tango_quant_job).
struct QuantJob {
    Tensor t;
    int mode;
    uint64_t seed, call;
    int64_t align = 16;
    Tensor scale;         // given scale; undefined: max|t| / 127
    Tensor gate;          // t counts only where gate > 0
    Tensor row_scale;
    bool colsum = false;
    Tensor times[2];
    int times_job = -1;   // product[0] = this scale * the scale of that job
    Tensor clear, clear2; // set to zero by the launch (4-byte elements), for the kernels behind it that accumulate
};
// A job with the rounding mode configured for the stand-alone quantizer, drawing a call number when it is stochastic.
QuantJob quant_job(const Tensor &t, int64_t align = 16);
// One launch for up to four jobs.
std::vector<Quantized> quantize_all(const std::vector<QuantJob> &jobs);
Quantized quantize(const QuantJob &job);
inline Quantized quantize(const Tensor &t, int64_t align = 16) { return quantize(quant_job(t, align)); }
Tensor absmax_scale(const Tensor &t, const Tensor &row_scale = {});

// ---- GEMMs
// Y = act(acc * scales * row_scale[r] + bias).  Here and below a `scale_out`, if given, holds 0 and receives max|.| / 127.
Tensor gemm_nt(const Quantized &x, const Quantized &w, const Tensor &bias, const Tensor &scale_out = {},
               const Tensor &row_scale = {}, bool relu = false);
Tensor gemm_dx(const Quantized &dy, const Quantized &w, const Tensor &row_scale = {}, const Tensor &scale_out = {});
// `scratch`: from dw_scratch, cleared by a launch in front
Tensor dw_scratch(int64_t m, int64_t n, int64_t k, const Tensor &like);
Tensor gemm_dw(const Quantized &dy, const Quantized &x, const Tensor &scratch);

// ---- graph operators
// Scratch of an aggregation of `f` features (undefined if it needs none): cleared by a launch in front (QuantJob.clear), the
// aggregation is then a single launch; without it, it clears and finishes its own.
Tensor spmm_scratch(const Graph &g, bool reverse, int64_t f, const Tensor &like);
Tensor spmm_copy_u(const Graph &g, bool reverse, const Quantized &n, const Tensor &scratch, const Tensor &row_scale = {},
                   const Tensor &bias = {}, bool relu = false, const Tensor &scale_out = {});
// `n` int8 [N, H, D], `e` int8 [E, H]; `scale` multiplies the integer sums
Tensor spmm_u_mul_e(const Graph &g, bool reverse, const Tensor &n, const Tensor &e, const Tensor &scale, const Tensor &scratch,
                    const Tensor &bias = {});
Tensor incidence_sum(const Graph &g, bool reverse, const Quantized &z, const Tensor &scratch);
// op: "dot", "add", "sub", "mul", "div"; U and V 2-D or 3-D; `scale` (optional, holding 0) receives max|out| / 127
Tensor sddmm(const Graph &g, const std::string &op, const Tensor &u, const Tensor &v, const Tensor &su,
             const Tensor &sv, const Tensor &scale, bool reverse);

}  // namespace tango_host
