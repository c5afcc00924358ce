// The differentiable operators and fused layers of the host layer (torch_autograd.cpp).
#pragma once
#include "torch_ops.h"

namespace tango_host {

// QLinear (cuda/QLinear.py:28-72 of the reference).  With `xq` / `sx` given the input's int8 copy is re-used instead of
// quantizing X again.  Returns (Y, scale of Y or undefined, Xq, sX).
std::tuple<Tensor, Tensor, Tensor, Tensor> qlinear(const Tensor &x, const Tensor &w, const Tensor &b, bool want_scale,
                                                   const Tensor &xq, const Tensor &sx);

// Layers that read the same input: X and up to three weights quantized in one launch, one GEMM each.
std::vector<Tensor> qlinear_group(const Tensor &x, const std::vector<Tensor> &w, const std::vector<Tensor> &b);

Tensor spmm_copy_u_fn(const GraphPtr &g, const Tensor &n, const Tensor &scale);
Tensor spmm_u_mul_e_fn(const GraphPtr &g, const Tensor &n, const Tensor &e, const Tensor &scale_e);
Tensor sddmm_u_add_v_fn(const GraphPtr &g, const Tensor &u, const Tensor &v, const Tensor &su, const Tensor &sv);
Tensor sddmm_u_dot_v_fn(const GraphPtr &g, const Tensor &u, const Tensor &v);

// One graph convolution, norm='both', the linear layer or the aggregation first:
// act((A . Q(Q(X * out_norm) W^T)) * in_norm + b)  or  act((Q(A . Q(X * out_norm)) W^T) * in_norm + b).
Tensor gcn_conv_fn(const GraphPtr &g, const Tensor &x, const Tensor &w, const Tensor &b, const Tensor &out_norm,
                   const Tensor &in_norm, bool relu, bool linear_first);

// softmax(z * factor) over the incoming edges of every destination; (weights, max|weight| / 127).
std::tuple<Tensor, Tensor> edge_softmax_fn(const GraphPtr &g, const Tensor &z, double factor);
// edge_softmax(leaky_relu(Q(el)[src] + Q(er)[dst])); (weights [E, H, 1], max|weight| / 127).
std::tuple<Tensor, Tensor> gat_attention_fn(const GraphPtr &g, const Tensor &el, const Tensor &er, double slope);
// A whole GAT layer behind its linear projection: el = <ft, al>, er = <ft, ar> per head, the weights above, and their
// aggregation of Q(ft) plus bias.  int8_weights: without an fp32 copy of the weights.
Tensor gat_layer_fn(const GraphPtr &g, const Tensor &ft, const Tensor &al, const Tensor &ar, const Tensor &bias, double slope,
                    bool int8_weights);

}  // namespace tango_host
