"""The native operators as a user's program meets them: differentiable entry points against the CPU oracle at the sizes where
the fused quantizer, the GEMMs and the single-launch aggregation can go wrong, and the autograd features around them
(saved-tensor hooks, tracing, forward mode, functorch, module hooks, copies and files of a model)."""
import copy
import io

import numpy as np
import pytest
import torch
import torch.nn.functional as F

from oracle import tango_oracle as O

pytestmark = pytest.mark.gpu


def _np(t):
    return t.detach().cpu().numpy()


def _graph(n=1500, e=20000, seed=3):
    import tango_b200 as T
    from tango_b200.graph import rmat_graph
    return T.graph_preprocess(rmat_graph(n, e, seed, device="cuda"))


def _star(n, hub_edges):
    """Two rows far above the slicing threshold, rows of 0..70 neighbours, and rows with one."""
    import tango_b200 as T
    from tango_b200.graph import Graph
    rng = np.random.default_rng(5)
    deg = np.concatenate([[hub_edges, hub_edges // 2], np.arange(71), np.full(n - 73, 1)])
    dst = np.repeat(np.arange(n), deg)
    src = rng.integers(0, n, dst.size)
    order = rng.permutation(dst.size)
    g = Graph(torch.from_numpy(src[order].astype(np.int32)), torch.from_numpy(dst[order].astype(np.int32)), n).to("cuda")
    return T.graph_preprocess(g)


def _index(g, fmt):
    return [_np(t).astype(np.int64) for t in (g.adj_csr if fmt == "csr" else g.adj_csc)]


@pytest.mark.parametrize("m,k,n", [(1, 1, 1), (1, 5, 1), (1, 100, 32), (7, 100, 1), (1, 33, 20), (2, 1, 2), (3, 5, 2), (127, 16, 33), (129, 130, 41), (1000, 602, 64), (4099, 31, 257),
                                   (700, 5, 40000)])         # too many columns for the partial sums of one launch
@pytest.mark.parametrize("expanded", [False, True])
def test_linear_layer_against_oracle(cuda, m, k, n, expanded):
    """Forward, dX and dW bit for bit; the bias gradient is an fp32 sum, in any order within m * 2^-24 * sum|dY|."""
    import tango_b200 as T
    rng = np.random.default_rng(m + k + n)
    x, dy = rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal((m, n)).astype(np.float32)
    if expanded:
        dy[:] = dy[:1]
    layer = T.QLinear(k, n).cuda()
    xt = torch.from_numpy(x).cuda().requires_grad_()
    y = layer(xt)
    grad = torch.from_numpy(dy).cuda()
    y.backward(grad[:1].expand(m, n) if expanded else grad)
    ry, xq, wq, sx, sw, *_ = O.qgemm_forward(x, _np(layer.weight), _np(layer.bias))
    sdy = O.absmax_scale(dy)
    dyq = O.quantize(dy, sdy)
    np.testing.assert_array_equal(_np(y), ry)
    np.testing.assert_array_equal(_np(xt.grad), O.qgemm_backward_dx(dyq, wq, sdy, sw))
    np.testing.assert_array_equal(_np(layer.weight.grad), O.qgemm_backward_dw(dyq, xq, sdy, sx))
    d64 = dy.astype(np.float64)
    assert (np.abs(_np(layer.bias.grad) - d64.sum(0)) <= m * 2.0 ** -24 * np.abs(d64).sum(0)).all()


@pytest.mark.parametrize("m,k,n", [(1, 100, 32), (7, 100, 1), (1, 5, 1)])
def test_reference_gemm_calls_with_one_row(cuda, m, k, n):
    """The one-row operands of the kernel module's own calls: a padded pitch, although the tensor counts as contiguous."""
    from tango_b200 import kernels as K
    rng = np.random.default_rng(m + n)
    x, w, dy = (rng.standard_normal(s).astype(np.float32) for s in ((m, k), (n, k), (m, n)))
    xt, wt = torch.from_numpy(x).cuda(), torch.from_numpy(w).cuda()
    sx, sw = K.cuda_kernels.get_scale(xt), K.cuda_kernels.get_scale(wt)
    xq, wq = K.alloc_int8(xt.shape, xt.device), K.alloc_int8(wt.shape, wt.device)
    y = K.QGEMM_forward(xt, xq, sx, wt, wq, sw, None, False)
    ry, rxq, rwq, rsx, rsw, *_ = O.qgemm_forward(x, w)
    np.testing.assert_array_equal(_np(y), ry)
    dyq, sdy = K.quantize(torch.from_numpy(dy).cuda())
    dx, dw = K.QGEMM_backward(dyq, xq, wq, sdy, sx, sw)
    rdyq = O.quantize(dy, O.absmax_scale(dy))
    np.testing.assert_array_equal(_np(dx), O.qgemm_backward_dx(rdyq, rwq, sdy.item(), rsw))
    np.testing.assert_array_equal(_np(dw), O.qgemm_backward_dw(rdyq, rxq, sdy.item(), rsx))


@pytest.mark.parametrize("f", [1, 4, 16, 17, 41, 64, 128, 130, 513, 602])
def test_neighbour_sum_of_all_row_classes(cuda, f):
    """Sliced, long, short and one-neighbour rows in one launch; twice, as the second finds the first one's scratch."""
    import tango_b200 as T
    g = _star(2000, 9000)
    x = np.random.default_rng(f).standard_normal((2000, f)).astype(np.float32)
    dz = np.random.default_rng(f + 1).standard_normal((2000, f)).astype(np.float32)
    csc, csr = _index(g, "csc"), _index(g, "csr")
    sx, sz = O.absmax_scale(x), O.absmax_scale(dz)
    for _ in range(2):
        xt = torch.from_numpy(x).cuda().requires_grad_()
        out = T.spmm_copy_u.apply(g, xt)
        out.backward(torch.from_numpy(dz).cuda())
        np.testing.assert_array_equal(_np(out), O.spmm_copy_u(csc[0], csc[1], O.quantize(x, sx), sx))
        np.testing.assert_array_equal(_np(xt.grad), O.spmm_copy_u(csr[0], csr[1], O.quantize(dz, sz), sz))


@pytest.mark.parametrize("h,d", [(1, 16), (1, 41), (2, 8), (2, 24), (4, 4), (4, 32), (3, 5), (8, 16)])
def test_weighted_sum_of_all_row_classes(cuda, h, d):
    """One, two and four heads take their weights as a word, the others byte by byte; edge sums stream contiguous rows."""
    import tango_b200 as T
    g = _star(1500, 5000)
    rng = np.random.default_rng(h * d)
    x = rng.standard_normal((1500, h, d)).astype(np.float32)
    e = rng.standard_normal((g.num_edges(), h, 1)).astype(np.float32)
    out = T.spmm_u_mul_e.apply(g, torch.from_numpy(x).cuda(), torch.from_numpy(e).cuda())
    csc = _index(g, "csc")
    sx, se = O.absmax_scale(x), O.absmax_scale(e)
    ref = O.spmm_u_mul_e(csc[0], csc[1], csc[2], O.quantize(x, sx), O.quantize(e[:, :, 0], se), np.float32(sx * se))
    np.testing.assert_array_equal(_np(out), ref)
    v = torch.zeros(1500, h, 1, device="cuda", requires_grad=True)
    T.sddmm_u_add_v.apply(g, torch.zeros_like(v), v).backward(torch.from_numpy(e).cuda())
    eq = O.quantize(e.reshape(-1, h), se)
    np.testing.assert_array_equal(_np(v.grad)[:, :, 0], O.spmm_incidence(csc[0], csc[2], eq, se))


def _models(g):
    from tango_b200.gnn import GAT, GCN, HGT
    torch.manual_seed(0)
    yield "gcn", GCN(g, 40, 24, 30, 1).cuda()          # a layer that narrows the features and one that does not
    yield "gat", GAT(g, 2, 40, 8, 5, [4, 1]).cuda()
    yield "gat int8", GAT(g, 2, 40, 8, 5, [4, 1], fused="int8").cuda()
    hgt = HGT(40, 32, 4).cuda()
    hgt.graph = g
    yield "hgt", hgt


def _forward(m, x):
    return m(m.graph, x) if type(m).__name__ == "HGT" else m(x)


def _step(m, x):
    m.zero_grad(set_to_none=True)
    out = _forward(m, x)
    out.square().sum().backward()
    return [out.detach()] + [p.grad for p in m.parameters()]


def test_saved_tensor_hooks_and_copies_of_models(cuda):
    g = _graph()
    x = torch.randn(g.num_nodes(), 40, device="cuda")
    for name, m in _models(g):
        want = _step(m, x)
        seen = []
        with torch.autograd.graph.saved_tensors_hooks(lambda t: seen.append(t.dtype) or t.cpu(), lambda t: t.cuda()):
            got = _step(m, x)
        assert all(torch.equal(a, b) for a, b in zip(want, got)), name
        # the fused layers' int8 operands are offloaded too; the single operators that hgt is made of keep theirs on the node,
        # as the reference's Functions do, and allow a second backward pass
        assert name == "hgt" or torch.int8 in seen, name
        for other in (copy.deepcopy(m), torch.load(io.BytesIO(_saved(m)), weights_only=False)):
            assert all(torch.equal(a, b) for a, b in zip(want, _step(other, x))), name
        out = _forward(m, x).sum()
        out.backward(retain_graph=True)
        out.backward()
        if name != "hgt":
            with pytest.raises(RuntimeError, match="backward through the graph a second time"):
                out.backward()


def _saved(m):
    b = io.BytesIO()
    torch.save(m, b)
    return b.getvalue()


def test_tracing_and_transforms_see_the_operators(cuda):
    import tango_b200 as T
    g = _graph(300, 3000)
    layer = T.QLinear(40, 8).cuda()
    a, b = torch.randn(2, 300, 40, device="cuda")
    ops = {"linear": layer, "spmm": lambda t: T.spmm_copy_u.apply(g, t),
           "dot": lambda t: T.sddmm_u_dot_v.apply(g, t.view(300, 4, 10), t.view(300, 4, 10))}
    for name, op in ops.items():
        with torch.no_grad():
            traced = torch.jit.trace(op, a, check_trace=False)
            assert torch.equal(traced(b), op(b)), name
        with torch.autograd.forward_ad.dual_level(), pytest.raises(RuntimeError):
            op(torch.autograd.forward_ad.make_dual(a, b))
        with pytest.raises(RuntimeError):
            torch.func.grad(lambda t: op(t).sum())(a)
        with pytest.raises(RuntimeError):
            torch.vmap(op)(torch.stack([a, b]))
        with torch.autograd.forward_ad.dual_level():               # no tangent: an ordinary pass
            x1, x2 = a.clone().requires_grad_(), a.clone().requires_grad_()
            y1 = op(x1)
        y2 = op(x2)
        assert torch.equal(y1, y2)
        dy = torch.randn_like(y1)
        y1.backward(dy)
        y2.backward(dy)
        assert torch.equal(x1.grad, x2.grad), name


@pytest.mark.parametrize("share", [False, True])
def test_module_hooks_of_projections_that_share_their_input(cuda, share):
    from tango_b200 import config
    from tango_b200.gnn import HGT
    g = _graph(400, 4000)
    m = HGT(40, 32, 4).cuda()
    x = torch.randn(400, 40, device="cuda")
    config.share_quantized_inputs(share)
    try:
        plain = m(g, x)
        seen = []
        m.k_linear.register_forward_pre_hook(lambda mod, args: seen.append(len(args)))
        m.q_linear.register_forward_hook(lambda mod, args, out: out * 1.0)
        assert torch.equal(m(g, x), plain) and seen == [1]
        m.v_linear.register_forward_pre_hook(lambda mod, args: (args[0] * 2,))
        assert not torch.equal(m(g, x), plain)
    finally:
        config.share_quantized_inputs(False)


def test_linear_layer_with_a_strided_bias(cuda):
    import tango_b200 as T
    x, w = torch.randn(33, 24, device="cuda"), torch.randn(16, 24, device="cuda")
    b = torch.randn(32, device="cuda")[::2].requires_grad_()
    assert torch.equal(T.Qlinear_func.apply(x, w, b), T.Qlinear_func.apply(x, w, b.detach().contiguous()))


def test_widths_that_do_not_match_are_refused(cuda):
    from tango_b200.gnn import QGraphConv
    g = _graph(300, 3000)
    for feats, hidden in ((40, 8), (8, 40)):
        with pytest.raises(AssertionError):
            QGraphConv(feats, hidden).cuda()(g, torch.randn(300, feats - 1, device="cuda"))
    # what broadcasts or promotes in a layer that aggregates first is taken by the operators, the rest refused by them
    m = QGraphConv(8, 40).cuda()
    x = torch.randn(300, 8, device="cuda").half()
    assert torch.equal(m(g, x), m(g, x.float()))
    assert torch.equal(m(g, x[:1].float()), m(g, x[:1].float().repeat(300, 1)))
    for rows in (299, 301):
        with pytest.raises(RuntimeError):
            m(g, torch.randn(rows, 8, device="cuda"))
    y = m(g, x.float())
    m.bias = torch.nn.Parameter(torch.full((1,), 2.0, device="cuda"))
    assert torch.equal(m(g, x.float()), y + 2)
    m.bias = torch.nn.Parameter(torch.zeros(39, device="cuda"))
    with pytest.raises(RuntimeError):
        m(g, x.float())


@pytest.mark.parametrize("heads", [1, 2, 3, 4, 5, 8])
@pytest.mark.parametrize("order", ["rows", "shuffled"])
def test_edge_softmax_of_row_lengths_around_the_trips(cuda, heads, order):
    """Rows of 0 to 3000 edges, with the edge numbers along the rows and not.  __expf of an argument of at most 40 is off by
    40 * 2^-23 + 2^-21 relative, the sum of up to 3000 positive terms by less than that again: 2e-5 in all."""
    import tango_b200 as T
    from tango_b200.gnn import edge_softmax
    from tango_b200.graph import Graph
    deg = np.array([0, 1, 2, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 257, 1023, 1024, 1025, 2049, 3000])
    dst = np.repeat(np.arange(deg.size), deg)
    rng = np.random.default_rng(heads)
    if order == "shuffled":
        dst = rng.permutation(dst)
    src = rng.integers(0, deg.size, dst.size)
    g = T.graph_preprocess(Graph(torch.from_numpy(src.astype(np.int32)), torch.from_numpy(dst.astype(np.int32)), deg.size).to("cuda"))
    z = rng.uniform(-20, 20, (dst.size, heads, 1)).astype(np.float32)
    z[rng.random(z.shape) < 0.02] = -np.inf
    z[dst == 1] = 0.5
    da = rng.standard_normal(z.shape).astype(np.float32)
    zt = torch.from_numpy(z).cuda().requires_grad_()
    a, sa = edge_softmax(g, zt, 0.5, True)
    a.backward(torch.from_numpy(da).cuda())
    want, grad, size = (np.zeros(z.shape) for _ in range(3))
    for v in range(deg.size):
        e = dst == v
        if e.any():
            w = np.exp(z[e] * 0.5 - (z[e] * 0.5).max(0))
            want[e] = w = w / w.sum(0)
            dot = (w * da[e]).sum(0)
            grad[e] = w * (da[e] - dot) * 0.5
            size[e] = w * (np.abs(da[e]) + (w * np.abs(da[e])).sum(0)) * 0.5
    tiny = 1e-37                                        # (weights below the normal range are flushed)
    assert (np.abs(_np(a) - want) <= 2e-5 * want + tiny).all()
    assert (np.abs(_np(zt.grad) - grad) <= 4e-5 * size + tiny).all()
    assert sa.item() == np.float32(_np(a).max()) / np.float32(127)


@pytest.mark.parametrize("n,h,d", [(1, 1, 1), (5, 3, 5), (130, 4, 64), (1000, 8, 8), (257, 1, 41), (63, 2, 600), (3001, 4, 63)])
@pytest.mark.parametrize("offset", [0, 1])
def test_attention_projection_gradients(cuda, n, h, d, offset):
    """Sums of k terms within k * 2^-24 of the sum of their magnitudes, any order; offset: only 4-byte aligned features."""
    from tango_b200 import _lib
    rng = np.random.default_rng(n + d)

    def dev(*shape):
        t = torch.empty(offset + int(np.prod(shape)), device="cuda")[offset:].view(shape)
        return t.copy_(torch.from_numpy(rng.standard_normal(shape).astype(np.float32)))

    x, al, ar, dl, dr, dx0 = dev(n, h, d), dev(h, d), dev(h, d), dev(n, h), dev(n, h), dev(n, h, d)
    dx, dal, dar = dx0.clone(), dev(h, d), dev(h, d)
    scratch = torch.empty(_lib.lib.tango_gat_project_bwd_scratch_bytes(n, h, d) // 4, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    p = [t.data_ptr() for t in (x, al, ar, dl, dr, dx, dal, dar, scratch)]
    _lib.check(_lib.lib.tango_gat_project_bwd(p[0], n, h, d, *p[1:], scratch.numel() * 4, stream), "project_bwd")
    chain = (dx0 + dr[:, :, None] * ar) + dl[:, :, None] * al            # the gradients meet as in the operator chain
    assert torch.equal(dx, chain)
    x, dl, dr = (_np(t).astype(np.float64) for t in (x, dl, dr))
    u = 2.0 ** -24

    def close(got, terms, axis, k):
        assert (np.abs(_np(got) - terms.sum(axis)) <= (k + 1) * u * np.abs(terms).sum(axis)).all()

    close(dal, dl[:, :, None] * x, 0, n)
    close(dar, dr[:, :, None] * x, 0, n)


@pytest.mark.parametrize("residual,bias", [(False, True), (True, True), (False, False)])
@pytest.mark.parametrize("heads,dim", [(1, 7), (2, 1), (4, 16), (8, 8), (3, 5)])
def test_gat_layer_as_one_node_against_the_chain(cuda, residual, bias, heads, dim):
    """int8 weights, fp32 weights and the operator-by-operator chain give the same layer bit for bit: every value that is
    quantized comes out of the same sums.  The gradients of attn_l, attn_r and the bias are sums over all nodes that end the
    chain; the operators add them in another order.  (With one feature per head the gradient of a weight is one product, which
    the chain dequantizes factor by factor and the int8 form as a dot product.)"""
    from tango_b200.gnn import QGATConv
    g = _graph(600, 6000)
    x0 = torch.randn(600, 24, device="cuda")
    res = []
    for fused in (True, "int8", False):
        torch.manual_seed(1)
        m = QGATConv(24, dim, heads, residual=residual, bias=bias, activation=F.elu, fused=fused).cuda()
        if bias:
            torch.nn.init.normal_(m.bias)
        x = x0.clone().requires_grad_()
        out = m(g, x)
        torch.manual_seed(2)
        out.backward(torch.randn_like(out))
        res.append({"out": out, "x": x.grad, **{k: p.grad for k, p in m.named_parameters()}})
        for p in m.parameters():
            p.requires_grad_(False)
        assert not m(g, x0).requires_grad and torch.equal(m(g, x0), out)
    for k, c in res[2].items():
        if dim > 1:
            assert torch.equal(res[0][k], res[1][k]), k
        else:
            assert (res[0][k] - res[1][k]).norm() <= 1e-2 * c.norm(), k
        if k in ("attn_l", "attn_r", "bias"):
            assert (res[0][k] - c).norm() <= 1e-2 * c.norm(), k
        else:
            assert torch.equal(res[0][k], c), k


@pytest.mark.parametrize("heads", [1, 2, 4, 5, 8])
def test_edge_softmax_of_a_row_does_not_depend_on_the_rows_beside_it(cuda, heads):
    """Four short rows share a warp, and what is short depends on the longest of them: a row of k edges gives the same bits
    among its equals, beside long rows and in a graph that is a hundred times larger (its weights are quantized next, where
    one ulp can move every code)."""
    import tango_b200 as T
    from tango_b200.gnn import edge_softmax
    from tango_b200.graph import Graph
    rng = np.random.default_rng(heads)
    lengths = [1, 2, 7, 8, 9, 15, 16, 17, 24, 31, 32, 33, 40, 63, 64, 65, 130, 300, 700, 1024]

    def weights(deg, z, da):
        dst = np.repeat(np.arange(deg.size), deg).astype(np.int32)
        g = T.graph_preprocess(Graph(torch.from_numpy(np.zeros_like(dst)), torch.from_numpy(dst), deg.size).to("cuda"))
        zt = torch.from_numpy(z).cuda().requires_grad_()
        a = edge_softmax(g, zt, 0.5)
        a.backward(torch.from_numpy(da).cuda())
        return _np(a), _np(zt.grad)

    large = rng.integers(1, 1025, 8000)
    zl, dl = rng.standard_normal((2, large.sum(), heads, 1)).astype(np.float32)
    for k in lengths:
        z, da = rng.standard_normal((2, 4 * k, heads, 1)).astype(np.float32)
        equals = weights(np.full(4, k), z, da)
        zb, db = rng.standard_normal((2, 3 * 1024, heads, 1)).astype(np.float32)
        beside = weights(np.array([k, 1024, 1024, 1024]), np.concatenate([z[:k], zb]), np.concatenate([da[:k], db]))
        among = weights(np.concatenate([[k], large]), np.concatenate([z[:k], zl]), np.concatenate([da[:k], dl]))
        for i in range(2):
            np.testing.assert_array_equal(equals[i][:k], beside[i][:k], err_msg=str(k))
            np.testing.assert_array_equal(equals[i][:k], among[i][:k], err_msg=str(k))


def test_scale_switch_of_the_weighted_sum_is_read_in_the_backward_pass(cuda, monkeypatch):
    """Flipped between forward and backward, dN is the integer sum times the forward scales; also inside a GAT layer."""
    import tango_b200 as T
    from tango_b200.gnn import QGATConv
    g = _graph(200, 2000)
    n0, e = torch.randn(200, 2, 8, device="cuda"), torch.rand(g.num_edges(), 2, 1, device="cuda")
    dz = torch.randn(200, 2, 8, device="cuda") * 3
    layer = QGATConv(24, 8, 2).cuda()
    x0 = torch.randn(200, 24, device="cuda")

    def grads(forward, backward):
        monkeypatch.setattr(T.spmm_u_mul_e, "compat_dn_scale", forward)
        n, x = n0.clone().requires_grad_(), x0.clone().requires_grad_()
        out, y = T.spmm_u_mul_e.apply(g, n, e), layer(g, x)
        monkeypatch.setattr(T.spmm_u_mul_e, "compat_dn_scale", backward)
        out.backward(dz)
        y.backward(dz)
        return n.grad, x.grad

    off, on = grads(False, False), grads(True, True)
    assert not torch.equal(off[0], on[0]) and not torch.equal(off[1], on[1])
    for forward in (False, True):
        assert all(torch.equal(a, b) for a, b in zip(off, grads(forward, False)))
        assert all(torch.equal(a, b) for a, b in zip(on, grads(forward, True)))
    ratio = T.kernels.cuda_kernels.get_scale(n0) / T.kernels.cuda_kernels.get_scale(dz)
    torch.testing.assert_close(on[0], off[0] * ratio, rtol=1e-6, atol=0)
    monkeypatch.undo()
    assert T.spmm_u_mul_e.compat_dn_scale is False


def test_wide_layer_behind_relu_sums_its_columns_apart(cuda):
    """40,000 outputs: gate, column sums and quantisation of the gradient are separate kernels; same layer as the operators."""
    from tango_b200.gnn import QGraphConv
    g = _graph(700, 4000)
    x0 = torch.randn(700, 8, device="cuda")
    res = []
    for fused in (True, False):
        torch.manual_seed(1)
        m = QGraphConv(8, 40000, activation=F.relu, fused=fused).cuda()
        torch.nn.init.normal_(m.bias)
        x = x0.clone().requires_grad_()
        out = m(g, x)
        torch.manual_seed(2)
        dy = torch.randn_like(out)
        out.backward(dy)
        res.append((out, x.grad, m.weight.grad))
        d64 = torch.where(out > 0, dy, 0).double()
        assert ((m.bias.grad - d64.sum(0)).abs() <= 700 * 2.0 ** -24 * d64.abs().sum(0)).all()
    assert all(torch.equal(a, b) for a, b in zip(*res))


@pytest.mark.parametrize("rows,cols", [(1, 5), (300, 7), (2001, 130), (70000, 64)])
@pytest.mark.parametrize("mode", [0, 1, 2])
def test_quantizer_in_two_launches_equals_the_cooperative_one(cuda, rows, cols, mode):
    """What a context with too few SMs for the grid barrier runs: gate, row factor, column sums, products and clears."""
    from tango_b200 import _lib
    ld = (cols + 15) // 16 * 16
    x, gate, y = torch.randn(3, rows, cols, device="cuda")
    factor = torch.rand(rows, device="cuda") + 0.5
    res = []
    for entry in (_lib.lib.tango_quantize_fused, _lib.lib.tango_quantize_two_launches):
        q = torch.full((2, rows, ld), 99, dtype=torch.int8, device="cuda")
        scales, product, colsum = torch.zeros(2, device="cuda"), torch.zeros(2, device="cuda"), torch.zeros(cols, device="cuda")
        words = torch.full((1000,), 7, dtype=torch.int32, device="cuda")
        jobs = (_lib.QuantJob * 2)(
            _lib.QuantJob(x=x.data_ptr(), rows=rows, cols=cols, ldx=cols, gate=gate.data_ptr(), ldgate=cols,
                          row_scale=factor.data_ptr(), scale=scales[0:].data_ptr(), times_job=-1, colsum=colsum.data_ptr(),
                          clear=(words.data_ptr(), None), clear_words=(999, 0), q=q[0].data_ptr(), ldq=ld, mode=mode, seed=3, call=1),
            _lib.QuantJob(x=y.data_ptr(), rows=rows, cols=cols, ldx=cols, scale=scales[1:].data_ptr(), times_job=0,
                          times=(None, factor.data_ptr()), product=(product[0:].data_ptr(), product[1:].data_ptr()),
                          q=q[1].data_ptr(), ldq=ld, mode=mode, seed=3, call=2))
        n = _lib.lib.tango_quantize_fused_scratch_bytes(jobs, 2)
        scratch = torch.empty(n, dtype=torch.uint8, device="cuda")
        _lib.check(entry(jobs, 2, None, scratch.data_ptr(), n, torch.cuda.current_stream().cuda_stream), "quantize")
        res.append((q, scales, product, colsum, words))
    assert all(torch.equal(a, b) for a, b in zip(*res))
    q, scales, product, colsum, words = (_np(t) for t in res[1])
    masked = np.where(_np(gate) > 0, _np(x), np.float32(0))
    assert scales[0] == O.absmax_scale(masked * _np(factor)[:, None]) and scales[1] == O.absmax_scale(_np(y))
    assert product[0] == scales[1] * scales[0] and product[1] == scales[1] * _np(factor)[0]
    assert (words == np.concatenate([np.zeros(999), [7]])).all() and (q[:, :, cols:] == 0).all()
    assert (np.abs(colsum - masked.astype(np.float64).sum(0)) <= rows * 2.0 ** -24 * np.abs(masked).astype(np.float64).sum(0)).all()
    if mode == 1:
        np.testing.assert_array_equal(q[1, :, :cols], O.quantize(_np(y), scales[1]))


def test_vector_beyond_the_indices_of_the_fused_quantizer(cuda):
    """2^32 + 8 elements (17 GB): scale and codes as the fused kernel gives them piece by piece."""
    from tango_b200 import kernels as K
    n, step = 2 ** 32 + 8, 2 ** 28
    x = torch.empty(n, device="cuda")
    for i in range(0, n, step):
        x[i:i + step].normal_()
    x[-1] = -40.0
    q, s = K.quantize(x)
    assert s.item() == np.float32(40) / np.float32(127)
    for i in range(0, n, step):
        assert torch.equal(q[i:i + step], K.quantize(x[i:i + step], s)[0])



@pytest.mark.parametrize("out", [40, 41])
def test_infinities_and_nan_go_through_a_convolution_as_through_the_operators(cuda, out):
    """An infinite feature gives infinite scales and NaN sums; ReLU keeps a NaN and lets its gradient pass."""
    from tango_b200.gnn import QGraphConv
    g = _graph(200, 1000)
    x0 = torch.randn(200, 8, device="cuda")
    x0[3, 2] = float("inf")
    res = []
    for fused in (True, False):
        torch.manual_seed(1)
        m = QGraphConv(8, out, activation=F.relu, fused=fused).cuda()
        x = x0.clone().requires_grad_()
        y = m(g, x)
        torch.manual_seed(2)
        y.backward(torch.randn_like(y))
        res.append((y, x.grad, m.weight.grad, m.bias.grad))
    assert res[0][0].isnan().any()
    for a, b in zip(*res):
        torch.testing.assert_close(a, b, rtol=0, atol=0 if a is not res[0][3] else 1e-4, equal_nan=True)


@pytest.mark.parametrize("m,n,k", [(1, 1, 16), (129, 41, 100), (700, 256, 602)])
@pytest.mark.parametrize("relu", [0, 1])
def test_gemm_epilogue_options(cuda, m, n, k, relu):
    """Row factor, bias, ReLU and the output maximum with its own factor, operation for operation."""
    import tango_b200 as T
    from tango_b200 import _lib
    rng = np.random.default_rng(m)
    x, w = rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal((n, k)).astype(np.float32)
    row, bias, factor = (rng.standard_normal(s).astype(np.float32) for s in (m, n, m))
    (xq, sx), (wq, sw) = T.kernels.quantize(torch.from_numpy(x).cuda()), T.kernels.quantize(torch.from_numpy(w).cuda())
    y, sy, st = torch.empty(m, n, device="cuda"), torch.zeros(1, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    rt, bt, ft = (torch.from_numpy(t).cuda() for t in (row, bias, factor))
    p = [t.data_ptr() for t in (xq, wq, sx, sw, rt, bt, y, sy, ft, st)]
    ld = (k + 15) // 16 * 16
    _lib.check(_lib.lib.tango_qgemm_layer(p[0], ld, p[1], ld, m, n, k, p[2], p[3], p[4], p[5], relu, p[6], n, p[7], p[8], p[9],
                                          torch.cuda.current_stream().cuda_stream), "qgemm_layer")
    acc = _np(xq).astype(np.int64) @ _np(wq).astype(np.int64).T
    want = acc.astype(np.float32) * (_np(sx) * _np(sw)) * row[:, None] + bias
    want = np.maximum(want, np.float32(0)) if relu else want
    np.testing.assert_array_equal(_np(y), want)
    assert sy.item() == np.float32(np.abs(want * factor[:, None]).max()) / np.float32(127) and st.item() == 0
