"""Decode-sized products fetch their weights ahead of the kernel before them, except behind one that wrote weights: the kinds of edges
in a captured graph, which is where the launches' order can be read, and training steps whose weights change from step to step."""

import ctypes

import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops(lib_built):
    from t81lib_b200 import _capi, ops
    assert _capi.device_available(), _capi.last_error()
    return ops


class _EdgeData(ctypes.Structure):
    _fields_ = [("from_port", ctypes.c_ubyte), ("to_port", ctypes.c_ubyte), ("type", ctypes.c_ubyte), ("reserved", ctypes.c_ubyte * 5)]


def _edge_kinds(graph):
    """Of a graph that is one chain: True for each edge, first to last, on which the later kernel starts early."""
    cuda, handle, n = ctypes.CDLL("libcuda.so.1"), ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_size_t(0)
    assert cuda.cuGraphGetEdges_v2(handle, None, None, None, ctypes.byref(n)) == 0
    a, b, kinds = (ctypes.c_void_p * n.value)(), (ctypes.c_void_p * n.value)(), (_EdgeData * n.value)()
    assert cuda.cuGraphGetEdges_v2(handle, a, b, kinds, ctypes.byref(n)) == 0
    following = {a[i]: (b[i], kinds[i].type == 1) for i in range(n.value)}
    assert len(following) == n.value
    node, early = (set(a) - set(b)).pop(), []
    while node in following:
        node, kind = following[node]
        early.append(kind)
    return early


def _captured(work):
    work()  # plans and kernel attributes outside the capture
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        work()
    return _edge_kinds(graph)


# write the weights, multiply twice: the first product waits for the writer, the second overlaps the first
@pytest.mark.parametrize("writer", ["pack_t2", "qat_quantize_t2", "quantize_pack", "tq_to_packed", "qat_quantize_pack", "of the caller's"])
@pytest.mark.parametrize("tokens", [1, 16])
def test_a_product_behind_new_weights_waits_for_them(ops, writer, tokens):
    from t81lib_b200 import _capi
    rows, K = 256, 768
    w, x = torch.randn(rows, K, device="cuda"), torch.randn(tokens, K, device="cuda", dtype=torch.bfloat16)
    packed, scale = ops.quantize_pack(w, 0.45, "absmean")
    t2, blocks = ops.pack_t2(packed, rows, K), ops.packed_to_tq(packed, rows, K, "TQ2_0", scale)
    limbs = lambda p: ops.gemm_trit(p, x, M=rows, K=K, layout="nk", row_scale=scale)
    codes = lambda t: ops.linear_t2(t, rows, x, K, scale, None)

    def work():
        if writer == "pack_t2":
            product, weight = codes, ops.pack_t2(packed, rows, K)
        elif writer == "qat_quantize_t2":
            product, weight = codes, ops.qat_quantize_t2(w, 0.45, scale[:1], transposed=False)[0]
        elif writer == "quantize_pack":
            product, weight = limbs, ops.quantize_pack(w, 0.45, "absmean")[0]
        elif writer == "tq_to_packed":
            product, weight = limbs, ops.tq_to_packed(blocks, rows, K, "TQ2_0")[0]
        elif writer == "qat_quantize_pack":
            product, weight = limbs, ops.qat_quantize_pack(w, 0.45, scale[:1])[0]
        else:
            product, weight = codes, t2.bitwise_or(0)
            _capi.lib.t81b200_weights_written(torch.cuda.current_stream().cuda_stream)
        product(weight)
        product(weight)
    early = _captured(work)
    assert early[-2:] == [False, True]
    assert _capi.kernel_status(reset=True) == 0


# scales and biases may come from the kernel directly ahead, with copies and threads fetching them (rows of no multiple of a tile)
@pytest.mark.parametrize("rows", [256, 250, 2000])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_scales_and_biases_of_the_kernel_ahead(ops, rows, dtype):
    K = 576
    gen = torch.Generator(device="cuda").manual_seed(rows)
    trits = torch.randint(-1, 2, (rows, K), generator=gen, device="cuda").float()
    t2 = ops.pack_t2(ops.quantize_pack(trits, 0.5, "fixed")[0], rows, K)
    x = torch.randint(-3, 4, (5, K), generator=gen, device="cuda").to(dtype)
    exact = x.double() @ trits.double().t()
    scale, bias = torch.zeros(rows, device="cuda"), torch.zeros(rows, device="cuda")
    for step in range(1, 20):
        scale.fill_(step / 8)
        bias.fill_(-step)
        got = ops.linear_t2(t2, rows, x, K, scale, bias, torch.float32)
        assert torch.equal(got, (exact * (step / 8) - step).float())  # eighths: exact


@pytest.mark.parametrize("tokens", [1, 3, 16])
def test_decode_sized_training_steps_follow_their_weights(ops, tokens):
    from t81lib_b200.nn import Linear
    rows, K = 130, 500
    layer = Linear(K, rows, bias=False, device="cuda").train()
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    x = torch.randint(-3, 4, (tokens, K), generator=gen, device="cuda").to(torch.bfloat16).float()
    for _ in range(12):
        with torch.no_grad():
            layer.weight.copy_(torch.randn(rows, K, generator=gen, device="cuda"))
        y = layer(x)
        scale = float(layer.training_scale)
        trits = oracle.qat_quantize(layer.weight.detach().cpu().numpy(), np.float32(scale), 0.45)
        want = (x.cpu().numpy().astype(np.float64) @ trits.T) * scale
        # whole numbers below 2^24, times the scale: one rounding
        np.testing.assert_allclose(y.detach().cpu().numpy(), want, rtol=2.0 ** -23, atol=0)


# Products of one input captured one after the other read it early; whatever lies between them, and inputs, scales and biases that
# come from the product ahead, take the order that the stream gives.
@pytest.mark.parametrize("dtype,tokens", [(torch.bfloat16, 8), (torch.float16, 13), (torch.float32, 3)])
def test_captured_products_of_one_input(ops, dtype, tokens):
    from t81lib_b200 import _capi
    K, rows = 1024, 1024
    gen = torch.Generator(device="cuda").manual_seed(tokens)

    def weight():
        trits = torch.randint(-1, 2, (rows, K), generator=gen, device="cuda").float()
        trits *= torch.rand(rows, K, generator=gen, device="cuda") < 0.02  # results stay small whole numbers: exact in every type
        return trits, ops.pack_t2(ops.quantize_pack(trits, 0.5, "fixed")[0], rows, K)
    weights = [weight() for _ in range(10)]
    x = torch.empty(tokens, K, device="cuda", dtype=dtype)
    vector, shared = torch.zeros(rows, device="cuda"), torch.zeros(tokens, K, device="cuda", dtype=dtype)

    def chain(product):
        one = [product(i, x) for i in range(3)]               # q, k, v
        shared.copy_(one[0].clamp(-2, 2))                     # another kernel between two products
        two = [product(3, shared), product(4, shared)]
        again = product(5, two[1].clamp(-2, 2))               # and products of the one ahead
        follows = [product(6, again), product(7, again)]
        follows.append(product(8, x))
        vector.copy_(follows[2][0].float())
        return one + two + [again] + follows + [product(9, x, vector)]

    def device(i, a, bias=None):
        return ops.linear_t2(weights[i][1], rows, a, K, None, bias)

    def expected(i, a, bias=None):
        y = a.double() @ weights[i][0].double().t()
        return (y if bias is None else y + bias.double()).to(dtype)
    x.zero_()
    chain(device)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = chain(device)
    for _ in range(20):
        x.copy_(torch.randint(-1, 2, (tokens, K), generator=gen, device="cuda"))
        graph.replay()
        got_now = [g.clone() for g in got]
        for g, want in zip(got_now, chain(expected)):
            assert torch.equal(g, want)
    assert _capi.kernel_status(reset=True) == 0


# The result of one product lies in the input of the next, or the next one's result over its input: no early reading, no early writing.
@pytest.mark.parametrize("overlap", ["reads what is written", "writes what is read", "apart"])
def test_captured_products_whose_buffers_touch(ops, overlap):
    from t81lib_b200 import _capi
    K = rows = 512
    gen = torch.Generator(device="cuda").manual_seed(3)
    trits = torch.randint(-1, 2, (rows, K), generator=gen, device="cuda").float() * (torch.rand(rows, K, generator=gen, device="cuda") < 0.01)
    t2 = ops.pack_t2(ops.quantize_pack(trits, 0.5, "fixed")[0], rows, K)
    a, b, c = (torch.zeros(4, K, device="cuda", dtype=torch.bfloat16) for _ in range(3))
    into = lambda x, y: _capi.check(_capi.lib.t81b200_linear_t2(
        t2.data_ptr(), None, None, y.data_ptr(), rows, x.data_ptr(), _capi.BF16, K, _capi.BF16, rows, 4, K, 1.0, 0.0, 2, None, 0,
        torch.cuda.current_stream().cuda_stream))
    steps = {"reads what is written": [(a, b), (b, c), (a, b), (b, a)], "writes what is read": [(a, b), (c, a), (a, c), (b, a)],
             "apart": [(a, b), (a, c), (a, b), (a, c)]}[overlap]
    into(a, b)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for x, y in steps:
            into(x, y)
    for _ in range(20):
        for t in (a, b, c):
            t.copy_(torch.randint(-1, 2, (4, K), generator=gen, device="cuda"))
        buffers = {id(t): t.double() for t in (a, b, c)}
        graph.replay()
        for x, y in steps:
            buffers[id(y)] = (buffers[id(x)] @ trits.double().t()).to(torch.bfloat16).double()
        for t in (a, b, c):
            assert torch.equal(t.double(), buffers[id(t)])
