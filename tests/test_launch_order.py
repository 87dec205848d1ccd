"""Decode-sized products fetch their weights ahead of the kernel before them, except behind one that wrote weights: the kinds of edges
in a captured graph, which is where the launches' order can be read, and training steps whose weights change from step to step."""

import contextlib
import ctypes

import numpy as np
import pytest
import torch

import oracle
from _graph_nodes import capture, kernels

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


def _products(graph):
    """The parameter blocks of a graph's streaming products, in the order of their capture."""
    return [parameter(3) for name, parameter in kernels(graph) if "gemv_trit_lut_kernel" in name]  # three tensor maps, then the block


@pytest.fixture(scope="module")
def forms(ops):
    """What a graph's products do, in order: "waits" before anything, "reads" early and waits before it stores, or "runs" on the caller's
    word.  Where a parameter block says so is found from one product captured twice, whose second launch differs in that alone."""
    trits = torch.ones(32, 192, device="cuda")
    t2, x, y = ops.pack_t2(ops.quantize_pack(trits, 0.5, "fixed")[0], 32, 192), torch.ones(1, 192, device="cuda", dtype=torch.bfloat16), []
    out = torch.empty(1, 32, device="cuda", dtype=torch.bfloat16)
    a, b = _products(capture(lambda: [ops.gemm_trit_t2([t2], [32], x, K=192, outs=[out]) for _ in range(2)]))
    (at,) = np.nonzero(a != b)[0]
    assert (a[at], b[at]) == (0, 2)
    return lambda graph: [("waits", "runs", "reads")[block[at]] for block in _products(graph)]


class _Weights:
    """Sparse weights, in either layout: products of small whole numbers are small whole numbers, exact in every type and order."""

    def __init__(self, ops, layout, n=4, size=512):
        gen = torch.Generator(device="cuda").manual_seed(size)
        self.ops, self.layout, self.size = ops, layout, size
        self.trits = [torch.randint(-1, 2, (size, size), generator=gen, device="cuda").float() * (torch.rand(size, size, generator=gen, device="cuda") < 0.01)
                      for _ in range(n)]
        packed = [ops.quantize_pack(t, 0.5, "fixed")[0] for t in self.trits]
        self.packed = packed if layout == "limbs" else [ops.pack_t2(p, size, size) for p in packed]

    def __call__(self, i, x, out, scale=None, bias=None, beta=0.0):
        if self.layout == "limbs":
            return self.ops.gemm_trit(self.packed[i], x, M=self.size, K=self.size, layout="nk", row_scale=scale, bias=bias, C=out, beta=beta)
        return self.ops.gemm_trit_t2([self.packed[i]], [self.size], x, K=self.size, row_scales=[scale], biases=[bias], outs=[out], beta=beta)[0]

    def want(self, i, x, out=None, scale=None, bias=None, beta=0.0):
        y = (x.double() @ self.trits[i].double().t()) * (1.0 if scale is None else scale.double()) + (0.0 if bias is None else bias.double())
        return y if beta == 0.0 else y + beta * out.double()


def _replayed(graph, tensors, check, seed=0):
    """Replays on new whole numbers in every tensor; `check` gets copies of what they held before."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    for _ in range(20):
        for t in tensors:
            t.copy_(torch.randint(-1, 2, t.shape, generator=gen, device="cuda"))
        before = [t.clone() for t in tensors]
        graph.replay()
        check(*before)


# Calls of more than 16 rows are slices of the kernel; behind a product that writes the rows of a later slice, and one whose input lies
# where a later slice stores, no slice runs on the word of the call alone.
@pytest.mark.parametrize("layout", ["limbs", "codes"])
@pytest.mark.parametrize("case", ["reads", "stores", "adds"])
def test_slices_behind_a_captured_product(ops, forms, layout, case):
    w, bf = _Weights(ops, layout), torch.bfloat16
    x, buf, out = (torch.zeros(r, w.size, device="cuda", dtype=bf) for r in (16, 32, 32))
    first = torch.empty(16, w.size, device="cuda", dtype=bf)
    if case == "reads":      # the second slice's input is the product's result
        work = lambda: (w(0, x, buf[16:]), w(1, buf, out))
    elif case == "stores":   # the second slice's result lies over the product's input
        work = lambda: (w(0, out[16:], first), w(1, buf, out))
    else:                    # and adds to what the product wrote
        work = lambda: (w(0, x, out[16:]), w(1, buf, out, beta=1.0))
    graph = capture(work)

    def check(x0, buf0, out0):
        if case == "reads":
            buf0[16:] = w.want(0, x0).to(bf)
            assert torch.equal(buf, buf0) and torch.equal(out, w.want(1, buf0).to(bf))
        elif case == "stores":
            assert torch.equal(first, w.want(0, out0[16:]).to(bf)) and torch.equal(out, w.want(1, buf0).to(bf))
        else:
            out0[16:] = w.want(0, x0).to(bf)
            assert torch.equal(out, w.want(1, buf0, out0, beta=1.0).to(bf))
    assert forms(graph) == {"reads": ["waits", "reads", "waits"], "stores": ["waits", "reads", "reads"], "adds": ["waits", "reads", "reads"]}[case]
    _replayed(graph, (x, buf, out), check)


# From five slices on the first one waits, and the others run beside it.
def test_many_slices_behind_a_captured_product(ops, forms):
    w = _Weights(ops, "codes")
    x, buf, out = (torch.zeros(r, w.size, device="cuda", dtype=torch.bfloat16) for r in (16, 80, 80))
    graph = capture(lambda: (w(0, x, buf[64:]), w(1, buf, out)))
    assert forms(graph) == ["waits", "waits", "runs", "runs", "runs", "runs"]

    def check(x0, buf0, _):
        buf0[64:] = w.want(0, x0).to(torch.bfloat16)
        assert torch.equal(out, w.want(1, buf0).to(torch.bfloat16))
    _replayed(graph, (x, buf, out), check)


# A hint speaks of the kernels back to the last unhinted one: it is taken at its word behind one that waited first, not behind one that
# started early, nor behind what another thread captured.
@pytest.mark.parametrize("layout", ["limbs", "codes"])
def test_hints_behind_captured_products(ops, forms, layout):
    w = _Weights(ops, layout)
    x, a, b, c, d = (torch.zeros(8, w.size, device="cuda", dtype=torch.bfloat16) for _ in range(5))
    hinted = ops.independent_of_previous

    def chain(*steps):
        def work():
            for i, (hint, src, dst) in enumerate(steps):
                with hinted() if hint else contextlib.nullcontext():
                    w(i, src, dst)

        graph = capture(work)

        def check(*before):
            held = {t.data_ptr(): v for t, v in zip((x, a, b, c, d), before)}
            for i, (_, src, dst) in enumerate(steps):
                held[dst.data_ptr()] = w.want(i, held[src.data_ptr()]).to(torch.bfloat16)
            for t in (x, a, b, c, d):
                assert torch.equal(t, held[t.data_ptr()])
        _replayed(graph, (x, a, b, c, d), check)
        return forms(graph)
    assert chain((0, x, a), (0, x, b), (1, a, c)) == ["waits", "reads", "waits"]
    assert chain((0, x, a), (0, x, b), (1, x, c), (1, x, d)) == ["waits", "reads", "reads", "reads"]
    assert chain((0, x, a), (0, x, b), (1, a, c), (1, x, d)) == ["waits", "reads", "waits", "runs"]
    assert chain((0, x, a), (1, x, b), (1, x, c), (0, x, d)) == ["waits", "runs", "runs", "waits"]

    import threading

    def work():
        stream = torch.cuda.current_stream()

        def other():
            with torch.cuda.stream(stream), hinted():
                w(2, a, c)
        w(0, x, a)
        w(1, x, b)
        thread = threading.Thread(target=other)
        thread.start()
        thread.join()
    assert forms(capture(work)) == ["waits", "reads", "waits"]


# Scales and biases that a product in flight writes, of one matrix and of any of a group's; groups of which nothing touches it read early.
@pytest.mark.parametrize("touch", ["scale", "bias", "a group's scale", "a group's bias", "nothing"])
def test_vectors_of_a_captured_product(ops, forms, touch):
    w = _Weights(ops, "codes")
    x = torch.zeros(1, w.size, device="cuda")
    vector, y, z = (torch.zeros(1, w.size, device="cuda") for _ in range(3))
    at = lambda kind: vector[0] if kind in touch else None

    def work():
        w(0, x, vector)
        if "group" in touch or touch == "nothing":
            ops.gemm_trit_t2(w.packed[1:3], [w.size] * 2, x, K=w.size, outs=[y, z], row_scales=[None, at("scale")], biases=[None, at("bias")])
        else:
            w(2, x, z, scale=at("scale"), bias=at("bias"))
    graph = capture(work)
    assert forms(graph) == ["waits", "reads" if touch == "nothing" else "waits"]

    def check(x0, *_):
        held = w.want(0, x0)
        assert torch.equal(vector, held.float())
        scale, bias = (held[0] if kind in touch else None for kind in ("scale", "bias"))
        assert torch.equal(z, w.want(2, x0, scale=scale, bias=bias).float())
        if "group" in touch or touch == "nothing":
            assert torch.equal(y, w.want(1, x0).float())
    _replayed(graph, (x, vector, y, z), check)


# Two streams in one capture: what follows a join, or another stream's product, waits.
def test_captured_streams_that_fork_and_join(ops, forms):
    w = _Weights(ops, "codes", n=6)
    x, a, b, c, d, e, f = (torch.zeros(8, w.size, device="cuda", dtype=torch.bfloat16) for _ in range(7))
    side = torch.cuda.Stream()

    def work():
        main = torch.cuda.current_stream()
        w(0, x, a)
        side.wait_stream(main)
        w(1, x, b)
        with torch.cuda.stream(side):
            w(2, a, c)
            w(3, a, d)
        main.wait_stream(side)
        w(4, d, e)
        w(5, b, f)
    graph = capture(work)
    assert forms(graph) == ["waits", "reads", "waits", "reads", "waits", "reads"]

    def check(x0, *_):
        held = [w.want(0, x0).to(torch.bfloat16), w.want(1, x0).to(torch.bfloat16)]
        held += [w.want(i, held[0]).to(torch.bfloat16) for i in (2, 3)]
        held += [w.want(4, held[3]).to(torch.bfloat16), w.want(5, held[1]).to(torch.bfloat16)]
        for got, want in zip((a, b, c, d, e, f), held):
            assert torch.equal(got, want)
    _replayed(graph, (x, a, b, c, d, e, f), check)
