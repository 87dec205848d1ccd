"""Parity of the tcgen05 tensor-core kernel (prefill-shaped TRIT mode: more than 16
tokens, bf16 activations, token-major layout) with the CPU oracle."""

import numpy as np
import pytest
import torch

import oracle
from _graph_nodes import capture, kernels

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev(lib_built):
    from t81lib_b200 import _capi
    assert _capi.device_available(), _capi.last_error()
    return torch.device("cuda", 0)


def cuda(a, dev, dtype=None):
    t = torch.from_numpy(np.ascontiguousarray(a)).to(dev)
    return t if dtype is None else t.to(dtype)


def rel_err(got, want):
    want = np.asarray(want, np.float64)
    return float(np.max(np.abs(np.asarray(got, np.float64) - want)) / (np.sqrt(np.mean(want ** 2)) + 1e-30))


def case(rng, out_f, in_f, tokens):
    w = rng.normal(0, 0.02, (out_f, in_f)).astype(np.float32)
    packed, scale = oracle.pack_dense_matrix_absmean(w, 0.45)
    x = rng.normal(size=(tokens, in_f)).astype(np.float32)
    bias = rng.normal(0, 0.01, out_f).astype(np.float32)
    return packed, scale, x, bias


# one tile; ragged rows / tokens / K; several tiles per CTA; K below one atom; K spanning many super-blocks
SHAPES = [(128, 192, 256), (384, 1000, 200), (100, 130, 33), (130, 70, 300), (512, 512, 512), (257, 4096, 700),
          (1024, 3072, 2048), (64, 48, 17), (300, 14336, 40)]


@pytest.mark.parametrize("out_f,in_f,tokens", SHAPES)
def test_tc_gemm_matches_oracle(dev, out_f, in_f, tokens):
    from t81lib_b200 import _capi, ops
    rng = np.random.default_rng(out_f + 31 * in_f + 977 * tokens)
    packed, scale, x, bias = case(rng, out_f, in_f, tokens)
    xb = cuda(x, dev, torch.bfloat16)
    oracle.set_num_threads(8)
    want = oracle.linear_forward(packed, scale, bias, xb.float().cpu().numpy(), in_f)
    oracle.set_num_threads(1)
    y = ops.gemm_trit(cuda(packed, dev), xb, M=out_f, K=in_f, layout="nk", row_scale=cuda(scale, dev),
                      bias=cuda(bias, dev), out_dtype=torch.float32)
    assert _capi.kernel_status(reset=True) == 0
    # exact bf16 products, fp32 accumulation in TMEM: only the summation order differs
    assert rel_err(y.cpu().numpy(), want) < 2e-5
    yb = ops.gemm_trit(cuda(packed, dev), xb, M=out_f, K=in_f, layout="nk", row_scale=cuda(scale, dev),
                       bias=cuda(bias, dev))
    assert yb.dtype == torch.bfloat16
    np.testing.assert_allclose(yb.float().cpu().numpy(), want, rtol=1e-2, atol=1e-2 * float(np.sqrt(np.mean(want ** 2))))


def test_tc_gemm_alpha_beta_and_column_slice(dev):
    from t81lib_b200 import _capi, ops
    rng = np.random.default_rng(5)
    packed, scale, x, bias = case(rng, 256, 500, 100)
    xb = cuda(x, dev, torch.bfloat16)
    base = oracle.linear_forward(packed, None, None, xb.float().cpu().numpy(), 500)
    c0 = rng.normal(size=(100, 256)).astype(np.float32)
    C = cuda(c0, dev)
    ops.gemm_trit(cuda(packed, dev), xb, M=256, K=500, layout="nk", C=C, alpha=0.5, beta=2.0)
    assert rel_err(C.cpu().numpy(), 0.5 * base + 2.0 * c0) < 2e-5
    wide = torch.zeros(100, 600, device=dev)
    ops.gemm_trit(cuda(packed, dev), xb, M=256, K=500, layout="nk", C=wide[:, 200:456])
    assert rel_err(wide[:, 200:456].cpu().numpy(), base) < 2e-5
    assert not wide[:, :200].any() and not wide[:, 456:].any()
    assert _capi.kernel_status(reset=True) == 0


def test_prefill_shape_linearity_at_full_size(dev):
    """A 2048-token prefill of the Phi-3-mini qkv layer (3072 -> 9216): checked through linearity,
    y(a*x1 + x2) == a*y(x1) + y(x2), and a sampled comparison with the oracle."""
    from t81lib_b200 import _capi, ops
    gen = torch.Generator(device="cpu").manual_seed(4)
    out_f, in_f, tokens = 9216, 3072, 2048
    w = torch.randn(out_f, in_f, generator=gen) * 0.02
    packed, scale = ops.quantize_pack(w.to(dev), 0.45, "absmean")
    x1 = torch.randn(tokens, in_f, generator=gen).to(dev).to(torch.bfloat16)
    x2 = torch.randn(tokens, in_f, generator=gen).to(dev).to(torch.bfloat16)
    # powers of two keep a*x1 exact in bf16; x1 + x2 is rounded, so compare against y of the rounded sum
    xs = (2.0 * x1.float() + x2.float()).to(torch.bfloat16)
    bias = (torch.randn(out_f, generator=gen) * 0.01).to(dev)
    y1 = ops.gemm_trit(packed, x1, M=out_f, K=in_f, layout="nk", row_scale=scale, out_dtype=torch.float32)
    y2 = ops.gemm_trit(packed, x2, M=out_f, K=in_f, layout="nk", row_scale=scale, out_dtype=torch.float32)
    resid = (xs.float() - (2.0 * x1.float() + x2.float())).to(torch.bfloat16)  # exactly representable rounding error
    ys = ops.gemm_trit(packed, xs, M=out_f, K=in_f, layout="nk", row_scale=scale, out_dtype=torch.float32)
    yr = ops.gemm_trit(packed, resid, M=out_f, K=in_f, layout="nk", row_scale=scale, out_dtype=torch.float32)
    lhs, rhs = ys - yr, 2.0 * y1 + y2
    assert float((lhs - rhs).abs().max() / rhs.pow(2).mean().sqrt()) < 1e-4
    # 64 sampled rows x 48 sampled tokens against the oracle, with the bias
    rows = torch.randperm(out_f, generator=gen)[:64]
    toks = torch.randperm(tokens, generator=gen)[:48]
    yb = ops.gemm_trit(packed, x1, M=out_f, K=in_f, layout="nk", row_scale=scale, bias=bias, out_dtype=torch.float32)
    want = oracle.linear_forward(packed[rows.to(dev)].cpu().numpy(), scale[rows.to(dev)].cpu().numpy(),
                                 bias[rows.to(dev)].cpu().numpy(), x1[toks.to(dev)].float().cpu().numpy(), in_f)
    got = yb[toks.to(dev)][:, rows.to(dev)].cpu().numpy()
    assert rel_err(got, want) < 2e-5
    assert _capi.kernel_status(reset=True) == 0


# ---- activations that need the staging pre-pass (scratch workspace): fp32 / fp16 values, (K, N) layout


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("out_f,in_f,tokens", [(384, 1000, 200), (130, 700, 300), (512, 4096, 129)])
def test_tc_gemm_staged_activations_token_major(dev, dtype, out_f, in_f, tokens):
    from t81lib_b200 import _capi, ops
    rng = np.random.default_rng(out_f + in_f + tokens)
    packed, scale, x, bias = case(rng, out_f, in_f, tokens)
    xd = cuda(x, dev, dtype)
    oracle.set_num_threads(8)
    want = oracle.linear_forward(packed, scale, bias, xd.float().cpu().numpy(), in_f)
    oracle.set_num_threads(1)
    assert _capi.lib.t81b200_gemm_trit_workspace_bytes(_capi.F32 if dtype == torch.float32 else _capi.F16,
                                                        _capi.LAYOUT_NK, _capi.F32, out_f, tokens, in_f) > 0
    y = ops.gemm_trit(cuda(packed, dev), xd, M=out_f, K=in_f, layout="nk", row_scale=cuda(scale, dev),
                      bias=cuda(bias, dev), out_dtype=torch.float32)
    assert _capi.kernel_status(reset=True) == 0
    # two bf16 planes carry 16 mantissa bits of each activation: 1e-3 asked for fp32, ~1e-5 achieved
    assert rel_err(y.cpu().numpy(), want) < 1e-3
    assert rel_err(y.cpu().numpy(), want) < 5e-5


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_tc_gemm_reference_argument_order(dev, dtype):
    """(K, N) dense operand and (M, N) result, the layout of t81::linalg::gemm_ternary."""
    from t81lib_b200 import _capi, ops
    rng = np.random.default_rng(77)
    M, N, K = 300, 260, 1000
    trits = rng.integers(-1, 2, (M, K)).astype(np.int8)
    A = oracle.pack_trits_rowwise(trits)
    B = cuda(rng.normal(size=(K, N)).astype(np.float32), dev, dtype)
    C0 = rng.normal(size=(M, N)).astype(np.float32)
    oracle.set_num_threads(8)
    want = oracle.gemm_trit(A, B.float().cpu().numpy(), C0, M, N, K, 1.5, 0.5)
    oracle.set_num_threads(1)
    C = cuda(C0, dev)
    ops.gemm_trit(cuda(A, dev), B, M=M, K=K, layout="kn", C=C, alpha=1.5, beta=0.5)
    assert _capi.kernel_status(reset=True) == 0
    assert rel_err(C.cpu().numpy(), want) < 5e-5


def test_host_pointer_entry_point(dev):
    """t81b200_gemm_trit_host: what the C++ span overload of gemm_ternary binds to."""
    import ctypes
    from t81lib_b200 import _capi
    rng = np.random.default_rng(78)
    M, N, K = 128, 64, 480
    trits = rng.integers(-1, 2, (M, K)).astype(np.int8)
    A = oracle.pack_trits_rowwise(trits)
    B = rng.normal(size=(K, N)).astype(np.float32)
    C = rng.normal(size=(M, N)).astype(np.float32)
    want = oracle.gemm_trit(A, B, C, M, N, K, 2.0, -1.0)
    vp = ctypes.c_void_p
    rc = _capi.lib.t81b200_gemm_trit_host(A.ctypes.data_as(vp), B.ctypes.data_as(vp), C.ctypes.data_as(vp), M, N, K, 2.0, -1.0)
    assert rc == 0, _capi.last_error()
    assert rel_err(C, want) < 5e-5
    rc = _capi.lib.t81b200_gemm_trit_host(A.ctypes.data_as(vp), B.ctypes.data_as(vp), C.ctypes.data_as(vp), -1, N, K, 1.0, 0.0)
    assert rc == _capi.EINVAL and "non-negative" in _capi.last_error()


# 16-bit results whose rows start anywhere, and activations whose rows do: widths around words, warps and tiles, tokens around blocks.
# Whole numbers below 256 throughout, so that every type holds them exactly.
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("out_f,in_f,tokens", [(1, 577, 33), (2, 576, 40), (63, 201, 100), (65, 203, 64), (127, 385, 31), (129, 1001, 300), (255, 66, 257), (257, 95, 1000),
                                               (386, 833, 2100), (4093, 301, 50), (1999, 2047, 90)])
def test_tc_rows_off_boundaries(dev, dtype, out_f, in_f, tokens):
    from t81lib_b200 import _capi, ops
    gen = torch.Generator(device="cuda").manual_seed(out_f + tokens)
    trits = torch.randint(-1, 2, (out_f, in_f), generator=gen, device="cuda").float()
    t2 = ops.pack_t2(ops.quantize_pack(trits, 0.5, "fixed")[0], out_f, in_f)
    x = torch.randint(-1, 2, (tokens, in_f), generator=gen, device="cuda").to(dtype)
    x[torch.rand(tokens, in_f, generator=gen, device="cuda") < 0.5] = 0
    want = (x.double() @ trits.double().t()).to(dtype)
    got = ops.linear_t2(t2, out_f, x, in_f, None, None)
    assert torch.equal(got, want)
    wide = torch.full((tokens, in_f + 3), float("nan"), device="cuda", dtype=dtype)  # nothing beside the rows is used
    wide[:, 1:in_f + 1] = x
    assert torch.equal(ops.linear_t2(t2, out_f, wide[:, 1:in_f + 1], in_f, None, None), want)
    assert _capi.kernel_status(reset=True) == 0


# Staged 16-bit rows: four k a thread up to a size, eight beyond it; less where four leave many lanes idle (513: 130 pieces on 160 lanes).
@pytest.mark.parametrize("in_f,tokens,width", [(1023, 1536, 4), (1023, 1537, 8), (513, 1008, 4), (513, 1009, 8), (2047, 17, 4), (2047, 768, 4), (2047, 769, 8), (703, 2000, 4),
                                               (513, 2000, 8)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_staged_rows_by_size(dev, in_f, tokens, width, dtype):
    from t81lib_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    trits = torch.randint(-1, 2, (130, in_f), generator=gen, device="cuda").float()
    t2 = ops.pack_t2(ops.quantize_pack(trits, 0.5, "fixed")[0], 130, in_f)
    x = torch.randint(-1, 2, (tokens, in_f), generator=gen, device="cuda").to(dtype)
    x[torch.rand(tokens, in_f, generator=gen, device="cuda") < 0.8] = 0
    got = []
    staging = [name for name, _ in kernels(capture(lambda: got.append(ops.linear_t2(t2, 130, x, in_f, None, None)))) if "stage_rows_kernel" in name]
    assert len(staging) == 1 and f"Li0ELi{width}E" in staging[0]
    assert torch.equal(got[0], (x.double() @ trits.double().t()).to(dtype))


# 16-bit results that TMA cannot write have a kernel of their own; everything else stays out of it.
@pytest.mark.parametrize("out_f,dtype,out_dtype,own", [(256, torch.bfloat16, None, 0), (255, torch.bfloat16, None, 1), (260, torch.float16, None, 1),
                                                       (255, torch.bfloat16, torch.float32, 0), (255, torch.float32, torch.bfloat16, 1), (264, torch.float32, torch.float16, 0)])
def test_rows_off_boundaries_have_their_own_kernel(dev, out_f, dtype, out_dtype, own):
    from t81lib_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(out_f)
    trits = torch.randint(-1, 2, (out_f, 192), generator=gen, device="cuda").float()
    t2 = ops.pack_t2(ops.quantize_pack(trits, 0.5, "fixed")[0], out_f, 192)
    x, got = torch.randint(-1, 2, (70, 192), generator=gen, device="cuda").to(dtype), []
    names = [name for name, _ in kernels(capture(lambda: got.append(ops.linear_t2(t2, out_f, x, 192, None, None, out_dtype)))) if "gemm_trit_tc_kernel" in name]
    assert len(names) == 1 and f"ELb{own}EEE" in names[0], names
    assert torch.equal(got[0], (x.double() @ trits.double().t()).to(out_dtype or dtype))


# The planes of float32 activations side by side in one product (up to 96 tokens a tile), apart (128) and wide (192 to 256, tiles alone):
# tokens at the edges of the widths, one tile, tiles that follow one another and a contraction split over a cluster.
@pytest.mark.parametrize("planes", [2, 3])
@pytest.mark.parametrize("out_f,in_f,tokens", [(300, 700, 17), (256, 4000, 32), (300, 4000, 33), (260, 4000, 64), (5000, 3000, 65), (20000, 200, 96), (20000, 200, 97), (300, 9000, 128),
                                               (2600, 1000, 513), (20000, 193, 129), (5530, 6000, 249), (20000, 500, 250), (700, 130, 6000)])
def test_planes_of_float32_by_width(dev, out_f, in_f, tokens, planes):
    from t81lib_b200 import _capi, ops
    gen = torch.Generator(device="cuda").manual_seed(out_f + tokens)
    trits = torch.randint(-1, 2, (out_f, in_f), generator=gen, device="cuda").float()
    t2 = ops.pack_t2(ops.quantize_pack(trits, 0.5, "fixed")[0], out_f, in_f)
    x = torch.randn(tokens, in_f, generator=gen, device="cuda")
    # small planes say much: values whose second and third plane are of one sign
    x = (x.bfloat16().float() * (1.0 + 2.0 ** -9 + 2.0 ** -18)).contiguous()
    want = x.double() @ trits.double().t()
    got = ops.linear_t2(t2, out_f, x, in_f, None, None, torch.float32, planes)
    # two planes leave 2^-17 of a value out, three 2^-25; an accumulator is cut off at 2^-23 of its sum, which grows with its root, every
    # 16 columns: the first plane's with the values' 8 bits hardly ever, the others' always, but they are 2^-8 of it
    err = float((got.double() - want).norm() / want.norm())
    assert err < (2.0 ** -16 if planes == 2 else 2.0 ** -20)
    assert _capi.kernel_status(reset=True) == 0


# Every form in which planes meet (Mode): side by side in one product, apart and wide, of tiles alone, one after the other and split over a
# cluster.  The form is read from what was launched, so that other step costs cannot drop one unseen.
TC_PARAM_WIDTH, TC_PARAM_SPLITS, TC_PARAM_M_TILES, TC_PARAM_N_TILES = 21, 27, 19, 20  # TcParams in 32-bit words
SIDE, APART, WIDE = 1, 2, 3


@pytest.mark.parametrize("planes", [2, 3])
@pytest.mark.parametrize("out_f,in_f,tokens,mode,split,alone", [
    (2600, 1000, 513, SIDE, False, True), (5000, 3000, 65, SIDE, True, True), (20000, 200, 96, SIDE, False, False),
    (10152, 11900, 114, APART, False, True), (7391, 13254, 101, APART, True, True), (20000, 500, 250, APART, False, False),
    (700, 130, 6000, WIDE, False, True), (2807, 9347, 475, WIDE, True, True)])
def test_planes_of_float32_in_every_form(dev, out_f, in_f, tokens, mode, split, alone, planes):
    from t81lib_b200 import _capi, ops
    gen = torch.Generator(device="cuda").manual_seed(out_f + tokens)
    trits = torch.randint(-1, 2, (out_f, in_f), generator=gen, device="cuda").float()
    t2 = ops.pack_t2(ops.quantize_pack(trits, 0.5, "fixed")[0], out_f, in_f)
    x = torch.randn(tokens, in_f, generator=gen, device="cuda")
    x = (x.bfloat16().float() * (1.0 + 2.0 ** -9 + 2.0 ** -18)).contiguous()
    got = []
    graph = capture(lambda: got.append(ops.linear_t2(t2, out_f, x, in_f, None, None, torch.float32, planes)))  # its parameters live as long as it does
    launched = [(name, params(3)) for name, params in kernels(graph) if "gemm_trit_tc_kernel" in name]
    graph.replay()
    assert len(launched) == 1 and f"ModeE{mode}E" in launched[0][0], launched[0][0]
    words = launched[0][1]
    assert (words[TC_PARAM_SPLITS] > 1) == split and words[TC_PARAM_WIDTH] in ((), (32, 64, 96), (128,), (192, 224, 256))[mode]
    assert (split or words[TC_PARAM_M_TILES] * words[TC_PARAM_N_TILES] <= 74) == alone
    want = x.double() @ trits.double().t()
    for y in got:  # the call before the capture, and the captured one
        assert float((y.double() - want).norm() / want.norm()) < (2.0 ** -16 if planes == 2 else 2.0 ** -20)  # as above
    assert _capi.kernel_status(reset=True) == 0


# Products of every tile width one behind the other, each in a part of the chip's pairs so that the next one's set-up runs beside it; the
# last pair's odd CTA has no weights.  A wait that runs out shows in the status, and in sums that are not whole.
def test_products_of_every_width_one_behind_the_other(dev):
    from t81lib_b200 import _capi, ops
    gen = torch.Generator(device="cuda").manual_seed(160)
    shapes = [(11392, 10808, (143,)), (11392, 2056, (30, 60, 90, 120, 143, 190, 220, 250)), (5504, 4104, (160, 288, 130, 448))]
    work = []
    for out_f, in_f, rows in shapes:
        trits = torch.randint(-1, 2, (out_f, in_f), generator=gen, device="cuda").float()
        t2 = ops.pack_t2(ops.quantize_pack(trits, 0.5, "fixed")[0], out_f, in_f)
        for tokens in rows:
            x = torch.randint(-1, 2, (tokens, in_f), generator=gen, device="cuda").bfloat16()
            work.append((t2, out_f, x, in_f, (x.double() @ trits.double().t()).bfloat16()))
        del trits
    for _ in range(20):
        for t2, out_f, x, in_f, want in work:
            assert torch.equal(ops.linear_t2(t2, out_f, x, in_f, None, None), want)
    for step in (1, 5):  # without anything between the products
        got = []
        graph = capture(lambda: got.append([ops.linear_t2(*work[step * i % len(work)][:4], None, None) for i in range(2 * len(work))]))
        for _ in range(20):
            graph.replay()
            torch.cuda.synchronize()
        for i, y in enumerate(got[-1]):
            assert torch.equal(y, work[step * i % len(work)][4])
    assert _capi.kernel_status(reset=True) == 0
