"""The paired tensor-core kernel behind ``ops.linear_t2`` (decode-stream layout) and ``ops.gemm_trit`` (limbs) at the
edges of its tiles, contraction splits and staging rules, against the CPU oracle."""

import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev(lib_built):
    from t81lib_b200 import _capi
    assert _capi.device_available(), _capi.last_error()
    return torch.device("cuda", 0)


# (rows, K, tokens): one row and column; 17 tokens on a 32-token tile; two CTAs with the second one empty (rows <= 128) or
# nearly so (129, 257); K below, at and just past an atom (64) and a chunk (192); splits of 2 to 4 with unequal shares; a
# 224- and a 256-token tile; several tiles per cluster with a ragged last one in both directions;
# 192-, 224- and 160-token tiles whose chunks go behind one barrier, the last chunk of one step
SHAPES = [(1, 1, 17), (128, 64, 32), (129, 65, 33), (257, 192, 64), (256, 193, 96), (300, 385, 97), (512, 1001, 129),
          (1024, 4096, 40), (4096, 1536, 80), (100, 14336, 18), (260, 256, 777), (9500, 200, 1100),
          (2048, 577, 1500), (9728, 400, 200), (12000, 130, 450)]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("rows,K,tokens", SHAPES)
def test_products_match_the_oracle(dev, rows, K, tokens, dtype):
    from t81lib_b200 import _capi, ops
    rng = np.random.default_rng(rows + 31 * K + 977 * tokens)
    trits = rng.integers(-1, 2, (rows, K)).astype(np.int8)
    limbs = oracle.pack_trits_rowwise(trits)
    scale, bias = rng.uniform(0.01, 0.03, rows).astype(np.float32), rng.normal(0, 0.01, rows).astype(np.float32)
    packed, sd, bd = (torch.from_numpy(a).to(dev) for a in (limbs, scale, bias))
    t2 = ops.pack_t2(packed, rows, K)
    wide = torch.from_numpy(rng.normal(size=(tokens, K + 3)).astype(np.float32)).to(dev).to(dtype)
    # products are exact, sums fp32 in another order: about sqrt(K) ulp of the sum's size; fp32 activations enter with 16
    # mantissa bits (2^-17 each, averaging out over K)
    tol = 2e-5 if dtype != torch.float32 else 5e-5
    for x in (wide[:, :K].contiguous(), wide[:, 1:K + 1]):  # rows on 16-byte boundaries where K allows, and not
        want = (x.double().cpu().numpy() @ trits.T.astype(np.float64)) * scale + bias
        rms = float(np.sqrt(np.mean(want ** 2)))
        y = ops.linear_t2(t2, rows, x, K, sd, bd, torch.float32)
        z = ops.gemm_trit(packed, x, M=rows, K=K, layout="nk", row_scale=sd, bias=bd, out_dtype=torch.float32)
        assert np.abs(y.cpu().numpy() - want).max() < tol * rms
        assert np.abs(z.cpu().numpy() - want).max() < tol * rms
        # 16-bit results: one rounding of the fp32 ones (TMA-store epilogue where rows are a multiple of 8)
        h = ops.linear_t2(t2, rows, x, K, sd, bd, torch.bfloat16)
        assert torch.equal(h, y.to(torch.bfloat16))
    assert _capi.kernel_status(reset=True) == 0


# decode-sized calls whose rows lie on 16-byte, 4-byte and odd 2-byte places, and end inside a group of eight
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("rows,K,tokens", [(40, 7, 1), (70, 1905, 16), (100, 130, 5), (33, 1538, 9), (64, 14336, 16)])
def test_decode_rows_off_boundaries(dev, rows, K, tokens, dtype):
    from t81lib_b200 import _capi, ops
    rng = np.random.default_rng(rows + K)
    trits = rng.integers(-1, 2, (rows, K)).astype(np.int8)
    t2 = ops.pack_t2(torch.from_numpy(oracle.pack_trits_rowwise(trits)).to(dev), rows, K)
    wide = torch.from_numpy(rng.normal(size=(tokens, K + 3)).astype(np.float32)).to(dev).to(dtype)
    tol = 2e-5 if dtype != torch.float32 else 1e-4  # as above; short contractions average fp32's 2^-17 roundings less
    for x in (wide[:, :K].contiguous(), wide[:, 1:K + 1], wide[:, 2:K + 2]):
        want = x.double().cpu().numpy() @ trits.T.astype(np.float64)
        y = ops.linear_t2(t2, rows, x, K, None, None, torch.float32)
        assert np.abs(y.cpu().numpy() - want).max() < tol * float(np.sqrt(np.mean(want ** 2)))
    assert _capi.kernel_status(reset=True) == 0


# launch shapes of short rows: K from 4 to 9 chunks with up to and past three 32-row CTAs per SM, 10 to 18 chunks with up to
# and past one pair of 64-row CTAs per SM; long rows in eight slices, and a row too many for them
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,K,tokens", [(33, 584, 1), (1000, 1728, 16), (14208, 768, 5), (14240, 768, 9), (3200, 1736, 9),
                                           (129, 3456, 16), (9472, 1920, 12), (9536, 1920, 12), (449, 8208, 3),
                                           (2048, 14336, 8), (2049, 8208, 1)])
def test_decode_short_rows(dev, rows, K, tokens, dtype):
    from t81lib_b200 import _capi, ops
    rng = np.random.default_rng(rows + K)
    trits = rng.integers(-1, 2, (rows, K)).astype(np.int8)
    t2 = ops.pack_t2(torch.from_numpy(oracle.pack_trits_rowwise(trits)).to(dev), rows, K)
    x = torch.from_numpy(rng.normal(size=(tokens, K)).astype(np.float32)).to(dev).to(dtype)
    want = x.double().cpu().numpy() @ trits.T.astype(np.float64)
    y = ops.linear_t2(t2, rows, x, K, None, None, torch.float32)
    assert np.abs(y.cpu().numpy() - want).max() < 2e-5 * float(np.sqrt(np.mean(want ** 2)))  # exact products, fp32 sums
    assert _capi.kernel_status(reset=True) == 0


# fp32 rows in three planes, weights without zeros to thin the sums out: tiles alone, split over a cluster, several per cluster and
# the widest the two accumulators of a tile leave room for
@pytest.mark.parametrize("rows,K,tokens", [(100, 512, 33), (512, 1537, 1000), (9500, 700, 1100), (300, 4096, 257), (2048, 14336, 600)])
def test_three_planes_are_as_exact_as_fp32(dev, rows, K, tokens):
    from t81lib_b200 import _capi, ops
    gen = torch.Generator(device="cuda").manual_seed(rows + K)
    trits = torch.randint(0, 2, (rows, K), generator=gen, device=dev).float() * 2 - 1
    t2 = ops.pack_t2(ops.quantize_pack(trits, 0.5, "fixed")[0], rows, K)
    x = torch.randn(tokens, K, generator=gen, device=dev)
    want = x.double() @ trits.double().t()
    rms = lambda y: float((y.double() - want).norm() / want.norm())
    plain = rms(torch.cat([x[i:i + 256] @ trits.t() for i in range(0, tokens, 256)]))  # fp32 on CUDA cores
    assert rms(ops.linear_t2(t2, rows, x, K, None, None, torch.float32, 3)) <= plain
    assert _capi.kernel_status(reset=True) == 0


# small fp32 products keep every mantissa bit on either layout: more than 128 rows, and 17 to 128 where slices of the streaming
# kernel would be the slower way (K short against the number of slices)
@pytest.mark.parametrize("rows,K,tokens", [(256, 256, 128), (64, 512, 100), (128, 100, 300), (16, 512, 1000), (2000, 8, 500), (64, 64, 40), (64, 128, 64)])
def test_small_fp32_products_are_exact(dev, rows, K, tokens):
    from t81lib_b200 import _capi, ops
    gen = torch.Generator(device="cuda").manual_seed(rows + K)
    trits = torch.randint(-1, 2, (rows, K), generator=gen, device=dev).float()
    packed = ops.quantize_pack(trits, 0.5, "fixed")[0]
    t2 = ops.pack_t2(packed, rows, K)
    wide = torch.randn(tokens, K + 1, generator=gen, device=dev)
    for x in (wide[:, :K].contiguous(), wide[:, 1:]):
        want = x.double() @ trits.double().t()
        for y in (ops.linear_t2(t2, rows, x, K, None, None, torch.float32), ops.gemm_trit(packed, x, M=rows, K=K, layout="nk")):
            # a rounding of up to half an ulp of the running sum per addition, K of them at random
            assert float((y.double() - want).norm() / want.norm()) < 2.0 ** -25 * (K ** 0.5 + 1)
    assert _capi.kernel_status(reset=True) == 0


# two planes on either layout: 16 mantissa bits leave 2^-17 / sqrt(3) of a value at most, whatever the length of the sums; tiles of
# one and two accumulators' widths, alone, split and several per cluster, and the rows that slices of the streaming kernel served
@pytest.mark.parametrize("rows,K,tokens", [(512, 1537, 1000), (9500, 700, 1100), (300, 4096, 257), (2048, 14336, 250), (4096, 14336, 100), (512, 6000, 17)])
def test_two_planes_lose_only_the_inputs_bits(dev, rows, K, tokens):
    from t81lib_b200 import _capi, ops
    gen = torch.Generator(device="cuda").manual_seed(rows + K)
    trits = torch.randint(-1, 2, (rows, K), generator=gen, device=dev).float()
    packed = ops.quantize_pack(trits, 0.5, "fixed")[0]
    t2 = ops.pack_t2(packed, rows, K)
    x = torch.randn(tokens, K, generator=gen, device=dev)
    want = x.double() @ trits.double().t()
    for y in (ops.linear_t2(t2, rows, x, K, None, None, torch.float32), ops.gemm_trit(packed, x, M=rows, K=K, layout="nk"),
              ops.gemm_trit(packed, x.t().contiguous(), M=rows, K=K, layout="kn").t()):
        assert float((y.double() - want).norm() / want.norm()) < 2.0 ** -17 / 3 ** 0.5
    assert _capi.kernel_status(reset=True) == 0


# an infinity among fp32 activations reaches the results as it does in fp32 arithmetic (signs kept, no number where a trit is zero), and
# large values keep their size, on the limbs next to the largest there is (the other layout's codes are twice the trits): three planes,
# two planes, both layouts
@pytest.mark.parametrize("tokens,K", [(40, 96), (300, 96), (400, 1000)])
def test_infinities_and_the_largest_values(dev, tokens, K):
    from t81lib_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    trits = torch.randint(-1, 2, (256, K), generator=gen, device=dev).float()
    packed = ops.quantize_pack(trits, 0.5, "fixed")[0]
    t2 = ops.pack_t2(packed, 256, K)
    x = torch.randn(tokens, K, generator=gen, device=dev)
    x[1, 3], x[2, 5], x[5] = float("inf"), float("-inf"), 0.0
    for largest in (1.5e38, 3.4e38):  # rounds to infinity in bf16; the very largest does with 16 mantissa bits too
        x[5, 7] = -largest
        want = x.double() @ trits.double().t()
        outs = [ops.gemm_trit(packed, x.t().contiguous(), M=256, K=K, layout="kn").t()]
        if largest < 1.7e38:
            outs += [ops.linear_t2(t2, 256, x, K, None, None, torch.float32, planes) for planes in (2, 3)]
        _compare_beyond_finite(outs, want)


def _compare_beyond_finite(outs, want):
    for y in outs:
        assert torch.equal(y.isnan(), want.isnan()) and torch.equal(torch.where(y.isinf(), y, 0.0).double(), torch.where(want.isinf(), want, 0.0))
        torch.testing.assert_close(y[5].double(), want[5], rtol=2.0 ** -16, atol=0)
