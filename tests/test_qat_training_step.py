"""The two kernels of the fused training step at the edges of their tiles: the quantiser that writes the decode-stream
layout of a weight and of its transpose (bytes, against the oracle), and the weight gradient on the tensor cores (against
float64 sums of the same operands)."""

import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols", [(1, 1), (32, 192), (33, 100), (193, 385), (700, 161), (192, 384)])
@pytest.mark.parametrize("threshold", [0.0, 0.45, 1.0])
def test_quantiser_bytes(lib_built, rows, cols, threshold):
    from t81lib_b200 import ops
    rng = np.random.default_rng(rows * 7 + cols)
    w = rng.normal(0, 0.03, (rows, cols)).astype(np.float32)
    scale = np.float32(np.abs(w).max())
    # values whose quotient rounds onto the threshold, from either side, and zeros of both signs
    near = np.float32(threshold) * scale
    w.flat[:6] = [near, -near, np.nextafter(near, np.float32(0)), np.nextafter(near, np.float32(9)), 0.0, -0.0][:w.size]
    want = oracle.qat_quantize(w, scale, threshold)
    wd = torch.from_numpy(w).cuda()
    wide = torch.zeros(rows, cols + 5, device="cuda")
    wide[:, :cols] = wd
    for src in (wd, wide[:, :cols]):
        t2, t2_t, scales = ops.qat_quantize_t2(src, threshold, torch.tensor([scale]).cuda())
        assert np.array_equal(t2.cpu().numpy(), oracle.pack_t2(want))
        assert np.array_equal(t2_t.cpu().numpy(), oracle.pack_t2(np.ascontiguousarray(want.T)))
        assert scales.numel() == max(rows, cols) and bool((scales == float(scale)).all())


# one output; columns of a 128- and a 256-column tile and one past them; tokens below, at and past a 64-token step;
# tokens split over a cluster; several tiles per cluster; fp32 tokens in two segments
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("tokens,rows,cols", [(1, 1, 1), (63, 128, 64), (64, 256, 256), (65, 257, 129), (1000, 200, 300), (130, 2050, 1537),
                                              (70, 4000, 4096), (1100, 4000, 4300)])
def test_weight_gradient(lib_built, tokens, rows, cols, dtype):
    from t81lib_b200 import _capi, ops
    gen = torch.Generator(device="cuda").manual_seed(tokens + rows + cols)
    w = torch.randn(rows, cols, device="cuda", generator=gen) * 0.03
    scale = w.abs().amax().reshape(1)
    w.view(-1)[0] = scale[0] * 0.5  # exactly on the surrogate's edge: no gradient
    g = torch.randn(tokens, rows + 1, device="cuda", generator=gen).to(dtype)
    x = torch.randn(tokens, cols + 1, device="cuda", generator=gen).to(dtype)
    slope = ((w / scale).abs() < 0.5).double() * 2.0
    for gs, xs in ((g[:, :rows].contiguous(), x[:, :cols].contiguous()), (g[:, 1:], x[:, 1:])):  # read in place, and staged
        got = ops.qat_weight_grad(gs, xs, w, scale)
        sums = gs.double().t() @ xs.double()
        # exact products (fp32: to an ulp), accumulated in fp32 16 tokens at a time: each of those steps may cut up to an
        # ulp (2^-23) of the running sum, which stays within about five times the root mean square of the results; the
        # slope doubles it, and the last addition of the two fp32 accumulators (or of a split's shares) adds two more ulps
        bound = 2 * 5 * (tokens / 16 + 3) * 2.0 ** -23
        err = (got.double() - sums * slope).abs().max() / sums.pow(2).mean().sqrt()
        assert float(err) < bound
        assert bool((got[slope == 0] == 0).all())
    assert _capi.kernel_status(reset=True) == 0


# no further from the exact sums than fp32 on CUDA cores, whatever the number of tokens: segments of every length, in one and in
# several accumulators a tile, tiles alone, split over a cluster and several per cluster
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("tokens,rows,cols", [(256, 512, 512), (500, 4000, 4300), (777, 1537, 1001), (1000, 2050, 1537), (4096, 1024, 1024),
                                              (8192, 512, 512), (8192, 128, 100), (3000, 4000, 4300)])
def test_weight_gradient_is_as_exact_as_fp32(lib_built, tokens, rows, cols, dtype):
    from t81lib_b200 import _capi, ops
    gen = torch.Generator(device="cuda").manual_seed(tokens + rows + cols)
    w, scale = torch.zeros(rows, cols, device="cuda"), torch.ones(1, device="cuda")  # slope 2 everywhere
    g, x = (torch.randn(tokens, n, device="cuda", generator=gen).to(dtype) for n in (rows, cols))
    want = 2.0 * (g.double().t() @ x.double())
    rms = lambda t: float((t.double() - want).norm() / want.norm())
    assert rms(ops.qat_weight_grad(g, x, w, scale)) <= rms(2.0 * (g.float().t() @ x.float()))
    assert _capi.kernel_status(reset=True) == 0


# weights and scales that are not finite quantise as the division does: infinite weights keep their sign under a finite scale, and
# nothing reaches the threshold under an infinite one
@pytest.mark.parametrize("scale", [0.05, float("inf"), float("nan")])
@pytest.mark.parametrize("threshold", [0.0, 0.45, 1.0])
def test_quantiser_bytes_beyond_finite_values(lib_built, scale, threshold):
    from t81lib_b200 import ops
    w = np.random.default_rng(0).normal(0, 0.03, (40, 200)).astype(np.float32)
    w.flat[:5] = [np.inf, -np.inf, np.nan, 3e38, -3e38]
    with np.errstate(invalid="ignore", over="ignore"):
        want = oracle.qat_quantize(w, np.float32(scale), threshold)
    t2, t2_t, _ = ops.qat_quantize_t2(torch.from_numpy(w).cuda(), threshold, torch.tensor([scale]).cuda())
    assert np.array_equal(t2.cpu().numpy(), oracle.pack_t2(want))
    assert np.array_equal(t2_t.cpu().numpy(), oracle.pack_t2(np.ascontiguousarray(want.T)))


# weights whose rows TMA reads, with and without gaps, and rows that go word by word: blocks at the edges of the matrix, slots that are
# filled again inside a tile and for the tile that follows, three and two of them, tokens split over a cluster
@pytest.mark.parametrize("gap,skip", [(0, 0), (4, 0), (4, 1), (3, 0)])
@pytest.mark.parametrize("tokens,rows,cols", [(64, 33, 36), (130, 300, 1540), (70, 4000, 4340), (300, 4000, 4340), (2100, 4000, 4341), (20, 4100, 700)])
def test_weight_gradient_of_strided_weights(lib_built, tokens, rows, cols, gap, skip):
    from t81lib_b200 import _capi, ops
    gen = torch.Generator(device="cuda").manual_seed(tokens + rows + cols + gap)
    w = (torch.randn(rows, cols + gap, device="cuda", generator=gen) * 0.03)[:, skip:skip + cols]
    scale = w.abs().amax().reshape(1)
    g, x = (torch.randn(tokens, n, device="cuda", generator=gen).bfloat16() for n in (rows, cols))
    slope = ((w / scale).abs() < 0.5).double() * 2.0
    sums = g.double().t() @ x.double()
    got = ops.qat_weight_grad(g, x, w, scale)
    bound = 2 * 5 * (tokens / 16 + 3) * 2.0 ** -23  # as above
    assert float((got.double() - sums * slope).abs().max() / sums.pow(2).mean().sqrt()) < bound
    assert _capi.kernel_status(reset=True) == 0


# an infinity in either fp32 operand comes out where and as it does in fp32 arithmetic
@pytest.mark.parametrize("tokens", [20, 600])
def test_weight_gradient_of_infinities(lib_built, tokens):
    from t81lib_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    w = torch.randn(70, 90, device="cuda", generator=gen) * 0.03
    scale = w.abs().amax().reshape(1)
    g, x = torch.randn(tokens, 70, device="cuda", generator=gen), torch.randn(tokens, 90, device="cuda", generator=gen)
    g[3, 4], x[5, 6] = float("inf"), float("-inf")
    want = (g.double().t() @ x.double()) * (((w / scale).abs() < 0.5).double() * 2.0)
    got = ops.qat_weight_grad(g, x, w, scale)
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(torch.where(got.isinf(), got, 0.0).double(), torch.where(want.isinf(), want, 0.0))
    finite = want.isfinite()
    torch.testing.assert_close(got[finite].double(), want[finite], rtol=1e-5, atol=1e-4)  # fp32 sums of up to 600 products
