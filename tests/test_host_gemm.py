"""``gemm_ternary`` on numpy buffers at the sizes where its staging changes: single copies, pieces, helper threads."""

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


# B of 2 MiB and one row less and more of it (helpers on the way up), C of 1 MiB and a row more (on the way down), rows of no
# multiple of 16 bytes, one element, and more than one piece in both directions
@pytest.mark.parametrize("M,N,K", [(1, 1, 48), (64, 33, 48), (128, 1024, 480), (128, 1024, 528), (96, 993, 528), (512, 512, 96),
                                   (513, 512, 96), (300, 4097, 576), (2048, 1500, 96)])
@pytest.mark.parametrize("beta", [0.0, 0.5])
def test_host_buffers(lib_built, M, N, K, beta):
    from t81lib_b200 import t81lib
    rng = np.random.default_rng(M + N + K)
    trits = rng.integers(-1, 2, (M, K)).astype(np.int8)
    b, c = rng.normal(size=(K, N)).astype(np.float32), rng.normal(size=(M, N)).astype(np.float32)
    want = 1.5 * (trits.astype(np.float64) @ b) + beta * c
    t81lib.gemm_ternary(oracle.pack_trits_rowwise(trits), b, c, M, N, K, alpha=1.5, beta=beta)
    # fp32 activations enter with 16 mantissa bits (2^-17 each, averaging out over K), as in the device tests; relative to the
    # product's root mean square
    assert np.abs(c - want).max() < 5e-5 * 1.5 * float(np.sqrt(np.mean(np.abs(trits).sum(1))))


def test_operands_that_the_default_stream_still_writes(lib_built):
    """A page-locked operand whose copy from the device is queued on the default stream: the call stands behind it."""
    import torch
    from t81lib_b200 import t81lib
    M, N, K = 64, 96, 96
    rng = np.random.default_rng(0)
    trits = rng.integers(-1, 2, (M, K)).astype(np.int8)
    a, c = oracle.pack_trits_rowwise(trits), np.zeros((M, N), np.float32)
    b = torch.zeros(K, N, pin_memory=True)
    there = torch.from_numpy(rng.integers(-3, 4, (K, N)).astype(np.float32)).cuda()
    t81lib.gemm_ternary(a, b.numpy(), c, M, N, K)  # buffers and plans
    busy = torch.ones(16384, 16384, device="cuda")
    torch.cuda.synchronize()
    for _ in range(4):
        busy.mul_(1.0)  # a millisecond of work ahead of the copy
    b.copy_(there, non_blocking=True)
    t81lib.gemm_ternary(a, b.numpy(), c, M, N, K)
    assert np.array_equal(c, trits.astype(np.float32) @ there.cpu().numpy())  # small whole numbers: exact


def test_read_only_operands_leave_the_warning_filters_alone(lib_built, monkeypatch):
    """bytes and read-only arrays are taken without a warning, and without touching what other threads' warnings depend on."""
    import warnings

    import torch
    from t81lib_b200 import t81lib
    M, N, K = 8, 5, 96
    rng = np.random.default_rng(1)
    trits = rng.integers(-1, 2, (M, K)).astype(np.int8)
    b = rng.integers(-3, 4, (K, N)).astype(np.float32)
    from_numpy, seen = torch.from_numpy, []
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        filters = list(warnings.filters)
        monkeypatch.setattr(torch, "from_numpy", lambda a: (seen.append(warnings.filters == filters), from_numpy(a))[1])
        limbs = oracle.pack_trits_rowwise(trits)
        limbs.flags.writeable = False
        for a in (limbs, limbs.tobytes()):
            c = torch.zeros(M, N, device="cuda")  # not all numpy: the general path
            t81lib.gemm_ternary(a, b, c, M, N, K)
            assert np.array_equal(c.cpu().numpy(), trits.astype(np.float32) @ b)
    assert seen and all(seen)
