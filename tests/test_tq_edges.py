"""The device transcoders between packed limbs and GGUF ternary blocks where rows end inside a block, a limb or a group of
three blocks, where several short rows share a warp's run or a row takes more than one, and on buffers that start on odd
addresses or between two 16-byte boundaries: bytes, against the numpy restatement."""

import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", ["TQ1_0", "TQ2_0"])
@pytest.mark.parametrize("rows,cols", [(1, 1), (3, 255), (2, 257), (5, 768), (4, 769), (3, 1537), (700, 2304)])
def test_transcoders(lib_built, rows, cols, fmt):
    from t81lib_b200 import ops
    rng = np.random.default_rng(rows + cols)
    trits = rng.integers(-1, 2, (rows, cols)).astype(np.int8)
    trits[0] = 0  # blocks without a non-zero trit have scale 0
    scale = rng.uniform(0.01, 2.0, rows).astype(np.float32)
    limbs, want = oracle.pack_trits_rowwise(trits), oracle.tq_encode(trits, scale, fmt)
    junk = rng.integers(0, 256, want.shape).astype(np.uint8)  # any bytes decode: TQ2_0 digit 3 reads as 2
    if fmt == "TQ1_0":
        junk = want
    back, d = oracle.tq_decode(junk, rows, cols, fmt)
    sd = torch.from_numpy(scale).cuda()
    for shift in (0, 1):
        def placed(a):
            buf = torch.empty(a.size + shift, dtype=torch.uint8, device="cuda")
            buf[shift:] = torch.from_numpy(np.ascontiguousarray(a).reshape(-1)).cuda()
            return buf[shift:].view(a.shape)
        assert np.array_equal(ops.packed_to_tq(placed(limbs), rows, cols, fmt, sd).cpu().numpy(), want)
        packed, scales = ops.tq_to_packed(placed(junk), rows, cols, fmt)
        assert np.array_equal(packed.cpu().numpy(), oracle.pack_trits_rowwise(back))
        assert np.array_equal(scales.cpu().numpy(), d, equal_nan=True)


@pytest.mark.parametrize("fmt", ["TQ1_0", "TQ2_0"])
@pytest.mark.parametrize("rows,cols", [(9500, 200), (28416, 256), (4801, 300), (2500, 2049), (3, 6145), (2, 12300), (5, 18433)])
def test_runs_of_rows_and_pieces(lib_built, rows, cols, fmt):
    """Rows of 1, 2 and 9 blocks taken together (the last run incomplete), rows of 25, 49 and 73 blocks in pieces of 24; limbs on
    8-byte boundaries, blocks on every even address of a 16-byte word."""
    from t81lib_b200 import ops
    rng = np.random.default_rng(rows + cols)
    trits = rng.integers(-1, 2, (rows, cols)).astype(np.int8)
    trits[rng.integers(0, rows, rows // 4 + 1), :256] = 0
    scale = rng.uniform(0.01, 2.0, rows).astype(np.float32)
    limbs, want = oracle.pack_trits_rowwise(trits), oracle.tq_encode(trits, scale, fmt)
    sd = torch.from_numpy(scale).cuda()
    for at_limbs, at_blocks in ((0, 0), (8, 2), (8, 14), (0, 8)):
        def placed(a, shift):
            buf = torch.empty(a.size + shift, dtype=torch.uint8, device="cuda")
            buf[shift:] = torch.from_numpy(np.ascontiguousarray(a).reshape(-1)).cuda()
            return buf[shift:].view(a.shape)
        assert np.array_equal(ops.packed_to_tq(placed(limbs, at_limbs), rows, cols, fmt, sd).cpu().numpy(), want)
        packed, scales = ops.tq_to_packed(placed(want, at_blocks), rows, cols, fmt)
        assert np.array_equal(packed.cpu().numpy(), limbs)
        assert np.array_equal(scales.cpu().numpy(), oracle.tq_decode(want, rows, cols, fmt)[1])
