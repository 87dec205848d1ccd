"""Quantise + pack where rows are staged in shared memory off 16-byte boundaries: every distance of a row from a boundary, rows that end
inside a group, first and last rows at the edges of their tensor, and the sizes at which one form takes over from the next.  Bytes
and scales against the oracle."""

import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


def _check(view, rule, threshold=0.45):
    from t81lib_b200 import _capi, ops
    packed, scale = ops.quantize_pack(view, threshold, rule)
    host = np.ascontiguousarray(view.float().cpu().numpy())
    if rule == "fixed":
        want = oracle.pack_dense_matrix(host, threshold)
    else:
        want, want_scale = oracle.pack_dense_matrix_absmean(host, threshold)
        assert np.array_equal(scale.cpu().numpy(), want_scale, equal_nan=True)
    assert np.array_equal(packed.cpu().numpy(), want)
    assert _capi.kernel_status(reset=True) == 0


# columns: less than a group, around a group, a chunk of 384 and four of them; then rows of which 24 just fit beside each other and
# just do not, and the same for the ring's six teams and four (bf16: 4720 / 4730, 9640 / 9650, 28900; fp32: half)
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("cols", [1, 3, 5, 47, 383, 385, 1537, 2355, 2369, 4705, 4737, 9633, 9665, 14465])
@pytest.mark.parametrize("rule", ["fixed", "absmean"])
def test_rows_off_boundaries(lib_built, dtype, cols, rule):
    rows = 301  # distances of the rows from a boundary: all there are
    gen = torch.Generator(device="cuda").manual_seed(cols)
    w = (torch.randn(rows, cols, generator=gen, device="cuda") * (0.02 if rule == "absmean" else 0.5)).to(dtype)
    w[7] = 0.0
    if cols > 3:
        w[11, 2] = float("nan")
        w[12, cols - 1] = float("inf")
    _check(w, rule)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("cols,ld,offset", [(100, 103, 1), (1000, 1008, 3), (2001, 2001, 5), (5003, 5009, 7), (4096, 4104, 8), (6, 6, 1), (7, 9, 2)])
def test_views(lib_built, dtype, cols, ld, offset):
    """Rows with gaps between them, in a buffer that starts and ends with the view: nothing outside it is looked at (it holds other values
    right up to the view, and those in the gaps are infinite)."""
    rows = 300
    gen = torch.Generator(device="cuda").manual_seed(cols)
    buffer = torch.full((offset + (rows - 1) * ld + cols,), float("inf"), device="cuda").to(dtype)
    view = buffer[offset:].as_strided((rows, cols), (ld, 1))
    view.copy_(torch.randn(rows, cols, generator=gen, device="cuda") * 0.02)
    _check(view, "absmean")
    _check(view, "fixed", 0.0)
