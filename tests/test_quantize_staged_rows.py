"""Quantise + pack where rows are staged in shared memory off 16-byte boundaries: every distance of a row from a boundary, rows that end
inside a group, first and last rows at the edges of their tensor, and the sizes at which one form takes over from the next.  Bytes
and scales against the oracle."""

import math

import numpy as np
import pytest
import torch

import oracle
from _graph_nodes import capture, kernels

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


# columns: less than a group, around a group, a chunk of 384 and four of them, and wide rows.  At 301 rows the row kernel has the narrow ones;
# the staged forms are met in test_form_by_size, from enough rows on.
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


# Which of the three forms takes a matrix, on both sides of each line of the rule, in rows an SM; and its bytes.  Off 16-byte boundaries: odd
# widths; "warps" and "teams" there are met with enough rows for them.
@pytest.mark.parametrize("per_sm,cols,dtype,rule,form", [
    (2, 1024, torch.float32, "absmean", "warp"), (2, 1540, torch.float32, "absmean", "ring"), (5, 1536, torch.float32, "absmean", "warp"),
    (4.9, 1536, torch.float32, "absmean", "ring"), (24, 2048, torch.float32, "absmean", "warp"), (23.9, 2048, torch.float32, "absmean", "ring"),
    (27, 2048, torch.float32, "absmean", "ring"), (32, 2048, torch.float32, "absmean", "warp"), (2, 2048, torch.float32, "fixed", "warp"),
    (5, 2304, torch.bfloat16, "absmean", "warp"), (4.9, 2304, torch.bfloat16, "absmean", "ring"), (3, 3072, torch.bfloat16, "fixed", "warp"),
    (2.9, 3072, torch.bfloat16, "fixed", "ring"), (23.9, 4096, torch.bfloat16, "fixed", "ring"), (2, 9600, torch.bfloat16, "absmean", "ring"),
    (4.9, 1025, torch.float32, "absmean", "row"), (5, 1025, torch.float32, "absmean", "warp"), (6, 1537, torch.float32, "absmean", "row"),
    (6.1, 1537, torch.float32, "absmean", "warp"), (6, 2049, torch.float32, "absmean", "row"), (6.1, 2049, torch.float32, "absmean", "ring"),
    (24, 2049, torch.float32, "absmean", "warp"), (27, 2305, torch.float32, "absmean", "ring"), (4.9, 4801, torch.float32, "absmean", "row"),
    (5, 4801, torch.float32, "absmean", "ring"), (2, 6001, torch.float32, "absmean", "ring"), (2, 5001, torch.float32, "fixed", "row"),
    (3.9, 1025, torch.float32, "fixed", "row"), (4, 1025, torch.float32, "fixed", "warp"), (6, 2305, torch.float32, "fixed", "row"), (6.1, 2305, torch.float32, "fixed", "warp"),
    (4.9, 513, torch.bfloat16, "absmean", "row"), (5, 513, torch.bfloat16, "absmean", "warp"), (3.3, 2049, torch.bfloat16, "absmean", "row"),
    (3.4, 2049, torch.bfloat16, "absmean", "ring"), (3.3, 513, torch.bfloat16, "fixed", "row"), (3.4, 513, torch.bfloat16, "fixed", "warp"),
    (3.4, 513, torch.float32, "fixed", "warp"), (8, 2049, torch.bfloat16, "absmean", "warp"), (8, 2305, torch.bfloat16, "absmean", "ring"),
    (24, 3077, torch.bfloat16, "absmean", "warp"), (2, 4097, torch.bfloat16, "absmean", "ring"), (8, 4097, torch.bfloat16, "fixed", "ring"),
    # where six teams' rows no longer fit, nor 24 rows beside each other, nor two slots for each of these: slots of 19200, 9472 and 4736 bytes
    (2, 4800, torch.float32, "absmean", "ring6"), (2, 4804, torch.float32, "absmean", "ring4"), (2, 9600, torch.bfloat16, "fixed", "ring6"),
    (2, 9608, torch.bfloat16, "fixed", "ring4"), (5, 4791, torch.float32, "absmean", "ring6"), (5, 4793, torch.float32, "absmean", "ring4"),
    (2, 9585, torch.bfloat16, "absmean", "ring6"), (2, 9587, torch.bfloat16, "absmean", "ring4"), (24, 2359, torch.float32, "absmean", "warp"),
    (24, 2361, torch.float32, "absmean", "ring6"), (24, 4721, torch.bfloat16, "absmean", "warp"), (24, 4723, torch.bfloat16, "absmean", "ring6"),
    (8, 1175, torch.float32, "absmean", "warp"), (8, 1177, torch.float32, "absmean", "warp"), (4, 2353, torch.bfloat16, "fixed", "warp"),
    (4, 2355, torch.bfloat16, "fixed", "ring6"), (8, 2355, torch.bfloat16, "fixed", "warp"),
    (2, 14457, torch.float32, "absmean", "row"), (2, 14455, torch.float32, "absmean", "ring4"),
    (4, 2049, torch.float16, "fixed", "warp"), (8, 3077, torch.float16, "fixed", "warp"), (1.9, 4097, torch.bfloat16, "absmean", "row")])
def test_form_by_size(lib_built, per_sm, cols, dtype, rule, form):
    from t81lib_b200 import ops
    rows = math.ceil(per_sm * torch.cuda.get_device_properties(0).multi_processor_count - 1e-9)
    gen = torch.Generator(device="cuda").manual_seed(cols + rows)
    w = (torch.randn(rows, cols, generator=gen, device="cuda") * (0.02 if rule == "absmean" else 0.5)).to(dtype)
    names = [name for name, _ in kernels(capture(lambda: ops.quantize_pack(w, 0.45, rule)))]
    kind, teams = form[:4].rstrip("0123456789"), form[4:]
    assert len(names) == 1 and f"quantize_pack_{kind}_kernel" in names[0] and (not teams or f"Li{teams}E" in names[0]), names
    _check(w, rule)
