"""Decode-sized products that read what peers stored, without a kernel's end between the stores and the reads: rows of every kind that
the kernel takes (whole 16-byte pieces, rows that are moved into place, float32).  The peer is this GPU itself: its second result is the
next layer's input and its flags are set by the kernel before, which has ended by the time the next one looks at them."""

import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", ["t2", "limbs"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("widths", [(520, 768, 512, 256), (775, 521, 1030, 193), (521, 769, 2, 100)])
@pytest.mark.parametrize("tokens", [1, 7, 16])
def test_chained_layers_behind_an_exchange(lib_built, fmt, dtype, widths, tokens):
    from t81lib_b200 import _capi, ops
    dev = torch.device("cuda", 0)
    words = torch.zeros(_capi.SYNC_WORDS, dtype=torch.int32, device=dev)

    class Flags:
        local_ptr = words.data_ptr()
        slot_ptrs = (ctypes.c_void_p * 1)(words.data_ptr() + 64)  # where "the peer" publishes: this rank's own slot

    gen = torch.Generator(device=dev).manual_seed(sum(widths) + tokens)
    x = torch.randint(-1, 2, (tokens, widths[0]), generator=gen, device=dev).to(dtype)
    layers = []
    for k, rows in zip(widths, widths[1:]):
        trits = torch.randint(-1, 2, (rows, k), generator=gen, device=dev).float()
        packed = ops.quantize_pack(trits, 0.5, "fixed")[0]
        layers.append((k, rows, trits, packed, ops.pack_t2(packed, rows, k), torch.empty(tokens, rows, device=dev, dtype=dtype),
                       torch.empty(tokens, rows, device=dev, dtype=dtype)))
    y = x
    for k, rows, _, packed, t2, out, peer in layers:
        if fmt == "t2":
            ops.gemm_trit_t2([t2], [rows], y, K=k, outs=[out], peers=[peer], sync=Flags)
        else:
            ops.gemm_trit(packed, y, M=rows, K=k, layout="nk", C=out, peers=[peer], sync=Flags)
        y = peer
    for _, _, trits, _, _, out, peer in layers:  # whole numbers below 2^24: exact sums in any order, one rounding
        assert torch.equal(out, (x.double() @ trits.double().t()).to(dtype))
        assert torch.equal(peer, out)
        x = peer
    assert int(words[1].item()) == len(layers)
    assert _capi.kernel_status(reset=True) == 0
