"""Rings whose slots are filled by copies and read by several groups of warps in turn.  A wait on an mbarrier tells phases by parity, so it is
right only for a waiter that knows the slot's use before to have landed.  The model: every copy lands at once but for one, which lands
when nobody can go on without it; whoever is let through to a chunk that has not landed reads something else."""

import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "t81lib_b200", "csrc")


def read_too_early(slots, groups, chunks, late, barriers=None):
    """The first chunk that a group takes before it has landed, or None.  Group g takes chunks g, g + groups, .., chunk k from slot k % slots,
    whose arrival barrier k % barriers (one per slot by default) tells, and hands the slot back; chunk k + slots is fetched once chunk
    k's slot is free."""
    barriers = barriers or slots
    landed, issued, freed, phases, at = set(), 0, set(), [0] * barriers, list(range(groups))
    while any(k < chunks for k in at):
        moved = False
        while issued < chunks and (issued < slots or issued - slots in freed):
            if issued != late:
                landed.add(issued)
                phases[issued % barriers] += 1
            issued += 1
            moved = True
        for g in range(groups):
            k = at[g]
            if k < chunks and phases[k % barriers] & 1 != (k // barriers) & 1:  # the barrier's wait for the parity of use k // barriers
                if k not in landed:
                    return k
                freed.add(k)
                at[g] += groups
                moved = True
        if not moved:
            assert late not in landed, "stuck"
            landed.add(late)
            phases[late % barriers] += 1
    return None


def test_model_finds_slots_that_change_hands():
    assert read_too_early(3, 2, 12, 0) == 3
    assert read_too_early(10, 4, 40, 2) is not None
    assert all(read_too_early(n, g, 40, late) is None for n, g in ((4, 2), (8, 4), (12, 4), (16, 8), (5, 1)) for late in range(40))


def test_packed_weights_of_the_tensor_core_product():
    source = open(os.path.join(CSRC, "gemm_trit_tc.cu")).read()
    slots = int(re.search(r"constexpr int RAW_STAGES = (\d+);", source).group(1))
    barriers = slots * int(re.search(r"constexpr int RAW_BARRIERS = (\d+) \* RAW_STAGES;", source).group(1))
    assert all(read_too_early(slots, 2, 24, late, barriers) is None for late in range(24))


# GemvLutParams in 32-bit words
ROW_WARPS, K_WARPS, LIMBS, STAGES = 57, 58, 59, 60


@pytest.mark.gpu
@pytest.mark.parametrize("fmt", ["t2", "limbs"])
@pytest.mark.parametrize("tokens", [1, 8, 16])
def test_rings_of_decode_sized_products(lib_built, tokens, fmt):
    import torch
    from _graph_nodes import capture, kernels
    from t81lib_b200 import _capi, ops
    reused = 0
    for rows, k in ((256, 14336), (600, 14330), (1024, 8200), (2048, 14336), (4096, 4096), (4096, 14336), (9216, 3072), (14336, 4096), (14336, 14336)):
        packed = torch.full((rows, (k + 47) // 48, 16), 13, dtype=torch.uint8, device="cuda")  # zero trits
        t2 = ops.pack_t2(packed, rows, k)
        x = torch.ones(tokens, k, device="cuda", dtype=torch.bfloat16)
        graph = capture(lambda: ops.linear_t2(t2, rows, x, k) if fmt == "t2" else ops.gemm_trit(packed, x, M=rows, K=k, layout="nk"))
        (words,) = [params(3) for name, params in kernels(graph) if "gemv_trit_lut_kernel" in name]
        stages, kw, chunks = int(words[STAGES]), int(words[K_WARPS]), int(words[LIMBS]) // 4
        assert 1 <= words[ROW_WARPS] <= 8 and 1 <= kw <= 8 and 1 <= stages <= chunks
        reused += stages < chunks
        assert stages == chunks or stages % kw == 0, (rows, k, stages, kw, chunks)
        assert all(read_too_early(stages, kw, chunks, late) is None for late in range(chunks))
    assert reused > 0
    assert _capi.kernel_status(reset=True) == 0
