"""The rings of csrc/w4_gemm.cu, replayed on the host for the launches its planner chooses: which blocks and steps each
group of dequantising warps goes through, in the kernel's order."""
import ctypes
import itertools

import pytest

from turbopi_b200 import _lib


def _plan(M, N, K, sms=148):
    info = _lib.W4GemmPlanInfo()
    assert _lib.load().tpb200_w4_gemm_plan(M, N, K, sms, ctypes.byref(info)) == 0
    return info


def _launches(sms):
    """Distinct (plan, weight blocks, steps) of a CTA over the sizes the GEMM is used for."""
    seen = set()
    tokens = [1, 4, 16, 17, 33, 48, 49, 50, 64, 65, 96, 100, 128, 129, 200, 256, 257, 397, 500, 712, 1000]
    rows = [8, 128, 264, 512, 1024, 1152, 2048, 2560, 4096, 4304, 8192, 16384, 32768]
    for M, N, K in itertools.product(tokens, rows, [16, 64, 256, 592, 1024, 1152, 1536, 2048, 4096, 4304, 8192, 16384]):
        p = _plan(M, N, K, sms)
        for rank in range(p.splits):
            lo, hi = rank * p.k_blocks // p.splits, (rank + 1) * p.k_blocks // p.splits
            steps = (min(hi * 4, p.k_steps) - lo * 4 + p.parts - 1) // p.parts
            seen.add((p.groups, p.parts, p.weight_slots, p.step_slots, hi - lo, steps))
    return seen


@pytest.mark.parametrize("sms", [148, 132, 40])
def test_a_group_waits_for_every_use_of_the_slots_it_reads(sms):
    """A parity wait tells a phase from the one before it only.  So a group that reads block j out of a slot must have
    waited for block j - slots, the slot's previous content; and a slot is handed back by the four warps of every group
    that reads it, 16 / parts arrivals in all."""
    launches = _launches(sms)
    assert any(parts == 2 and groups == 4 and blocks > slots for groups, parts, slots, _, blocks, _ in launches)
    for groups, parts, w_slots, s_slots, blocks, steps in launches:
        readers = [[] for _ in range(blocks)]
        for g in range(groups):
            visited = set()
            for i in range(g, steps, groups):
                j = i * parts >> 2
                assert j < w_slots or j in visited or j - w_slots in visited, (groups, parts, w_slots, blocks, steps)
                visited.add(j)
                readers[j].append(g)
        assert all(len(r) * 4 == 16 // parts for r in readers[:-1])
        # operand steps: before step i a group has waited for the MMAs of step i - groups - slots, and they complete in
        # order; that covers step i - 2 * slots, the phase that its next wait could mistake for the one it asks for
        assert s_slots >= min(groups, steps), (groups, parts, s_slots, steps)


def test_plan_refuses_what_the_launch_refuses():
    assert _lib.load().tpb200_w4_gemm_plan(1, 8, 16, 148, None) == -1
    info = _lib.W4GemmPlanInfo()
    for M, N, K, sms in ((0, 8, 16, 148), (1, 0, 16, 148), (1, 8, 0, 148), (1, 8, 16, 0)):
        assert _lib.load().tpb200_w4_gemm_plan(M, N, K, sms, ctypes.byref(info)) == -2
