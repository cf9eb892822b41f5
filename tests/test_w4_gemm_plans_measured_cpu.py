"""Launch plans of csrc/w4_gemm.cu against measured times, and the operand ring with several units per step, on the host."""
import ctypes
import itertools

import pytest

from turbopi_b200 import _lib

INT4, NVFP4, NONE, PDL = _lib.W4_INT4_KBLOCK, _lib.W4_NVFP4_TILED, _lib.FLAG_NONE, _lib.FLAG_PDL

# weights, M, N, K, the best of all plans on a B200 (us; INT4 as plain launches, NVFP4 in a chain of dependent ones), and every plan
# within 10 % of it: (tokens per tile, K ranges, CTAs per SM)
MEASURED = [
    (INT4, 712, 2048, 16384, 49.2, [(192, 2, 1), (240, 2, 1)]),
    (INT4, 712, 16384, 2048, 51.4, [(240, 1, 1)]),
    (INT4, 397, 2048, 16384, 31.5, [(208, 4, 1)]),
    (INT4, 397, 16384, 2048, 33.4, [(208, 1, 1)]),
    (INT4, 705, 2048, 16384, 49.3, [(192, 2, 1), (240, 2, 1)]),
    (INT4, 720, 2048, 16384, 48.9, [(192, 2, 1), (240, 2, 1)]),
    (INT4, 50, 2048, 2048, 7.8, [(32, 4, 1), (32, 4, 2), (64, 4, 1), (64, 4, 2)]),
    (INT4, 64, 8192, 2048, 11.7, [(64, 2, 1), (64, 2, 2), (64, 4, 2)]),
    (INT4, 1000, 2048, 16384, 55.3, [(256, 2, 1)]),
    (INT4, 239, 12448, 1408, 14.8, [(240, 1, 1)]),
    (INT4, 157, 2432, 2432, 11.6, [(64, 2, 1), (64, 2, 2), (80, 2, 1), (160, 4, 1)]),
    (INT4, 75, 7224, 2176, 11.8, [(80, 2, 1)]),
    (NVFP4, 50, 1024, 4096, 5.4, [(32, 4, 1), (32, 8, 2), (64, 8, 2)]),
    (NVFP4, 343, 2048, 2048, 7.4, [(96, 1, 1)]),
    (NVFP4, 1, 32768, 2048, 15.7, [(16, 1, 2)]),
    (NVFP4, 712, 2048, 16384, 39.6, [(192, 2, 1)]),
    (NVFP4, 50, 8192, 1024, 5.8, [(64, 1, 1), (64, 2, 2)]),
    (NVFP4, 4, 8576, 2048, 6.7, [(16, 1, 1), (16, 2, 2)]),
]


def _describe(M, N, K, fmt, flags=NONE, sms=148):
    info = _lib.W4GemmLaunchInfo()
    assert _lib.load().tpb200_w4_gemm_describe(M, N, K, fmt, flags, sms, ctypes.byref(info)) == 0
    return info


@pytest.mark.parametrize("fmt,M,N,K,best_us,plans", MEASURED)
def test_the_chosen_plan_is_among_the_fast_ones(fmt, M, N, K, best_us, plans):
    p = _describe(M, N, K, fmt)
    assert (p.tokens_per_tile, p.splits, p.ctas_per_sm) in plans, best_us
    q = _describe(M, N, K, fmt, PDL)                 # the same bits under every launch flag
    assert bytes(p) == bytes(q)


@pytest.mark.parametrize("M,N,K,ranges", [(50, 2560, 1024, 2), (50, 1024, 2048, 4), (50, 8192, 1024, 1), (50, 1024, 4096, 4), (50, 32, 1024, 2),
                                          (10, 1024, 1024, 2), (3, 2560, 1024, 2), (10, 8192, 1024, 1), (512, 3456, 1152, 1),
                                          (512, 1152, 4304, 2), (256, 1152, 4304, 2), (712, 2560, 2048, 1), (343, 2048, 2048, 1)])
def test_sums_of_the_pipeline_keep_their_order(M, N, K, ranges):
    """K ranges are added in rank order: another number of them rounds every action of the pipeline differently."""
    assert _describe(M, N, K, NVFP4).splits == ranges


def test_plans_at_the_limits():
    """One of everything, the most tokens and SM counts far from 148: a plan that the kernel can run."""
    for M, N, K, fmt, sms in itertools.product([1, 65535 * 256], [8, 1 << 20], [16, 256, 1 << 20], [NVFP4, INT4], [1, 20, 148, 1000]):
        p = _describe(M, N, K, fmt, NONE, sms)
        assert p.tokens_per_tile % 16 == 0 and 16 <= p.tokens_per_tile <= (128 if p.ctas_per_sm == 2 else 256)
        assert p.splits in (1, 2, 4, 8) and p.splits <= p.k_blocks and -(-M // p.tokens_per_tile) <= 65535
        assert p.smem_bytes <= 226 * 1024 and p.weight_slots >= 1 and p.step_slots >= 1


@pytest.mark.parametrize("fmt", [NVFP4, INT4])
def test_rings_with_several_units_per_step(fmt):
    """The replay of the kernel's loop: group g takes the units g, g + groups, ... of `parts` 64-K parts each, units_per_step of
    them make an operand step, zero units fill the last one."""
    tokens = [1, 17, 33, 50, 64, 65, 96, 100, 129, 200, 256, 397, 712, 1000]
    rows = [8, 128, 512, 1024, 2048, 2560, 4304, 8192, 16384]
    seen = set()
    for M, N, K in itertools.product(tokens, rows, [16, 64, 592, 1024, 1152, 2048, 4304, 8192, 9024, 16384]):
        p = _describe(M, N, K, fmt)
        for rank in range(p.splits):
            lo, hi = rank * p.k_blocks // p.splits, (rank + 1) * p.k_blocks // p.splits
            seen.add((p.groups, p.parts, p.units_per_step, p.weight_slots, p.step_slots, hi - lo, min(hi * 4, p.k_steps) - lo * 4))
    assert any(merge == 2 and live % (parts * merge) for _, parts, merge, _, _, _, live in seen)       # a padded last step
    assert any(merge == 2 and parts == 2 for _, parts, merge, _, _, _, _ in seen)
    for at in seen:
        groups, parts, merge, w_slots, s_slots, blocks, live = at
        steps = -(-live // (parts * merge))
        in_step, arrivals = [0] * steps, [0] * blocks
        for g in range(groups):
            visited = set()
            for i in range(g, steps * merge, groups):
                step, block = i // merge, i * parts >> 2
                assert block < blocks, at                        # a padded unit waits for a block that does arrive
                assert block < w_slots or block in visited or block - w_slots in visited, at
                visited.add(block)
                arrivals[block] += 4
                in_step[step] += 1
                # a wait on `empty` asks for the MMAs of step - s_slots; the one of the unit before covered the step before that
                # in the slot, whose phase has the same parity
                assert step < 2 * s_slots or (i >= groups and (i - groups) // merge - s_slots >= step - 2 * s_slots), at
        assert all(n == merge for n in in_step) and all(n == 16 // parts for n in arrivals[:-1]), at
