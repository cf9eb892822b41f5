"""Rules by which launches share tensor memory, checked where a GPU run could only hang: in the sources and in the launch plans."""
import ctypes
import itertools
import re
from pathlib import Path

import pytest

from turbopi_b200 import _lib

CSRC = Path(__file__).resolve().parent.parent / "turbopi_b200" / "csrc"


def _functions(text):
    """Bodies of the device functions, comments removed (a body starts at a line that ends in `{` in the first column's scope)."""
    text = re.sub(r"//[^\n]*", "", text)
    return re.findall(r"^[^\s#}][^\n;]*\([^;{}]*\)\s*\{\n(.*?)^\}", text, re.S | re.M)


@pytest.mark.parametrize("source", sorted(p.name for p in CSRC.glob("*.cu") if "tmem_alloc(" in p.read_text()))
def test_dependents_are_let_in_behind_the_allocation(source):
    """A kernel that lets the next launch in before its own allocation is complete can lose the columns to a CTA that keeps
    them until this kernel ends."""
    checked = 0
    for body in _functions((CSRC / source).read_text()):
        if "tmem_alloc(" not in body or "pdl_launch_dependents()" not in body:
            continue
        allocated = body.index("tmem_alloc(")
        barrier = body.index("__syncthreads()", allocated)
        assert body.index("pdl_launch_dependents()") > barrier, source
        checked += 1
    assert checked >= {"attention.cu": 2}.get(source, 1), source


SM_BYTES, CTA_BYTES = 228 * 1024, 1024          # shared memory of an SM, and what of it the system keeps per CTA


def _check_sharing(launches):
    """`launches`: (columns, dynamic shared memory) of launches whose CTAs wait for one another while they hold tensor memory,
    in any two streams: no mix of them that fits an SM's shared memory wants more than its 512 columns."""
    assert {c for c, _ in launches} <= {256, 512} and max(b for _, b in launches) <= 227 * 1024
    least = {c: min(b for cols, b in launches if cols == c) + CTA_BYTES for c in {c for c, _ in launches}}
    half, whole = least.get(256, SM_BYTES), least.get(512, SM_BYTES)
    assert 3 * half > SM_BYTES and whole + min(half, whole) > SM_BYTES, least


def test_waiting_launches_never_share_an_sm_beyond_its_tensor_memory():
    lib, launches = _lib.load(), set()
    for sms, M, N, K in itertools.product([148, 132], [1, 16, 33, 50, 64, 100, 128, 200, 397, 712, 1000], [128, 1024, 2560, 4304, 8192, 32768],
                                          [256, 1024, 1152, 2048, 4096, 16384]):
        for fmt, flags in itertools.product([_lib.W4_NVFP4_TILED, _lib.W4_INT4_KBLOCK], [_lib.FLAG_NONE, _lib.FLAG_PDL]):
            info = _lib.W4GemmLaunchInfo()
            assert lib.tpb200_w4_gemm_describe(M, N, K, fmt, flags, sms, ctypes.byref(info)) == 0
            if info.splits > 1:
                launches.add((info.tmem_columns, info.smem_bytes))
    assert {c for c, _ in launches} == {256, 512}
    for rows, keys, dim in itertools.product([1, 50, 400, 1500, 2744, 5696], [129, 256, 300, 762, 1024, 1100], [8, 64, 72, 128, 192, 200, 256]):
        info = _lib.AttentionLaunchInfo()
        assert lib.tpb200_attention_describe(rows, keys, dim, 1, 0, ctypes.byref(info)) == 0
        if info.cluster_ctas:
            launches.add((info.tmem_columns, info.smem_bytes))
    _check_sharing(launches)


def test_describe_refuses_what_the_launch_refuses():
    lib, w4, at = _lib.load(), _lib.W4GemmLaunchInfo(), _lib.AttentionLaunchInfo()
    assert lib.tpb200_w4_gemm_describe(1, 8, 16, 1, 0, 148, None) == -1 and lib.tpb200_attention_describe(1, 1, 8, 1, 0, None) == -1
    for M, N, K, fmt, flags, sms, status in ((0, 8, 16, 1, 0, 148, -2), (1, 0, 16, 1, 0, 148, -2), (1, 8, 0, 1, 0, 148, -2),
                                             (1, 8, 16, 1, 0, 0, -2), (1, 8, 16, -1, 0, 148, -4), (1, 8, 16, 9, 0, 148, -4),
                                             (1, 8, 16, 1, 2, 148, -4)):
        assert lib.tpb200_w4_gemm_describe(M, N, K, fmt, flags, sms, ctypes.byref(w4)) == status
    for rows, keys, dim in ((0, 1, 8), (1, 0, 8), (1, 1, 12), (1, 1, 264)):
        assert lib.tpb200_attention_describe(rows, keys, dim, 1, 0, ctypes.byref(at)) == -2
