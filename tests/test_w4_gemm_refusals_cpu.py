"""Refusals of the dequantising GEMM that come before any CUDA call (fake aligned pointers, no device needed)."""
import ctypes

import pytest

from turbopi_b200 import _lib

LINEAR = dict(x=256, ldx=512, format=_lib.W4_NVFP4_TILED, w=256, alpha=1.0, out=256, out_dtype=_lib.F32, ldo=32, M=50, N=32, K=512)


@pytest.mark.parametrize("norm", [dict(copy_out=256), dict(in_shift=256), dict(in_shift=256, in_parts=4, copy_out=256)])
def test_parts_of_a_folded_norm_without_its_sums(norm):
    """The result would leave without the shift, or without its copy."""
    call = _lib.load().tpb200_w4_gemm_norm
    assert call(ctypes.byref(_lib.W4GemmArgs(**LINEAR)), ctypes.byref(_lib.W4NormArgs(**norm)), None) == -1
