"""The RMS norms folded into the GEMM that dequantises weights in tensor memory (tpb200_w4_gemm_norm)."""
import ctypes
import re
from pathlib import Path

import pytest
import torch

from test_w4_gemm_gpu import _check, _nvfp4


def test_argument_struct_and_refusals():
    from turbopi_b200 import _lib
    header = (Path(__file__).resolve().parent.parent / "include" / "turbopi_b200.h").read_text()
    body = re.search(r"typedef struct\s*\{([^}]*)\}\s*tpb200_w4_norm_args\s*;", header, re.S).group(1)
    fields = [part.strip().split()[-1].lstrip("*") for d in body.split(";") if d.strip() for part in d.split(",")]
    assert fields == [f[0] for f in _lib.W4NormArgs._fields_]
    call, p = _lib.load().tpb200_w4_gemm_norm, 4096                       # refused before anything is read
    a = dict(x=p, ldx=1024, format=_lib.W4_NVFP4_TILED, w=p, out=p, out_dtype=_lib.BF16, ldo=512, M=4, N=512, K=1024)
    assert call(ctypes.byref(_lib.W4GemmArgs(**a)), None, None) == -1
    for change, norm, status in (({}, dict(in_sumsq=p, in_parts=6), -2), ({}, dict(in_sumsq=p + 4, in_parts=8), -3),
                                 (dict(N=520, ldo=520), dict(h_out=p, scale=p, out_sumsq=p), -2),
                                 ({}, dict(h_out=p, out_sumsq=p), -1), (dict(activation=1), dict(h_out=p, scale=p, out_sumsq=p), -4),
                                 (dict(format=_lib.W4_INT4_KBLOCK, w_scales=p), dict(in_sumsq=p, in_parts=8), -4)):
        st = call(ctypes.byref(_lib.W4GemmArgs(**{**a, **change})), ctypes.byref(_lib.W4NormArgs(**norm)), None)
        assert st == status, (change, norm)


def _args(x, b, sf, N, out, alpha, **kw):
    from turbopi_b200 import _lib, ops
    p = ops._ptr
    return _lib.W4GemmArgs(x=p(x), ldx=x.stride(0), format=_lib.W4_NVFP4_ROWMAJOR, w=p(b), w_pitch=b.stride(0), w_scales=p(sf),
                           alpha=alpha, out=p(out), out_dtype=ops._dt(out), ldo=out.stride(0), M=x.shape[0], N=N, K=x.shape[1], **kw)


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K", [(1, 128, 512), (50, 2560, 1024), (50, 8192, 1024), (33, 136, 2048), (130, 256, 4608)])
def test_norm_in_front(cuda_device, M, N, K):
    from turbopi_b200 import _lib, ops
    b, sf, w = _nvfp4(N, K, cuda_device, M + N + K)
    g = torch.Generator().manual_seed(M)
    x = torch.randn((M, K), generator=g).to(torch.bfloat16).to(cuda_device)
    ss = (torch.rand((M, K // 128), generator=g) * 256).to(cuda_device)
    shift, bias = torch.randn((2, N), generator=g).to(cuda_device)
    norm = _lib.W4NormArgs(in_sumsq=ops._ptr(ss), in_shift=ops._ptr(shift), in_parts=K // 128, in_eps=1e-6)
    y = torch.empty((M, N), dtype=torch.float32, device=cuda_device)
    ops._w4_gemm(_args(x, b, sf, N, y, 0.25, bias=ops._ptr(bias)), cuda_device, norm)
    r = torch.rsqrt(ss.double().sum(1, keepdim=True) / K + 1e-6)
    ref = 0.25 * r * (x.double() @ w.t())
    mag = r * (x.double().abs() @ w.abs().t())                            # rsqrtf and the sum of squares: 4 ulp of fp32
    _check(y, ref + (shift + bias).double(), mag + (shift.abs() + bias.abs()).double(), 2.0 ** -21)
    if N % 256 == 0:                                                      # the gated form sees the same two halves
        a = 0.25 / float(ref.std())
        norm.in_shift = ops._ptr(shift * a)
        gu, h = torch.empty((M, N), dtype=torch.bfloat16, device=cuda_device), torch.empty((M, N // 2), dtype=torch.bfloat16, device=cuda_device)
        keep = shift * a
        norm.in_shift = ops._ptr(keep)
        ops._w4_gemm(_args(x, b, sf, N, gu, a), cuda_device, norm)
        ops._w4_gemm(_args(x, b, sf, N, h, a, activation=_lib.ACT_SILU, gated=1), cuda_device, norm)
        gate, up = gu[:, :N // 2].double(), gu[:, N // 2:].double()
        want = torch.nn.functional.silu(gate).to(torch.bfloat16).double() * up
        # K is summed in another split: either projection may round to its neighbour, as the activation and the product
        assert bool(((h.double() - want).abs() <= 4 * 2.0 ** -8 * (want.abs() + 1.1 * (gate * up).abs()) + 1e-6).all())
    assert _lib.load().tpb200_device_error(0) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K", [(1, 128, 32), (50, 1024, 32), (50, 1024, 2048), (50, 1024, 4096), (130, 512, 1040)])
@pytest.mark.parametrize("with_res,with_gate", [(False, False), (True, False), (True, True)])
def test_residual_behind(cuda_device, M, N, K, with_res, with_gate):
    """The same bits as the linear, the residual and the scaling one after the other in bf16; in place on the residual."""
    from turbopi_b200 import _lib, ops
    b, sf, w = _nvfp4(N, K, cuda_device, M + N + K)
    g = torch.Generator().manual_seed(K)
    x, res = (torch.randn(s, generator=g).to(torch.bfloat16).to(cuda_device) for s in ((M, K), (M, N)))
    gate, scale = (torch.randn(N, generator=g).to(torch.bfloat16).to(cuda_device) for _ in range(2))
    alpha, p = 2.0 ** -9, ops._ptr
    y = torch.empty((M, N), dtype=torch.bfloat16, device=cuda_device)
    ops._w4_gemm(_args(x, b, sf, N, y, alpha), cuda_device)
    want = y * gate if with_gate else y
    want = res + want if with_res else want
    h, out = res.clone(), torch.empty_like(y)
    ss = torch.empty((M, N // 128), dtype=torch.float32, device=cuda_device)
    ops._w4_gemm(_args(x, b, sf, N, out, alpha), cuda_device,
                 _lib.W4NormArgs(res_in=p(h) if with_res else 0, gate=p(gate) if with_gate else 0, scale=p(scale), h_out=p(h),
                                 out_sumsq=p(ss)))
    assert torch.equal(h, want)
    assert torch.equal(out, (want.float() * (1 + scale.float())).to(torch.bfloat16))
    ref = want.double().square().view(M, -1, 128).sum(2)
    assert bool(((ss.double() - ref).abs() <= 128 * 2.0 ** -24 * ref).all())
    assert _lib.load().tpb200_device_error(0) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K", [(33, 8, 16), (65, 136, 2064), (100, 4304, 1152), (241, 264, 528), (712, 2560, 2176)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_tiles_stored_from_tensor_memory(cuda_device, M, N, K, dtype):
    """Unsplit plain tiles: ragged token and row tiles, a K whose last operand step has parts past its end, strided rows."""
    from turbopi_b200 import _lib, ops
    b, sf, w = _nvfp4(N, K, cuda_device, M + N + K)
    g = torch.Generator().manual_seed(N)
    x = torch.randn((M, K), generator=g).to(torch.bfloat16).to(cuda_device)
    bias = torch.randn(N, generator=g).to(cuda_device)
    out = torch.full((M + 1, N + 8), 7.0, dtype=dtype, device=cuda_device)
    ops.w4_gemm(x, b, N, _lib.W4_NVFP4_ROWMAJOR, sf, alpha=2.0 ** -8, bias=bias, activation=_lib.ACT_SILU, out=out[:M, :N])
    z = 2.0 ** -8 * (x.double() @ w.t()) + bias.double()
    mag = 2.0 ** -8 * (x.double().abs() @ w.abs().t()) + bias.double().abs()
    eps = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11, torch.float32: 2.0 ** -21}[dtype]
    # SiLU's slope is at most 1.1; the hardware exponential and division are good to 2^-20 of the result
    _check(out[:M, :N], torch.nn.functional.silu(z), 1.1 * mag + 1e-2, eps + 2.0 ** -20)
    assert bool((out[M] == 7).all()) and bool((out[:, N:] == 7).all())
    assert _lib.load().tpb200_device_error(0) == 0
