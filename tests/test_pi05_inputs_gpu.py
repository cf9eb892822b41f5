"""The pipeline's input kernels, and the Euler update in the last linear's epilogue."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("images,size,patch,pitch", [(1, 14, 14, 588), (2, 56, 14, 592), (2, 224, 14, 592), (3, 8, 2, 16)])
def test_patches_equal_the_elementwise_ops(cuda_device, images, size, patch, pitch):
    from turbopi_b200 import _lib, ops
    x = torch.randint(0, 256, (images, size, size, 3), dtype=torch.uint8, device=cuda_device)
    n = size // patch
    out = torch.full((images * n * n, pitch), 7.0, dtype=torch.bfloat16, device=cuda_device)
    assert ops._run(x, _lib.load().tpb200_pi05_patches, x.data_ptr(), out.data_ptr(), images, size, patch, pitch, 0) == 0
    ref = x.float().div_(127.5).sub_(1.0).view(images, n, patch, n, patch, 3).permute(0, 1, 3, 5, 2, 4).reshape(images * n * n, -1)
    assert torch.equal(out[:, :ref.shape[1]], ref.to(torch.bfloat16)) and bool((out[:, ref.shape[1]:] == 7).all())


@pytest.mark.parametrize("tokens,width", [(1, 2), (87, 512), (200, 2048)])
def test_embedding_equals_the_elementwise_ops(cuda_device, tokens, width):
    from turbopi_b200 import _lib, ops
    table = torch.randn(300, width, device=cuda_device).to(torch.bfloat16)
    idx = torch.randint(-300, 300, (tokens,), device=cuda_device)
    out = torch.empty((tokens, width), dtype=torch.bfloat16, device=cuda_device)
    call = lambda i: ops._run(table, _lib.load().tpb200_pi05_embed, i.data_ptr(), table.data_ptr(), out.data_ptr(), tokens, 300,  # noqa: E731
                              width, math.sqrt(width), 0)
    assert call(idx) == 0
    assert torch.equal(out, table[idx] * math.sqrt(width))
    assert call(torch.full_like(idx, 300)) == 0 and bool((out == 0).all())
    assert _lib.load().tpb200_pi05_embed(idx.data_ptr(), table.data_ptr(), out.data_ptr(), 0, 300, width, 1.0, 0, None) == -2


@pytest.mark.parametrize("M,N,K", [(1, 32, 1024), (50, 32, 1024), (33, 136, 512)])
def test_update_and_copy(cuda_device, M, N, K):
    from test_w4_gemm_gpu import _check, _nvfp4
    from test_w4_gemm_norm_gpu import _args
    from turbopi_b200 import _lib, ops
    b, sf, w = _nvfp4(N, K, cuda_device, M + N)
    g = torch.Generator().manual_seed(M)
    x = torch.randn((M, K), generator=g).to(torch.bfloat16).to(cuda_device)
    ss, shift, y0 = (torch.rand(s, generator=g).to(cuda_device) for s in ((M, K // 128), (N,), (M, N)))
    y, copy = y0.clone(), torch.empty((M, N), dtype=torch.bfloat16, device=cuda_device)
    norm = _lib.W4NormArgs(in_sumsq=ops._ptr(ss), in_shift=ops._ptr(shift), in_parts=K // 128, in_eps=1e-6, copy_out=ops._ptr(copy))
    ops._w4_gemm(_args(x, b, sf, N, y, -2.0 ** -9, beta=1.0), cuda_device, norm)
    r = torch.rsqrt(ss.double().sum(1, keepdim=True) / K + 1e-6) * 2.0 ** -9
    _check(y, y0.double() + shift.double() - r * (x.double() @ w.t()), r * (x.double().abs() @ w.abs().t()) + 2, 2.0 ** -21)
    assert torch.equal(copy, y.to(torch.bfloat16))
