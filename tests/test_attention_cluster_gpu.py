"""Attention with the key tiles of a row tile merged inside a thread-block cluster, against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [8, 64, 72, 128, 200, 256])
@pytest.mark.parametrize("R,S", [(1, 129), (400, 762), (129, 256), (127, 385), (1500, 300), (130, 1024), (130, 1025)])
def test_against_float64(cuda_device, R, S, D):
    """2 to 8 key tiles, ragged rows and keys, every cut of head_dim, widths it cannot be cut for; 1025 keys are past it."""
    from turbopi_b200 import _lib, ops
    g = torch.Generator().manual_seed(R + S + D)
    q, k, v = (torch.randn(n, D, generator=g).to(torch.bfloat16).to(cuda_device) for n in (R, S, S))
    bias = torch.where(torch.rand(S, generator=g) < 0.2, -2.3819763e38, 0.0)
    bias[:min(S, 130)] = -2.3819763e38 if S > 256 else 0.0               # a whole key tile masked
    bias[-1] = 0.0
    bias = bias.to(torch.bfloat16).to(cuda_device)
    out = torch.full((R + 1, D), 7.0, dtype=torch.bfloat16, device=cuda_device)
    ops.attention(q, k, v, out[:R], D ** -0.5, bias)
    p = torch.softmax(q.double() @ k.double().t() * D ** -0.5 + bias.double(), -1)
    ref, mag = p @ v.double(), p @ v.double().abs()
    # probabilities relative to a tile's maximum are rounded to bf16 (2^-9 each, in the sum as well), the result once more
    assert bool(((out[:R].double() - ref).abs() <= 2.0 ** -8 * (mag + ref.abs()) + 1e-5).all())
    assert bool((out[R] == 7).all()) and _lib.load().tpb200_device_error(0) == 0


def test_every_key_masked(cuda_device):
    """The finite mask value on all keys: the mean of the values, keys past the end not among them."""
    from turbopi_b200 import ops
    q, k, v = (torch.randn(n, 256, device=cuda_device).to(torch.bfloat16) for n in (40, 300, 300))
    bias = torch.full((300,), -2.3819763e38, device=cuda_device).to(torch.bfloat16)
    out = torch.empty_like(q)
    ops.attention(q, k, v, out, 256 ** -0.5, bias)
    assert bool(((out.double() - v.double().mean(0)).abs() <= 2.0 ** -8 * v.double().abs().mean(0)).all())


def test_strided_groups_and_repeats(cuda_device):
    """Groups as strided views, and the same bits from launches that overlap under programmatic dependent launch."""
    from turbopi_b200 import ops
    x = torch.randn(2, 200, 3, 4, 64, device=cuda_device).to(torch.bfloat16)
    q, k, v = x.permute(2, 0, 3, 1, 4)
    o = torch.empty(2, 200, 4, 64, dtype=torch.bfloat16, device=cuda_device)
    ops.attention(q, k, v, o.permute(0, 2, 1, 3), 0.125)
    ref = torch.softmax(q.double() @ k.double().transpose(-1, -2) * 0.125, -1) @ v.double()
    assert bool(((o.permute(0, 2, 1, 3).double() - ref).abs() <= 2.0 ** -7 * (ref.abs() + v.double().abs().mean(-2, keepdim=True))).all())
    outs = [torch.empty_like(o) for _ in range(8)]
    with ops.launch_flags(ops.FLAG_PDL):
        for y in outs:
            ops.attention(q, k, v, y.permute(0, 2, 1, 3), 0.125)
    assert all(torch.equal(y, o) for y in outs)
