"""Attention where the finite mask value lies on every key: the mean of the values, keys past the end not among them, whatever
form the launch takes."""
import pytest
import torch

pytestmark = pytest.mark.gpu

MASKED = -2.3819763e38          # the additive mask of the reference (pi0_pytorch.py:185-188)


def _inputs(R, S, D, device):
    g = torch.Generator().manual_seed(R + S + D)
    q, k, v = (torch.randn(n, D, generator=g).to(torch.bfloat16).to(device) for n in (R, S, S))
    return q, k, v + 1, torch.full((S,), MASKED, device=device).to(torch.bfloat16)


@pytest.mark.parametrize("R,S,D", [(40, 100, 256),          # one ragged key tile
                                   (40, 300, 256),          # three, merged inside a cluster
                                   (40, 1100, 72),          # nine: too many for a cluster
                                   (8200, 300, 64), (8200, 200, 256),   # two key tiles per CTA, the second ragged / alone
                                   (8200, 600, 128)])
def test_every_key_masked(cuda_device, R, S, D):
    from turbopi_b200 import _lib, ops
    q, k, v, bias = _inputs(R, S, D, cuda_device)
    out = torch.empty_like(q)
    ops.attention(q, k, v, out, D ** -0.5, bias)
    # the weights are equal and exact; the mean is summed in fp32 and rounded to bf16 once
    assert bool(((out.double() - v.double().mean(0)).abs() <= 2.0 ** -8 * v.double().abs().mean(0)).all())
    assert _lib.load().tpb200_device_error(0) == 0


@pytest.mark.parametrize("L,S,heads", [(50, 100, 8), (50, 300, 8), (1000, 300, 8)])
def test_fused_operand_of_masked_keys(cuda_device, L, S, heads):
    """attention(quant=) is still attention followed by the row kernel."""
    from turbopi_b200 import _lib, ops
    D = 256
    q, k, v, bias = _inputs(L * heads, S, D, cuda_device)
    out = torch.empty_like(q)
    ops.attention(q, k, v, out, D ** -0.5, bias)
    two_step, fused = (ops.QuantBuf(L, heads * D, 3, cuda_device, tiled=True) for _ in range(2))
    ops.rowop(_lib.ROW_NONE, out.view(L, heads * D), heads * D, two_step)
    ops.attention(q, k, v, None, D ** -0.5, bias, quant=fused, rows_per_token=heads)
    assert torch.equal(fused.packed, two_step.packed) and torch.equal(fused.row_scale, two_step.row_scale)
