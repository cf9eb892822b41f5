"""The calls of csrc/calls.cpp against the Python forms they stand in for: the same bits, and the other forms left alone."""
import pytest
import torch

pytestmark = pytest.mark.gpu


class _None:
    """Recognises nothing: every call takes its Python form."""

    def __getattr__(self, name):
        return lambda *args: None


def _both(call, monkeypatch):
    from turbopi_b200 import _lib
    taken = call()
    with monkeypatch.context() as m:
        m.setattr(_lib, "_native", _None())
        python = call()
    a, b = (v if isinstance(v, tuple) else (v,) for v in (taken, python))
    assert len(a) == len(b)
    for x, y in zip(a, b):
        assert x.dtype == y.dtype and x.shape == y.shape and torch.equal(x, y)


@pytest.mark.parametrize("shape", [(1, 256), (3, 5, 256), (256,), (40, 256), (2, 20, 256)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32, torch.float64])
@pytest.mark.parametrize("bias", [False, True])
def test_int4_linear(cuda_device, monkeypatch, shape, dtype, bias):
    from turbopi_b200.w4a16 import W4A16Linear
    layer = W4A16Linear.from_linear(torch.nn.Linear(256, 136, bias=bias).to(cuda_device))
    x = torch.randn(shape, device=cuda_device).to(dtype)
    for v in (x, x.expand(2, *shape) if dtype == torch.float16 else x, x.flip(-1)):
        if v.dim() >= 2 or shape != (256,):
            _both(lambda: layer(v), monkeypatch)                                   # noqa: B023


@pytest.mark.parametrize("T", [1, 17, 50, 300])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_packed_mlp_and_linears(cuda_device, monkeypatch, T, dtype):
    from turbopi_b200 import ops
    from turbopi_b200.nvfp4_linear import NVFP4Linear
    from turbopi_b200.nvfp4_packed import NVFP4PackedLinear, NVFP4PackedMLP

    class Gemma(torch.nn.Module):
        def __init__(self):
            super().__init__()
            self.gate_proj, self.up_proj = (torch.nn.Linear(256, 512, bias=False) for _ in range(2))
            self.down_proj = torch.nn.Linear(512, 256, bias=False)

    mlp = NVFP4PackedMLP.from_gemma_mlp(Gemma().to(cuda_device), gate_activation="gelu", fmt="nvfp4")
    lin = NVFP4PackedLinear.from_linear(torch.nn.Linear(256, 512).to(cuda_device), activation="gelu", fmt="nvfp4")
    w4a4 = NVFP4Linear.from_linear(torch.nn.Linear(256, 16384).to(cuda_device), use_mse_search=False)
    x = torch.randn(T, 256, device=cuda_device).to(dtype)
    for v in (x, x.view(1, T, 256), torch.cat([x, x], 1)[:, :256]):
        _both(lambda: mlp(v), monkeypatch)                                         # noqa: B023
        _both(lambda: lin(v), monkeypatch)                                         # noqa: B023
        _both(lambda: w4a4(v), monkeypatch)                                        # noqa: B023
    _both(lambda: ops.quantize_activation_to_fp8(x), monkeypatch)


def test_attention_forms_and_refusals(cuda_device, monkeypatch):
    from turbopi_b200 import ops
    from turbopi_b200._lib import TurboPiError
    x = torch.randn(2, 100, 3, 4, 64, device=cuda_device).to(torch.bfloat16)
    q, k, v = x.permute(2, 0, 3, 1, 4)
    ws = ops.attention_workspace(100, 100, 64, 8, cuda_device)
    _both(lambda: ops.attention(q, k, v, torch.empty(2, 100, 4, 64, dtype=q.dtype, device=cuda_device).permute(0, 2, 1, 3), 0.125,
                                None, ws), monkeypatch)
    flat = x.view(-1, 64)[:600].clone()
    bias = torch.zeros(600, device=cuda_device).to(torch.bfloat16)
    ws = ops.attention_workspace(600, 600, 64, 1, cuda_device)
    _both(lambda: ops.attention(flat, flat, flat, torch.empty_like(flat), 0.125, bias, ws), monkeypatch)
    for args in ((flat.float(), flat, flat, flat, 0.125, bias, ws), (flat, flat, flat[:5], flat, 0.125, bias, ws),
                 (flat, flat, flat, torch.empty_like(flat), 0.125, bias, ws[:1024]), (flat.cpu(), flat, flat, flat, 0.125, bias, ws)):
        with pytest.raises(TurboPiError):
            ops.attention(*args)
