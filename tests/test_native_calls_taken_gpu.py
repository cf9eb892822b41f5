"""Which calls csrc/calls.cpp takes and which it leaves to the Python forms."""
import pytest
import torch

pytestmark = pytest.mark.gpu


class _Recorder:
    """Passes every call on and notes whether it was taken."""

    def __init__(self, native):
        self._native, self.taken = native, []

    def __getattr__(self, name):
        def call(*args):
            done = getattr(self._native, name)(*args)
            self.taken.append((name, done is not None))
            return done
        return call


@pytest.fixture
def recorder(cuda_device, monkeypatch):
    from turbopi_b200 import _lib
    r = _Recorder(_lib.native())
    monkeypatch.setattr(_lib, "_native", r)
    return r


def test_a_layer_without_inputs_is_refused(cuda_device, recorder):
    """in_features 0: no division by it on the way to the refusal."""
    from turbopi_b200._lib import TurboPiError
    from turbopi_b200.w4a16 import W4A16Linear
    layer = W4A16Linear(0, 8, device=cuda_device)
    with pytest.raises(TurboPiError):
        layer(torch.zeros(1, 0, dtype=torch.float16, device=cuda_device))
    assert recorder.taken == [("w4a16_linear", False)]


def _calls(device):
    """(name, plain call, calls of the same function that are left to the Python forms)"""
    from turbopi_b200 import _lib, ops
    from turbopi_b200.nvfp4_linear import NVFP4Linear
    from turbopi_b200.nvfp4_packed import NVFP4PackedLinear, NVFP4PackedMLP
    from turbopi_b200.w4a16 import W4A16Linear

    class Gemma(torch.nn.Module):
        def __init__(self):
            super().__init__()
            self.gate_proj, self.up_proj = (torch.nn.Linear(256, 512, bias=False) for _ in range(2))
            self.down_proj = torch.nn.Linear(512, 256)

    x = torch.randn(40, 256, device=device).to(torch.bfloat16)
    strided = torch.cat([x, x], 1)[:, :256]
    int4 = W4A16Linear.from_linear(torch.nn.Linear(256, 136).to(device))
    mlp = NVFP4PackedMLP.from_gemma_mlp(Gemma().to(device), gate_activation="gelu", fmt="nvfp4")
    w4a4 = NVFP4Linear.from_linear(torch.nn.Linear(256, 16384).to(device), use_mse_search=False)
    packed = NVFP4PackedLinear.from_linear(torch.nn.Linear(256, 512).to(device), fmt="nvfp4")
    rows = torch.randn(600, 64, device=device).to(torch.bfloat16)
    ws = ops.attention_workspace(600, 600, 64, 1, device)
    attend = lambda q, workspace=ws: ops.attention(q, rows, rows, torch.empty_like(rows), 0.125, None, workspace)     # noqa: E731
    return [
        ("w4a16_linear", lambda: int4(x), [lambda: int4(strided), lambda: int4(x.double())]),
        ("w4a16_linear", lambda: int4(x[:1].half()), [lambda: int4(strided[:2])]),
        ("mlp", lambda: mlp(x), []),
        ("nvfp4_linear", lambda: w4a4(torch.cat([x] * 8)), []),
        ("w4_gemm", lambda: packed(x), []),
        ("w4_gemm", lambda: ops.w4_gemm(strided, packed._tc_state()[0], 512, _lib.W4_NVFP4_TILED), []),
        ("quantize_fp8", lambda: ops.quantize_activation_to_fp8(x),
         [lambda: ops.quantize_activation_to_fp8(strided), lambda: ops.quantize_activation_to_fp8(x.float())]),
        ("attention", lambda: attend(rows), []),
    ]


@pytest.mark.parametrize("which", range(8))
def test_plain_calls_are_taken(cuda_device, recorder, which):
    name, plain, others = _calls(cuda_device)[which]
    recorder.taken.clear()
    plain()
    assert recorder.taken == [(name, True)]
    for other in others:
        recorder.taken.clear()
        other()
        assert recorder.taken == [(name, False)]
