"""Modules whose bias or buffers are not where they were registered (replicas, pruning, parametrisations): forward finds them.
No GPU: a recorder stands in for the native calls, and the modules' own refusal of CPU tensors ends the call behind it."""
import pytest
import torch
from torch.nn.utils import parametrize, prune

from turbopi_b200 import _lib
from turbopi_b200.nvfp4_packed import NVFP4PackedLinear, NVFP4PackedMLP
from turbopi_b200.w4a16 import W4A16Linear


class _Same(torch.nn.Module):
    def forward(self, t):
        return t


def _replica(layer):
    """What nn.DataParallel makes of a module: no registered parameters, the copies plain attributes."""
    r = layer._replicate_for_data_parallel()
    for name, p in layer._parameters.items():
        setattr(r, name, None if p is None else p.detach().clone())
    return r


def _pruned(layer):
    return prune.identity(layer, "bias")


def _parametrised_bias(layer):
    parametrize.register_parametrization(layer, "bias", _Same())
    return layer


def _parametrised_scales(layer):
    parametrize.register_parametrization(layer, "scales" if hasattr(layer, "scales") else "weight_scales", _Same())
    return layer


CHANGES = [_replica, _pruned, _parametrised_bias, _parametrised_scales]


@pytest.mark.parametrize("change", CHANGES)
def test_w4a16_linear(monkeypatch, change):
    layer = W4A16Linear.from_linear(torch.nn.Linear(64, 16))
    bias, scales, seen = layer.bias.detach().clone(), layer.scales.clone(), []

    class Recorder:
        def w4a16_linear(self, *args):
            seen.append(args)
            return "done"
    monkeypatch.setattr(_lib, "_native", Recorder())
    assert change(layer)(torch.zeros(1, 64)) == "done"
    assert torch.equal(seen[0][3], bias) and torch.equal(seen[0][2], scales)


@pytest.mark.parametrize("change", CHANGES)
def test_packed_linear_and_mlp(change):
    """On the CPU the packed modules end in a refusal; the attributes are found before it."""
    lin = NVFP4PackedLinear.from_linear(torch.nn.Linear(64, 16), fmt="nvfp4")
    with pytest.raises(_lib.TurboPiError):
        change(lin)(torch.zeros(1, 64))

    class Gemma(torch.nn.Module):
        def __init__(self):
            super().__init__()
            self.gate_proj, self.up_proj = (torch.nn.Linear(64, 128) for _ in range(2))
            self.down_proj = torch.nn.Linear(128, 64)
    mlp = NVFP4PackedMLP.from_gemma_mlp(Gemma(), gate_activation="gelu", fmt="nvfp4")
    for name in ("gate_proj", "up_proj", "down_proj"):
        setattr(mlp, name, change(getattr(mlp, name)))
    with pytest.raises(_lib.TurboPiError):
        mlp(torch.zeros(1, 64))


@pytest.mark.parametrize("change", CHANGES[:3])
def test_packed_mlp_hands_the_bias_on(monkeypatch, change):
    class Gemma(torch.nn.Module):
        def __init__(self):
            super().__init__()
            self.gate_proj, self.up_proj = (torch.nn.Linear(64, 128, bias=False) for _ in range(2))
            self.down_proj = torch.nn.Linear(128, 64)
    mlp = NVFP4PackedMLP.from_gemma_mlp(Gemma(), gate_activation="gelu", fmt="nvfp4")
    bias, seen = mlp.down_proj.bias.detach().clone(), []
    if change is _replica:
        for name in ("gate_proj", "up_proj"):
            setattr(mlp, name, change(getattr(mlp, name)))
    mlp.down_proj = change(mlp.down_proj)

    class Recorder:
        def mlp(self, x, gate_up, down, d_bias, *rest):
            seen.append(d_bias)
            return torch.zeros(1, 64, dtype=torch.bfloat16)
    monkeypatch.setattr(_lib, "_native", Recorder())
    monkeypatch.setattr(NVFP4PackedLinear, "tensor_core_ready", lambda self: True)
    monkeypatch.setattr(NVFP4PackedMLP, "_tiled", lambda self, *a: (None, None, True))
    monkeypatch.setattr(NVFP4PackedLinear, "_tiled", lambda self, *a: (None, None, True))
    assert mlp(torch.zeros(1, 64)).shape == (1, 64) and torch.equal(seen[0], bias)
