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
