"""A prompt token outside the embedding table is an error, never a plausible action."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@torch.no_grad()
@pytest.mark.parametrize("token", [1000, 2 ** 40, -1001])
@pytest.mark.parametrize("use_graph", [False, True])
def test_unknown_token(cuda_device, token, use_graph):
    from turbopi_b200 import _lib
    from turbopi_b200._lib import TurboPiError
    from turbopi_b200.pi05 import Pi05, Pi05Config
    cfg = Pi05Config(image_size=28, patch=14, vision_layers=1, vision_width=128, vision_mlp=272, vision_heads=2,
                     prefix_layers=1, width=256, mlp=512, text_len=24, vocab=1000, expert_layers=1, expert_width=128,
                     expert_mlp=256, max_seq=128)
    model = Pi05(cfg, cuda_device, seed=1)
    images, noise = torch.zeros((2, 28, 28, 3), dtype=torch.uint8), torch.ones(50, 32)
    good = torch.arange(-12, 12)
    good[:2] = torch.tensor([-1000, 999])
    run = lambda t: model.infer(images, t, noise, num_steps=2, use_graph=use_graph).clone()      # noqa: E731
    first = run(good)
    assert bool(first.isfinite().all()) and _lib.load().tpb200_device_error(0) == 0
    bad = good.clone()
    bad[5] = token
    with pytest.raises(TurboPiError):
        run(bad)
    assert bool(run(bad.to(cuda_device)).isnan().all())
    assert _lib.load().tpb200_device_error(1) == 401
    assert torch.equal(run(good.to(cuda_device)), first) and _lib.load().tpb200_device_error(0) == 0
