"""Weights written in place after the first inference: what the pipeline keeps of products of them follows, also for a graph
captured before the write."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _model(device, expert_width):
    from turbopi_b200.pi05 import Pi05, Pi05Config
    cfg = Pi05Config(image_size=28, patch=14, vision_layers=1, vision_width=128, vision_mlp=272, vision_heads=2,
                     prefix_layers=2, width=256, mlp=512, text_len=24, vocab=1000, expert_layers=2, expert_width=expert_width,
                     expert_mlp=256, max_seq=128)
    return Pi05(cfg, device, seed=1)


WRITES = {
    "qkv": lambda m: m.expert[1]["qkv"].b, "qkv scales": lambda m: m.expert[0]["qkv"].sf, "gate_up": lambda m: m.expert[0]["gate_up"].b,
    "action_out": lambda m: m.action_out.b, "action_out bias": lambda m: m.action_out.bias, "positions": lambda m: m.pos_emb,
    "ada": lambda m: m.ada_dense.b,
}


def _moved(w):
    """Other values of the same kind: rows reversed, images of bytes turned by 512, vectors by one."""
    return w.flip(0) if w.dim() > 1 else w.roll(512 if w.dtype == torch.uint8 else 1)


@torch.no_grad()
@pytest.mark.parametrize("expert_width", [128, 512])           # row kernels / the norms in the linears' epilogues
@pytest.mark.parametrize("use_graph", [False, True])
@pytest.mark.parametrize("what", WRITES)
def test_written_weights_are_followed(cuda_device, expert_width, use_graph, what):
    from turbopi_b200.pi05 import Pi05
    model = _model(cuda_device, expert_width)
    g = torch.Generator().manual_seed(2)
    images = torch.randint(0, 256, (2, 28, 28, 3), generator=g, dtype=torch.uint8)
    tokens, noise = torch.randint(0, 1000, (24,), generator=g), torch.randn(50, 32, generator=g)
    run = lambda m: m.infer(images, tokens, noise, num_steps=2, use_graph=use_graph).clone()     # noqa: E731
    before = run(model)
    w = WRITES[what](model)
    w.copy_(_moved(w))
    after = run(model)
    fresh = run(Pi05.sharing_weights(model))                   # the same weights, tables of its own
    assert torch.equal(after, fresh) and not torch.equal(after, before)
    w.data.copy_(_moved(w.data))      # a write that no version counter sees
    model.weights_changed()
    assert torch.equal(run(model), run(Pi05.sharing_weights(model)))


@torch.no_grad()
def test_a_capture_after_a_write_holds_the_new_tables(cuda_device):
    from turbopi_b200 import ops
    from turbopi_b200.pi05 import Pi05
    model = _model(cuda_device, 512)
    args = (torch.zeros((2, 28, 28, 3), dtype=torch.uint8), torch.arange(24), torch.ones(50, 32), 2)
    model.infer(*args, use_graph=False)
    model.expert[0]["qkv"].b.copy_(model.expert[0]["qkv"].b.flip(0))
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph), ops.launch_flags(model.launch_flags):
        model.denoise_loop(2)
    graph.replay()
    assert torch.equal(model.actions, Pi05.sharing_weights(model).infer(*args, use_graph=False))
    assert torch.equal(model.infer(*args, use_graph=False), model.actions)
