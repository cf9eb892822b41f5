"""The tiled images of NVFP4PackedLinear / NVFP4PackedMLP follow their weights: written in place, replaced, moved, and under
captured graphs, whose image must outlive every later call."""
import copy
import io
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu

# the routes on an image: 1 and 8 tokens (the MLP's two launches; the linear's GEMV from 5 on), 40 (dequantising GEMM), and
# token counts above its limit (three-piece GEMM)
TOKENS = [1, 8, 40, 200]


@pytest.fixture(params=["linear", "mlp", "mlp_pieces"])
def kind(request):
    return request.param


def _pair(kind, device, monkeypatch):
    from turbopi_b200 import nvfp4_packed
    if kind == "mlp_pieces":                                # the routes above the size limit
        monkeypatch.setattr(nvfp4_packed, "_dense_is_faster", lambda *a: False)
    torch.manual_seed(7)
    mods = []
    for _ in range(2):
        if kind == "linear":
            mods.append(nvfp4_packed.NVFP4PackedLinear.from_linear(torch.nn.Linear(128, 256, device=device), fmt="nvfp4"))
        else:
            p = {n: torch.nn.Linear(*s, bias=False, device=device)
                 for n, s in (("gate_proj", (128, 256)), ("up_proj", (128, 256)), ("down_proj", (256, 128)))}
            mods.append(nvfp4_packed.NVFP4PackedMLP.from_gemma_mlp(SimpleNamespace(**p), gate_activation="gelu", fmt="nvfp4"))
    return mods


def _linears(m):
    return [x for x in m.modules() if hasattr(x, "weight_packed")]


def _load(dst, src):
    for a, b in zip(_linears(dst), _linears(src)):
        a.weight_packed.copy_(b.weight_packed)
        a.weight_scales.copy_(b.weight_scales)
        a.global_scale = b.global_scale
        if a.bias is not None:
            a.bias.copy_(b.bias)


def _scribble(device):
    torch.cuda.synchronize()
    for n in (1 << 12, 1 << 16, 1 << 20):
        held = [torch.full((n,), 255, dtype=torch.uint8, device=device) for _ in range(64)]
        del held


@torch.no_grad()
@pytest.mark.parametrize("T", TOKENS)
def test_capture_after_a_warm_up(cuda_device, monkeypatch, kind, T):
    """Warm up, capture, write, one eager call: the replay reads an image that is still there, and the new weights."""
    a, b = _pair(kind, cuda_device, monkeypatch)
    for m, n in zip(_linears(a), _linears(b)):
        n.global_scale = m.global_scale                     # a scalar argument, which a capture keeps
    x = torch.randn(T, 128, device=cuda_device).to(torch.bfloat16)
    old, want = a(x), b(x)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = a(x)
    graph.replay()
    assert torch.equal(y, old)
    for _ in range(2):
        _load(a, b)
        assert torch.equal(a(x), want) and not torch.equal(old, want)
        _scribble(cuda_device)
        graph.replay()
        assert torch.equal(y, want)


@torch.no_grad()
@pytest.mark.parametrize("T", TOKENS)
@pytest.mark.parametrize("warm", [False, True])
def test_capture_without_a_current_image(cuda_device, monkeypatch, kind, T, warm):
    """A first call that is captured, or one after weights were written: the tiling is part of the capture."""
    a, b = _pair(kind, cuda_device, monkeypatch)
    for m, n in zip(_linears(a), _linears(b)):
        n.global_scale = m.global_scale
    x = torch.randn(T, 128, device=cuda_device).to(torch.bfloat16)
    want = b(x)
    if warm:
        a(x)
        for m in _linears(a):                               # written, no eager call: the image is behind
            m.weight_packed.copy_(m.weight_packed.clone())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = a(x)
    old = a(x)
    graph.replay()
    assert torch.equal(y, old)
    _load(a, b)
    _scribble(cuda_device)
    graph.replay()
    assert torch.equal(y, want) and not torch.equal(old, want)


@torch.no_grad()
@pytest.mark.parametrize("T", TOKENS)
def test_moved_replaced_copied(cuda_device, monkeypatch, kind, T):
    a, b = _pair(kind, cuda_device, monkeypatch)
    x = torch.randn(T, 128, device=cuda_device).to(torch.bfloat16)
    before, want = a(x), b(x)
    c = copy.deepcopy(a)
    store = io.BytesIO()
    torch.save(a, store)
    host = copy.deepcopy(b).cpu()
    a.cpu()
    _load(a, host)
    a.to(cuda_device)                                       # the caching allocator may hand the freed addresses out again
    assert torch.equal(a(x), want)
    for m, n in zip(_linears(a), _linears(c)):              # and does, where the old buffers go first
        codes, scales = n.weight_packed.cpu(), n.weight_scales.cpu()
        m.global_scale = n.global_scale
        address = m.weight_packed.data_ptr()
        m.weight_packed = None
        m.weight_packed = codes.to(cuda_device)
        m.weight_scales = None
        m.weight_scales = scales.to(cuda_device)
        if m.bias is not None:
            m.bias.copy_(n.bias)
    assert m.weight_packed.data_ptr() == address
    assert torch.equal(a(x), before)
    assert torch.equal(c(x), before)
    for m, n in zip(_linears(c), _linears(b)):
        m.weight_packed, m.weight_scales, m.global_scale = n.weight_packed.clone(), n.weight_scales.clone(), n.global_scale
        if m.bias is not None:
            m.bias.copy_(n.bias)
    assert torch.equal(c(x), want)
    store.seek(0)
    d = torch.load(store, weights_only=False)
    assert torch.equal(d(x), before)
    for m in _linears(d):
        m.weight_packed.data = m.weight_packed.data.clone()     # the same object on other memory
    assert torch.equal(d(x), before)


@torch.no_grad()
@pytest.mark.parametrize("H,I", [(2048, 14144), (2048, 14208), (2048, 16384)])
def test_one_token_inside_a_capture(cuda_device, H, I):
    """Either side of the size from which a captured single token takes the GEMVs: both against float64."""
    from turbopi_b200.nvfp4_packed import NVFP4PackedMLP, unpack_nvfp4
    g = torch.Generator(device=cuda_device).manual_seed(I)
    w = {n: torch.randn(s, generator=g, device=cuda_device) * 0.02
         for n, s in (("gate_proj", (I, H)), ("up_proj", (I, H)), ("down_proj", (H, I)))}
    lin = {n: torch.nn.Linear(v.shape[1], v.shape[0], bias=False, device="meta") for n, v in w.items()}
    for n, l in lin.items():
        l.weight = torch.nn.Parameter(w[n], requires_grad=False)
    mlp = NVFP4PackedMLP.from_gemma_mlp(SimpleNamespace(**lin), gate_activation="gelu", fmt="nvfp4")
    x = torch.randn((1, H), generator=g, device=cuda_device).to(torch.bfloat16)
    eager = mlp(x)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = mlp(x)
    graph.replay()

    def dense(m):
        s = m.weight_scales.view(torch.float8_e4m3fn).double().repeat_interleave(16, 1)
        return unpack_nvfp4(m.weight_packed, m.out_features, m.in_features).double() * s * m.global_scale

    gate, up = x.double() @ dense(mlp.gate_proj).t(), x.double() @ dense(mlp.up_proj).t()
    h = torch.nn.functional.gelu(gate, approximate="tanh") * up
    wd = dense(mlp.down_proj)
    ref = h @ wd.t()
    # gate, up, the activation and the product round to bf16, each by 2^-8 / sqrt(3) of its value in the mean square: together
    # less than 4 * 2^-9 of the 2-norm of the terms; five times that, and the last rounding
    tol = 5 * 4 * 2.0 ** -9 * ((h * h) @ (wd * wd).t()).sqrt() + 2.0 ** -8 * ref.abs()
    for out in (eager, y):
        assert bool(((out.double() - ref).abs() <= tol).all())
    assert torch.equal(eager, y) == (2 * I * H < 58_000_000)


@torch.no_grad()
def test_scratch_of_a_capture(cuda_device, monkeypatch):
    """Operand buffers and split-K scratch: those a captured graph uses outlive calls with other token counts; those made
    inside a capture, whose zeros only a replay writes, serve no other call."""
    a, b = _pair("mlp_pieces", cuda_device, monkeypatch)
    xs = {T: torch.randn(T, 128, device=cuda_device).to(torch.bfloat16) for T in (1, 200, 300, 17, 33, 65, 130, 260, 390)}
    for m, n in zip(_linears(a), _linears(b)):
        n.global_scale = m.global_scale
    _load(b, a)
    want = {T: b(x) for T, x in xs.items()}
    a(xs[1])
    a(xs[200])
    graphs, ys = {}, {}
    for T in (200, 300):                                    # warmed up, and not
        graphs[T] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graphs[T]):
            ys[T] = a(xs[T])
    for m in _linears(a):
        assert all(key[0] != 300 for key in m.__dict__.get("_operands", {}))
    assert torch.equal(a(xs[300]), want[300])
    for T in (17, 33, 65, 130, 260, 390):
        assert torch.equal(a(xs[T]), want[T])
    _scribble(cuda_device)
    for _ in range(2):
        for T, graph in graphs.items():
            graph.replay()
            assert torch.equal(ys[T], want[T])
    from turbopi_b200 import _lib
    assert _lib.load().tpb200_device_error(0) == 0
