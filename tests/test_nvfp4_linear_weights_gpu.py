"""NVFP4Linear multiplies with the weights its buffers hold when the kernels run: written in place, through `.data`, moved
off the GPU and back, or changed between a capture and its replays."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# either side of the rule on output tiles, and the ragged edges of the 128 x 256 form
FEATURES = [256, 25600, 25352]


def _pair(device, features, K=288):
    from turbopi_b200.nvfp4_linear import TILED_MIN_TILES, NVFP4Linear
    torch.manual_seed(features)
    a, b = (NVFP4Linear.from_linear(torch.nn.Linear(K, features, bias=True, device=device), use_mse_search=False) for _ in range(2))
    assert (a._tiles(8) >= TILED_MIN_TILES) == (features > 256)
    return a, b, torch.randn(8, K, device=device).to(torch.bfloat16)


def _load(dst, src, through_data=False):
    for name, t in [*dst.named_buffers(), *dst.named_parameters()]:
        (t.data if through_data else t).copy_(dict([*src.named_buffers(), *src.named_parameters()])[name])


@torch.no_grad()
@pytest.mark.parametrize("features", FEATURES)
def test_written_behind_the_version_counter(cuda_device, features):
    a, b, x = _pair(cuda_device, features)
    before, want = a(x), b(x)
    _load(a, b, through_data=True)
    assert torch.equal(a(x), want) and not torch.equal(before, want)


@torch.no_grad()
@pytest.mark.parametrize("features", FEATURES)
def test_moved_off_the_gpu_loaded_and_moved_back(cuda_device, features):
    a, b, x = _pair(cuda_device, features)
    want = b(x)
    a(x)
    for _ in range(3):                      # the caching allocator hands the freed addresses out again
        a.cpu()
        _load(a, b.cpu())
        a.to(cuda_device)
        assert torch.equal(a(x), want)
        b.to(cuda_device)


@torch.no_grad()
@pytest.mark.parametrize("features", FEATURES)
@pytest.mark.parametrize("eager_between", [False, True])
def test_replay_of_a_capture_sees_later_writes(cuda_device, features, eager_between):
    a, b, x = _pair(cuda_device, features)
    a(x)                                    # the warm-up call before a capture
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = a(x)
    want = b(x)
    _load(a, b)
    if eager_between:
        assert torch.equal(a(x), want)
        scribble = [torch.full((1 << 20,), 255, dtype=torch.uint8, device=cuda_device) for _ in range(64)]
        del scribble
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, want)


@torch.no_grad()
def test_first_pass_is_like_the_next_and_nothing_is_kept(cuda_device):
    a, _, x = _pair(cuda_device, 25600)
    held = torch.cuda.memory_allocated()
    first = a(x)
    del first
    assert torch.cuda.memory_allocated() == held
    with torch.inference_mode():
        c = type(a).from_linear(torch.nn.Linear(288, 25600, device=cuda_device), use_mse_search=False)
        assert torch.equal(c(x), c(x))


@pytest.mark.parametrize("M,N,K", [(1, 8, 16), (8, 264, 272), (129, 128, 272), (129, 136, 1040), (200, 1000, 1040), (712, 4096, 2048),
                                   (300, 20480, 512)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_row_major_weights_under_wide_tiles(cuda_device, M, N, K, dtype):
    """The same bits as from the tiled weight image, which holds the same codes and scales."""
    from turbopi_b200 import _lib, ops
    g = torch.Generator().manual_seed(M + N + K)
    b = torch.zeros((N, ops.packed_pitch(K)), dtype=torch.uint8)
    b[:, :K // 2] = torch.randint(0, 256, (N, K // 2), generator=g, dtype=torch.uint8)
    b, sf = b.to(cuda_device), ops.swizzle_scales(torch.randint(0, 0x7F, (N, K // 16), generator=g, dtype=torch.uint8)).to(cuda_device)
    x = torch.randn((M, K), generator=g).to(dtype).to(cuda_device)
    bias = torch.randn(N, generator=g).to(cuda_device)
    for out_dtype in (torch.bfloat16, torch.float32):
        want = ops.nvfp4_linear_tiled(x, ops.tile_weights(b, sf, N, K), N, 0.25, bias, _lib.ACT_GELU, out_dtype)
        assert torch.equal(ops.nvfp4_linear_tiled(x, b, N, 0.25, bias, _lib.ACT_GELU, out_dtype, b_sf=sf), want)
    assert _lib.load().tpb200_device_error(0) == 0
