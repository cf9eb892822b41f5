"""The GEMM that dequantises 4-bit weights into tensor memory, against float64 on the dequantised weights."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _nvfp4(N, K, device, seed):
    """(codes [N, pitch], scale atoms, dequantised float64 [N, K])"""
    from turbopi_b200 import ops
    from turbopi_b200.nvfp4_packed import unpack_nvfp4
    g = torch.Generator().manual_seed(seed)
    codes = torch.randint(0, 256, (N, K // 2), generator=g, dtype=torch.uint8)
    scales = torch.randint(0, 0x7F, (N, K // 16), generator=g, dtype=torch.uint8)      # every finite UE4M3 value
    w = unpack_nvfp4(codes, N, K).double() * scales.view(torch.float8_e4m3fn).double().repeat_interleave(16, 1)
    b = torch.zeros((N, ops.packed_pitch(K)), dtype=torch.uint8)
    b[:, :K // 2] = codes
    return b.to(device), ops.swizzle_scales(scales).to(device), w.to(device)


def _check(y, ref, mag, out_eps):
    """|y - ref| <= half an ulp of the output type + fp32 accumulation (mag = sum |x w|, K terms in any order)"""
    err = (y.double() - ref).abs()
    assert bool((err <= out_eps * ref.abs() + 2e-6 * mag + 1e-30).all()), float((err / (ref.abs() + mag)).max())


@pytest.mark.parametrize("M,N,K", [(1, 8, 16), (17, 128, 64), (50, 1024, 4096), (50, 2560, 1024), (64, 136, 272),
                                   (128, 1152, 592), (129, 4304, 1152), (256, 264, 4304), (257, 128, 2048), (712, 2048, 2048)])
@pytest.mark.parametrize("tiled", [False, True])
def test_nvfp4(cuda_device, M, N, K, tiled):
    from turbopi_b200 import _lib, ops
    b, sf, w = _nvfp4(N, K, cuda_device, M + N + K)
    x = torch.randn((M, K + 8), generator=torch.Generator().manual_seed(M)).to(torch.bfloat16).to(cuda_device)[:, :K]
    bias = torch.randn(N, generator=torch.Generator().manual_seed(N)).to(cuda_device)
    ref, mag = x.double() @ w.t(), x.double().abs() @ w.abs().t()
    weight = (ops.tile_weights(b, sf, N, K), N, _lib.W4_NVFP4_TILED) if tiled else (b, N, _lib.W4_NVFP4_ROWMAJOR, sf)
    y = ops.w4_gemm(x, *weight, alpha=0.25, out_dtype=torch.float32)
    _check(y, 0.25 * ref, mag, 2.0 ** -22)
    y = ops.w4_gemm(x, *weight, alpha=0.25, bias=bias)
    _check(y, 0.25 * ref + bias.double(), mag, 2.0 ** -8)
    out = torch.randn((M, N + 8), device=cuda_device).to(torch.float16)
    old = out.clone()
    ops.w4_gemm(x, *weight, alpha=2.0 ** -8, beta=0.5, out=out[:, :N])
    _check(out[:, :N], 2.0 ** -8 * ref + 0.5 * old[:, :N].double(), 2.0 ** -8 * mag + old[:, :N].double().abs(), 2.0 ** -10)
    assert torch.equal(out[:, N:], old[:, N:])
    assert _lib.load().tpb200_device_error(0) == 0


@pytest.mark.parametrize("M,I,K", [(1, 64, 64), (50, 4096, 1024), (130, 192, 304), (300, 448, 1024)])
@pytest.mark.parametrize("tiled", [False, True])
def test_gated(cuda_device, M, I, K, tiled):
    from turbopi_b200 import _lib, ops
    b, sf, w = _nvfp4(2 * I, K, cuda_device, M + I + K)
    x = torch.randn((M, K), generator=torch.Generator().manual_seed(M)).to(torch.bfloat16).to(cuda_device)
    a = 1.0 / float((x.double() @ w.t()).std())
    weight = (ops.tile_weights(b, sf, 2 * I, K), 2 * I, _lib.W4_NVFP4_TILED) if tiled else (b, 2 * I, _lib.W4_NVFP4_ROWMAJOR, sf)
    gu = ops.w4_gemm(x, *weight, alpha=a)                                  # checked above
    for act, fn in ((_lib.ACT_GELU, lambda v: torch.nn.functional.gelu(v, approximate="tanh")),
                    (_lib.ACT_SILU, torch.nn.functional.silu)):
        y = ops.w4_gemm(x, *weight, alpha=a, activation=act, gated=True).double()
        g = fn(gu[:, :I].double())
        ref = g.to(torch.bfloat16).double() * gu[:, I:].double()
        # the activation may round to the neighbouring bf16 (2^-8 of it), the product rounds once more (2^-9)
        assert bool(((y - ref).abs() <= 1.6 * 2.0 ** -8 * ref.abs() + 1e-6).all())


@pytest.mark.parametrize("M", [1, 50, 177])
def test_qkv_epilogue_equals_the_piecewise_gemm(cuda_device, M):
    """Same projection, rotation and cache rows as the e2m1-piece GEMM's epilogue, up to its activation rounding."""
    from turbopi_b200 import _lib, ops
    K, q_dim, N = 1024, 2048, 2560
    b, sf, _ = _nvfp4(N, K, cuda_device, 3)
    x = torch.randn((M, K), generator=torch.Generator().manual_seed(M)).to(torch.bfloat16).to(cuda_device)
    cos, sin = ops.rope_tables(1024, device=cuda_device)
    pos = torch.randperm(1024, generator=torch.Generator().manual_seed(1))[:M].to(torch.int32).to(cuda_device)
    kv = torch.zeros((4, M + 2, 256), dtype=torch.bfloat16, device=cuda_device)
    ref = ops.fused_qkv_rope_append(x, b, sf, q_dim, kv[0], kv[1], pos, cos, sin, 2.0 ** -9, 4)
    q = torch.empty_like(ref)
    p = ops._ptr
    ops._w4_gemm(_lib.W4GemmArgs(x=p(x), ldx=K, format=_lib.W4_NVFP4_ROWMAJOR, w=p(b), w_pitch=b.stride(0), w_scales=p(sf),
                                 alpha=2.0 ** -9, out=p(q), out_dtype=_lib.BF16, ldo=q_dim, M=M, N=N, K=K, qkv_q_dim=q_dim,
                                 qkv_k_rows=p(kv[2]), qkv_v_rows=p(kv[3]), qkv_positions=p(pos), qkv_rope_cos=p(cos),
                                 qkv_rope_sin=p(sin)), cuda_device)
    for a, c in ((q, ref), (kv[2], kv[0]), (kv[3], kv[1])):
        # four pieces leave 3e-3 of a row's largest entry; two more bf16 roundings
        assert float((a.double() - c.double()).abs().max()) <= 8e-3 * float(c.double().abs().max())
    assert float((kv[2:, M:]).abs().max()) == 0


@pytest.mark.parametrize("M", [1, 50, 177])
@pytest.mark.parametrize("tiled", [False, True])
def test_qkv_epilogue_against_float64(cuda_device, M, tiled):
    from turbopi_b200 import _lib, ops
    K, q_dim, N = 1024, 2048, 2560
    b, sf, w = _nvfp4(N, K, cuda_device, M)
    x = torch.randn((M, K), generator=torch.Generator().manual_seed(M)).to(torch.bfloat16).to(cuda_device)
    cos, sin = ops.rope_tables(1024, device=cuda_device)
    pos = torch.randperm(1024, generator=torch.Generator().manual_seed(1))[:M].to(torch.int32).to(cuda_device)
    kv = torch.zeros((2, M + 2, 256), dtype=torch.bfloat16, device=cuda_device)
    q = torch.empty((M, q_dim), dtype=torch.bfloat16, device=cuda_device)
    p, alpha = ops._ptr, 2.0 ** -9
    image = ops.tile_weights(b, sf, N, K)
    weight = (dict(format=_lib.W4_NVFP4_TILED, w=p(image)) if tiled
              else dict(format=_lib.W4_NVFP4_ROWMAJOR, w=p(b), w_pitch=b.stride(0), w_scales=p(sf)))
    ops._w4_gemm(_lib.W4GemmArgs(x=p(x), ldx=K, alpha=alpha, out=p(q), out_dtype=_lib.BF16, ldo=q_dim, M=M, N=N, K=K,
                                 qkv_q_dim=q_dim, qkv_k_rows=p(kv[0]), qkv_v_rows=p(kv[1]), qkv_positions=p(pos),
                                 qkv_rope_cos=p(cos), qkv_rope_sin=p(sin), **weight), cuda_device)
    rows = torch.empty_like(w)
    rows[ops.qkv_tile_permutation(q_dim).to(cuda_device)] = w              # the kernel's rows are permuted by tile
    ref, mag = alpha * (x.double() @ rows.t()), alpha * (x.double().abs() @ rows.abs().t())
    c, s = cos[pos.long()].double()[:, None], sin[pos.long()].double()[:, None]
    heads, hm = ref[:, :q_dim + 256].view(M, -1, 2, 128), mag[:, :q_dim + 256].view(M, -1, 2, 128)
    lo, hi, ml, mh = heads[:, :, 0], heads[:, :, 1], hm[:, :, 0], hm[:, :, 1]
    got = torch.cat([q, kv[0, :M]], 1).double().view(M, -1, 2, 128)
    u = 2.0 ** -8                                                          # unit roundoff of bf16 (eight significant bits)
    for y, r, m, ms in ((got[:, :, 0], lo * c - hi * s, (lo * c).abs() + (hi * s).abs(), (ml * c.abs()) + (mh * s.abs())),
                        (got[:, :, 1], hi * c + lo * s, (hi * c).abs() + (lo * s).abs(), (mh * c.abs()) + (ml * s.abs()))):
        # both projections, both products and the sum round once each; fp32 sums of K terms
        assert bool(((y - r).abs() <= 1.02 * u * (2 * m + r.abs()) + 2e-6 * ms + 1e-30).all())
    v, mv = ref[:, q_dim + 256:], mag[:, q_dim + 256:]
    assert bool(((kv[1, :M].double() - v).abs() <= 1.02 * u * v.abs() + 2e-6 * mv + 1e-30).all())
    assert float(kv[:, M:].abs().max()) == 0
    assert _lib.load().tpb200_device_error(0) == 0


@pytest.mark.parametrize("M,N,K", [(17, 8, 128), (50, 1032, 1024), (200, 136, 384), (257, 512, 2048), (712, 2048, 1024)])
@pytest.mark.parametrize("plugin", [False, True])
def test_int4(cuda_device, M, N, K, plugin):
    from turbopi_b200 import _lib, ops
    from turbopi_b200.w4a16 import _codes_to_words
    g = torch.Generator().manual_seed(M + N + K)
    codes = torch.randint(0, 16, (N, K), generator=g, dtype=torch.uint8)
    x = torch.randn((M, K), generator=g).to(torch.bfloat16)
    q = codes.double() - 8
    words = _codes_to_words(codes)
    if plugin:
        sc = (torch.rand((N, K // 128), generator=g) * 0.1).to(torch.bfloat16)
        zp = (torch.randn((N, K // 128), generator=g) * 0.1).to(torch.bfloat16)
        w = (q * sc.double().repeat_interleave(128, 1) + zp.double().repeat_interleave(128, 1)).float().to(torch.bfloat16)
        packed = (words.view(torch.uint8).reshape(N, K // 2) ^ 0x88).to(cuda_device)      # two's-complement nibbles
        args = (packed, N, _lib.W4_INT4_PLUGIN, sc.to(cuda_device), zp.to(cuda_device))
    else:
        sc = (torch.rand((N, K // 32), generator=g) * 0.1).half()
        w = (q * sc.double().repeat_interleave(32, 1)).float().to(torch.bfloat16)         # exact in fp32, one rounding
        packed = words.reshape(N, K // 32, 4).permute(1, 0, 2).contiguous().to(cuda_device)
        args = (packed, N, _lib.W4_INT4_KBLOCK, sc.t().contiguous().to(cuda_device))
    xd, wd = x.to(cuda_device), w.double().to(cuda_device)
    y = ops.w4_gemm(xd, *args, out_dtype=torch.float32)
    _check(y, xd.double() @ wd.t(), xd.double().abs() @ wd.abs().t(), 2.0 ** -22)
    if not plugin:                                                                        # scales that TMA cannot fetch
        odd = torch.empty(args[3].numel() + 1, dtype=torch.float16, device=cuda_device)[1:].view(args[3].shape)
        assert odd.copy_(args[3]).data_ptr() % 16 == 2
        assert torch.equal(ops.w4_gemm(xd, *args[:3], odd, out_dtype=torch.float32), y)
    assert _lib.load().tpb200_device_error(0) == 0


def _ring_wraps(M, N, K):
    """Whether the launch has narrow token tiles, an SM per CTA and more weight blocks than ring slots."""
    import ctypes
    from turbopi_b200 import _lib
    p = _lib.W4GemmPlanInfo()
    assert _lib.load().tpb200_w4_gemm_plan(M, N, K, 148, ctypes.byref(p)) == 0
    return p.parts == 2 and p.groups == 4 and -(-p.k_blocks // p.splits) > p.weight_slots


def _repeat_cold(call, y, device):
    """The same bits again under programmatic dependent launch, with the operands out of L2 and in it."""
    from turbopi_b200 import _lib, ops
    flush = torch.empty(256 << 20, dtype=torch.uint8, device=device)
    for _ in range(4):
        flush.zero_()
        with ops.launch_flags(ops.FLAG_PDL):
            ys = [call() for _ in range(3)]
        assert all(torch.equal(v, y) for v in ys)
    assert _lib.load().tpb200_device_error(0) == 0


@pytest.mark.parametrize("M,N,K", [(1, 2048, 16384), (17, 2048, 16384), (50, 2048, 16384), (64, 2048, 16384), (17, 16384, 2048),
                                   (64, 16384, 2048), (50, 8192, 1280), (512, 1152, 4304)])
def test_few_tokens_and_a_long_k(cuda_device, M, N, K):
    """K ranges of more 256-K blocks than the weight ring holds, with each group of warps on every second block."""
    from turbopi_b200 import _lib, ops
    assert _ring_wraps(M, N, K)
    b, sf, w = _nvfp4(N, K, cuda_device, M + N + K)
    x = torch.randn((M, K), generator=torch.Generator().manual_seed(M)).to(torch.bfloat16).to(cuda_device)
    ref, mag = x.double() @ w.t(), x.double().abs() @ w.abs().t()
    for weight in ((ops.tile_weights(b, sf, N, K), N, _lib.W4_NVFP4_TILED), (b, N, _lib.W4_NVFP4_ROWMAJOR, sf)):
        call = lambda: ops.w4_gemm(x, *weight, alpha=0.25, out_dtype=torch.float32)      # noqa: E731
        y = call()
        _check(y, 0.25 * ref, mag, 2.0 ** -22)
        _repeat_cold(call, y, cuda_device)


@pytest.mark.parametrize("M,I,K", [(1, 8192, 2048), (50, 8192, 2048), (64, 1024, 8192)])
def test_gated_few_tokens_and_a_long_k(cuda_device, M, I, K):
    from turbopi_b200 import _lib, ops
    assert _ring_wraps(M, 2 * I, K)
    b, sf, w = _nvfp4(2 * I, K, cuda_device, M + I + K)
    x = torch.randn((M, K), generator=torch.Generator().manual_seed(M)).to(torch.bfloat16).to(cuda_device)
    gu = x.double() @ w.t()
    a = 1.0 / float(gu.std())
    image = ops.tile_weights(b, sf, 2 * I, K)
    call = lambda: ops.w4_gemm(x, image, 2 * I, _lib.W4_NVFP4_TILED, alpha=a, activation=_lib.ACT_GELU, gated=True)   # noqa: E731
    y = call()
    r16 = lambda v: v.to(torch.bfloat16).double()      # noqa: E731
    gate, up = r16(a * gu[:, :I]), r16(a * gu[:, I:])
    ref = r16(torch.nn.functional.gelu(gate, approximate="tanh")) * up
    # gate may round to its neighbour, 2^-8 of it, which GELU passes on with a slope of at most 1.13; up, the activation and
    # the product round likewise; the fp32 sums of K terms are off by 2e-6 * mag before all that
    mag = a * (x.double().abs() @ w.abs().t())
    tol = 2.0 ** -8 * (1.13 * (gate * up).abs() + 3 * ref.abs()) + 2e-6 * 1.13 * (mag[:, :I] * up.abs() + mag[:, I:] * gate.abs())
    assert bool(((y.double() - ref).abs() <= tol + 1e-6).all())
    _repeat_cold(call, y, cuda_device)


@pytest.mark.parametrize("M,N,K", [(17, 2048, 16384), (64, 2048, 16384), (17, 16384, 2048), (64, 16384, 2048)])
@pytest.mark.parametrize("plugin", [False, True])
def test_int4_few_tokens_and_a_long_k(cuda_device, M, N, K, plugin):
    from turbopi_b200 import ops
    assert _ring_wraps(M, N, K)
    xd, args, wd = _int4(M, N, K, plugin, cuda_device)
    call = lambda: ops.w4_gemm(xd, *args, out_dtype=torch.float32)      # noqa: E731
    y = call()
    _check(y, xd.double() @ wd.t(), xd.double().abs() @ wd.abs().t(), 2.0 ** -22)
    _repeat_cold(call, y, cuda_device)


def _int4(M, N, K, plugin, device):
    """(bf16 activations, operands of w4_gemm, dequantised float64 weights)"""
    from turbopi_b200 import _lib
    from turbopi_b200.w4a16 import _codes_to_words
    g = torch.Generator().manual_seed(M + N + K)
    codes = torch.randint(0, 16, (N, K), generator=g, dtype=torch.uint8)
    x = torch.randn((M, K), generator=g).to(torch.bfloat16)
    q = codes.double() - 8
    words = _codes_to_words(codes)
    if plugin:
        sc = (torch.rand((N, K // 128), generator=g) * 0.1).to(torch.bfloat16)
        zp = (torch.randn((N, K // 128), generator=g) * 0.1).to(torch.bfloat16)
        w = (q * sc.double().repeat_interleave(128, 1) + zp.double().repeat_interleave(128, 1)).float().to(torch.bfloat16)
        packed = (words.view(torch.uint8).reshape(N, K // 2) ^ 0x88).to(device)               # two's-complement nibbles
        args = (packed, N, _lib.W4_INT4_PLUGIN, sc.to(device), zp.to(device))
    else:
        sc = (torch.rand((N, K // 32), generator=g) * 0.1).half()
        w = (q * sc.double().repeat_interleave(32, 1)).float().to(torch.bfloat16)             # exact in fp32, one rounding
        packed = words.reshape(N, K // 32, 4).permute(1, 0, 2).contiguous().to(device)
        args = (packed, N, _lib.W4_INT4_KBLOCK, sc.t().contiguous().to(device))
    return x.to(device), args, w.double().to(device)


@pytest.mark.parametrize("M,N,K", [(1, 64, 512), (1, 72, 1024), (2, 136, 8192), (5, 1000, 4096), (1, 2048, 16384), (16, 8, 2080),
                                   (3, 61, 1056)])
def test_kblock_gemv_with_k_cut_over_a_cluster(cuda_device, M, N, K):
    """Few output tiles, K ranges of unequal length, ragged N (scales by TMA or not)."""
    from turbopi_b200 import _lib, ops
    from turbopi_b200.w4a16 import _codes_to_words
    g = torch.Generator().manual_seed(M + N + K)
    codes = torch.randint(0, 16, (N, K), generator=g, dtype=torch.uint8)
    sc = (torch.rand((N, K // 32), generator=g) * 0.1).half()
    x = torch.randn((M, K), generator=g).half()
    bias = torch.randn(N, generator=g)
    w = (codes.double() - 8) * sc.double().repeat_interleave(32, 1)
    words = _codes_to_words(codes).reshape(N, K // 32, 4).permute(1, 0, 2).contiguous().to(cuda_device)
    out = torch.empty((M, N), dtype=torch.float32, device=cuda_device)
    ops.w4a16_gemv_out(x.to(cuda_device), words, sc.t().contiguous().to(cuda_device), out, bias.to(cuda_device))
    ref = x.double() @ w.t() + bias.double()
    # chains of four fp16 products (2^-11 each of their magnitude), then fp32
    mag = x.double().abs() @ w.abs().t() + bias.double().abs()
    assert bool(((out.cpu().double() - ref).abs() <= 2.0 ** -10 * mag).all())
    assert _lib.load().tpb200_device_error(0) == 0


@pytest.mark.parametrize("M,N,K,shift", [(1, 16, 16, 0), (50, 272, 1040, 0), (130, 144, 272, 0), (256, 2048, 2048, 0),
                                         (65, 264, 528, 0), (33, 256, 512, 4)])
def test_w4a8_forward_on_transposed_weights(cuda_device, M, N, K, shift):
    """The plugin's transposed codes read as they are (N a multiple of 16, aligned pointers) or re-laid out first."""
    from oracle import w4a8
    from turbopi_b200 import _lib, ops
    lib = _lib.load()
    g = torch.Generator().manual_seed(M + N + K)
    w = (torch.randn((N, K), generator=g) * 0.05).to(torch.bfloat16).to(cuda_device)
    x = torch.randn((M, K), generator=g).to(torch.bfloat16).to(cuda_device)
    wp_t, ws_t = ops.quantize_weight_to_nvfp4(w)
    a8, sa = ops.quantize_activation_to_fp8(x)
    held = torch.empty(wp_t.numel() + 16, dtype=torch.uint8, device=cuda_device)
    held[shift:shift + wp_t.numel()] = wp_t.reshape(-1)                       # `shift` bytes off a 16-byte boundary
    out = torch.empty((M, N), dtype=torch.bfloat16, device=cuda_device)
    nws = lib.getW4A8GemmWorkspaceSize(M, N, K)
    ws = torch.empty(nws, dtype=torch.uint8, device=cuda_device)
    torch.cuda.synchronize()
    lib.w4a8GemmForward(a8.data_ptr(), sa.data_ptr(), held.data_ptr() + shift, ws_t.data_ptr(), out.data_ptr(), M, N, K, 0.5,
                        ws.data_ptr(), nws, torch.cuda.current_stream().cuda_stream)
    _lib.check_void("w4a8GemmForward")
    ref = torch.from_numpy(np.asarray(w4a8.gemm(a8.cpu().numpy(), sa.cpu().numpy(), wp_t.cpu().numpy(), ws_t.cpu().numpy(), 0.5)))
    # exact products in bf16 x bf16, fp32 sums, one rounding to bf16
    assert bool(((out.cpu().double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-5 * ref.abs().max()).all())
    assert lib.tpb200_device_error(0) == 0


@pytest.mark.parametrize("M,N,K", [(1, 8, 16), (129, 264, 272), (200, 1000, 1040), (712, 4096, 2048)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_w4a4_tiled_operands_equal_the_row_major_form(cuda_device, M, N, K, dtype):
    from turbopi_b200 import _lib, ops
    b, sf, _ = _nvfp4(N, K, cuda_device, M + N + K)
    x = torch.randn((M, K), generator=torch.Generator().manual_seed(M)).to(dtype).to(cuda_device)
    bias = torch.randn(N, generator=torch.Generator().manual_seed(N)).to(cuda_device)
    a, a_sf = ops.nvfp4_quantize_act(x)
    want = ops.nvfp4_gemm(a, a_sf, b, sf, M, N, K, alpha=0.25, bias=bias, activation=_lib.ACT_GELU, out_dtype=torch.float32)
    got = ops.nvfp4_linear_tiled(x, ops.tile_weights(b, sf, N, K), N, 0.25, bias, _lib.ACT_GELU, torch.float32)
    # the same products; fp32 sums may associate differently
    assert float((got - want).abs().max()) <= 2e-6 * float(want.abs().max())
    assert _lib.load().tpb200_device_error(0) == 0


@torch.no_grad()
def test_nvfp4_linear_notices_weights_written_in_place(cuda_device):
    from turbopi_b200.nvfp4_linear import NVFP4Linear
    torch.manual_seed(3)
    l1, l2 = (torch.nn.Linear(256, 25600, bias=False, device=cuda_device) for _ in range(2))
    a, b = NVFP4Linear.from_linear(l1, use_mse_search=False), NVFP4Linear.from_linear(l2, use_mse_search=False)
    x = torch.randn(8, 256, device=cuda_device).to(torch.bfloat16)
    before, want = a(x), b(x)
    a.load_state_dict(b.state_dict())
    assert torch.equal(a(x), want) and not torch.equal(before, want)


@torch.no_grad()
@pytest.mark.parametrize("T", [1, 8, 40])
def test_packed_mlp_notices_weights_loaded_in_place(cuda_device, T):
    from types import SimpleNamespace
    from turbopi_b200.nvfp4_packed import NVFP4PackedMLP
    torch.manual_seed(5)
    mods = []
    for _ in range(2):
        p = {n: torch.nn.Linear(*s, bias=False, device=cuda_device) for n, s in (("gate_proj", (128, 256)), ("up_proj", (128, 256)), ("down_proj", (256, 128)))}
        mods.append(NVFP4PackedMLP.from_gemma_mlp(SimpleNamespace(**p), gate_activation="gelu", fmt="nvfp4"))
    a, b = mods
    x = torch.randn(T, 128, device=cuda_device).to(torch.bfloat16)
    before, want = a(x), b(x)
    for la, lb in ((a.gate_proj, b.gate_proj), (a.up_proj, b.up_proj), (a.down_proj, b.down_proj)):
        la.weight_packed.copy_(lb.weight_packed)
        la.weight_scales.copy_(lb.weight_scales)
        la.global_scale = lb.global_scale
    assert torch.equal(a(x), want) and not torch.equal(before, want)


@torch.no_grad()
@pytest.mark.parametrize("features", [256, 25600])           # either side of the rule on output tiles
def test_nvfp4_linear_reads_the_weights_it_has_now(cuda_device, features):
    """A module built in inference mode; a first call that is captured."""
    from turbopi_b200.nvfp4_linear import TILED_MIN_TILES, NVFP4Linear
    torch.manual_seed(4)
    l1, l2 = (torch.nn.Linear(256, features, bias=False, device=cuda_device) for _ in range(2))
    a, b = NVFP4Linear.from_linear(l1, use_mse_search=False), NVFP4Linear.from_linear(l2, use_mse_search=False)
    assert (a._tiles(8) >= TILED_MIN_TILES) == (features == 25600)
    x = torch.randn(8, 256, device=cuda_device).to(torch.bfloat16)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = a(x)
    want = b(x)
    # the forms may sum in another order (fp32), then each rounds to bf16
    tol = 2e-6 * float(want.abs().max())
    for name, buf in a.named_buffers():
        buf.copy_(dict(b.named_buffers())[name])
    assert torch.equal(a(x), want)
    with torch.inference_mode():
        c = NVFP4Linear.from_linear(l2, use_mse_search=False)
        assert torch.allclose(c(x).float(), want.float(), rtol=2.0 ** -7, atol=tol)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.allclose(y.float(), want.float(), rtol=2.0 ** -7, atol=tol)
