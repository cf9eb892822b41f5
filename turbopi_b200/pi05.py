"""Pi0.5-shaped inference pipeline on the turbopi_b200 kernels.

SigLIP-So400m/14 vision tower -> Gemma-2B prefix (image + text tokens, fills the KV cache) ->
Gemma-300M action expert running N flow-matching Euler steps over 50 action tokens against that
cache (`PI0Pytorch.sample_actions`, openpi/src/openpi/models_pytorch/pi0_pytorch.py:876-937;
cached denoise step :524-654; adaptive RMSNorm / gated residual / MLP,
transformers_replace/models/gemma/modeling_gemma.py:49-129,212-230).

Every linear layer runs as NVFP4 weights x bf16 activations on the tensor cores.  The two large prefix MLP
matrices take the block-scaled e2m1 GEMM (activations as residual e2m1 pieces, written by the row kernels);
every other linear takes the GEMM that dequantises its weights into tensor memory and reads the bf16
activations as they are (csrc/w4_gemm.cu): no quantiser in front of it, GELU(gate) * up and Q/K/V + RoPE +
KV-cache append in its epilogue.  Norms and residuals are the fused row kernels, in the action expert the
epilogues of the linears around them; attention is the tensor-core kernel of csrc/attention.cu (`ops.attention`).  All buffers are
allocated once, so the whole inference (or just the denoise loop) replays as ONE CUDA graph.

Weights come from a reference-named state dict (`Pi05.from_state_dict`, tensor names of
`PI0Pytorch.state_dict()`), from a prepared container file (`Pi05.save` / `Pi05.from_file`,
turbopi_b200/weights.py) or, for benchmarks, from a seeded random initialisation.

Padding follows the reference: prefix tokens that do not exist (a missing camera, the padded tail of the
prompt) are never attended to, position ids are `cumsum(valid) - 1`, and the action tokens continue at
`sum(valid)` (pi0_pytorch.py:80-108,442,571-579,791-866).  The valid mask only changes small device
buffers (positions, additive key bias), so one captured graph serves every mask.
"""
import ctypes
import math
import operator
from dataclasses import dataclass

import torch

from . import _lib, ops, weights
from ._lib import ACT_GELU, ACT_NONE, ACT_SILU, TurboPiError
from .nvfp4_packed import quantize_nvfp4_two_level


@dataclass
class Pi05Config:
    # SigLIP-So400m/14
    image_size: int = 224
    patch: int = 14
    vision_layers: int = 27
    vision_width: int = 1152
    vision_mlp: int = 4304
    vision_heads: int = 16
    num_images: int = 2
    # Gemma-2B prefix
    prefix_layers: int = 18
    width: int = 2048
    mlp: int = 16384
    heads: int = 8
    head_dim: int = 256
    text_len: int = 200
    vocab: int = 257152
    # Gemma-300M action expert
    expert_layers: int = 18
    expert_width: int = 1024
    expert_mlp: int = 4096
    action_horizon: int = 50
    action_dim: int = 32
    max_seq: int = 1024
    pieces: int = 3          # residual e2m1 pieces of the prefix MLP's activations (every other linear takes them in bf16)
    eps: float = 1e-6

    @property
    def image_tokens(self):
        return (self.image_size // self.patch) ** 2

    @property
    def prefix_len(self):
        return self.num_images * self.image_tokens + self.text_len

    @property
    def q_dim(self):
        return self.heads * self.head_dim


QuantBuf, rowop = ops.QuantBuf, ops.rowop


class TcLinear:
    """One NVFP4 weight matrix prepared for the tensor-core GEMM (standard NVFP4: E4M3 scale per 16 and
    an fp32 global scale), the global scale, an optional fp32 bias, in one of the GEMM's two operand forms:
    the tiled image (`sf is None`; 128 x 256 output tiles, one contiguous block per K stage: the form for the
    large prefix MLP matrices), or
    row-major codes [N, pitch] + swizzled scale atoms.  A call with a `QuantBuf` (in the weight's form) runs the
    block-scaled GEMM; `dense` / `dense_qkv` take bf16 activations and dequantise the weights inside the kernel.
    `raw` keeps the reference-layout codes / scale bytes for dequantisation in tests."""

    def __init__(self, image, g, N, K, bias=None, raw=None, sf=None):
        self.b, self.sf, self.g, self.N, self.K = image, sf, float(g), int(N), int(K)
        self.bias = None if bias is None else bias.float().contiguous()
        if raw is not None:
            self.raw = raw
        self.ws = None            # split-K scratch, set by the owning pipeline

    @property
    def rowmajor(self):
        return self.sf is not None

    @classmethod
    def from_weight(cls, weight, bias=None, row_perm=None, keep_raw=False, rowmajor=False):
        N, K = weight.shape
        packed, scales, g = quantize_nvfp4_two_level(weight, 16)
        raw = (packed.clone(), scales.clone(), g) if keep_raw else None
        if row_perm is not None:
            packed, scales = packed[row_perm], scales[row_perm]
        if rowmajor:
            b = torch.zeros((N, ops.packed_pitch(K)), dtype=torch.uint8, device=packed.device)
            b[:, :K // 2] = packed
            return cls(b, g, N, K, bias, raw, sf=ops.swizzle_scales(scales.contiguous()))
        return cls(weights.tile_weights_host(packed, scales), g, N, K, bias, raw)

    def _args(self, q, M):
        if q.tiled == self.rowmajor:
            raise TurboPiError("activation operand and weight are in different operand forms")
        p = ops._ptr
        if self.rowmajor:
            return _lib.GemmArgs(a_packed=p(q.packed), a_pitch=q.pitch, a_sf=p(q.sf), a_pieces=q.pieces,
                                 a_piece_rows=q.piece_rows, a_row_scale=p(q.row_scale), b_packed=p(self.b),
                                 b_pitch=self.b.stride(0), b_sf=p(self.sf), alpha=float(self.g), M=M, N=self.N, K=self.K,
                                 layout=ops.OPERANDS_ROWMAJOR)
        return _lib.GemmArgs(a_packed=p(q.packed), a_pieces=q.pieces, a_row_scale=p(q.row_scale), b_packed=p(self.b),
                             alpha=float(self.g), M=M, N=self.N, K=self.K, layout=ops.OPERANDS_TILED)

    def __call__(self, q, out, activation=ACT_NONE, M=None):
        args = self._args(q, q.M if M is None else M)
        args.bias, args.activation = ops._ptr(self.bias), int(activation)
        args.out, args.out_dtype, args.ldo = ops._ptr(out), ops._dt(out), out.stride(0)
        ops._gemm_ex(args, out.device, self.ws)
        return out

    def _w4_args(self, x, M, out, ldo):
        p = ops._ptr
        return _lib.W4GemmArgs(x=p(x), ldx=x.stride(0), format=_lib.W4_NVFP4_ROWMAJOR if self.rowmajor else _lib.W4_NVFP4_TILED,
                               w=p(self.b), w_pitch=self.b.stride(0) if self.rowmajor else 0, w_scales=p(self.sf),
                               alpha=float(self.g), out=p(out), out_dtype=ops._dt(out), ldo=ldo, M=M, N=self.N, K=self.K)

    def dense(self, x, out, activation=ACT_NONE, gated=False, norm=None, bias=True, scale=1.0, beta=0.0):
        """out = act(scale * x W^T + bias) + beta * out for bf16 x [M, >= K]; `gated`: W = [gate; up], out = act(gate) * up.
        `norm` (_lib.W4NormArgs): the RMS norms around the linear, see tpb200_w4_gemm_norm."""
        args = self._w4_args(x, x.shape[0], out, out.stride(0))
        args.alpha, args.beta = float(self.g) * scale, beta
        args.bias, args.activation, args.gated = ops._ptr(self.bias if bias else None), int(activation), int(gated)
        ops._w4_gemm(args, out.device, norm)
        return out

    def dense_qkv(self, x, q_out, k_rows, v_rows, positions, cos, sin, q_dim, norm=None):
        M = x.shape[0]
        if k_rows.shape[0] < M or v_rows.shape[0] < M or positions.numel() < M:
            raise TurboPiError("fused QKV: cache rows / positions shorter than the token count")
        p = ops._ptr
        args = self._w4_args(x, M, q_out, q_out.stride(0))
        args.qkv_q_dim, args.qkv_k_rows, args.qkv_v_rows, args.qkv_positions = q_dim, p(k_rows), p(v_rows), p(positions)
        args.qkv_rope_cos, args.qkv_rope_sin = p(cos), p(sin)
        ops._w4_gemm(args, q_out.device, norm)
        return q_out


def sinusoidal_time_embedding(t, dim, min_period=4e-3, max_period=4.0):
    """openpi/src/openpi/models_pytorch/pi0_pytorch.py:53-70 (float64)."""
    frac = torch.linspace(0.0, 1.0, dim // 2, dtype=torch.float64)
    period = min_period * (max_period / min_period) ** frac
    ang = (1.0 / period * 2 * math.pi)[None, :] * t.to(torch.float64)[:, None]
    return torch.cat([torch.sin(ang), torch.cos(ang)], dim=1)


_version = operator.attrgetter("_version")


class _Marks:
    """The tensors a kept table was made from, with their version counters (inference tensors count no versions) and the
    plain numbers beside them."""

    def __init__(self, tensors, numbers=()):
        self.tensors, self.numbers = tensors, numbers
        self.counting = [t for t in tensors if not t.is_inference()]
        self.versions = list(map(_version, self.counting))

    @classmethod
    def of(cls, linears):
        return cls([t for l in linears for t in (l.b, l.sf, l.bias) if t is not None], [l.g for l in linears])

    def written(self):
        return list(map(_version, self.counting)) != self.versions

    def same(self, other):
        return (self.versions == other.versions and self.numbers == other.numbers
                and all(map(operator.is_, self.tensors, other.tensors)))


class Pi05:
    """Pi0.5-shaped model; `infer(images_u8, tokens, noise, num_steps)` -> actions [50, 32].

    Pi05(cfg, device, seed=...)            seeded random weights (benchmarks, tests)
    Pi05.from_state_dict(sd, cfg, device)  tensors under the reference's names (weights.reference_state_dict_names)
    Pi05.from_file(path, device)           a container written by `save()`
    """

    def __init__(self, cfg: Pi05Config, device, seed=0, keep_raw=False, pdl=True, state_dict=None, _prepared=None):
        self.cfg, self.device = cfg, device
        c = cfg
        if c.prefix_len + c.action_horizon > c.max_seq:
            raise TurboPiError(f"prefix ({c.prefix_len}) + action horizon ({c.action_horizon}) exceed the KV cache "
                               f"({c.max_seq} rows)")
        # programmatic dependent launch across the GEMM / row-kernel chain: each kernel's launch and set-up
        # overlap the tail of the one before it
        self.launch_flags = ops.FLAG_PDL if pdl else ops.FLAG_NONE
        self.keep_raw = keep_raw
        self.patch_k = (3 * c.patch * c.patch + 15) // 16 * 16
        self.n_norms = 2 * c.expert_layers + 1
        self.workspace = ops.gemm_workspace(device)       # split-K scratch of THIS pipeline's launches
        if _prepared is not None:
            self._from_prepared(_prepared)
        else:
            self._from_tensors(self._random_source(seed) if state_dict is None else self._dict_source(state_dict))
        self.cos, self.sin = ops.rope_tables(c.max_seq, c.head_dim, device=device)
        if self.cos.shape[0] != c.max_seq:
            raise TurboPiError("RoPE table and KV cache disagree on the number of positions")
        self._alloc()
        self._graph = None
        self._graph_steps = None
        self._time_emb = {}
        self._mod = {}            # per step count: the adaptive norms' modulation tables, and the weights they follow
        self._pos_marks = _Marks([self.pos_emb])
        # The expert's norms ride in the epilogues of the linears around them where a row's sums of squares come in
        # whole 16-byte groups of 128-column parts; other widths take the row kernel between two linears.
        self.fold_norms = cfg.expert_width % 512 == 0 and cfg.expert_mlp % 64 == 0
        self.set_valid()

    @classmethod
    def from_state_dict(cls, state_dict, cfg: Pi05Config, device, **kw):
        return cls(cfg, device, state_dict=state_dict, **kw)

    @classmethod
    def from_file(cls, path, device, **kw):
        tensors, meta = weights.load_container(path, device)
        if meta.get("kind") != "pi05":
            raise TurboPiError(f"{path}: not a Pi0.5 weight container")
        return cls(Pi05Config(**meta["config"]), device, _prepared=(tensors, meta), **kw)

    # ------------------------------------------------------------------ weights
    def _random_source(self, seed):
        g = torch.Generator(device=self.device).manual_seed(seed)
        shapes = weights.reference_state_dict_names(self.cfg)

        def get(name):
            shape = shapes[name]
            norm = len(shape) == 1 and ("layernorm" in name or "layer_norm" in name)
            # norm parameters: small random values so that the norms are not the identity
            t = torch.randn(shape, generator=g, device=self.device) * (0.1 if norm else 0.02)
            if norm and name.endswith(".weight") and ("layer_norm" in name or "post_layernorm" in name):
                t = t + 1.0
            return t
        return get

    def _dict_source(self, sd):
        shapes = weights.reference_state_dict_names(self.cfg)
        missing = [n for n in shapes if n not in sd]
        if missing:
            raise TurboPiError(f"state dict lacks {len(missing)} tensors, e.g. {missing[:3]}")

        def get(name):
            t = sd[name]
            if tuple(t.shape) != tuple(shapes[name]):
                raise TurboPiError(f"{name}: shape {tuple(t.shape)}, expected {tuple(shapes[name])}")
            return t.to(self.device).float()
        return get

    def _from_tensors(self, get):
        """Quantise, permute and tile every linear; norms, embeddings and tables go to bf16."""
        c, kr = self.cfg, self.keep_raw
        bf = torch.bfloat16
        V = "paligemma_with_expert.paligemma.model.vision_tower.vision_model."
        PG = "paligemma_with_expert.paligemma.model."
        EX = "paligemma_with_expert.gemma_expert.model."

        # Operand form per linear: the tiled image for the large prefix MLP matrices (gate_up, down: 712 x 32768 x 2048 in
        # 61 us + 28 us of row kernel against 107 us on the dequantising GEMM, 712 x 2048 x 16384 in 35 against 47), row-major
        # for everything else (the vision tower, the attention projections, the action expert, the small projections).
        def lin(wname, bias=True, perm=None, rm=True):
            return TcLinear.from_weight(get(wname + ".weight"), get(wname + ".bias") if bias else None, perm, kr, rm)

        def stacked(names, bias, perm=None, rm=True):
            w = torch.cat([get(n + ".weight") for n in names], 0)
            b = torch.cat([get(n + ".bias") for n in names], 0) if bias else None
            return TcLinear.from_weight(w, b, perm, kr, rm)

        vw = c.vision_width
        wp = torch.zeros(vw, self.patch_k, device=self.device)
        wp[:, :3 * c.patch * c.patch] = get(V + "embeddings.patch_embedding.weight").reshape(vw, -1)   # (c, i, j)
        self.patch_embed = TcLinear.from_weight(wp, get(V + "embeddings.patch_embedding.bias"), None, kr, True)
        self.pos_emb = get(V + "embeddings.position_embedding.weight").to(bf)
        self.vision = []
        for i in range(c.vision_layers):
            L = f"{V}encoder.layers.{i}."
            self.vision.append(dict(
                ln1_w=get(L + "layer_norm1.weight").to(bf), ln1_b=get(L + "layer_norm1.bias").to(bf),
                qkv=stacked([L + "self_attn.q_proj", L + "self_attn.k_proj", L + "self_attn.v_proj"], True),
                out=lin(L + "self_attn.out_proj"),
                ln2_w=get(L + "layer_norm2.weight").to(bf), ln2_b=get(L + "layer_norm2.bias").to(bf),
                fc1=lin(L + "mlp.fc1"), fc2=lin(L + "mlp.fc2")))
        self.post_ln_w, self.post_ln_b = get(V + "post_layernorm.weight").to(bf), get(V + "post_layernorm.bias").to(bf)
        self.projector = lin(PG + "multi_modal_projector.linear")

        perm = ops.qkv_tile_permutation(c.q_dim).to(self.device)
        self.embed_tokens = get(PG + "language_model.embed_tokens.weight").to(bf)

        def decoder(prefix, mlp_rm):
            a = prefix + "self_attn."
            return dict(qkv=stacked([a + "q_proj", a + "k_proj", a + "v_proj"], False, perm),
                        o=lin(a + "o_proj", False),
                        gate_up=stacked([prefix + "mlp.gate_proj", prefix + "mlp.up_proj"], False, rm=mlp_rm),
                        down=lin(prefix + "mlp.down_proj", False, rm=mlp_rm))

        self.prefix = []
        for i in range(c.prefix_layers):
            L = f"{PG}language_model.layers.{i}."
            d = decoder(L, False)
            d["in_norm"] = get(L + "input_layernorm.weight").to(bf)
            d["post_norm"] = get(L + "post_attention_layernorm.weight").to(bf)
            self.prefix.append(d)

        self.action_in = lin("action_in_proj")
        self.action_out = lin("action_out_proj")
        self.time_mlp_in = lin("time_mlp_in")
        self.time_mlp_out = lin("time_mlp_out")
        self.expert, dense = [], []
        for i in range(c.expert_layers):
            L = f"{EX}layers.{i}."
            self.expert.append(decoder(L, True))
            dense += [L + "input_layernorm.dense", L + "post_attention_layernorm.dense"]
        self.ada_dense = stacked(dense + [EX + "norm.dense"], True)    # every adaptive norm's dense(cond), stacked

    _LINEAR_SLOTS = ("qkv", "out", "fc1", "fc2", "o", "gate_up", "down")

    def _named_parts(self):
        """(name, object) of everything `save()` stores: TcLinear objects and plain tensors."""
        yield "patch_embed", self.patch_embed
        yield "pos_emb", self.pos_emb
        for group, layers in (("vision", self.vision), ("prefix", self.prefix), ("expert", self.expert)):
            for i, L in enumerate(layers):
                for k, v in L.items():
                    yield f"{group}.{i}.{k}", v
        for k in ("post_ln_w", "post_ln_b", "projector", "embed_tokens", "action_in", "action_out", "time_mlp_in",
                  "time_mlp_out", "ada_dense"):
            yield k, getattr(self, k)

    def _export(self):
        """(tensors, meta) of the prepared model: what `save` writes and `_from_prepared` reads.  The tensors are
        the model's own, not copies."""
        tensors, linears = {}, {}
        for name, obj in self._named_parts():
            if isinstance(obj, TcLinear):
                if obj.rowmajor:
                    tensors[name + ".codes"] = obj.b
                    tensors[name + ".scale_atoms"] = obj.sf
                else:
                    tensors[name + ".image"] = obj.b
                if obj.bias is not None:
                    tensors[name + ".bias"] = obj.bias
                linears[name] = {"N": obj.N, "K": obj.K, "global_scale": obj.g,
                                 "form": "rowmajor" if obj.rowmajor else "tiled"}
            else:
                tensors[name] = obj
        cfgd = {k: getattr(self.cfg, k) for k in self.cfg.__dataclass_fields__}
        return tensors, {"kind": "pi05", "config": cfgd, "linears": linears}

    def save(self, path):
        """Write the prepared model (4-bit operands in the form each linear runs in, bf16 tables) to a container file."""
        tensors, meta = self._export()
        return weights.save_container(path, tensors, meta)

    @classmethod
    def sharing_weights(cls, other, **kw):
        """A second pipeline over `other`'s weights (the same device tensors, no copy) with buffers, KV cache,
        split-K and attention scratch of its own: two such pipelines can run at the same time on two streams of
        one GPU (every kernel's scratch is per pipeline, split-K launches are cooperative launches)."""
        kw.setdefault("pdl", other.launch_flags == ops.FLAG_PDL)
        return cls(other.cfg, other.device, _prepared=other._export(), **kw)

    def _from_prepared(self, prepared):
        tensors, meta = prepared
        lins = meta["linears"]

        def part(name):
            if name in lins:
                e = lins[name]
                if e.get("form", "tiled") == "rowmajor":
                    return TcLinear(tensors[name + ".codes"], e["global_scale"], e["N"], e["K"], tensors.get(name + ".bias"),
                                    sf=tensors[name + ".scale_atoms"])
                return TcLinear(tensors[name + ".image"], e["global_scale"], e["N"], e["K"], tensors.get(name + ".bias"))
            return tensors[name]

        c = self.cfg
        self.patch_embed, self.pos_emb = part("patch_embed"), part("pos_emb")
        self.vision = [{k: part(f"vision.{i}.{k}") for k in ("ln1_w", "ln1_b", "qkv", "out", "ln2_w", "ln2_b", "fc1", "fc2")}
                       for i in range(c.vision_layers)]
        self.prefix = [{k: part(f"prefix.{i}.{k}") for k in ("qkv", "o", "gate_up", "down", "in_norm", "post_norm")}
                       for i in range(c.prefix_layers)]
        self.expert = [{k: part(f"expert.{i}.{k}") for k in ("qkv", "o", "gate_up", "down")}
                       for i in range(c.expert_layers)]
        for k in ("post_ln_w", "post_ln_b", "projector", "embed_tokens", "action_in", "action_out", "time_mlp_in",
                  "time_mlp_out", "ada_dense"):
            setattr(self, k, part(k))

    # ------------------------------------------------------------------ buffers
    def _alloc(self):
        c, d, P = self.cfg, self.device, self.cfg.pieces
        bf = torch.bfloat16
        T = c.num_images * c.image_tokens
        vw = c.vision_width
        S = c.prefix_len
        A = c.action_horizon
        ew = c.expert_width
        self.cache = torch.zeros((c.prefix_layers, 2, c.max_seq, c.head_dim), dtype=bf, device=d)
        self.b = dict(
            # vision
            patches=torch.zeros((T, self.patch_k), dtype=bf, device=d), pos=self.pos_emb.repeat(c.num_images, 1),
            vh=torch.empty((T, vw), dtype=bf, device=d), vy=torch.empty((T, vw), dtype=bf, device=d),
            vx=torch.empty((T, vw), dtype=bf, device=d), v_qkv=torch.empty((T, 3 * vw), dtype=bf, device=d),
            v_attn=torch.empty((T, vw), dtype=bf, device=d),
            v_fc1=torch.empty((T, c.vision_mlp), dtype=bf, device=d),
            # prefix
            ph=torch.empty((S, c.width), dtype=bf, device=d), py=torch.empty((S, c.width), dtype=bf, device=d),
            q_p=QuantBuf(S, c.width, P, d), px=torch.empty((S, c.width), dtype=bf, device=d),
            p_q=torch.empty((S, c.q_dim), dtype=bf, device=d), p_attn=torch.empty((S, c.q_dim), dtype=bf, device=d), p_gu=torch.empty((S, 2 * c.mlp), dtype=bf, device=d),
            q_pmlp=QuantBuf(S, c.mlp, P, d), pos_prefix=torch.arange(S, dtype=torch.int32, device=d),
            # expert
            x_t=torch.zeros((A, c.action_dim), dtype=torch.float32, device=d),
            x_bf=torch.zeros((A, c.action_dim), dtype=bf, device=d),
            eh=torch.empty((A, ew), dtype=bf, device=d), ey=torch.empty((A, ew), dtype=bf, device=d),
            ex=torch.empty((A, ew), dtype=bf, device=d), e_q=torch.empty((A, c.q_dim), dtype=bf, device=d),
            e_attn=torch.empty((A, c.q_dim), dtype=bf, device=d), e_mlp=torch.empty((A, c.expert_mlp), dtype=bf, device=d),
            e_gu=torch.empty((A if c.expert_mlp % 64 else 0, 2 * c.expert_mlp), dtype=bf, device=d),
            e_ss=torch.empty((A, max(1, ew // 128)), dtype=torch.float32, device=d),
            v_out=torch.empty((A, c.action_dim), dtype=torch.float32, device=d),
            pos_suffix=torch.arange(S, S + A, dtype=torch.int32, device=d),
        )
        for _, obj in self._named_parts():
            if isinstance(obj, TcLinear):
                obj.ws = self.workspace
        # additive attention bias per key (0 or the reference's mask value) over the cache rows
        self.key_bias = torch.zeros((c.max_seq,), dtype=bf, device=d)
        # scratch of the attention kernel (partial results of the key tiles), sized for the largest call
        lib = _lib.load()
        hd_v = c.vision_width // c.vision_heads
        need = max(lib.tpb200_attention_workspace_size(S * c.heads, S, c.head_dim, 1),
                   lib.tpb200_attention_workspace_size(A * c.heads, S + A, c.head_dim, 1),
                   lib.tpb200_attention_workspace_size(c.image_tokens, c.image_tokens, hd_v, c.num_images * c.vision_heads))
        self.attn_ws = torch.empty(int(need), dtype=torch.uint8, device=d)
        self.tokens = torch.zeros((c.text_len,), dtype=torch.long, device=d)
        self.images = torch.zeros((c.num_images, c.image_size, c.image_size, 3), dtype=torch.uint8, device=d)
        self.noise = torch.zeros((A, c.action_dim), dtype=torch.float32, device=d)
        self.actions = torch.zeros((A, c.action_dim), dtype=torch.float32, device=d)

    # ------------------------------------------------------------------ stages
    def set_valid(self, image_valid=None, prompt_len=None):
        """Declare which prefix tokens exist: `image_valid[i]` per camera, and the number of prompt tokens
        before the padding.  Updates the position ids (`cumsum(valid) - 1`; action tokens continue at
        `sum(valid)`) and the additive key bias in place, so a captured graph picks them up on its next replay."""
        c = self.cfg
        image_valid = [True] * c.num_images if image_valid is None else [bool(v) for v in image_valid]
        prompt_len = c.text_len if prompt_len is None else int(prompt_len)
        if len(image_valid) != c.num_images or not 0 <= prompt_len <= c.text_len:
            raise TurboPiError("set_valid: one flag per camera and 0 <= prompt_len <= text_len")
        key = (tuple(image_valid), prompt_len)
        if getattr(self, "_valid_key", None) == key:       # the same mask as last time: the device tables stand
            return
        valid = torch.cat([torch.full((c.image_tokens,), v) for v in image_valid] + [torch.arange(c.text_len) < prompt_len])
        if not bool(valid.any()):
            raise TurboPiError("set_valid: at least one prefix token must be valid")
        pos = (torch.cumsum(valid.long(), 0) - 1).clamp_min(0)
        first = int(valid.sum())
        S, A = c.prefix_len, c.action_horizon
        bias = torch.zeros(c.max_seq, dtype=torch.float32)
        bias[:S][~valid] = -2.3819763e38                      # the reference's mask value (pi0_pytorch.py:185-188)
        self.b["pos_prefix"].copy_(pos.to(torch.int32))
        self.b["pos_suffix"].copy_(torch.arange(first, first + A, dtype=torch.int32))
        self.key_bias.copy_(bias.to(torch.bfloat16))
        self.valid = valid
        self._valid_key = key

    def _attention(self, q, k, v, out):
        """q [L, H*D] -> softmax(q k^T / sqrt(D) + key bias) v, all heads sharing one K/V head.  Prefix
        tokens see every valid prefix token, action tokens see the valid prefix and each other.  The
        (token, head) pairs are rows of one [L * H, D] problem for the tensor-core kernel."""
        c = self.cfg
        L = q.shape[0]
        ops.attention(q.view(L * c.heads, c.head_dim), k, v, out.view(L * c.heads, c.head_dim), c.head_dim ** -0.5,
                      self.key_bias, self.attn_ws)

    def weights_changed(self):
        """Weights may be written in place at any time; what is kept of products of them (the positions once per image, the
        adaptive norms' modulation and the linears' share of their shifts) is made again, in its own memory, when PyTorch's
        version counters have moved.  After a write that they do not see (through `.data`, from another library, to
        tensors made in inference mode) call this: the next inference makes the tables again, also for a captured graph."""
        self._pos_marks = None
        self._mod = {n: (mod, shift, None) for n, (mod, shift, _) in self._mod.items()}

    def _positions(self):
        """The position embeddings, once per image: the first LayerNorm's row kernel adds them."""
        marks = _Marks([self.pos_emb])
        if self._pos_marks is None or not marks.same(self._pos_marks):
            c = self.cfg
            self.b["pos"].view(c.num_images, c.image_tokens, c.vision_width).copy_(self.pos_emb)
            if not torch.cuda.is_current_stream_capturing():
                self._pos_marks = marks
        return self.b["pos"]

    def vision_tower(self):
        c, b = self.cfg, self.b
        pos = self._positions()
        T, vw = c.num_images * c.image_tokens, c.vision_width
        st = ops._run_on(self.images.device, _lib.load().tpb200_pi05_patches, ops._ptr(self.images), ops._ptr(b["patches"]),
                         c.num_images, c.image_size, c.patch, self.patch_k, ops._flags.value)
        _lib.check(st, "tpb200_pi05_patches")
        self.patch_embed.dense(b["patches"], b["vh"])
        hd = vw // c.vision_heads
        first = True
        for L in self.vision:
            if first:
                rowop(_lib.ROW_LAYERNORM, b["vh"], vw, y_out=b["vx"], res_in=pos, h_out=b["vh"], w0=L["ln1_w"], w1=L["ln1_b"],
                      eps=c.eps)
                first = False
            else:
                rowop(_lib.ROW_LAYERNORM, b["vy"], vw, y_out=b["vx"], res_in=b["vh"], h_out=b["vh"], w0=L["ln1_w"],
                      w1=L["ln1_b"], eps=c.eps)
            L["qkv"].dense(b["vx"], b["v_qkv"])
            qkv = b["v_qkv"].view(c.num_images, c.image_tokens, 3, c.vision_heads, hd).permute(2, 0, 3, 1, 4)
            ops.attention(qkv[0], qkv[1], qkv[2],
                          b["v_attn"].view(c.num_images, c.image_tokens, c.vision_heads, hd).permute(0, 2, 1, 3),
                          hd ** -0.5, None, self.attn_ws)
            L["out"].dense(b["v_attn"], b["vy"])
            rowop(_lib.ROW_LAYERNORM, b["vy"], vw, y_out=b["vx"], res_in=b["vh"], h_out=b["vh"], w0=L["ln2_w"], w1=L["ln2_b"],
                  eps=c.eps)
            L["fc1"].dense(b["vx"], b["v_fc1"], ACT_GELU)
            L["fc2"].dense(b["v_fc1"], b["vy"])
        rowop(_lib.ROW_LAYERNORM, b["vy"], vw, y_out=b["vx"], res_in=b["vh"], h_out=b["vh"], w0=self.post_ln_w,
              w1=self.post_ln_b, eps=c.eps)
        self.projector.dense(b["vx"], b["ph"][:T])                                          # image tokens of the prefix

    def prefix_pass(self):
        c, b = self.cfg, self.b
        T, S = c.num_images * c.image_tokens, c.prefix_len
        if c.text_len:
            st = ops._run_on(self.tokens.device, _lib.load().tpb200_pi05_embed, ops._ptr(self.tokens), ops._ptr(self.embed_tokens),
                             ops._ptr(b["ph"][T:]), c.text_len, self.embed_tokens.shape[0], c.width, math.sqrt(c.width),
                             ops._flags.value | _lib.FLAG_STRICT_TOKENS)
            _lib.check(st, "tpb200_pi05_embed")
        first = True
        for l, L in enumerate(self.prefix):
            if first:
                rowop(_lib.ROW_RMSNORM, b["ph"], c.width, y_out=b["px"], w0=L["in_norm"], eps=c.eps)
                first = False
            else:
                rowop(_lib.ROW_RMSNORM, b["py"], c.width, y_out=b["px"], res_in=b["ph"], h_out=b["ph"], w0=L["in_norm"],
                      eps=c.eps)
            L["qkv"].dense_qkv(b["px"], b["p_q"], self.cache[l, 0], self.cache[l, 1], b["pos_prefix"], self.cos, self.sin,
                               c.q_dim)
            self._attention(b["p_q"], self.cache[l, 0, :S], self.cache[l, 1, :S], b["p_attn"])
            L["o"].dense(b["p_attn"], b["py"])
            rowop(_lib.ROW_RMSNORM, b["py"], c.width, b["q_p"], res_in=b["ph"], h_out=b["ph"], w0=L["post_norm"],
                  eps=c.eps)
            # GELU(gate) * up rides in the row kernel: in the GEMM's epilogue (ACT_GEGLU) it would sit between
            # the accumulator reads of a 128 x 256 tile and hold up the next tile's MMAs
            L["gate_up"](b["q_p"], b["p_gu"])
            rowop(_lib.ROW_GELU_MUL, b["p_gu"], c.mlp, b["q_pmlp"])
            L["down"](b["q_pmlp"], b["py"])

    def _ada_modulation(self, num_steps, out=None):
        """adarms_cond per step and every adaptive norm's (scale, shift, gate): [steps, n_norms, 3, width]
        (pi0_pytorch.py:817-839; GemmaRMSNorm.dense, modeling_gemma.py:96-103)."""
        c, d = self.cfg, self.device
        ew = c.expert_width
        if num_steps not in self._time_emb:      # host-side constants: made once, outside any graph capture
            dt = -1.0 / num_steps
            ts = torch.tensor([1.0 + i * dt for i in range(num_steps)], dtype=torch.float32)
            self._time_emb[num_steps] = sinusoidal_time_embedding(ts, ew).to(torch.bfloat16).to(d)
        emb = self._time_emb[num_steps]
        t1 = torch.empty((2, num_steps, ew), dtype=torch.bfloat16, device=d)
        self.time_mlp_in.dense(emb, t1[0], ACT_SILU)
        self.time_mlp_out.dense(t1[0], t1[1], ACT_SILU)
        mod = torch.empty((num_steps, self.n_norms * 3 * ew), dtype=torch.bfloat16, device=d) if out is None else out.view(num_steps, -1)
        self.ada_dense.dense(t1[1], mod)
        return mod.view(num_steps, self.n_norms, 3, ew)

    def _shifts(self, mod, out=None):
        """W * shift of every linear behind an adaptive norm, per step: what is left of the norm's shift when its RMS
        factor is applied behind the linear.  fp32, alpha included; rows in the order of the weights."""
        c, n = self.cfg, mod.shape[0]
        if out is None:
            empty = lambda lin: torch.empty((n, lin.N), dtype=torch.float32, device=self.device)    # noqa: E731
            out = dict(qkv=[empty(L["qkv"]) for L in self.expert], gate_up=[empty(L["gate_up"]) for L in self.expert],
                       out=empty(self.action_out))
        for l, L in enumerate(self.expert):
            L["qkv"].dense(mod[:, 2 * l, 1], out["qkv"][l], bias=False)
            L["gate_up"].dense(mod[:, 2 * l + 1, 1], out["gate_up"][l], bias=False)
        self.action_out.dense(mod[:, 2 * c.expert_layers, 1], out["out"]).mul_(-1.0 / n)             # times the Euler step
        return out

    def _norm_in(self, shift):
        b, c = self.b, self.cfg
        return _lib.W4NormArgs(in_sumsq=ops._ptr(b["e_ss"]), in_shift=ops._ptr(shift), in_parts=c.expert_width // 128, in_eps=c.eps)

    def _norm_out(self, scale, gate=None, first=False):
        b, p = self.b, ops._ptr
        return _lib.W4NormArgs(res_in=0 if first else p(b["eh"]), gate=p(gate), scale=p(scale), h_out=p(b["eh"]),
                               out_sumsq=p(b["e_ss"]))

    def denoise_step(self, mod, dt, shift=None):
        """One Euler step: v = expert(x_t | cache); x_t += dt * v.  `shift` (one row per linear, `_shifts`): the norms and the
        Euler update run in the epilogues of the linears around them, x_bf holds bf16(x_t) before and after; None: in row
        kernels between the linears."""
        c, b = self.cfg, self.b
        S, A, ew = c.prefix_len, c.action_horizon, c.expert_width
        if shift is None:
            b["x_bf"].copy_(b["x_t"])
            self._expert_with_row_kernels(mod)
            b["x_t"].add_(b["v_out"], alpha=dt)
        else:
            self.action_in.dense(b["x_bf"], b["ex"], norm=self._norm_out(mod[0, 0], first=True))
            for l, L in enumerate(self.expert):
                m_in, m_post = mod[2 * l], mod[2 * l + 1]
                L["qkv"].dense_qkv(b["ex"], b["e_q"], self.cache[l, 0, S:], self.cache[l, 1, S:], b["pos_suffix"], self.cos,
                                   self.sin, c.q_dim, norm=self._norm_in(shift["qkv"][l]))
                self._attention(b["e_q"], self.cache[l, 0, :S + A], self.cache[l, 1, :S + A], b["e_attn"])
                L["o"].dense(b["e_attn"], b["ex"], norm=self._norm_out(m_post[0], m_in[2]))
                L["gate_up"].dense(b["ex"], b["e_mlp"], ACT_GELU, gated=True, norm=self._norm_in(shift["gate_up"][l]))
                L["down"].dense(b["e_mlp"], b["ex"], norm=self._norm_out(mod[2 * l + 2, 0], m_post[2]))
            norm = self._norm_in(shift["out"])
            norm.copy_out = ops._ptr(b["x_bf"])
            self.action_out.dense(b["ex"], b["x_t"], norm=norm, bias=False, scale=dt, beta=1.0)

    def _expert_with_row_kernels(self, mod):
        c, b = self.cfg, self.b
        S, A, ew = c.prefix_len, c.action_horizon, c.expert_width
        self.action_in.dense(b["x_bf"], b["eh"])
        prev_gate = None
        for l, L in enumerate(self.expert):
            m_in, m_post = mod[2 * l], mod[2 * l + 1]
            if prev_gate is None:
                rowop(_lib.ROW_ADARMS, b["eh"], ew, y_out=b["ex"], w0=m_in[0], w1=m_in[1], eps=c.eps)
            else:
                rowop(_lib.ROW_ADARMS, b["ey"], ew, y_out=b["ex"], res_in=b["eh"], gate=prev_gate, h_out=b["eh"], w0=m_in[0],
                      w1=m_in[1], eps=c.eps)
            L["qkv"].dense_qkv(b["ex"], b["e_q"], self.cache[l, 0, S:], self.cache[l, 1, S:], b["pos_suffix"], self.cos,
                               self.sin, c.q_dim)
            self._attention(b["e_q"], self.cache[l, 0, :S + A], self.cache[l, 1, :S + A], b["e_attn"])
            L["o"].dense(b["e_attn"], b["ey"])
            rowop(_lib.ROW_ADARMS, b["ey"], ew, y_out=b["ex"], res_in=b["eh"], gate=m_in[2], h_out=b["eh"], w0=m_post[0],
                  w1=m_post[1], eps=c.eps)
            if c.expert_mlp % 64 == 0:
                L["gate_up"].dense(b["ex"], b["e_mlp"], ACT_GELU, gated=True)
            else:                       # the gated epilogue pairs 64 gate rows with 64 up rows
                L["gate_up"].dense(b["ex"], b["e_gu"])
                rowop(_lib.ROW_GELU_MUL, b["e_gu"], c.expert_mlp, y_out=b["e_mlp"])
            L["down"].dense(b["e_mlp"], b["ey"])
            prev_gate = m_post[2]
        m_f = mod[2 * c.expert_layers]
        rowop(_lib.ROW_ADARMS, b["ey"], ew, y_out=b["ex"], res_in=b["eh"], gate=prev_gate, h_out=b["eh"], w0=m_f[0], w1=m_f[1],
              eps=c.eps)
        self.action_out.dense(b["ex"], b["v_out"])

    def _modulation(self, num_steps):
        """The adaptive norms' (scale, shift, gate) for every step of an `num_steps` schedule.  They depend on
        the schedule and the weights only, not on the observation (the reference precomputes the per-step
        conditioning vectors for its graphs too: pi0_pytorch.py:770-839), so they are computed once per schedule -- by
        the warm-up pass that precedes a capture -- and stay out of the per-inference graph.  Made again in the same memory
        when a weight has been written since (a capture that finds them out of date contains the making)."""
        mod, shift, held = self._mod.get(num_steps, (None, None, None))
        linears = [self.time_mlp_in, self.time_mlp_out, self.ada_dense]
        if self.fold_norms:
            linears.append(self.action_out)
            for L in self.expert:
                linears += L["qkv"], L["gate_up"]
        marks = _Marks.of(linears)
        if held is None or not marks.same(held):
            capturing = torch.cuda.is_current_stream_capturing()
            if capturing and mod is None:
                raise TurboPiError("the modulation table of a new schedule must be built before the capture")
            mod = self._ada_modulation(num_steps, mod)
            shift = self._shifts(mod, shift) if self.fold_norms else None
            if not capturing:
                self._mod[num_steps] = (mod, shift, marks)
        return mod, shift

    def denoise_loop(self, num_steps):
        mod, shift = self._modulation(num_steps)
        self.b["x_t"].copy_(self.noise)
        self.b["x_bf"].copy_(self.noise)
        dt = -1.0 / num_steps
        for i in range(num_steps):
            at = None if shift is None else dict(qkv=[s[i] for s in shift["qkv"]], gate_up=[s[i] for s in shift["gate_up"]],
                                                 out=shift["out"][i])
            self.denoise_step(mod[i], dt, at)
        self.actions.copy_(self.b["x_t"])

    def forward(self, num_steps):
        with ops.launch_flags(self.launch_flags):
            self.vision_tower()
            self.prefix_pass()
            self.denoise_loop(num_steps)

    # ------------------------------------------------------------------ public API
    def capture(self, num_steps):
        """Capture vision + prefix + the whole denoise loop as one CUDA graph."""
        side = torch.cuda.Stream(device=self.device)
        side.wait_stream(torch.cuda.current_stream(self.device))     # the warm-up makes tables of weights written there
        with torch.cuda.stream(side):
            self.forward(num_steps)            # warm-up: attribute setup, allocator pools
        torch.cuda.synchronize(self.device)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=side):
            self.forward(num_steps)
        self._graph, self._graph_steps = g, num_steps

    @torch.no_grad()
    def infer(self, images_u8, tokens, noise, num_steps=10, use_graph=True, image_valid=None, prompt_len=None):
        """images_u8 [num_images, H, W, 3] uint8, tokens [text_len] int64, noise [horizon, action_dim] fp32
        (host or device tensors); `image_valid` / `prompt_len` as in `set_valid` (default: everything valid).
        A token outside the embedding table is refused where it lies on the host; on the device it makes every action NaN
        and is recorded (tpb200_device_error: 401).  Returns the device tensor of actions [horizon, action_dim] fp32."""
        if not tokens.is_cuda and tokens.numel():
            low, high = torch.aminmax(tokens)
            vocab = self.embed_tokens.shape[0]
            if low < -vocab or high >= vocab:
                raise TurboPiError(f"token ids {int(low)}..{int(high)} are outside the embedding table of {vocab} rows")
        if image_valid is not None or prompt_len is not None or not bool(self.valid.all()):
            self.set_valid(image_valid, prompt_len)
        self.images.copy_(images_u8, non_blocking=True)
        self.tokens.copy_(tokens, non_blocking=True)
        self.noise.copy_(noise, non_blocking=True)
        if use_graph:
            if self._graph is None or self._graph_steps != num_steps:
                self.capture(num_steps)
            else:                              # tables that a write has made stale: in the memory the graph reads them from
                if self._pos_marks is None or self._pos_marks.written():
                    self._positions()
                marks = self._mod[num_steps][2]
                if marks is None or marks.written():
                    self._modulation(num_steps)
            self._graph.replay()
        else:
            self.forward(num_steps)
        return self.actions
