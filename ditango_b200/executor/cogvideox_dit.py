"""Random-init CogVideoX-5B-shaped DiT driven by the sequence-parallel attention path.

A plain-PyTorch restatement of the reference's CogVideoX fork -- block structure of
executor/cogvideox/cogvideox_transformer_3d.py:139-190 (LayerNormZero modulation, joint text+video
attention, GELU-tanh feed-forward), model forward :447-543 (embed, shard tokens and rotary tables
over the sequence-parallel group with zero-padded uneven shards, blocks, gather, final norm / proj,
unpatchify), attention adapter executor/cogvideox/attention_processor.py:31-86 (use-ditango) and
baseline/ulysses.py:32-136 (use-ulysses), denoising loop pipeline_cogvideox.py:608-656 (in-batch
classifier-free guidance).  diffusers is not required.  Weights are random: this module exists to
measure per-step latency and exposed communication of the two attention modes inside a whole
denoising loop; projections and feed-forward are library GEMMs, the attention is this package's.
"""
import math
from dataclasses import dataclass
from typing import Tuple

import torch
import torch.nn as nn
import torch.nn.functional as F
from torch.autograd import forward_ad

from ..baseline.ulysses import heads_to_sequence, sequence_to_heads
from ..core.attention import proAttention
from ..utils import remove_padding_after_gather, split_tensor_uneven, update_timestep
from .. import ops as _engine


@dataclass
class DiTConfig:
    num_layers: int = 42
    num_heads: int = 48
    head_dim: int = 64
    in_channels: int = 16
    patch_size: int = 2
    text_dim: int = 4096
    time_dim: int = 512
    frames: int = 13
    height: int = 60
    width: int = 90
    text_len: int = 226

    @property
    def dim(self) -> int:
        return self.num_heads * self.head_dim

    @property
    def video_tokens(self) -> int:
        return self.frames * (self.height // self.patch_size) * (self.width // self.patch_size)


def rotary_tables(cfg: DiTConfig, device, dtype=torch.float32) -> Tuple[torch.Tensor, torch.Tensor]:
    """3-D rotary tables [video_tokens, head_dim]: head_dim split 1/4 : 3/8 : 3/8 over (t, h, w)."""
    d_t = cfg.head_dim // 4
    d_h = d_w = (cfg.head_dim - d_t) // 2
    gh, gw = cfg.height // cfg.patch_size, cfg.width // cfg.patch_size

    def axis(n, d):
        freqs = 1.0 / (10000.0 ** (torch.arange(0, d, 2, dtype=torch.float32) / d))
        ang = torch.outer(torch.arange(n, dtype=torch.float32), freqs)
        return ang.repeat_interleave(2, dim=1)                       # [n, d]
    t = axis(cfg.frames, d_t)[:, None, None, :].expand(cfg.frames, gh, gw, d_t)
    h = axis(gh, d_h)[None, :, None, :].expand(cfg.frames, gh, gw, d_h)
    w = axis(gw, d_w)[None, None, :, :].expand(cfg.frames, gh, gw, d_w)
    ang = torch.cat([t, h, w], dim=-1).reshape(-1, cfg.head_dim)
    return ang.cos().to(device=device, dtype=dtype), ang.sin().to(device=device, dtype=dtype)


def apply_rotary(x: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor) -> torch.Tensor:
    """x [B, S, H, D] with interleaved (real, imaginary) channel pairs; cos/sin [S, D]."""
    xr, xi = x.float().unflatten(-1, (-1, 2)).unbind(-1)
    rot = torch.stack([-xi, xr], dim=-1).flatten(-2)
    return (x.float() * cos[None, :, None, :] + rot * sin[None, :, None, :]).to(x.dtype)


def _unobserved(m: nn.Module, kind: type) -> bool:
    """True when calling `m` is running kind.forward and nothing else: no subclass, no hook, no replaced forward."""
    mod = nn.modules.module
    return (type(m) is kind and "forward" not in m.__dict__ and
            not (m._forward_hooks or m._forward_pre_hooks or m._backward_hooks or m._backward_pre_hooks) and
            not (mod._global_forward_hooks or mod._global_forward_pre_hooks or mod._global_backward_hooks or
                 mod._global_backward_pre_hooks))


_PLAIN_TYPES = (torch.Tensor, nn.Parameter)


def _addressable(*tensors: torch.Tensor) -> bool:
    """Whether a kernel that is given addresses sees all there is to `tensors`: values in memory of their own (no subclass,
    nothing that torch.func wraps) and no forward-mode tangent, which it would drop.  Alignment: 16 bytes."""
    # (outside of a dual level, the usual case, no tensor has a tangent; the level is not public: without it all are asked)
    duals = getattr(forward_ad, "_current_level", 0) >= 0
    try:
        for x in tensors:
            address = x.data_ptr()
            if type(x) not in _PLAIN_TYPES or address == 0 or address % 16 or (duals and forward_ad.unpack_dual(x).tangent is not None):
                return False
    except RuntimeError:        # no storage
        return False
    return True


def _plain_norm(norm: nn.Module, dim: int, device: torch.device) -> bool:
    """True for a bf16 LayerNorm over the last `dim` channels on `device` that a kernel may stand in for."""
    return (_unobserved(norm, nn.LayerNorm) and tuple(norm.normalized_shape) == (dim,) and
            norm.weight is not None and norm.bias is not None and norm.weight.dtype == norm.bias.dtype == torch.bfloat16 and
            norm.weight.device == norm.bias.device == device and _addressable(norm.weight, norm.bias))


def _plain_bf16(device: torch.device, *tensors: torch.Tensor) -> bool:
    return all(x.dtype == torch.bfloat16 and x.device == device and x.is_contiguous() for x in tensors) and _addressable(*tensors)


def _rotate_video(x, cos, sin, text_len: int) -> torch.Tensor:
    return torch.cat([x[:, :text_len], apply_rotary(x[:, text_len:], cos, sin)], dim=1)


class _NormRotate(torch.autograd.Function):
    """The kernel of norm_and_rotate with the gradient of the operations it stands in for: they are run again on the saved
    inputs."""

    @staticmethod
    def launch(q, k, q_weight, q_bias, k_weight, k_bias, cos, sin, q_eps, k_eps, text_len):
        return _engine.norm_rope(q, k, (q_weight, q_bias, q_eps), (k_weight, k_bias, k_eps), cos, sin, text_len)

    @staticmethod
    def forward(ctx, *args):
        ctx.save_for_backward(*args[:8])
        ctx.eps_and_len = args[8:]
        return _NormRotate.launch(*args)

    @staticmethod
    def backward(ctx, *grads):
        q_eps, k_eps, text_len = ctx.eps_and_len
        with torch.enable_grad(), torch.autocast("cuda", enabled=False):
            # an alias per argument: a tensor that is passed twice gets each argument's own share
            args = [x.view_as(x) for x in ctx.saved_tensors]
            q, k, q_weight, q_bias, k_weight, k_bias, cos, sin = args
            outs = [_rotate_video(F.layer_norm(x, x.shape[-1:], w, b, eps), cos, sin, text_len)
                    for x, w, b, eps in ((q, q_weight, q_bias, q_eps), (k, k_weight, k_bias, k_eps))]
        wanted = [x for x, need in zip(args, ctx.needs_input_grad) if need]
        pairs = [(o, g) for o, g in zip(outs, grads) if o.requires_grad]
        got = iter(torch.autograd.grad([o for o, _ in pairs], wanted, [g for _, g in pairs],
                                       create_graph=torch.is_grad_enabled(), allow_unused=True))
        return tuple(next(got) if need else None for need in ctx.needs_input_grad)


def norm_and_rotate(q, k, norm_q, norm_k, cos, sin, text_len: int) -> Tuple[torch.Tensor, torch.Tensor]:
    """norm_q / norm_k over the heads of q, k [B, S, H, D], then rotary embedding of the tokens behind the first
    text_len.  On a GPU in bf16 this is one kernel over both tensors (fp32 inside, one rounding at the end)."""
    D = q.shape[-1]
    if (q.is_cuda and D in (64, 128) and q.shape == k.shape and _plain_bf16(q.device, q, k) and
            _plain_norm(norm_q, D, q.device) and _plain_norm(norm_k, D, q.device) and
            all(x.dtype == torch.float32 and x.shape == (q.shape[1] - text_len, D) and x.is_contiguous() and
                x.device == q.device and (x.numel() == 0 or _addressable(x)) for x in (cos, sin)) and
            not torch.is_autocast_enabled("cuda")):
        args = (q, k, norm_q.weight, norm_q.bias, norm_k.weight, norm_k.bias, cos, sin, norm_q.eps, norm_k.eps, text_len)
        if torch.is_grad_enabled() and any(x.requires_grad for x in args[:8]):
            return _NormRotate.apply(*args)
        return _NormRotate.launch(*args)
    return tuple(_rotate_video(x, cos, sin, text_len).contiguous() for x in (norm_q(q), norm_k(k)))


def _plain_modulation(h: torch.Tensor, mod: torch.Tensor) -> bool:
    """Whether the kernels can take `mod`: one bf16 row per sequence of h.  (A row that broadcasts over the batch, another
    dtype or layout -- what a hook on, or a replacement of, the projection may return -- stays with the separate operations.)"""
    return tuple(mod.shape) == (h.shape[0], 6 * h.shape[-1]) and _plain_bf16(h.device, mod)


def gated_residual(h, enc, a, mod) -> Tuple[torch.Tensor, torch.Tensor]:
    """(h, enc) + gate * (their parts of the joint tensor a [B, text + video, dim], text first), gates from the modulation.
    For streams that LayerNormZero.fuses; one kernel where `a` and `mod` allow it."""
    text_len = enc.shape[1]
    if _plain_modulation(h, mod) and tuple(a.shape) == (h.shape[0], text_len + h.shape[1], h.shape[2]) and _plain_bf16(h.device, a):
        return _engine.gate_add(h, enc, a, mod)
    _, _, gate, _, _, e_gate = mod.chunk(6, dim=1)
    return h + gate[:, None] * a[:, text_len:], enc + e_gate[:, None] * a[:, :text_len]


class LayerNormZero(nn.Module):
    def __init__(self, time_dim: int, dim: int):
        super().__init__()
        self.linear = nn.Linear(time_dim, 6 * dim)
        self.norm = nn.LayerNorm(dim, eps=1e-5)

    def fuses(self, h, enc) -> bool:
        """Whether `joint` may stand in for forward(): bf16 streams on a GPU, no gradient to be recorded (the kernels have
        none), and no hook on the modules whose calls it skips."""
        dim = h.shape[-1]
        return (h.is_cuda and not torch.is_grad_enabled() and not torch.is_autocast_enabled("cuda") and
                dim % 256 == 0 and dim <= _engine.MOD_MAX_DIM and
                _plain_bf16(h.device, h, enc) and
                _unobserved(self, LayerNormZero) and _plain_norm(self.norm, dim, h.device))

    def joint(self, h, enc, temb):
        """([B, text + video, dim] normalised and modulated, text first; the modulation, whose gates gated_residual takes)."""
        mod = self.linear(F.silu(temb))
        if _plain_modulation(h, mod):
            return _engine.ln_modulate(h, enc, self.norm.weight, self.norm.bias, self.norm.eps, mod), mod
        nh, nenc, _, _ = self.modulate(h, enc, mod)
        return torch.cat([nenc, nh], dim=1), mod

    def forward(self, h, enc, temb):
        return self.modulate(h, enc, self.linear(F.silu(temb)))

    def modulate(self, h, enc, mod):
        shift, scale, gate, e_shift, e_scale, e_gate = mod.chunk(6, dim=1)
        h = self.norm(h) * (1 + scale)[:, None] + shift[:, None]
        enc = self.norm(enc) * (1 + e_scale)[:, None] + e_shift[:, None]
        return h, enc, gate[:, None], e_gate[:, None]


class DiTBlock(nn.Module):
    def __init__(self, cfg: DiTConfig, layer_id: int, group, mode: str):
        super().__init__()
        dim = cfg.dim
        self.cfg, self.mode, self.group = cfg, mode, group
        self.norm1 = LayerNormZero(cfg.time_dim, dim)
        self.to_q, self.to_k, self.to_v = (nn.Linear(dim, dim) for _ in range(3))
        self.norm_q = nn.LayerNorm(cfg.head_dim, eps=1e-6)
        self.norm_k = nn.LayerNorm(cfg.head_dim, eps=1e-6)
        self.to_out = nn.Linear(dim, dim)
        self.norm2 = LayerNormZero(cfg.time_dim, dim)
        self.ff_in = nn.Linear(dim, 4 * dim)
        self.ff_out = nn.Linear(4 * dim, dim)
        self.attention = proAttention(layer_id, group) if mode != "ulysses" else None

    def _attend(self, h, enc, rope):
        cfg = self.cfg
        B, text_len = h.shape[0], enc.shape[1]
        H, D = cfg.num_heads, cfg.head_dim
        if self.mode == "ulysses":
            # project the local shards, exchange heads for sequence per stream, then text before video
            def proj(x):
                return [f(x).view(B, x.shape[1], H, D) for f in (self.to_q, self.to_k, self.to_v)]
            q, k, v = heads_to_sequence(proj(h), self.group)
            eq, ek, ev = heads_to_sequence(proj(enc), self.group)
            text_all = eq.shape[1]
            q, k, v = (torch.cat([a, b], dim=1) for a, b in ((eq, q), (ek, k), (ev, v)))
            cos, sin = rope                                          # unsharded (padded) tables
            q, k = norm_and_rotate(q, k, self.norm_q, self.norm_k, cos, sin, text_all)
            out, _ = _engine.flash_partial(q, k, v.contiguous(), out_dtype=torch.bfloat16,
                                           softmax_scale=1.0 / math.sqrt(D))
            o_enc = sequence_to_heads(out[:, :text_all].contiguous(), self.group).flatten(2).to(h.dtype)
            o_vid = sequence_to_heads(out[:, text_all:].contiguous(), self.group).flatten(2).to(h.dtype)
            return self.to_out(o_vid), self.to_out(o_enc)
        out = self._attend_joint(torch.cat([enc, h], dim=1), text_len, rope)
        return out[:, text_len:], out[:, :text_len]

    def _attend_joint(self, x, text_len, rope):
        """Attention of the joint sequence x [B, text + video, dim], projected back."""
        B, H, D = x.shape[0], self.cfg.num_heads, self.cfg.head_dim
        q, k, v = (f(x).view(B, -1, H, D) for f in (self.to_q, self.to_k, self.to_v))
        cos, sin = rope                                              # this rank's slice of the tables
        q, k = norm_and_rotate(q, k, self.norm_q, self.norm_k, cos, sin, text_len)
        out = self.attention.attn(q, k, v.contiguous())
        return self.to_out(out.to(x.dtype).flatten(2))

    def forward(self, h, enc, temb, rope):
        text_len = enc.shape[1]
        # (a subclass's or an instance's own _attend takes the streams one by one)
        if self.mode != "ulysses" and getattr(self._attend, "__func__", None) is DiTBlock._attend and self.norm1.fuses(h, enc):
            x, mod = self.norm1.joint(h, enc, temb)
            h, enc = gated_residual(h, enc, self._attend_joint(x, text_len, rope), mod)
        else:
            nh, nenc, gate, e_gate = self.norm1(h, enc, temb)
            a_h, a_enc = self._attend(nh, nenc, rope)
            h = h + gate * a_h
            enc = enc + e_gate * a_enc
        if self.norm2.fuses(h, enc):
            x, mod = self.norm2.joint(h, enc, temb)
            return gated_residual(h, enc, self._feed_forward(x), mod)
        nh, nenc, gate, e_gate = self.norm2(h, enc, temb)
        ff = self._feed_forward(torch.cat([nenc, nh], dim=1))
        return h + gate * ff[:, text_len:], enc + e_gate * ff[:, :text_len]

    def _feed_forward(self, x):
        return self.ff_out(F.gelu(self.ff_in(x), approximate="tanh"))


class CogVideoXDiT(nn.Module):
    """mode: 'ditango' / 'ring' (proAttention; the stride schedule decides reuse) or 'ulysses'."""

    def __init__(self, cfg: DiTConfig, group, mode: str = "ditango"):
        super().__init__()
        self.cfg, self.group, self.mode = cfg, group, mode
        p = cfg.patch_size
        self.patch_embed = nn.Linear(cfg.in_channels * p * p, cfg.dim)
        self.text_proj = nn.Linear(cfg.text_dim, cfg.dim)
        self.time_embed = nn.Sequential(nn.Linear(cfg.dim, cfg.time_dim), nn.SiLU(), nn.Linear(cfg.time_dim, cfg.time_dim))
        self.blocks = nn.ModuleList(DiTBlock(cfg, i, group, mode) for i in range(cfg.num_layers))
        self.norm_final = nn.LayerNorm(cfg.dim, eps=1e-5)
        self.norm_out = nn.LayerNorm(cfg.dim, eps=1e-5, elementwise_affine=False)
        self.out_mod = nn.Linear(cfg.time_dim, 2 * cfg.dim)
        self.proj_out = nn.Linear(cfg.dim, cfg.in_channels * p * p)
        self._rope = None

    def _timestep_embedding(self, t: torch.Tensor) -> torch.Tensor:
        half = self.cfg.dim // 2
        freqs = torch.exp(-math.log(10000.0) * torch.arange(half, device=t.device, dtype=torch.float32) / half)
        ang = t.float()[:, None] * freqs[None]
        return torch.cat([ang.cos(), ang.sin()], dim=-1)

    def forward(self, latents: torch.Tensor, text: torch.Tensor, timestep: torch.Tensor) -> torch.Tensor:
        """latents [B, F, C, H, W], text [B, text_len, text_dim], timestep [B] -> noise prediction like latents."""
        cfg, p = self.cfg, self.cfg.patch_size
        B, Fr, C, Hh, Ww = latents.shape
        dtype = self.patch_embed.weight.dtype
        temb = self.time_embed(self._timestep_embedding(timestep).to(dtype))
        x = latents.reshape(B, Fr, C, Hh // p, p, Ww // p, p).permute(0, 1, 3, 5, 2, 4, 6).flatten(4).flatten(1, 3)
        h = self.patch_embed(x.to(dtype))
        enc = self.text_proj(text.to(dtype))
        N, r = self.group.world_size, self.group.rank_in_group
        if self._rope is None:
            self._rope = rotary_tables(cfg, latents.device)
        cos, sin = self._rope
        if N > 1:
            h = split_tensor_uneven(h, N, dim=1, tensor_name="hidden")[r]
            enc = split_tensor_uneven(enc, N, dim=1, tensor_name="encoder_hidden")[r]
            if self.mode == "ulysses":
                # full tables in the gathered order: every rank's shard keeps its zero padding
                cos = torch.cat(split_tensor_uneven(cos, N, dim=0), dim=0)
                sin = torch.cat(split_tensor_uneven(sin, N, dim=0), dim=0)
            else:
                cos, sin = split_tensor_uneven(cos, N, dim=0)[r], split_tensor_uneven(sin, N, dim=0)[r]
        for blk in self.blocks:
            h, enc = blk(h, enc, temb, (cos, sin))
        if N > 1:
            h = remove_padding_after_gather(self.group.all_gather(h.contiguous(), dim=1), "hidden")
            enc = remove_padding_after_gather(self.group.all_gather(enc.contiguous(), dim=1), "encoder_hidden")
        text_len = enc.shape[1]
        h = self.norm_final(torch.cat([enc, h], dim=1))[:, text_len:]
        shift, scale = self.out_mod(F.silu(temb)).chunk(2, dim=1)
        h = self.proj_out(self.norm_out(h) * (1 + scale)[:, None] + shift[:, None])
        out = h.reshape(B, Fr, Hh // p, Ww // p, -1, p, p).permute(0, 1, 4, 2, 5, 3, 6).flatten(5, 6).flatten(3, 4)
        return out


@torch.no_grad()
def denoise(model: CogVideoXDiT, latents: torch.Tensor, text_cond: torch.Tensor, text_uncond: torch.Tensor,
            num_steps: int, guidance_scale: float = 6.0, first_step: int = 0, on_step=None) -> torch.Tensor:
    """Denoising loop with in-batch classifier-free guidance and a plain Euler update (the scheduler is
    not part of the attention path).  Sets the global step index before every model call."""
    text = torch.cat([text_uncond, text_cond], dim=0)
    for i in range(first_step, first_step + num_steps):
        update_timestep(i)
        t = torch.full((2 * latents.shape[0],), 1000.0 * (1.0 - i / max(1, first_step + num_steps)), device=latents.device)
        noise = model(torch.cat([latents, latents], dim=0), text, t).float()
        n_uncond, n_text = noise.chunk(2)
        noise = n_uncond + guidance_scale * (n_text - n_uncond)
        latents = (latents.float() - noise / (first_step + num_steps)).to(latents.dtype)
        if on_step is not None:
            on_step(i)
    return latents
