"""The fused layer norm + modulation and the gated residual of the transformer block against the same steps in 64 bits.

The kernels round once, to bf16 (2^-9 relative); their fp32 arithmetic adds about 1e-6 of the terms' size."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _bf16(g, *shape, scale=1.0, shift=0.0):
    return (torch.randn(*shape, generator=g) * scale + shift).to(torch.bfloat16).cuda()


# The last four go round the kernels' grid-stride loops several times, with remainders: on 148 SMs a pass of ln_modulate
# covers 4736 / B rows and one of gate_add 1.2 M / B pieces of 8 values.
@pytest.mark.parametrize("B,Sv,St,dim", [(1, 1, 1, 256), (2, 9, 3, 512), (1, 8, 16, 768), (2, 333, 226, 3072), (1, 1500, 1, 1536), (3, 40, 77, 2816),
                                         (2, 17550, 226, 3072), (1, 9477, 5000, 1536), (1, 4737, 9479, 1792), (3, 3, 40001, 256)])
def test_ln_modulate_and_gate_add_match_exact(B, Sv, St, dim):
    from ditango_b200 import ops
    g = torch.Generator().manual_seed(dim + Sv)
    video, text = _bf16(g, B, Sv, dim, scale=3.0, shift=0.7), _bf16(g, B, St, dim)
    w, b, mod = _bf16(g, dim), _bf16(g, dim), _bf16(g, B, 6 * dim)
    a = _bf16(g, B, St + Sv, dim)
    m = mod.double().view(B, 6, 1, dim)

    def norm(x, shift, scale):
        x = x.double()
        x = (x - x.mean(-1, keepdim=True)) * torch.rsqrt(x.var(-1, unbiased=False, keepdim=True) + 1e-5) * w.double() + b.double()
        return x * (1 + scale) + shift

    got = ops.ln_modulate(video, text, w, b, 1e-5, mod).double()
    want = torch.cat([norm(text, m[:, 3], m[:, 4]), norm(video, m[:, 0], m[:, 1])], dim=1)
    assert ((got - want).abs() <= want.abs() * 2.0 ** -8 + 1e-4).all()
    gv, gt = ops.gate_add(video, text, a, mod)
    for got, want in ((gv, video.double() + m[:, 2] * a[:, St:].double()), (gt, text.double() + m[:, 5] * a[:, :St].double())):
        assert ((got.double() - want).abs() <= want.abs() * 2.0 ** -8 + 1e-5).all()


def test_block_takes_the_fused_path_only_where_nothing_observes_it():
    from ditango_b200 import ops
    from ditango_b200.core import redundancy_map as rmod
    from ditango_b200.core.config import init_config
    from ditango_b200.core.group_coordinate import SingleRankGroup
    from ditango_b200.executor.cogvideox_dit import DiTBlock, DiTConfig
    from ditango_b200.utils import update_timestep
    cfg = init_config(None, make_output_dir=False)
    cfg.num_layers, cfg.num_inference_steps = 1, 1
    rmod.destroy_redundancy_map()
    rmod.init_redundancy_map(cfg, world_size=1)
    update_timestep(0)
    torch.manual_seed(0)
    dc = DiTConfig(num_layers=1, num_heads=4, frames=1, height=8, width=8, text_len=5)
    block = DiTBlock(dc, 0, SingleRankGroup(torch.device("cuda", 0)), "ditango").cuda().to(torch.bfloat16)
    h, enc, temb = (torch.randn(s, device="cuda").to(torch.bfloat16) for s in ((2, 16, 256), (2, 5, 256), (2, 512)))
    rope = (torch.ones(16, 64, device="cuda"), torch.zeros(16, 64, device="cuda"))
    with torch.no_grad():
        n0 = ops.LaunchLog.count
        fused = block(h, enc, temb, rope)
        assert ops.LaunchLog.count - n0 == 6          # norm + gate twice, norm + rotary, attention
        hooks = [m.register_forward_hook(lambda m, i, o: None) for m in (block.norm1, block.norm2.norm, block.norm_q)]
        n0 = ops.LaunchLog.count
        plain = block(h, enc, temb, rope)
        assert ops.LaunchLog.count - n0 == 1
        for x in hooks:
            x.remove()
    n0 = ops.LaunchLog.count
    out = block(h, enc, temb, rope)
    assert out[0].requires_grad and ops.LaunchLog.count - n0 == 2      # gradients of the residual path stay
    for a, b, c in zip(fused, plain, out):            # bf16 roundings in between: a few units in the last place
        scale = b.float().abs().max()
        assert (a.float() - b.float()).abs().max() <= scale * 2.0 ** -5 and (c.float() - b.float()).abs().max() <= scale * 2.0 ** -5
    rmod.destroy_redundancy_map()


@pytest.fixture
def block_inputs():
    """A bf16 block of four heads, its streams (batch 2), a timestep embedding and unit rotary tables."""
    from ditango_b200.core import redundancy_map as rmod
    from ditango_b200.core.config import init_config
    from ditango_b200.core.group_coordinate import SingleRankGroup
    from ditango_b200.executor.cogvideox_dit import DiTBlock, DiTConfig
    from ditango_b200.utils import update_timestep
    cfg = init_config(None, make_output_dir=False)
    cfg.num_layers, cfg.num_inference_steps = 1, 1
    rmod.destroy_redundancy_map()
    rmod.init_redundancy_map(cfg, world_size=1)
    update_timestep(0)
    torch.manual_seed(1)
    dc = DiTConfig(num_layers=1, num_heads=4, frames=1, height=8, width=8, text_len=5)
    block = DiTBlock(dc, 0, SingleRankGroup(torch.device("cuda", 0)), "ditango").cuda().to(torch.bfloat16)
    h, enc, temb = (torch.randn(s, device="cuda").to(torch.bfloat16) for s in ((2, 16, 256), (2, 5, 256), (2, 512)))
    yield block, h, enc, temb, (torch.ones(16, 64, device="cuda"), torch.zeros(16, 64, device="cuda"))
    rmod.destroy_redundancy_map()


def _general(block, *args):
    """The block with its separate operations: a hook on the layers that the kernels would stand in for."""
    hooks = [m.register_forward_hook(lambda m, i, o: None) for m in (block.norm1, block.norm2, block.norm_q)]
    try:
        return block(*args)
    finally:
        for x in hooks:
            x.remove()


def _close(got, want):
    for a, b in zip(got, want):                       # bf16 roundings in between, as above
        assert a.dtype == b.dtype and a.shape == b.shape
        assert (a.float() - b.float()).abs().max() <= b.float().abs().max() * 2.0 ** -5


@torch.no_grad()
def test_one_timestep_for_the_whole_batch(block_inputs):
    block, h, enc, temb, rope = block_inputs
    _close(block(h, enc, temb[:1], rope), _general(block, h, enc, temb[:1], rope))
    _close(block(h, enc, temb[:1], rope), block(h, enc, temb[:1].expand(2, -1), rope))


def _strided(m, i, o):
    return torch.stack([o, o], dim=-1)[..., 0]


@torch.no_grad()
@pytest.mark.parametrize("where,hook", [
    ("to_out", _strided), ("ff_out", _strided), ("norm1.linear", _strided), ("norm2.linear", _strided),
    ("ff_out", lambda m, i, o: o.float()), ("ff_out", lambda m, i, o: o[:, :, :1]), ("to_out", lambda m, i, o: o[:1])])
def test_a_projection_whose_output_a_hook_replaces(block_inputs, where, hook):
    block, *args = block_inputs
    handle = block.get_submodule(where).register_forward_hook(hook)
    _close(block(*args), _general(block, *args))
    handle.remove()


@torch.no_grad()
@pytest.mark.parametrize("norm", ["norm1", "norm2"])
def test_a_modulation_without_a_weight_of_its_own(block_inputs, norm):
    block, *args = block_inputs
    plain = block(*args)
    layer = getattr(block, norm)
    layer.linear = torch.nn.Sequential(layer.linear)
    _close(block(*args), plain)


@torch.no_grad()
@pytest.mark.parametrize("which", range(3))
def test_forward_mode_tangents_are_not_dropped(block_inputs, which):
    """A tangent on the video stream, the text stream or the timestep embedding gives what the separate operations give: the
    same tangents, or torch's own error (its derivative of a bf16 layer norm is fp32, which a bf16 projection refuses)."""
    from torch.autograd import forward_ad
    block, *args = block_inputs

    def outcome(f):
        with forward_ad.dual_level():
            dual = list(args)
            dual[which] = forward_ad.make_dual(args[which], torch.ones_like(args[which]))
            try:
                return [forward_ad.unpack_dual(x).tangent for x in f(*dual)]
            except RuntimeError as e:
                return str(e)

    got, want = outcome(block), outcome(lambda *a: _general(block, *a))
    assert isinstance(got, str) == isinstance(want, str)
    if isinstance(want, str):
        assert got == want
    else:
        assert any(t is not None for t in want)
        for a, b in zip(got, want):
            assert (a is None) == (b is None) and (a is None or torch.equal(a, b))


@torch.no_grad()
def test_a_tangent_of_the_sublayer_output_is_not_dropped(block_inputs):
    """h + gate * a, with tangents that enter behind the norms."""
    from torch.autograd import forward_ad
    from ditango_b200.executor.cogvideox_dit import gated_residual
    _, h, enc, _, _ = block_inputs
    a, mod = torch.cat([enc, h], dim=1), torch.randn(2, 6 * 256, device="cuda").to(torch.bfloat16)
    with forward_ad.dual_level():
        vo, to = gated_residual(h, enc, forward_ad.make_dual(a, torch.ones_like(a)), mod)
        gate, e_gate = mod.chunk(6, dim=1)[2::3]
        assert torch.equal(forward_ad.unpack_dual(vo).tangent, gate[:, None].expand_as(h))
        assert torch.equal(forward_ad.unpack_dual(to).tangent, e_gate[:, None].expand_as(enc))


@torch.no_grad()
def test_a_replaced_attention_step_is_called(block_inputs):
    block, *args = block_inputs
    seen = []

    def attend(h, enc, rope):
        seen.append((h.shape, enc.shape))
        return torch.zeros_like(h), torch.zeros_like(enc)
    block._attend = attend
    _close(block(*args), _general(block, *args))
    assert seen == [(args[0].shape, args[1].shape)] * 2
