"""The fused query / key norm + rotary kernel against the same steps in 64 bits.

Inputs are the same bf16 values; the kernel rounds once, to bf16: half a unit in the last place is 2^-9 relative, and the
fp32 arithmetic before it adds about 1e-6 of the row's scale."""
import pytest
import torch
import torch.nn as nn

pytestmark = pytest.mark.gpu


def _exact(x, w, b, eps, cos, sin, text_len):
    x = x.double()
    x = (x - x.mean(-1, keepdim=True)) * torch.rsqrt(x.var(-1, unbiased=False, keepdim=True) + eps) * w.double() + b.double()
    v = x[:, text_len:]
    rot = torch.stack([-v[..., 1::2], v[..., 0::2]], dim=-1).flatten(-2)
    v = v * cos.double()[None, :, None] + rot * sin.double()[None, :, None]
    return torch.cat([x[:, :text_len], v], dim=1)


@pytest.mark.parametrize("B,S,H,D,text_len", [(1, 1, 1, 64, 0), (1, 1, 1, 128, 1), (2, 37, 3, 64, 5), (2, 33, 7, 128, 33),
                                              (1, 300, 48, 64, 226), (2, 129, 50, 64, 0), (1, 65, 24, 128, 17), (1, 2500, 2, 64, 9)])
def test_norm_rope_matches_exact(B, S, H, D, text_len):
    from ditango_b200 import ops
    g = torch.Generator().manual_seed(S)
    q, k = ((torch.randn(B, S, H, D, generator=g) * 2 + 0.5).to(torch.bfloat16).cuda() for _ in range(2))
    qn, kn = ((torch.randn(D, generator=g).to(torch.bfloat16).cuda(), torch.randn(D, generator=g).to(torch.bfloat16).cuda(), e)
              for e in (1e-6, 1e-3))
    ang = torch.randn(S - text_len, D, generator=g) * 3
    cos, sin = ang.cos().cuda(), ang.sin().cuda()
    qo, ko = ops.norm_rope(q, k, qn, kn, cos, sin, text_len)
    for got, x, n in ((qo, q, qn), (ko, k, kn)):
        want = _exact(x, n[0], n[1], n[2], cos, sin, text_len)
        assert ((got.double() - want).abs() <= want.abs() * 2.0 ** -8 + 1e-5).all()


def test_the_fused_path_and_the_general_one_agree_and_hooks_keep_the_general_one():
    from ditango_b200 import ops
    from ditango_b200.executor.cogvideox_dit import norm_and_rotate
    torch.manual_seed(0)
    q, k = (torch.randn(2, 50, 4, 64, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    nq, nk = (nn.LayerNorm(64, eps=1e-6).cuda().to(torch.bfloat16) for _ in range(2))
    ang = torch.randn(44, 64, device="cuda")
    with torch.no_grad():
        n0 = ops.LaunchLog.count
        fused = norm_and_rotate(q, k, nq, nk, ang.cos(), ang.sin(), 6)
        assert ops.LaunchLog.count == n0 + 1
        seen = []
        nk.register_forward_hook(lambda m, i, o: seen.append(1))
        plain = norm_and_rotate(q, k, nq, nk, ang.cos(), ang.sin(), 6)
        assert ops.LaunchLog.count == n0 + 1 and seen
        strided = norm_and_rotate(q.transpose(1, 2).contiguous().transpose(1, 2), k, nq, nk, ang.cos(), ang.sin(), 6)
    for a, b, c in zip(fused, plain, strided):       # the general path rounds to bf16 twice more
        assert (a.float() - b.float()).abs().max() <= 2.0 ** -7 * b.float().abs().max() and torch.equal(b, c)


@torch.no_grad()
def test_tensors_without_an_address_and_tangents_take_the_general_path():
    from torch.autograd import forward_ad
    from ditango_b200 import ops
    from ditango_b200.executor.cogvideox_dit import norm_and_rotate
    torch.manual_seed(0)
    q, k = (torch.randn(2, 9, 4, 64, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    nq, nk = (nn.LayerNorm(64, eps=1e-6).cuda().to(torch.bfloat16) for _ in range(2))
    ang = torch.randn(7, 64, device="cuda")
    f = lambda a, b: norm_and_rotate(a, b, nq, nk, ang.cos(), ang.sin(), 2)
    n0 = ops.LaunchLog.count
    nq.register_forward_hook(lambda m, i, o: None)
    want = f(q, k)
    nq._forward_hooks.clear()
    assert ops.LaunchLog.count == n0
    for got in (torch.func.vmap(lambda a, b: f(a[None], b[None]))(q, k), torch.func.jvp(f, (q, k), (q, k))[0]):
        assert all(torch.equal(a.view(b.shape), b) for a, b in zip(got, want))
    with forward_ad.dual_level():
        got = f(forward_ad.make_dual(q, torch.ones_like(q)), k)
        assert forward_ad.unpack_dual(got[0]).tangent is not None and torch.equal(got[1], want[1])
    for shape in ((0, 9, 4, 64), (2, 9, 0, 64)):
        e = torch.empty(shape, device="cuda", dtype=torch.bfloat16)
        assert all(x.shape == shape for x in f(e, e))
    assert ops.LaunchLog.count == n0


@pytest.mark.parametrize("same", [False, True])
def test_gradients_are_those_of_the_separate_operations(same):
    """First and second derivatives through the kernel's path and through the general one; also with one tensor as q and k."""
    from ditango_b200 import ops
    from ditango_b200.executor.cogvideox_dit import norm_and_rotate
    torch.manual_seed(0)
    q, k = (torch.randn(2, 11, 3, 64, device="cuda", dtype=torch.bfloat16, requires_grad=True) for _ in range(2))
    k = q if same else k
    nq, nk = (nn.LayerNorm(64, eps=1e-6).cuda().to(torch.bfloat16) for _ in range(2))
    nq.weight.data.normal_()
    ang = torch.randn(7, 64, device="cuda")
    g = [torch.randn(2, 11, 3, 64, device="cuda", dtype=torch.bfloat16) for _ in range(3)]
    inputs = [q, nq.weight, nq.bias, nk.weight, nk.bias] + ([] if same else [k])

    def derivatives():
        n0 = ops.LaunchLog.count
        outs = norm_and_rotate(q, k, nq, nk, ang.cos(), ang.sin(), 4)
        first = torch.autograd.grad(outs, inputs, g[:2], create_graph=True)
        return ops.LaunchLog.count - n0, list(first) + list(torch.autograd.grad(first[0], inputs[:2], g[2]))

    launches, got = derivatives()
    nq.register_forward_hook(lambda m, i, o: None)
    general, want = derivatives()
    assert (launches, general) == (1, 0)
    for a, b in zip(got, want):                # the same operations in the same types; sums may be taken in another order
        assert a.shape == b.shape and (a.float() - b.float()).abs().max() <= 2.0 ** -6 * b.float().abs().max()


def test_a_differentiable_attention_behind_the_norms_reaches_the_projections():
    from ditango_b200.executor.cogvideox_dit import norm_and_rotate
    torch.manual_seed(0)
    proj = nn.Linear(64, 64, device="cuda", dtype=torch.bfloat16)
    nq, nk = (nn.LayerNorm(64, eps=1e-6).cuda().to(torch.bfloat16) for _ in range(2))
    x = torch.randn(1, 10, 2, 64, device="cuda", dtype=torch.bfloat16)
    cos, sin = torch.ones(10, 64, device="cuda"), torch.zeros(10, 64, device="cuda")
    q, k = norm_and_rotate(proj(x), x, nq, nk, cos, sin, 0)
    nn.functional.scaled_dot_product_attention(*(t.transpose(1, 2) for t in (q, k, x))).float().pow(2).sum().backward()
    assert all(p.grad is not None and p.grad.abs().sum() > 0 for p in (proj.weight, nq.weight, nk.weight))
