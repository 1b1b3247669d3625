"""The attention kernel at the sizes where its 128-key tiles, its two-part hand-over and its polynomial exponentials can go
wrong, against softmax in 64 bits.

Tolerances: probabilities are rounded to bf16 (relative 2^-9) before they meet V, so a result differs from exact by at
most 2^-9 of the largest |V| of its row plus fp32 accumulation, here 2^-8 in all.  lse is fp32: the exponentials carry a
relative error below 3e-7 (either unit) and the sum's rounding is of the same order, so |d lse| <= 1e-6 (1 + |lse|)."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _qkv(B, Sq, Sk, H, D, scale=1.0, seed=0):
    g = torch.Generator().manual_seed(seed)
    q, k, v = (torch.randn(B, S, H, D, generator=g) for S in (Sq, Sk, Sk))
    return (q * scale).to(torch.bfloat16).cuda(), k.to(torch.bfloat16).cuda(), v.to(torch.bfloat16).cuda()


def _exact(q, k, v):
    s = torch.einsum("bqhd,bkhd->bhqk", q.double(), k.double()) / math.sqrt(q.shape[-1])
    return torch.einsum("bhqk,bkhd->bqhd", torch.softmax(s, -1), v.double()), torch.logsumexp(s, -1)


def _check(got, want, v):
    (o, l), (ro, rl) = got, want
    assert (o.double() - ro).abs().max() <= v.double().abs().max() * 2.0 ** -8
    assert ((l.double() - rl).abs() <= 1e-6 * (1 + rl.abs())).all()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("Sq,Sk,scale", [
    (1, 1, 1.0), (127, 63, 1.0), (128, 64, 1.0), (129, 65, 1.0), (255, 127, 4.0), (256, 128, 1.0), (257, 129, 1.0),
    (300, 191, 1.0), (100, 192, 8.0), (513, 255, 1.0), (64, 256, 30.0), (200, 257, 1.0), (256, 384, 100.0), (130, 1409, 1.0)])
def test_tile_edges(D, Sq, Sk, scale):
    from ditango_b200 import ops
    q, k, v = _qkv(2, Sq, Sk, 3, D, scale)
    want = _exact(q, k, v)
    _check(ops.flash_partial(q, k, v), want, v)
    if Sk > 1:                                    # the same keys in two launches, the second merged into the first
        h = Sk // 3 + 1
        a, b, c, d = (x.contiguous() for x in (k[:, :h], v[:, :h], k[:, h:], v[:, h:]))
        o, l = ops.flash_partial(q, a, b)
        if c.shape[1]:
            ops.flash_partial(q, c, d, out=o, lse=l, accumulate=True, overlap_previous=True)
        _check((o, l), want, v)
    assert ops.read_status() == 0


@pytest.mark.parametrize("D", [64, 128])
def test_rising_scores_rescale_at_every_tile(D):
    """Scores whose weights rise 2^4.3-fold with every key tile (a rescale in every second one) and 2^52-fold (in every one)."""
    from ditango_b200 import ops
    q, k, v = _qkv(1, 256, 640, 2, D)
    q = torch.ones_like(q)
    step = torch.arange(640, device="cuda") // 128
    for gain in (0.25, 3.0):
        kk = (k.float() * 0.01 + (gain * 12.0 / math.sqrt(D)) * step[None, :, None, None]).to(torch.bfloat16)
        _check(ops.flash_partial(q, kk, v), _exact(q, kk, v), v)
    assert ops.read_status() == 0


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("key", range(112, 144))
def test_a_nan_key_reaches_every_row(D, key):
    """Whichever unit exponentiates a column, a NaN score must not turn into a weight of zero."""
    from ditango_b200 import ops
    q, k, v = _qkv(1, 130, 200, 1, D)
    k[0, key, 0, 3] = float("nan")
    o, l = ops.flash_partial(q, k, v)
    assert torch.isnan(o).all() and torch.isnan(l).all()
    assert ops.read_status() == 0


@pytest.mark.parametrize("D", [64, 128])
def test_a_launch_of_empty_sequences_does_not_break_a_chain_of_overlapping_ones(D):
    """Three overlapping launches on one state, the middle one without a single query row: same bits as separate launches."""
    from ditango_b200 import ops
    q, k, v = (x.flatten(0, 1) for x in _qkv(1, 3000, 3000, 6, D))
    full = torch.tensor([0, 3000], dtype=torch.int32, device="cuda")
    none = torch.zeros(2, dtype=torch.int32, device="cuda")

    def chain(overlap):
        o, l = ops.flash_partial(q, k, v, cu_seqlens_q=full, cu_seqlens_k=full)
        for cu in (none, full):
            ops.flash_partial(q, v, k, cu_seqlens_q=cu, cu_seqlens_k=full, out=o, lse=l, accumulate=True, overlap_previous=overlap)
        return o, l

    want = chain(False)
    torch.cuda.synchronize()
    for _ in range(5):
        got = chain(True)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    assert ops.read_status() == 0


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("Sk", [1, 15, 16, 17, 63, 64, 65, 100, 127, 128, 129, 192, 255, 270])
def test_a_neighbour_that_is_not_finite_stays_outside(D, Sk):
    """The last key tile of a sequence reads rows of whatever lies behind it: the next batch item, the next packed segment,
    rows past the last offset.  Infinities and NaN there must not change a bit of the result."""
    from ditango_b200 import ops
    Sq = 200
    q, k, v = _qkv(2, Sq, Sk, 2, D)
    clean = ops.flash_partial(q, k, v)
    cu_q, cu_k = (torch.tensor([0, n, 2 * n], dtype=torch.int32, device="cuda") for n in (Sq, Sk))
    for bad in (float("nan"), float("inf")):
        kb, vb = k.clone(), v.clone()
        kb[1], vb[1] = bad, bad
        o, l = ops.flash_partial(q, kb, vb)                                          # dense, behind batch item 0
        assert torch.equal(o[0], clean[0][0]) and torch.equal(l[0], clean[1][0]) and torch.isnan(o[1]).all()
        qp, kp, vp = (x.flatten(0, 1) for x in (q, kb, vb))
        o, l = ops.flash_partial(qp, kp, vp, cu_seqlens_q=cu_q, cu_seqlens_k=cu_k)   # packed, behind segment 0
        assert torch.equal(o[:Sq], clean[0][0]) and torch.equal(l[:, :Sq], clean[1][0])
        o, l = ops.flash_partial(qp, kp, vp, cu_seqlens_q=cu_q[:2].contiguous(), cu_seqlens_k=cu_k[:2].contiguous())
        assert torch.equal(o[:Sq], clean[0][0]) and torch.equal(l[:, :Sq], clean[1][0])
    assert ops.read_status() == 0
