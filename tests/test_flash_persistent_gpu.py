"""The attention kernel whose CTAs stay and take one block of queries after another, at the sizes where that can go wrong.

A launch at D = 64 with enough blocks (256 query rows of one head) takes it; the same work head by head does not have them and
takes the kernel with one CTA per block.  Both do the same arithmetic in the same order, so results agree bit for bit;
the first cases are also held against softmax in 64 bits.  Tolerances there: probabilities are rounded to bf16 (relative 2^-9)
before they meet V, so a result differs from exact by at most 2^-9 of the largest |V| plus fp32 accumulation, 2^-8 in all; lse
is fp32 with exponentials good to 3e-7: |d lse| <= 1e-6 (1 + |lse|)."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _blocks(Sq, H, nseg):
    return -(-Sq // 256) * H * nseg


def _qkv(B, Sq, Sk, H, D, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return tuple(torch.randn(B, S, H, D, generator=g, device="cuda").to(torch.bfloat16) for S in (Sq, Sk, Sk))


def _sms():
    return torch.cuda.get_device_properties(0).multi_processor_count


def _by_head(q, k, v, **kw):
    """The same call in launches of one head each."""
    from ditango_b200 import ops
    parts = [ops.flash_partial(*(x[..., h:h + 1, :].contiguous() for x in (q, k, v)), **kw) for h in range(q.shape[-2])]
    return torch.cat([o for o, _ in parts], dim=-2), torch.cat([l for _, l in parts], dim=-2)


@pytest.mark.parametrize("D", [64])
@pytest.mark.parametrize("Sq,Sk", [(257, 1), (300, 63), (512, 64), (257, 65), (300, 127), (256, 128), (600, 129), (300, 200), (256, 256),
                                   (257, 257), (300, 391), (1000, 640), (300, 1409), (513, 2500)])
def test_a_full_grid_gives_the_bits_of_its_heads(D, Sq, Sk):
    from ditango_b200 import ops
    B, H = 2, 300
    q, k, v = _qkv(B, Sq, Sk, H, D)
    assert _blocks(Sq, H, B) > 4 * _sms() and _blocks(Sq, 1, B) <= _sms()
    o, l = ops.flash_partial(q, k, v)
    ho, hl = _by_head(q, k, v)
    assert torch.equal(o, ho) and torch.equal(l, hl)
    s = torch.einsum("bqhd,bkhd->bhqk", q[:, :, :3].double(), k[:, :, :3].double()) / math.sqrt(D)
    want = torch.einsum("bhqk,bkhd->bqhd", torch.softmax(s, -1), v[:, :, :3].double())
    assert (o[:, :, :3].double() - want).abs().max() <= v.double().abs().max() * 2.0 ** -8
    want = torch.logsumexp(s, -1)
    assert ((l[:, :3].double() - want).abs() <= 1e-6 * (1 + want.abs())).all()
    # folded into a state, overlapping the launch before it; bf16 result; the other lse layout
    o2, l2 = ops.flash_partial(q, k, v)
    ops.flash_partial(q, v, k, out=o2, lse=l2, accumulate=True, overlap_previous=True)
    for h in (0, H - 1):
        one = ops.flash_partial(*(x[:, :, h:h + 1].contiguous() for x in (q, k, v)))
        one = ops.flash_partial(*(x[:, :, h:h + 1].contiguous() for x in (q, v, k)), out=one[0], lse=one[1], accumulate=True)
        assert torch.equal(o2[:, :, h:h + 1], one[0]) and torch.equal(l2[:, h:h + 1], one[1])
    b, bl = ops.flash_partial(q, k, v, out_dtype=torch.bfloat16, lse_layout=ops.LSE_BSH)
    assert torch.equal(b, ho.to(torch.bfloat16)) and torch.equal(bl.transpose(-1, -2), hl)
    assert ops.read_status() == 0


@pytest.mark.parametrize("D", [64])
@pytest.mark.parametrize("keys", ["ragged", "short", "empty"])
def test_packed_sequences_of_all_lengths(D, keys):
    """Work items of very different lengths behind one another: no queries, no keys, one key, many tiles; neighbours that are not
    finite stay outside."""
    from ditango_b200 import ops
    H = 24
    lens_q = [256, 1, 0, 300, 0, 513, 40, 256, 129, 700, 0, 2, 255, 257, 90, 1000]
    lens_k = dict(ragged=[300, 0, 5, 129, 64, 1, 1300, 0, 15, 16, 17, 640, 128, 255, 0, 513],
                  short=[1, 2, 15, 16, 17, 31, 32, 33, 47, 63, 64, 65, 100, 127, 3, 1], empty=[0] * 15 + [7])[keys]
    cu_q, cu_k = (torch.tensor([0] + torch.tensor(n).cumsum(0).tolist(), dtype=torch.int32, device="cuda") for n in (lens_q, lens_k))
    q, k, v = (x[0] for x in _qkv(1, sum(lens_q), sum(lens_k), H, D, seed=1))
    assert sum(-(-n // 256) for n in lens_q) * H > 2 * _sms() and _blocks(1000, 1, len(lens_q)) <= _sms()
    kw = dict(cu_seqlens_q=cu_q, cu_seqlens_k=cu_k, max_seqlen_q=1000, max_seqlen_k=max(lens_k))
    o, l = ops.flash_partial(q, k, v, **kw)
    ho, hl = _by_head(q, k, v, **kw)
    assert torch.equal(o, ho) and torch.equal(l, hl)
    kb, vb = k.clone(), v.clone()
    start = int(cu_k[-2])                      # the last sequence's keys are the neighbours of those before
    kb[start:], vb[start:] = float("nan"), float("inf")
    ob, lb = ops.flash_partial(q, kb, vb, **kw)
    n = int(cu_q[-2])
    assert torch.equal(ob[:n], o[:n]) and torch.equal(lb[:, :n], l[:, :n])
    # folding further keys into the state: rows without keys keep it
    ops.flash_partial(q, k, v, out=o, lse=l, accumulate=True, overlap_previous=False, **kw)
    for s, (a, b) in enumerate(zip(lens_q, lens_k)):
        if a and not b:
            rows = slice(int(cu_q[s]), int(cu_q[s + 1]))
            assert torch.equal(o[rows], ho[rows]) and torch.equal(l[:, rows], hl[:, rows])
    assert ops.read_status() == 0


@pytest.mark.parametrize("D", [64])
def test_rising_scores_and_chains(D):
    """A reference that has to move at every key tile, over several work items per CTA; a chain of overlapping launches."""
    from ditango_b200 import ops
    q, k, v = _qkv(2, 700, 640, 60, D)
    q = torch.ones_like(q)
    step = torch.arange(640, device="cuda") // 128
    for gain in (0.25, 3.0):
        kk = (k.float() * 0.01 + (gain * 12.0 / math.sqrt(D)) * step[None, :, None, None]).to(torch.bfloat16)
        o, l = ops.flash_partial(q, kk, v)
        ho, hl = _by_head(q, kk, v)
        assert torch.equal(o, ho) and torch.equal(l, hl)

    chunks = [(k[:, i * 100:].contiguous(), v[:, i * 100:].contiguous()) for i in range(5)]

    def chain(overlap):
        o, l = ops.flash_partial(q, k, v)
        for kk, vv in chunks:
            ops.flash_partial(q, kk, vv, out=o, lse=l, accumulate=True, overlap_previous=overlap)
        return o, l
    want = chain(False)
    for _ in range(5):
        got = chain(True)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    assert ops.read_status() == 0


def test_a_posted_status_ends_the_launch():
    """CTAs that start after a failure elsewhere do no work, also where they would have taken several items."""
    from ditango_b200 import _capi, ops
    q, k, v = _qkv(2, 1000, 500, 60, 64)
    want = ops.flash_partial(q, k, v)
    lib = _capi.load()
    stream = torch.cuda.current_stream().cuda_stream
    assert lib.dtb_post_status(77, stream) == 0
    o, l = torch.full_like(want[0], 5.0), torch.full_like(want[1], 5.0)
    ops.flash_partial(q, k, v, out=o, lse=l)
    assert lib.dtb_read_status(stream) == 77
    assert (o == 5.0).all() and (l == 5.0).all()
    got = ops.flash_partial(q, k, v)
    assert ops.read_status() == 0 and torch.equal(got[0], want[0])


def _last_kernel(run):
    """Which of the two kernels the last attention launch of run() was."""
    from torch.profiler import ProfilerActivity, profile
    run()
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        run()
        torch.cuda.synchronize()
    seen = sorted((e for e in prof.events() if "flash_fwd" in e.name), key=lambda e: e.time_range.start)
    assert seen, "no attention kernel was recorded"
    return "stays" if "persistent" in seen[-1].name else "leaves"


# Blocks per SM (of 512 queries: two blocks a head), keys, folded into a state, overlapping the launch before.
@pytest.mark.parametrize("per_sm,Sk,accumulate,overlap,want", [
    (1, 640, False, False, "leaves"), (1.1, 640, False, False, "stays"), (1.1, 640, True, False, "stays"),
    (1.1, 128, False, False, "stays"), (1.1, 128, True, False, "leaves"), (1.1, 129, True, False, "stays"),
    (2, 640, True, True, "leaves"), (2.1, 640, True, True, "stays"), (2.1, 385, True, True, "stays"),
    (3, 384, True, True, "leaves"), (3.1, 384, True, True, "stays"), (3.1, 129, False, True, "stays"),
    (3, 128, False, True, "leaves"), (3.1, 128, False, True, "stays"), (4, 128, True, True, "leaves"), (4.1, 128, True, True, "stays"),
    (1.1, 24576, False, False, "stays"), (1.1, 24577, False, False, "leaves")])
def test_which_kernel_a_launch_takes(per_sm, Sk, accumulate, overlap, want):
    from ditango_b200 import ops
    H = int(per_sm * _sms()) // 2
    q, k, v = _qkv(1, 512, Sk, H, 64)
    o, l = ops.flash_partial(q, k, v)

    def run():
        ops.flash_partial(q, k, v, out=o, lse=l)
        ops.flash_partial(q, k, v, out=o, lse=l, accumulate=accumulate, overlap_previous=overlap)
    assert _last_kernel(run) == want
    assert ops.read_status() == 0


@pytest.mark.parametrize("overlap,H,lens,want", [(True, 24, [1975, 25], "leaves"), (True, 24, [3000, 25], "stays"),
                                                 (False, 24, [1000, 25], "leaves"), (False, 48, [500, 25], "leaves"),
                                                 (False, 24, [1600, 25], "stays"), (True, 48, [1300, 25], "stays")])
def test_blocks_without_queries_do_not_count(overlap, H, lens, want):
    """A valid and a pad sequence: almost half of the grid has no queries."""
    from ditango_b200 import ops
    cu = torch.tensor([0, lens[0], sum(lens)], dtype=torch.int32, device="cuda")
    q, k, v = (x[0] for x in _qkv(1, sum(lens), sum(lens), H, 64))
    kw = dict(cu_seqlens_q=cu, cu_seqlens_k=cu, max_seqlen_q=lens[0], max_seqlen_k=lens[0])
    assert _blocks(lens[0], H, 2) > (2 if overlap else 1) * _sms()
    o, l = ops.flash_partial(q, k, v, **kw)

    def run():
        ops.flash_partial(q, k, v, out=o, lse=l, **kw)
        ops.flash_partial(q, k, v, out=o, lse=l, accumulate=True, overlap_previous=overlap, **kw)
    assert _last_kernel(run) == want
    assert ops.read_status() == 0


def test_a_chain_through_both_kernels():
    """Overlapping launches of which some take one kernel and some the other: each waits for the one before it and, through it, for
    all others."""
    from ditango_b200 import ops
    H = int(2.1 * _sms()) // 2
    chunks = [_qkv(1, 512, Sk, H, 64, seed=i) for i, Sk in enumerate([640, 300, 1000, 128, 129, 640, 513, 1])]
    q = chunks[0][0]

    def chain(overlap):
        o, l = ops.flash_partial(q, *chunks[0][1:])
        for _, k, v in chunks[1:]:
            ops.flash_partial(q, k, v, out=o, lse=l, accumulate=True, overlap_previous=overlap)
        return o, l
    want = chain(False)
    torch.cuda.synchronize()
    for _ in range(10):
        got = chain(True)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    assert ops.read_status() == 0


def test_views_of_a_fused_projection():
    """q, k and v one behind the other in each token, the result among other things in a row of its own."""
    from ditango_b200 import ops
    B, S, H = 2, 700, 60
    x = torch.randn(B, S, 3, H, 64, device="cuda").to(torch.bfloat16)
    q, k, v = x.unbind(2)
    want = ops.flash_partial(*(t.contiguous() for t in (q, k, v)))
    for dtype in (torch.float32, torch.bfloat16):
        rows = torch.full((B, S, 2 * H, 64), 7.0, device="cuda", dtype=dtype)
        o, l = ops.flash_partial(q, k, v, out=rows[:, :, H:])
        assert torch.equal(o, want[0].to(dtype)) and torch.equal(l, want[1]) and (rows[:, :, :H] == 7.0).all()
    rows = torch.full((B, S, 2 * H, 64), 7.0, device="cuda")
    rows[:, :, :H] = want[0]
    l = want[1].clone()
    ops.flash_partial(q, v, k, out=rows[:, :, :H], lse=l, accumulate=True)
    ops.flash_partial(*(t.contiguous() for t in (q, v, k)), out=want[0], lse=want[1], accumulate=True)
    assert torch.equal(rows[:, :, :H], want[0]) and torch.equal(l, want[1]) and (rows[:, :, H:] == 7.0).all()
    assert ops.read_status() == 0


def test_two_streams_at_once():
    from ditango_b200 import ops
    work = [_qkv(2, 600, 500 + 300 * i, 60, 64, seed=i) for i in range(2)]
    want = [ops.flash_partial(*w) for w in work]
    streams = [torch.cuda.Stream() for _ in work]
    torch.cuda.synchronize()
    got = [[], []]
    for _ in range(10):
        for i, s in enumerate(streams):
            with torch.cuda.stream(s):
                got[i].append(ops.flash_partial(*work[i]))
    torch.cuda.synchronize()
    for w, results in zip(want, got):
        assert all(torch.equal(o, w[0]) and torch.equal(l, w[1]) for o, l in results)
    assert ops.read_status() == 0
