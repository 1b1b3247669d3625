"""The workloads this package is used for, as cases that can be timed and compared on ONE GPU.

Most of the package's work is the attention of one rank of a sequence-parallel group, called once per layer and
denoising step.  On one GPU a case is therefore what ONE rank of an N-rank job executes: the rank's own chunk plus
the other ranks' K/V chunks, which the copy-engine transport lands in this GPU's memory while earlier chunks are
attended.  `ResidentPeers` stands in for the group: the incoming chunks are already resident, nothing is sent, and
no transfer is timed.  (A Ulysses exchange becomes a device copy of the packed buffer onto itself's twin: every
rank is given this rank's data.)

Kinds of case:
  attn     proAttention.attn on a single rank: the whole sequence in one call
  ring     proAttention.attn / varlen_attn of one rank of N over a few denoising steps of a stride schedule
           (dividers 1 = full refresh, d = one of d blocks refreshed, the others taken from the cache)
  pairs    the same under a per-(source, destination) reuse map
  ulysses  ulysses_attention of one rank of N
  merge    update_out_and_lse, the two-state merge of the reference's API, chained over a few blocks
  profile  the profiling pass that fills the redundancy map from the layers' outputs
  dit      one denoising step of the CogVideoX-shaped transformer (classifier-free guidance in the batch)
"""
import math

import torch

from ditango_b200.baseline.ulysses import ulysses_attention
from ditango_b200.core.attention import proAttention
from ditango_b200.core.config import init_config
from ditango_b200.core.group_coordinate import SingleRankGroup
from ditango_b200.core.redundancy_map import RedundancyMap, destroy_redundancy_map, init_redundancy_map
from ditango_b200.core.schedule import plan_pair_step, plan_step
from ditango_b200.executor.cogvideox_dit import CogVideoXDiT, DiTConfig, denoise
from ditango_b200.utils import update_out_and_lse, update_timestep

BF16 = torch.bfloat16


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # A toy-sized layer (512 tokens per rank, four heads) over four steps with reuse: the smallest thing the
        # package is asked to do; launches and host work are all there is.
        dict(name="ring_tiny_2", kind="ring", world=2, rank=0, B=1, H=4, D=64, S=512, dividers="1,2,2,1",
             packed=False, pad=0, rms=False, out16=False, cache16=False),
        # CogVideoX-5B self-attention on one GPU: CFG batch 2, 17550 video + 226 text tokens, head dimension 64.
        dict(name="attn_cogvideox", kind="attn", B=2, H=48, D=64, S=17776, rms=False, out16=False),
        # HunyuanVideo 720p self-attention on one GPU: 118800 video + 256 text tokens, head dimension 128,
        # RMS-normalised q and k.  The largest call.
        dict(name="attn_hunyuan", kind="attn", B=1, H=24, D=128, S=119056, rms=True, out16=False),
        # CogVideoX on rank 3 of 8: full refresh, then the cache in 8, 4 and 2 blocks (short launches, merges).
        dict(name="ring_cogvideox_8", kind="ring", world=8, rank=3, B=2, H=48, D=64, S=2222, dividers="1,8,4,2",
             packed=False, pad=0, rms=False, out16=False, cache16=False),
        # HunyuanVideo on rank 5 of 8: the packed call its adapter makes (a valid and a pad segment per shard),
        # full refresh, then 4 and 2 blocks; bf16 result, which is what the adapter casts to.
        dict(name="ring_hunyuan_8", kind="ring", world=8, rank=5, B=1, H=24, D=128, S=14882, dividers="1,4,2",
             packed=True, pad=25, rms=True, out16=True, cache16=False),
        # The same model's dense call on rank 0 of 4 with nothing reused: plain ring, fp32 result.
        dict(name="ring_plain_4", kind="ring", world=4, rank=0, B=1, H=24, D=128, S=7201, dividers="1",
             packed=False, pad=0, rms=True, out16=False, cache16=False),
        # Stepvideo-T2V on rank 2 of 8: chunks more than two ring hops away come from the cache after the first
        # step; bf16 cache and bf16 result.
        dict(name="pairs_stepvideo_8", kind="pairs", world=8, rank=2, B=2, H=48, D=128, S=6851, steps=2, hops=2,
             rms=False, out16=True, cache16=True),
        # CogVideoX in Ulysses mode on one rank of 8: six heads of the whole sequence.
        dict(name="ulysses_cogvideox_8", kind="ulysses", world=8, B=2, H=48, D=64, S=2222, rms=False),
        # Merging partial states one after the other, as code written against the reference's helper does: bf16
        # blocks with [B,H,S] log-sum-exps folded into an fp32 state.
        dict(name="merge_hunyuan", kind="merge", B=1, H=24, D=128, S=14882, blocks=4),
        # Profiling pass: outputs of two layers at the CogVideoX chunk size of 4 ranks over three steps.
        dict(name="profile_cogvideox", kind="profile", B=2, H=48, D=64, S=4444, layers=2, steps=3),
        # One denoising step of the CogVideoX-5B-shaped transformer at full width, two of its layers.
        dict(name="dit_cogvideox", kind="dit", layers=2, heads=48, frames=13, height=60, width=90, text=226),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["attn", "attn", "ring", "ring", "ring", "pairs", "ulysses", "merge", "profile", "dit"])
    D = rng.choice([64, 128])
    B = rng.choice([1, 2])
    if kind == "attn":
        H = rng.choice([4, 8, 12, 24, 48])
        top = int(math.sqrt(6.0e13 / (4.0 * B * H * D)))
        return dict(kind=kind, B=B, H=H, D=D, S=_log_int(rng, 256, min(top, 60000)), rms=rng.random() < 0.5,
                    out16=rng.random() < 0.5)
    if kind == "ring":
        world = rng.choice([2, 4, 8])
        dividers = rng.choice({2: ["1", "1,2", "1,2,2"], 4: ["1", "1,4,2", "1,2", "1,4"],
                               8: ["1", "1,8,4", "1,4,2", "1,8", "1,2"]}[world])
        packed = rng.random() < 0.4
        S = _log_int(rng, 200, 9000)
        return dict(kind=kind, world=world, rank=rng.randrange(world), B=1 if packed else B,
                    H=rng.choice([4, 8, 24, 48]), D=D, S=S, dividers=dividers, packed=packed,
                    pad=rng.randrange(1, min(S // 4, 256)) if packed else 0, rms=rng.random() < 0.5,
                    out16=rng.random() < 0.5, cache16=rng.random() < 0.3)
    if kind == "pairs":
        world = rng.choice([4, 8])
        return dict(kind=kind, world=world, rank=rng.randrange(world), B=B, H=rng.choice([8, 24, 48]), D=D,
                    S=_log_int(rng, 300, 5000), steps=rng.choice([2, 3]), hops=rng.choice([1, 2]),
                    rms=rng.random() < 0.5, out16=rng.random() < 0.5, cache16=rng.random() < 0.5)
    if kind == "ulysses":
        world = rng.choice([2, 4, 8])
        return dict(kind=kind, world=world, B=B, H=rng.choice([8, 24, 48]), D=D, S=_log_int(rng, 250, 32000 // world),
                    rms=rng.random() < 0.5)
    if kind == "merge":
        return dict(kind=kind, B=B, H=rng.choice([4, 8, 24, 48]), D=D, S=_log_int(rng, 500, 15000),
                    blocks=rng.randint(2, 5))
    if kind == "profile":
        return dict(kind=kind, B=B, H=rng.choice([4, 24, 48]), D=D, S=_log_int(rng, 500, 9000),
                    layers=rng.randint(1, 3), steps=rng.randint(2, 4))
    return dict(kind="dit", layers=rng.randint(1, 2), heads=rng.choice([12, 24, 48]), frames=rng.randint(1, 13),
                height=2 * rng.randint(8, 30), width=2 * rng.randint(8, 45), text=rng.randint(16, 226))


# ------------------------------------------------------------------------------------------------ groups
class ResidentPeers:
    """One rank's view of an N-rank group whose K/V chunks have all arrived: `chunks[src]` is the payload tuple
    (K, V[, cu_seqlens]) of rank `src` for the current step."""
    wait_is_event_only = True

    def __init__(self, world, rank):
        self.world_size, self.rank_in_group, self.ranks, self.local_rank = world, rank, list(range(world)), 0
        self.device = torch.device("cuda", torch.cuda.current_device())
        self.chunks = None

    def p2p_prepare(self, tag, payload, slots):
        pass

    def p2p_isend(self, tensor, dst=None, slot=None):
        pass

    def p2p_irecv(self, size=None, dtype=None, src=None, out=None, slot=None):
        return self.chunks[src][slot[2]]

    def p2p_commit_batch(self):
        return []

    def p2p_wait_batch(self, handle):
        pass

    def all_to_all_single(self, output, input_):
        output.copy_(input_)


# ------------------------------------------------------------------------------------------------ inputs
def _normal(gen, *shape):
    return torch.randn(shape, generator=gen, device="cuda", dtype=torch.float32)


def _to_input(x, rms):
    if rms:                                    # the models that normalise q and k do it per head
        x = x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + 1e-6)
    return x.to(BF16)


def _qkv(gen, shape, rms):
    return tuple(_to_input(_normal(gen, *shape), rms and i < 2) for i in range(3))


def _drifting(gen, shape, rms, steps):
    """One tensor of a layer over consecutive denoising steps: N(0,1), then N(0, 0.05^2) added per step."""
    x = _normal(gen, *shape)
    seq = [_to_input(x, rms)]
    for _ in range(1, steps):
        x.add_(_normal(gen, *shape), alpha=0.05)
        seq.append(_to_input(x, rms))
    return seq


def _schedule(world, steps, layers=1):
    """The run's configuration and a schedule without reuse; returns the schedule."""
    cfg = init_config(None, make_output_dir=False)
    cfg.num_layers, cfg.num_inference_steps = layers, steps
    destroy_redundancy_map()
    return init_redundancy_map(cfg, world_size=world)


def _reusable(world, steps, hops):
    """reusable[t][0][src][dst]: pairs further apart than `hops` on the ring may be reused after the first step."""
    def far(src, dst):
        d = abs(src - dst)
        return min(d, world - d) > hops
    return [[[[t > 0 and far(s, d) for d in range(world)] for s in range(world)]] for t in range(steps)]


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    if kind in ("attn", "ring", "pairs"):
        B, H, D, S = case["B"], case["H"], case["D"], case["S"]
        if kind == "attn":
            world, rank, steps, packed = 1, 0, 1, False
            _schedule(1, 1)
        else:
            world, rank, packed = case["world"], case["rank"], kind == "ring" and case["packed"]
            if kind == "ring":
                dividers = [int(d) for d in case["dividers"].split(",")]
                steps = len(dividers)
                rm = _schedule(world, steps)
                for t, d in enumerate(dividers):
                    rm.divider_map[t, 0] = d
            else:
                steps = case["steps"]
                rm = _schedule(world, steps)
                rm.set_pair_map(_reusable(world, steps, case["hops"]))
        group = SingleRankGroup() if world == 1 else ResidentPeers(world, rank)
        layer = proAttention(0, group)
        if case["out16"]:
            layer.output_dtype = BF16
        if case.get("cache16"):
            layer.cache_dtype = layer.cache.store_dtype = BF16
        shape = (S, H, D) if packed else (B, S, H, D)
        q = _drifting(gen, shape, case["rms"], steps)
        kv = [(_drifting(gen, shape, case["rms"], steps), _drifting(gen, shape, False, steps)) for _ in range(world)]
        cu = [torch.tensor([0, S - case["pad"], S], dtype=torch.int32, device="cuda") for _ in range(world)] if packed else None
        chunks = [[(kv[r][0][t], kv[r][1][t]) + ((cu[r],) if packed else ()) for r in range(world)] for t in range(steps)]
        return dict(kind="steps", layer=layer, group=group, rank=rank, q=q, chunks=chunks, packed=packed, S=S)
    if kind == "ulysses":
        group = ResidentPeers(case["world"], 0)
        q, k, v = _qkv(gen, (case["B"], case["S"], case["H"], case["D"]), case["rms"])
        return dict(kind=kind, group=group, q=q, k=k, v=v)
    if kind == "merge":
        B, H, D, S = case["B"], case["H"], case["D"], case["S"]
        # partial states of equal-sized key chunks: values of attention outputs, log-sum-exps around log(chunk)
        blocks = [((0.1 * _normal(gen, B, S, H, D)).to(BF16), 9.0 + 0.3 * _normal(gen, B, H, S)) for _ in range(case["blocks"])]
        return dict(kind=kind, blocks=blocks)
    if kind == "profile":
        cfg = init_config(None, make_output_dir=False)
        cfg.num_layers, cfg.num_inference_steps = case["layers"], case["steps"]
        shape = (case["B"], case["S"], case["H"], case["D"])
        outs = []
        for _ in range(case["layers"]):
            x = 0.1 * _normal(gen, *shape)
            seq = [x]
            for _ in range(1, case["steps"]):
                seq.append(seq[-1] + 0.005 * _normal(gen, *shape))
            outs.append(seq)
        return dict(kind=kind, rm=RedundancyMap(cfg, world_size=1), outs=outs, layers=case["layers"], steps=case["steps"])
    if kind == "dit":
        _schedule(1, 1, case["layers"])
        cfg = DiTConfig(num_layers=case["layers"], num_heads=case["heads"], frames=case["frames"], height=case["height"],
                        width=case["width"], text_len=case["text"])
        torch.manual_seed(seed)
        with torch.device("cuda"):
            model = CogVideoXDiT(cfg, SingleRankGroup(), mode="ditango").to(BF16)
        latents = _normal(gen, 1, cfg.frames, cfg.in_channels, cfg.height, cfg.width).to(BF16)
        cond, uncond = (_normal(gen, 1, cfg.text_len, cfg.text_dim).to(BF16) for _ in range(2))
        return dict(kind=kind, model=model, latents=latents, cond=cond, uncond=uncond)
    raise ValueError(f"unknown kind {kind!r}")


# ------------------------------------------------------------------------------------------------ one pass
def run(state):
    kind = state["kind"]
    if kind == "steps":
        layer, outs = state["layer"], []
        for t, (q, chunks) in enumerate(zip(state["q"], state["chunks"])):
            update_timestep(t)
            state["group"].chunks = chunks
            own = chunks[state["rank"]]
            if state["packed"]:
                outs.append(layer.varlen_attn(q, own[0], own[1], cu_seqlens_q=own[2], cu_seqlens_kv=own[2],
                                              max_seqlen_q=state["S"], max_seqlen_kv=state["S"]))
            else:
                outs.append(layer.attn(q, own[0], own[1]))
        return outs + [layer.last_lse]
    if kind == "ulysses":
        return ulysses_attention(state["q"], state["k"], state["v"], group=state["group"])
    if kind == "merge":
        out = lse = None
        for block_out, block_lse in state["blocks"]:
            out, lse = update_out_and_lse(out, lse, block_out, block_lse)
        return out, lse
    if kind == "profile":
        rm = state["rm"]
        rm.enable_auto_setting()
        for t in range(state["steps"]):
            for layer in range(state["layers"]):
                rm.record_out_redundancy(t, layer, state["outs"][layer][t])
        rm.finished_one_round()
        rm.finish_auto_setting()
        return rm.redundancy_map
    return denoise(state["model"], state["latents"], state["cond"], state["uncond"], num_steps=1)


# ------------------------------------------------------------------------------------------------ what a pass needs
def work(case):
    kind = case["kind"]
    if kind == "dit":
        dim, p = case["heads"] * 64, 2
        tokens = 2 * (case["frames"] * (case["height"] // p) * (case["width"] // p) + case["text"])
        per_seq = tokens // 2
        layer_params = 12 * dim * dim + 2 * 512 * 6 * dim
        flops = case["layers"] * (2 * tokens * 12 * dim * dim + 2 * 4 * per_seq * per_seq * dim)
        params = case["layers"] * layer_params + dim * (4096 + 2 * 64 + 512 + 2 * 512)
        flops += 2 * 2 * case["text"] * 4096 * dim
        return dict(bytes=2 * params + 2 * 2 * 16 * case["frames"] * case["height"] * case["width"] + 2 * 2 * case["text"] * 4096,
                    flops=flops)
    B, H, D, S = case["B"], case["H"], case["D"], case["S"]
    rows, n = B * H * S, B * H * S * D
    if kind == "merge":
        return dict(bytes=case["blocks"] * (2 * n + 4 * rows) + 4 * n + 4 * rows, flops=case["blocks"] * 3 * n)
    if kind == "profile":
        # every step's output once (the first has nothing to be compared with, but is the second's past)
        return dict(bytes=4 * n * case["layers"] * case["steps"], flops=5 * n * case["layers"] * (case["steps"] - 1))
    if kind == "ulysses":
        S_all = S * case["world"]
        return dict(bytes=4 * 2 * n, flops=4 * B * (H // case["world"]) * S_all * S_all * D)
    pair = 4 * n * S                           # one query chunk against one key chunk
    if kind == "ring" and case["packed"]:
        valid = S - case["pad"]
        pair = 4 * H * D * (valid * valid + case["pad"] * case["pad"])
    if kind == "attn":
        attended, steps = 1, 1
    elif kind == "ring":
        world, rank, pointers, attended = case["world"], case["rank"], [0] * case["world"], 0
        dividers = [int(d) for d in case["dividers"].split(",")]
        steps = len(dividers)
        for d in dividers:
            plan = plan_step(world, world // d, pointers)
            attended += len(plan.ranks[rank].owners) + int(plan.ranks[rank].own_first)
            pointers = plan.pointers_after
    else:
        world, rank, steps, attended = case["world"], case["rank"], case["steps"], 0
        have = [set() for _ in range(world)]
        for flags in _reusable(world, steps, case["hops"]):
            attended += 1 + len(plan_pair_step(world, flags[0], have).ranks[rank].owners)
    out_bytes = 2 if case["out16"] else 4
    return dict(bytes=attended * 2 * 2 * n + steps * (2 * n + out_bytes * n) + 4 * rows, flops=attended * pair)


def tolerance(case):
    """About four times the distance between a pass and the same path in fp64 (transformer: in fp32)."""
    kind = case["kind"]
    if kind == "merge":
        return {"rel": 1e-6, "max": 8e-6}
    if kind == "profile":
        return {"rel": 1e-6}
    if kind == "dit":
        return {"rel": 3e-2, "max": 0.35}
    # probabilities are rounded to bf16 before they meet V (1.65e-3); a bf16 result and a bf16 cache add theirs (2.8e-3)
    if kind == "ulysses" or case["out16"] or case.get("cache16"):
        return {"rel": 1.1e-2, "max": 0.12}
    return {"rel": 6.5e-3, "max": 6e-2}
