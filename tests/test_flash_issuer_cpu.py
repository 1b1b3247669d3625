"""The MMA issuer of the attention kernel, replayed on the CPU.

The issuer's source is taken out of the kernel, compiled for the host against stubs that record every barrier wait, MMA and
commit, and run for a few numbers of key tiles.  What it does with the tensor core cannot be seen here; the order in which it
asks for things can."""
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ditango_b200", "csrc")

STUBS = r"""
#include <cstdint>
#include <cstdio>
#include <cstdlib>
%(constants)s
%(cfg)s
constexpr int D = %(head_dim)d;
using C = Cfg<D>;
constexpr int NB = C::kSBufs;
constexpr int kRing = C::kStages;
uint64_t q_full[2], kv_full[kRing], kv_empty[kRing], s_full[NB], p_lo[NB], p_hi[NB], pv_done[2], o_final[2], v_tail[1];
uint8_t s_q[1], s_kv[1];
struct { int* status; } p;
constexpr uint32_t idesc_bf16_f32(int, int, bool, bool) { return 0; }
uint32_t smem_u32(const void* x) { return x == s_q ? 0u : uint32_t(kQT * C::kTileBytes); }
uint64_t smem_desc_sw128(uint32_t addr, uint32_t, uint32_t) { return addr >> 4; }
void event(const char* what, const uint64_t* bar, int extra) {
#define BAR(b) if (bar >= b && bar < b + sizeof(b) / 8) std::printf("%%s %%s %%d %%d\n", what, #b, int(bar - b), extra)
  BAR(q_full); BAR(kv_full); BAR(kv_empty); BAR(s_full); BAR(p_lo); BAR(p_hi); BAR(pv_done); BAR(o_final); BAR(v_tail);
}
bool wait_or_abort(uint64_t* bar, uint32_t parity, int*, int) { event("wait", bar, int(parity)); return true; }
void mma_commit(uint64_t* bar) { event("commit", bar, 0); }
void mma_ss(uint32_t d, uint64_t, uint64_t b, uint32_t, uint32_t) { std::printf("S %%u %%llu\n", d, (unsigned long long)b); }
void mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t, uint32_t acc) {
  std::printf("PV %%u %%u %%llu %%u\n", d, a, (unsigned long long)b, acc);
}
void tc_fence_after() {}
bool elect_one() { return true; }
int main(int, char** argv) {
  const int k_len = std::atoi(argv[1]);
  const int n_tiles = (k_len + kBN - 1) / kBN;
  const int n_units = kQT * n_tiles;
  const int tail = k_len - (n_tiles - 1) * kBN;
  const int tail_steps = (tail + 15) >> 4;
  const uint32_t tmem_base = 0;
%(issuer)s
}
"""


def _block(text, start):
    """The text from the `{` behind position `start` to its matching `}`."""
    i = text.index("{", start)
    depth = 0
    for j in range(i, len(text)):
        depth += (text[j] == "{") - (text[j] == "}")
        if depth == 0:
            return text[i:j + 1]
    raise AssertionError("unbalanced braces")


@pytest.fixture(scope="module")
def replay(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no host compiler")
    kernel = open(os.path.join(CSRC, "flash_fwd_sm100.cu")).read()
    common = open(os.path.join(CSRC, "flash_common.cuh")).read()
    constants = "\n".join(re.findall(r"^constexpr int k\w+ = [^;]*;", common, re.M) + re.findall(r"^constexpr int k\w+ = [^;]*;", kernel, re.M))
    cfg = "template <int D>\nstruct Cfg " + _block(kernel, kernel.index("struct Cfg")) + ";"
    issuer = _block(kernel, kernel.index("if (elect_one())", kernel.index("- MMA issuer")))
    built = {}
    for head_dim in (64, 128):
        d = tmp_path_factory.mktemp("issuer")
        src, exe = str(d / "issuer.cpp"), str(d / "issuer")
        with open(src, "w") as f:
            f.write(STUBS % dict(constants=constants, cfg=cfg, issuer=issuer, head_dim=head_dim))
        r = subprocess.run([gxx, "-std=c++17", "-O0", "-w", src, "-o", exe], capture_output=True, text=True)
        assert r.returncode == 0, r.stderr
        built[head_dim] = exe

    def run(head_dim, k_len):
        r = subprocess.run([built[head_dim], str(k_len)], capture_output=True, text=True)
        assert r.returncode == 0
        return [line.split() for line in r.stdout.splitlines()]
    return run


@pytest.mark.parametrize("head_dim", [64, 128])
@pytest.mark.parametrize("tiles", [1, 2, 3, 4, 7, 12])
def test_no_arrival_is_left_behind_the_one_the_epilogue_waits_for(replay, head_dim, tiles):
    """Threads leave the CTA once both o_final barriers have completed.  Every other commit therefore has an MMA behind it
    that the last o_final commit covers, and none follows that."""
    ev = replay(head_dim, 128 * tiles)
    finals = [i for i, e in enumerate(ev) if e[:2] == ["commit", "o_final"]]
    assert [ev[i][2] for i in finals] == ["0", "1"] and finals[-1] == len(ev) - 1
    last_mma = max(i for i, e in enumerate(ev) if e[0] in ("S", "PV"))
    assert all(i < last_mma for i, e in enumerate(ev) if e[0] == "commit" and e[1] != "o_final")


@pytest.mark.parametrize("head_dim", [64, 128])
@pytest.mark.parametrize("tiles", [1, 2, 3, 4, 7, 12])
def test_every_wait_has_its_arrival(replay, head_dim, tiles):
    """The waits of the softmax warps and of the loads, counted against the issuer's commits."""
    ev = replay(head_dim, 128 * tiles)
    count = lambda name: sum(e[:2] == ["commit", name] for e in ev)
    stages = max(int(e[2]) for e in ev if e[1:2] == ["kv_full"]) + 1
    assert count("s_full") == 2 * tiles
    assert count("kv_empty") >= 2 * tiles - stages           # a slot is waited for before its next load
    if head_dim == 64:
        assert count("pv_done") >= 2 * (tiles - 1)           # a rescale in tile j waits for PV of tile j - 1
    loads = [(int(e[2]), int(e[3])) for e in ev if e[:2] == ["wait", "kv_full"]]
    ring = {64: 10, 128: 5}[head_dim]
    assert loads == [(i % ring, (i // ring) & 1) for i in range(2 * tiles)]


def test_every_way_out_of_the_kernel_waits_for_the_launch_it_may_overlap():
    """A launch that overlaps this one waits for this grid only, so no grid may complete before the one it overlaps: each
    early return waits first (of the blocks past a sequence's end the first of an empty sequence does: a grid in which every
    block returns there has only empty sequences)."""
    kernel = open(os.path.join(CSRC, "flash_fwd_sm100.cu")).read()
    body = _block(kernel, kernel.index("const FlashParams p) {\n  using C"))
    returns = [m.start() for m in re.finditer(r"\breturn;", body)]
    assert len(returns) == 2
    for at in returns:
        scope = body[body.rindex("{", 0, at):at]
        assert "grid_dependency_wait();" in scope, scope
    assert "if (blockIdx.x == 0) grid_dependency_wait();" in body[:returns[0]]
    tail = body[body.rindex("tear-down"):]
    assert tail.index("grid_dependency_wait();") < tail.index("__syncthreads();")


def test_every_tensor_memory_load_is_waited_for_with_its_registers():
    """tcgen05.wait::ld orders arithmetic on loaded registers only if they are operands of the wait."""
    kernel = open(os.path.join(CSRC, "flash_fwd_sm100.cu")).read()
    sources = {name: open(os.path.join(CSRC, name)).read() for name in os.listdir(CSRC) if name.endswith((".cu", ".cuh"))}
    assert sum(text.count('"tcgen05.wait::ld') for text in sources.values()) == 1      # one helper, which takes the registers
    helper = _block(sources["ptx_sm100.cuh"], sources["ptx_sm100.cuh"].index("void tmem_wait_ld(uint32_t* r)"))
    assert '"+r"(r[i])' in helper

    def where(arg):
        name, _, offset = arg.partition("+")
        return name.strip(), int(offset or 0)

    asked, events = {}, re.finditer(r"tmem_ld(\d+)\([^;]*, ([\w +]+)\);|tmem_wait_ld<(\d+)>\(([\w +]+)\);|tmem_wait_ld", kernel)
    for m in events:
        if m.group(1):
            name, at = where(m.group(2))
            asked.setdefault(name, set()).update(range(at, at + int(m.group(1))))
        else:
            assert m.group(3), "a wait without registers"
            name, at = where(m.group(4))
            covered = set(range(at, at + int(m.group(3))))
            assert covered <= asked[name]
            asked[name] -= covered
    assert asked and not any(asked.values())


@pytest.mark.parametrize("head_dim", [64, 128])
@pytest.mark.parametrize("k_len", [1, 15, 16, 17, 63, 64, 65, 112, 113, 127, 128, 129, 192, 255, 384, 391])
def test_pv_of_the_last_tile_stays_within_the_sequence(replay, head_dim, k_len):
    """PV covers all 128 keys of every tile but the last, there the steps of 16 keys that hold one; where the last step also
    holds foreign rows, the wait for their clearing is in front of it."""
    ev = replay(head_dim, k_len)
    tiles = -(-k_len // 128)
    per_tile = [8] * (tiles - 1) + [-(-(k_len - 128 * (tiles - 1)) // 16)]
    pv = [i for i, e in enumerate(ev) if e[0] == "PV"]
    assert len(pv) == 2 * sum(per_tile)
    last = pv[-2 * per_tile[-1]:]
    waits = [i for i, e in enumerate(ev) if e[:2] == ["wait", "v_tail"]]
    assert len(waits) == (1 if k_len % 16 else 0) and all(i < last[0] for i in waits)
    slot = lambda i: int(ev[i][3])
    for q_tile in range(2):                       # steps of one Q tile: K steps of 16 rows of 128 bytes, in units of 16 bytes
        mine = last[q_tile * per_tile[-1]:(q_tile + 1) * per_tile[-1]]
        assert [slot(i) - slot(mine[0]) for i in mine] == [128 * s for s in range(per_tile[-1])]
