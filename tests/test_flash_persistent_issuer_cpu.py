"""The MMA issuer of the attention kernel whose CTAs take several work items, replayed on the CPU: its source is taken out of the
kernel, compiled for the host against stubs that record every barrier wait, MMA, commit and arrival, and run over lists of items.
What it does with the tensor core cannot be seen here; the order in which it asks for things can."""
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
%(structs)s
struct {
  uint8_t s_q[1], s_kv[1];
  Item s_work[kWork];
  uint64_t q_full[4], q_empty[2], kv_full[C::kStages], kv_empty[C::kStages], s_full[NB], p_lo[NB], p_hi[NB], pv_done[2],
      o_final[2], o_free[2], work_empty[kWork], v_tail[kWork];
} sh;
struct { int* status; } p;
constexpr uint32_t idesc_bf16_f32(int, int, bool, bool) { return 0; }
uint32_t smem_u32(const void* x) { return x == sh.s_q ? 0u : uint32_t(C::kQBufs * kQT * C::kTileBytes); }
uint64_t smem_desc_sw128(uint32_t addr, uint32_t, uint32_t) { return addr >> 4; }
void event(const char* what, const uint64_t* bar, int extra) {
#define BAR(b) if (bar >= sh.b && bar < sh.b + sizeof(sh.b) / 8) std::printf("%%s %%s %%d %%d\n", what, #b, int(bar - sh.b), extra)
  BAR(q_full); BAR(q_empty); BAR(kv_full); BAR(kv_empty); BAR(s_full); BAR(p_lo); BAR(p_hi); BAR(pv_done); BAR(o_final); BAR(o_free);
  BAR(work_empty); BAR(v_tail);
}
bool wait_or_abort(uint64_t* bar, uint32_t parity, int*, int) { event("wait", bar, int(parity)); return true; }
void mma_commit(uint64_t* bar) { event("commit", bar, 0); }
void mbar_arrive(uint64_t* bar) { event("arrive", bar, 0); }
void mma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t, uint32_t) { std::printf("S %%u %%llu %%llu\n", d, (unsigned long long)a, (unsigned long long)b); }
void mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t, uint32_t acc) { std::printf("PV %%u %%u %%llu %%u\n", d, a, (unsigned long long)b, acc); }
void tc_fence_after() {}
bool elect_one() { return true; }
int main(int argc, char** argv) {
  uint32_t fetched = 0;
  const uint32_t tmem_base = 0;
  auto fetch = [&](auto&) {
    const int slot = fetched %% kWork, at = int(++fetched);
    if (at >= argc) return -1;
    sh.s_work[slot].k_len = std::atoi(argv[at]);
    sh.s_work[slot].n_tiles = (sh.s_work[slot].k_len + kBN - 1) / kBN;
    std::printf("item %%d %%d\n", slot, sh.s_work[slot].k_len);
    return slot;
  };
%(issuer)s
}
"""


def _block(text, start):
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
    kernel = open(os.path.join(CSRC, "flash_fwd_persistent_sm100.cu")).read()
    common = open(os.path.join(CSRC, "flash_common.cuh")).read()
    find = lambda text: re.findall(r"^constexpr int \w+ = [^;]*;", text, re.M)
    structs = "\n".join(f"struct {n} " + _block(kernel, kernel.index(f"struct {n} {{")) + ";" for n in ("C", "Item"))
    issuer = _block(kernel, kernel.index("if (elect_one())", kernel.index("- MMA issuer")))
    d = tmp_path_factory.mktemp("issuer")
    src, exe = str(d / "issuer.cpp"), str(d / "issuer")
    with open(src, "w") as f:
        f.write(STUBS % dict(constants="\n".join(find(common) + find(kernel)), structs=structs, issuer=issuer))
    r = subprocess.run([gxx, "-std=c++17", "-O0", "-w", src, "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr

    def run(items):
        r = subprocess.run([exe] + [str(k) for k in items], capture_output=True, text=True)
        assert r.returncode == 0
        return [line.split() for line in r.stdout.splitlines()]
    return run


ITEMS = [[1], [128], [129], [0, 200], [128, 128, 128], [1, 0, 0, 17, 300], [512, 64, 640, 1, 1, 1, 1000], [384, 0, 385, 391, 2222]]


@pytest.mark.parametrize("items", ITEMS, ids=str)
def test_units_run_through_all_items(replay, items):
    """Every barrier is waited for in the order of its phases, units take the S buffers in turn, S of a unit follows PV of the
    one that had its buffer, an item's first PV waits for the reads of the O before it, and what ends a CTA is o_final."""
    ev = replay(items)
    tiles = [-(-k // 128) for k in items if k]
    units = 2 * sum(tiles)
    waits = lambda name: [(int(e[2]), int(e[3])) for e in ev if e[:2] == ["wait", name]]
    turn = lambda n, size: [(i % size, (i // size) & 1) for i in range(n)]
    assert waits("kv_full") == turn(units, 8)
    assert waits("p_lo") == waits("p_hi") == turn(units, 3)
    assert waits("q_full") == [(2 * (i % 2) + t, (i // 2) & 1) for i in range(len(tiles)) for t in range(2)]
    assert waits("o_free") == [(t, (i - 1) & 1) for i in range(1, len(tiles)) for t in range(2)]
    commits = lambda name: [int(e[2]) for e in ev if e[:2] == ["commit", name]]
    assert commits("s_full") == [u % 3 for u in range(units)]
    assert commits("o_final") == [0, 1] * len(tiles)
    assert commits("q_empty") == [i % 2 for i in range(len(tiles))]
    assert sorted(commits("kv_empty")) == sorted(i % 8 for i in range(units - 1))      # all but the very last V
    assert commits("pv_done") == [0, 1] * (units // 2 - 1)
    assert ev[-1][:2] == ["commit", "o_final"]
    last_mma = max(i for i, e in enumerate(ev) if e[0] in ("S", "PV"))
    assert [e[:2] for e in ev[last_mma + 1:] if e[0] == "commit"] == [["commit", "o_final"]]
    assert len([e for e in ev if e[:2] == ["arrive", "work_empty"]]) == len(items)
    # PV: every K step of an item's tiles, the last tile's as far as it has keys; accumulating but for the first
    steps = [[8] * (n - 1) + [-(-(k - 128 * (n - 1)) // 16)] for n, k in zip(tiles, (k for k in items if k))]
    pv = [e for e in ev if e[0] == "PV"]
    assert len(pv) == 2 * sum(map(sum, steps))
    acc, want = [], []
    for e in pv:
        acc.append(int(e[4]))
    for s in steps:
        for j, n in enumerate(s):
            for tile in range(2):
                want += [0 if j == 0 and kk == 0 else 1 for kk in range(n)]
    assert acc == want
    # where in tensor memory: S(u) in buffer u mod 3, P(u) from there, 8 columns a K step, into the O of its Q tile
    assert [int(e[1]) for e in ev if e[0] == "S"] == [u % 3 * 128 for u in range(units) for _ in range(4)]
    at = []
    u = 0
    for s in steps:
        for n in s:
            for tile in range(2):
                at += [(384 + 64 * tile, u % 3 * 128 + 8 * kk) for kk in range(n)]
                u += 1
    assert [(int(e[1]), int(e[2])) for e in pv] == at
    # S of a unit is behind PV of the unit three before
    s_seen = pv_seen = 0
    for e in ev:
        if e[:2] == ["commit", "s_full"]:
            assert int(e[2]) == s_seen % 3
            assert s_seen < 3 or pv_seen > s_seen - 3
            s_seen += 1
        if e[:2] == ["wait", "p_hi"]:
            pv_seen += 1
    # the foreign rows of a ragged last tile are waited for
    assert len([e for e in ev if e[:2] == ["wait", "v_tail"]]) == sum(1 for k in items if k % 16)
