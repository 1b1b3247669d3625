"""What the warps of the attention kernels do when a bounded wait runs out, replayed on the CPU.

The lanes of a warp wait each for itself, so some of them may see the barrier's phase, or the status word, and others not.  A
role's source is taken out of its kernel, compiled for the host and run as 32 threads; every operation that a warp executes as a
whole is a meeting point of all of them.  A wait is made to fail in some lanes: the warp has to end together, since lanes that
left would be waited for without a bound by those that did not."""
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ditango_b200", "csrc")

STUBS = r"""
#include <cmath>
#include <condition_variable>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>
#define __device__
#define __forceinline__ inline
struct float2 { float x, y; };
float2 make_float2(float x, float y) { return {x, y}; }
struct uint4 { uint32_t x, y, z, w; };
uint4 make_uint4(uint32_t x, uint32_t y, uint32_t z, uint32_t w) { return {x, y, z, w}; }

// ---- the warp: lanes meet at every operation that all of them execute together
std::mutex mu;
std::condition_variable cv;
int arrived = 0, turn = 0, sum = 0, total = 0, where = 0;
thread_local int lane;
int meet(int line, bool vote) {
  std::unique_lock<std::mutex> lk(mu);
  if (arrived == 0) { where = line; sum = 0; }
  if (where != line) { std::printf("split %%d %%d\n", where, line); std::fflush(stdout); _Exit(0); }
  sum += vote;
  if (++arrived == 32) { arrived = 0; total = sum; ++turn; cv.notify_all(); return total; }
  const int mine = turn;
  cv.wait(lk, [&] { return turn != mine; });
  return total;
}
#define __syncwarp() meet(__LINE__, false)
#define __all_sync(m, v) (meet(__LINE__, v) == 32)
#define __any_sync(m, v) (meet(__LINE__, v) != 0)
int loads = 0;
void fill(uint32_t* r, int n) {              // scores that rise, so that every key tile moves the reference
  const float x = 1000.f * ++loads;
  for (int i = 0; i < n; ++i) std::memcpy(r + i, &x, 4);
}
#define tmem_ld32(a, r) (meet(__LINE__, false), fill(r, 32))
#define tmem_ld16(a, r) (meet(__LINE__, false), fill(r, 16))
#define tmem_st32(a, r) meet(__LINE__, false)
#define tmem_st16(a, r) meet(__LINE__, false)
template <int N> void tmem_wait_ld(uint32_t*) { meet(1000000 + N, false); }
void tmem_wait_st() { meet(2000000, false); }
void tc_fence_after() {}
void tc_fence_before() {}
void fence_proxy_async_smem() {}
void grid_dependency_wait() {}

// ---- barriers: wait number `fail_at` for `fail_code` never ends for the lanes of `fail_lanes`, and it is they whose limit runs out
int fail_code, fail_at;
uint32_t fail_lanes;
thread_local int waits = 0;
thread_local bool stuck = false;
thread_local bool failed = false;            // this lane is past that wait, whatever it saw of it
void begin(int code) {
  stuck = code == fail_code && ++waits == fail_at;
  failed |= stuck;
  stuck &= fail_lanes >> lane & 1;
}
bool mbar_try_wait(uint64_t*, uint32_t) { return !stuck; }
uint64_t globaltimer_ns() { static thread_local uint64_t t = 0; return stuck ? t += 2000000000ull : t; }
int atomicCAS(int* at, int, int code) { return *at = code; }
%(waits)s
#define wait_or_abort(b, parity, status, code) (begin(code), wait_or_abort(b, parity, status, code))
#define warp_wait_or_abort(b, parity, status, code) (begin(code), warp_wait_or_abort(b, parity, status, code))
uint8_t memory[1 << 18];
void mbar_arrive(uint64_t* bar) {
  if (failed) std::printf("arrive %%d\n", int(reinterpret_cast<uint8_t*>(bar) - memory));
}

float ex2(float x) { return x; }
float max3(float a, float b, float c) { return std::fmax(a, std::fmax(b, c)); }
float __uint_as_float(uint32_t x) { float f; std::memcpy(&f, &x, 4); return f; }
uint32_t __float_as_uint(float x) { uint32_t u; std::memcpy(&u, &x, 4); return u; }
uint64_t pack2(float, float) { return 0; }
void unpack2(uint64_t, float& a, float& b) { a = b = 0.f; }
uint64_t fma2(uint64_t, uint64_t, uint64_t) { return 0; }
uint64_t add2(uint64_t, uint64_t) { return 0; }
uint64_t exp2_poly2(uint64_t) { return 0; }
uint64_t exp2_mufu2(uint64_t) { return 0; }
uint32_t pack_bf16x2(float, float) { return 0; }
using std::fmax;
struct Params {
  int word = 0; int* status = &word; int accumulate = 0; int num_heads = 1; float scale_log2 = 1.f; float lse[1 << 16];
  const int* cu_q = nullptr;
} p;
int64_t lse_index(const Params&, int, int, int, int64_t) { return lane; }
void merge_weights(bool, float, float, float, float&, float&, float& lse) { lse = 0.f; }
struct OldRows {};
void load_old_rows32(const Params&, int64_t, int, int64_t, OldRows&) {}
#define store_rows32(...) (meet(__LINE__, false), failed ? void(std::printf("store\n")) : void())
template <int D> void write_empty_row(const Params&, int, int, int, int, int) {}
%(constants)s
%(structs)s
uint32_t opaque_zero() { return 0; }
int n_items;
char** lens;
void role(int warp, int thread) {
  struct { int x; } threadIdx{thread};
  uint8_t* smem = memory;
  const uint32_t tmem_base = 0;
  const int aborted = 0;
%(body)s
  meet(-1, false);
}
int main(int argc, char** argv) {
  const int warp = std::atoi(argv[1]);
  fail_code = std::atoi(argv[2]); fail_at = std::atoi(argv[3]); fail_lanes = std::strtoul(argv[4], nullptr, 16);
  n_items = argc - 5; lens = argv + 5;
  std::vector<std::thread> t;
  for (int i = 0; i < 32; ++i) t.emplace_back([=] { lane = i; role(warp, warp * 32 + i); if (i == 0) std::printf("together %%d\n", int(failed)); });
  for (auto& x : t) x.join();
}
"""

# A role of the kernel whose CTAs stay.  Its items are all in their slots beforehand (more slots than the kernel has).
STAY = r"""
  const Shared sh(smem);
  for (int i = 0; i <= n_items; ++i) {
    Item w{-1, 0, 0, 0, 0, 256, 0};
    if (i < n_items) { w.k_len = std::atoi(lens[i]); w.n_tiles = (w.k_len + kBN - 1) / kBN; }
    if (lane == 0) sh.s_work[i] = w;
  }
  meet(3000000, false);
%(fetch)s
%(role)s
"""


def _block(text, start):
    i = text.index("{", start)
    depth = 0
    for j in range(i, len(text)):
        depth += (text[j] == "{") - (text[j] == "}")
        if depth == 0:
            return text[i:j + 1]
    raise AssertionError("unbalanced braces")


def _strip(text):
    text = re.sub(r'asm volatile\("[^"]*"[^;]*\);', "", text)
    return re.sub(r"static_assert\([^;]*\);", "", text)


def _build(tmp_path, name, **parts):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no host compiler")
    src, exe = str(tmp_path / (name + ".cpp")), str(tmp_path / name)
    with open(src, "w") as f:
        f.write(STUBS % parts)
    r = subprocess.run([gxx, "-std=c++17", "-O0", "-w", "-pthread", src, "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return exe


def _read(name):
    with open(os.path.join(CSRC, name)) as f:
        return f.read()


def _constants(*texts):
    return "\n".join(c for t in texts for c in re.findall(r"^constexpr (?:int|float) \w+ = [^;]*;", t, re.M)).replace("kWork = 4;", "kWork = 16;")


@pytest.fixture(scope="module")
def programs(tmp_path_factory):
    common, stay, single = _read("flash_common.cuh"), _read("flash_fwd_persistent_sm100.cu"), _read("flash_fwd_sm100.cu")
    d = tmp_path_factory.mktemp("give_up")
    waits = common[common.index("__device__ __forceinline__ void report"):common.index("// ----", common.index("wait_or_abort"))]
    out = {}
    structs = "\n".join(f"struct {n} " + _block(stay, stay.index(f"struct {n} {{")) + ";" for n in ("C", "Item", "Shared"))
    fetch = stay[stay.index("uint32_t fetched = 0;"):stay.index("if (warp >= kTmaWarp) {")]
    for name, mark in (("softmax", "- softmax"), ("results", "- results"), ("tail", "- foreign rows of an item")):
        start = stay.index(mark)
        role = stay[start:stay.index("    } else {", start)] if name == "tail" else _block(stay, stay.index("if (!aborted)", start))
        if name == "tail":
            role = "{" + role[role.index("\n"):] + "}"
        out["stay", name] = _build(d, "stay_" + name, waits=waits, constants=_constants(common, stay), structs=structs,
                                   body=STAY % dict(fetch=fetch, role=_strip(role)))
    cfg = "template <int D>\nstruct Cfg " + _block(single, single.index("struct Cfg")) + ";"
    role = _block(single, single.rindex("{", 0, single.index("- softmax + epilogue")))
    for head_dim in (64, 128):
        body = """
  constexpr int D = %d;
  using C = Cfg<D>;
  constexpr int NB = C::kSBufs;
  uint8_t* s_q = smem;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + (1 << 17));
  uint64_t *s_full = bars, *p_lo = bars + NB, *p_hi = p_lo + NB, *pv_done = p_hi + NB, *o_final = pv_done + 2;
  const int k_len = std::atoi(lens[0]), n_tiles = (k_len + kBN - 1) / kBN, q0 = 0, q_len = 256, q_begin = 0, seg = 0, head = 0;
""" % head_dim
        out["single", head_dim] = _build(d, f"single_{head_dim}", waits=waits, constants=_constants(common, single), structs=cfg, body=body + _strip(role))
    return out


def _run(exe, warp, code, at, lanes, items):
    r = subprocess.run([exe, str(warp), str(code), str(at), f"{lanes:x}", *map(str, items)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stderr
    return r.stdout.split("\n")


ITEMS = [1, 300, 0, 129, 640, 128, 500, 77]
LANES = [0x80000000, 0xffff0000, 0xffffffff]


@pytest.mark.parametrize("lanes", LANES, ids=hex)
@pytest.mark.parametrize("role,warp,code,at", [
    ("softmax", 0, 51, 1), ("softmax", 5, 51, 4), ("softmax", 0, 31, 1), ("softmax", 0, 31, 3), ("softmax", 4, 32, 9),
    ("softmax", 0, 33, 1), ("softmax", 7, 34, 4), ("softmax", 0, 43, 1), ("softmax", 4, 43, 3),
    ("results", 8, 51, 1), ("results", 11, 51, 5), ("results", 8, 42, 1), ("results", 9, 42, 4), ("results", 8, 41, 1),
    ("results", 10, 41, 6), ("tail", 14, 51, 1), ("tail", 14, 51, 6), ("tail", 14, 16, 2), ("tail", 14, 12, 1)])
def test_a_warp_of_the_staying_kernel_gives_up_as_one(programs, role, warp, code, at, lanes):
    out = _run(programs["stay", role], warp, code, at, lanes, ITEMS)
    assert out[-2] == "together 1"
    # nothing is handed on and nothing is stored behind the failure; what result warps have read they may give back
    assert "store" not in out
    arrivals = [line for line in out if line.startswith("arrive")]
    assert len(arrivals) <= (1 if role == "results" and code == 42 else 0)


@pytest.mark.parametrize("lanes", LANES, ids=hex)
@pytest.mark.parametrize("D,warp,code,at", [(64, 0, 31, 1), (64, 5, 32, 3), (64, 0, 33, 2), (64, 4, 34, 1), (64, 0, 41, 1),
                                            (128, 0, 31, 1), (128, 7, 32, 4), (128, 3, 41, 1)])
def test_a_warp_of_the_other_kernel_gives_up_as_one(programs, D, warp, code, at, lanes):
    out = _run(programs["single", D], warp, code, at, lanes, [600])
    assert out == ["together 1", ""]


def test_without_a_failure_every_role_runs_through(programs):
    for (kind, name), exe in programs.items():
        warp = dict(softmax=0, results=8, tail=14).get(name, 0)
        assert _run(exe, warp, 0, 0, 0, ITEMS if kind == "stay" else [600])[-2] == "together 0"
