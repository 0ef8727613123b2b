"""The tickets of the decode kernel's in-launch merge. The device functions themselves (group_of, draw_piece and draw_group of
hkv_decode.cuh) are compiled for the host, with a thread for a CTA and a pause around every atomic, so that adds and subtractions of one
word interleave in any order; the partition arithmetic is modelled with the constants of the sources."""
import os
import re
import subprocess

import numpy as np
import pytest

from horizon_kernels_b200 import build

CU, CUH = (open(os.path.join(build.CSRC, f)).read() for f in ("hkv_decode.cu", "hkv_decode.cuh"))


def _constant(src, name):
    return int(re.search(rf"\b{name} = (\d+)", src).group(1))


MIN_PER, GROUP, GROUP_FROM = _constant(CU, "kMinPer"), _constant(CUH, "kGroup"), _constant(CUH, "kGroupFrom")
PIECE_COST = [int(x) for x in re.search(r"PIECE_COST = UB == 2 \? (\d+) : (\d+);", CU).groups()]

HARNESS = r"""
#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <numeric>
#include <random>
#include <thread>
#include <vector>
#define __device__
#define __forceinline__ inline
using std::min;
thread_local std::mt19937 rng;
static void pause_() { for (unsigned i = rng() % 4; i > 0; --i) std::this_thread::yield(); }
static void __threadfence() { std::atomic_thread_fence(std::memory_order_seq_cst); }
static int atomicAdd(int* p, int v) { pause_(); const int o = __atomic_fetch_add(p, v, __ATOMIC_SEQ_CST); pause_(); return o; }
static int atomicSub(int* p, int v) { return atomicAdd(p, -v); }
@CODE@
int main(int argc, char** argv) {
  const int P = atoi(argv[1]), runs = atoi(argv[2]), first = 5, last = first + P - 1, W = 8;
  std::vector<int> tickets(last + 2);
  for (int run = 0; run < runs; ++run) {
    std::vector<int> order(P);
    std::iota(order.begin(), order.end(), first);
    std::mt19937 g(run);
    std::shuffle(order.begin(), order.end(), g);
    std::vector<std::atomic<int>> done(last + 1), merged(last + 1);
    std::atomic<int> next{0}, finals{0}, bad{0};
    auto final_merge = [&](int step) {
      for (int p = first; p <= last; p += step) if (!(step == 1 ? done : merged)[p]) ++bad;
      ++finals;
    };
    std::vector<std::thread> ts;
    for (int w = 0; w < W; ++w)
      ts.emplace_back([&, w] {
        rng.seed(run * W + w);
        for (int i; (i = next++) < P;) {
          const int part = order[i];
          done[part] = 1;
          const Group gr = group_of(part, first, last);
          if (part < gr.first || part > gr.last || gr.first < first || gr.last > last) ++bad;
          if (!draw_piece(tickets.data(), gr)) continue;
          if (P <= kGroupFrom) { final_merge(1); continue; }
          for (int p = gr.first; p <= gr.last; ++p) if (!done[p]) ++bad;
          if ((gr.first - first) % kGroup || merged[gr.first]++) ++bad;
          if (draw_group(tickets.data(), first, last)) final_merge(kGroup);
        }
      });
    for (auto& t : ts) t.join();
    if (bad || finals != 1) { printf("run %d: %d bad, %d final merges\n", run, (int)bad, (int)finals); return 1; }
    for (int t : tickets) if (t) { printf("run %d: a counter is left at %d\n", run, t); return 1; }
  }
  return 0;
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    code = CUH[CUH.index("constexpr int kGroup = "):CUH.rindex("}  // namespace hkv")]
    d = tmp_path_factory.mktemp("tickets")
    (d / "t.cpp").write_text(HARNESS.replace("@CODE@", code))
    subprocess.run([os.environ.get("CXX", "g++"), "-O1", "-std=c++17", "-pthread", "-o", str(d / "t"), str(d / "t.cpp")], check=True)
    return str(d / "t")


@pytest.mark.parametrize("P", [1, 2, GROUP_FROM - 1, GROUP_FROM, GROUP_FROM + 1, 3 * GROUP - 1, 3 * GROUP, 3 * GROUP + 1, 444, 4096])
def test_every_group_and_the_sequence_are_merged_once(harness, P):
    r = subprocess.run([harness, str(P), str(max(3, min(200, 8000 // P)))], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout


@pytest.mark.parametrize("pc", PIECE_COST)
@pytest.mark.parametrize("seed", range(8))
def test_a_counter_serves_one_sequence(seed, pc):
    """with partitions of at least kMinPer slots: pieces of one split sequence lie in consecutive partitions without a gap, a partition
    has at most two, and the words a sequence counts in (the last partition of each group, and its own last partition) serve no other
    sequence"""
    assert "per = (int)max((long long)kMinPer, (total + n_parts - 1) / n_parts)" in CU
    rng = np.random.default_rng(seed)
    KVH, n_parts = int(rng.choice([1, 2, 8])), int(rng.choice([16, 148, 296, 444]))
    Us = np.maximum(1, np.exp(rng.uniform(0, 9, int(rng.integers(1, 40)))).astype(int))
    total = int((Us + pc).sum()) * KVH
    per = max(MIN_PER, -(-total // n_parts))
    assert -(-total // per) <= n_parts
    owner, slots, seq0, grouped = {}, {}, 0, 0
    for seq, U in enumerate(int(u) for u in np.repeat(Us, KVH)):
        u0 = seq0 + pc
        first, last = u0 // per, (u0 + U - 1) // per
        for part in range(first, last + 1):
            assert max(u0, part * per) < min(u0 + U, (part + 1) * per)          # no piece is empty
            if first != last:
                slot = 2 * part + (part == first and first * per < seq0)
                assert slots.setdefault(slot, seq) == seq
        if first != last:
            n = last - first + 1
            words = {last} if n <= GROUP_FROM else {min(first + i + GROUP - 1, last) for i in range(0, n, GROUP)}
            grouped += n > GROUP_FROM
            for w in words:
                assert owner.setdefault(w, seq) == seq
        seq0 += U + pc
    assert seq0 == total


def test_counts_fit_their_half_words():
    parts = _constant(open(os.path.join(build.CSRC, "hkv_common.cuh")).read(), "kMaxParts")
    assert GROUP_FROM < 1 << 16 and -(-parts // GROUP) < 1 << 15
