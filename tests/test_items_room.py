"""Sizes that the host's buffers and the kernels agree on (hg_items.h), compiled
for the CPU.

The bound pass's work list: whatever chunk length the device chooses, the items
it then writes fit the room the host gave the list, over explicit leaf layouts
and over random ones, for every chunk length that the tuning takes.

The survivor-pair list: warps that reserve blocks of it past its end leave a
counter that tells so, however many pairs they drop, and no slot is written
twice."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

SOURCE = r"""
#include <algorithm>
#include <cstdio>
#include <random>
#include <vector>
#include "hg_items.h"
using namespace hg;

static unsigned long long written(const std::vector<uint32_t>& use, const std::vector<uint32_t>& cnt, uint32_t btpi,
                                  uint64_t room) {
  unsigned long long work = 0, groups = 0, items = 0;
  for (size_t l = 0; l < use.size(); ++l) {
    const uint32_t g = (cnt[l] + kBatchBoundQueries - 1) / kBatchBoundQueries;
    groups += g;
    work += (unsigned long long)g * use[l];
  }
  const uint32_t b = bound_item_tiles(work, groups, btpi, room);
  if (b > btpi || b < 1) return ~0ull;
  for (size_t l = 0; l < use.size(); ++l)
    items += (unsigned long long)((cnt[l] + kBatchBoundQueries - 1) / kBatchBoundQueries) * ((use[l] + b - 1) / b);
  return items;
}

static int bad = 0;
static void check(const std::vector<uint32_t>& use, const std::vector<uint32_t>& cnt, uint32_t btpi) {
  uint32_t nq = 0, most = 0;
  for (uint32_t c : cnt) nq += c;
  for (uint32_t u : use) most = std::max(most, u);
  // the buffer may be one of an earlier, larger call: more room is as good
  for (uint64_t extra : {0ull, 1000ull}) {
    const uint64_t room = bound_items_room(nq, use.size(), most, btpi) + extra;
    const unsigned long long n = written(use, cnt, btpi, room);
    if (n > room && ++bad < 20)
      printf("%zu leaves, %u queries, btpi %u: %llu items, room %llu\n", use.size(), nq, btpi, n,
             (unsigned long long)room);
  }
}

int main() {
  for (uint32_t btpi = 2; btpi <= 64; ++btpi) {
    check(std::vector<uint32_t>(21, 169), std::vector<uint32_t>(21, 1), btpi);
    check(std::vector<uint32_t>(10, 355), std::vector<uint32_t>(10, 6), btpi);
    check({781, 700, 560, 500, 400, 302}, {11, 11, 11, 11, 10, 10}, btpi);
    check({4096}, {1}, btpi);
    check({0, 1}, {3, 5}, btpi);
    std::mt19937 rng(btpi);
    for (int r = 0; r < 3000; ++r) {
      const uint32_t nl = 1 + rng() % 120, scale = 1 + rng() % 4096, nq = 1 + rng() % 600;
      const bool even = rng() % 2;
      std::vector<uint32_t> use(nl), cnt(nl, 0);
      for (uint32_t& u : use) u = even ? scale - rng() % std::max(1u, scale / 50) : rng() % (scale + 1);
      for (uint32_t q = 0; q < nq; ++q) ++cnt[rng() % nl];
      check(use, cnt, btpi);
    }
  }
  // a list without room for shorter chunks keeps btpi
  if (bound_item_tiles(2 * kBatchItemTarget, 10, 64, 100) != 64) ++bad;
  return bad ? 1 : 0;
}
"""


PAIRS = r"""
#include <cstdio>
#include <vector>
#include "hg_items.h"
using namespace hg;

// `warps` warps push `votes` votes of n pairs each, in turn
static int run(uint32_t cap, uint32_t warps, uint64_t votes, uint32_t n) {
  std::vector<uint32_t> cur(warps, 0), end(warps, 0);
  std::vector<uint8_t> slots(cap, 0);
  uint32_t counter = 0;  // the device's, 32 bits
  uint64_t stored = 0;
  for (uint64_t v = 0; v < votes; ++v) {
    uint32_t &c = cur[v % warps], &e = end[v % warps];
    if (c + n > e) {
      if (pair_list_full(c, cap)) continue;
      for (uint32_t i = c; i < e; ++i) ++slots[i];  // closed with sentinels
      const uint32_t nb = counter;
      counter += kBatchPairBlock;
      pair_block(nb, cap, &c, &e);
    }
    for (uint32_t i = 0; i < n; ++i)
      if (c + i < e) {
        if (c + i >= cap) return printf("slot %u of %u\n", c + i, cap), 1;
        ++slots[c + i];
        ++stored;
      }
    c += n;
  }
  for (uint32_t w = 0; w < warps; ++w)
    for (uint32_t i = cur[w]; i < end[w]; ++i) ++slots[i];
  for (uint32_t i = 0; i < cap; ++i)
    if (slots[i] != (i < counter ? 1 : 0)) return printf("slot %u of %u written %d times\n", i, cap, slots[i]), 1;
  // the last block inside the list begins below cap; after it a warp takes one
  // more at most.  A list that is no multiple of a block (the library's are) says
  // "lost" as soon as its last block is begun.
  const bool lost = counter > cap, dropped = stored < votes * n;
  if ((dropped && !lost) || (lost && !dropped && cap % kBatchPairBlock == 0) ||
      counter > (uint64_t)cap + ((uint64_t)warps + 1) * kBatchPairBlock)
    return printf("cap %u, %u warps, %llu votes of %u: %llu stored, counter %u\n", cap, warps,
                  (unsigned long long)votes, n, (unsigned long long)stored, counter), 1;
  return 0;
}

int main() {
  int bad = 0;
  for (uint32_t cap : {1u, 1000u, 1024u, 4096u, 16384u + 1184u * 1024u})
    for (uint32_t n : {1u, 5u, 32u})
      for (uint64_t votes : {1ull, 31ull, 4096ull, 200000ull, 9000000ull})  // the last: past 2^32 blocks of counts
        for (uint32_t warps : {1u, 1184u}) bad += run(cap, warps, votes, n);
  return bad ? 1 : 0;
}
"""


@pytest.mark.parametrize("source", [SOURCE, PAIRS], ids=["bound pass items", "survivor pairs"])
def test_sizes_agree(tmp_path, source):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    src = tmp_path / "items.cpp"
    src.write_text(source)
    exe = str(tmp_path / "items")
    subprocess.run([cxx, "-O2", "-std=c++17", "-I" + os.path.join(ROOT, "hercules_b200", "csrc"), str(src), "-o", exe],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
