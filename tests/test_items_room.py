"""The bound pass's work list (hg_items.h): whatever chunk length the device
chooses, the items it then writes fit the room the host gave the list.  The
header is compiled for the CPU and both sides are run over explicit leaf
layouts and over random ones, for every chunk length that the tuning takes."""
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


def test_bound_pass_items_fit_their_room(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    src = tmp_path / "items.cpp"
    src.write_text(SOURCE)
    exe = str(tmp_path / "items")
    subprocess.run([cxx, "-O2", "-std=c++17", "-I" + os.path.join(ROOT, "hercules_b200", "csrc"), str(src), "-o", exe],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
