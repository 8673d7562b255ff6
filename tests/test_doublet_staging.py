"""The doublet count's staging (doublet_staging.cuh, compiled here) in a CPU model of the group loop: every item's
count is right, staged doublets are read only where they were stored, and what goes to the pool is each item's own."""
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "cms-julia_b200" / "csrc"

MODEL = r"""
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>
#include "doublet_staging.cuh"
using namespace pxl;
using Item = std::vector<char>;  // an item's survivors of the first cuts, in order: passes the remaining cuts or not

// k_doublets_count's loop over one group, a doublet as (owner, its number within the item)
bool group(const std::vector<Item>& items, const char* what) {
  struct Out { uint32_t o, k; };
  const uint32_t n = uint32_t(items.size());
  std::vector<Out> q, s_out(kGroupCells, Out{99, 0}), pool;
  for (uint32_t o = 0; o < n; ++o)
    for (char p : items[o]) q.push_back({o, uint32_t(p)});
  std::vector<uint32_t> truth(n), cnt(n, 0), over(n, 0), off(n, 0), seen(n, 0);
  for (uint32_t o = 0; o < n; ++o)
    for (char p : items[o]) truth[o] += p;
  std::vector<char> pooled(n, 0), written(n, 0);
  uint32_t nout = 0, done = 0, beyond = 0;
  size_t head = 0;
  for (bool last = false; !last;) {
    const size_t mm = std::min<size_t>(32, q.size() - head);
    last = head + mm == q.size() && mm < 32;
    for (size_t i = 0; i < mm; ++i) {
      const Out v = q[head + i];
      if (!v.k) continue;
      if (nout < uint32_t(kGroupCells)) s_out[nout] = Out{v.o, seen[v.o]};
      else ++over[v.o];
      ++nout;
      ++seen[v.o];
    }
    head += mm;
    if (!last && !staging_near_full(nout)) continue;
    const uint32_t nst = std::min<uint32_t>(nout, kGroupCells);
    const uint32_t keep = last ? 32u : s_out[nst - 1].o;
    if (!last && !staging_hands_over(nout, keep, done)) continue;
    std::vector<uint32_t> beg(33, 0), end(33, 0);
    for (uint32_t x = 0; x < nst; ++x) {
      if (x == 0 || s_out[x - 1].o != s_out[x].o) beg[s_out[x].o] = x;
      if (x + 1 == nst || s_out[x + 1].o != s_out[x].o) end[s_out[x].o] = x + 1;
    }
    const uint32_t ncopy = last ? nst : beg[keep];
    const bool keeps = nout > 0 && nout <= uint32_t(kGroupCells);
    uint32_t ex = 0;
    for (uint32_t o = done; o < n && o < keep; ++o) {
      written[o] += 1;
      cnt[o] = end[o] - beg[o] + over[o];
      pooled[o] = keeps;
      off[o] = uint32_t(pool.size()) + ex;
      ex += cnt[o];
    }
    if (keeps) pool.insert(pool.end(), s_out.begin(), s_out.begin() + ncopy);
    if (last) break;
    for (uint32_t x = ncopy; x < nout; ++x) {
      if (x >= uint32_t(kGroupCells)) ++beyond;  // what the kernel would read past its row
      else s_out[x - ncopy] = s_out[x];
    }
    nout -= ncopy;
    done = keep;
  }
  bool ok = beyond == 0;
  uint32_t most = 0;
  for (uint32_t o = 0; o < n; ++o) {
    ok = ok && written[o] == 1 && cnt[o] == truth[o];
    if (ok && pooled[o])
      for (uint32_t k = 0; k < cnt[o]; ++k) ok = ok && off[o] + k < pool.size() && pool[off[o] + k].o == o && pool[off[o] + k].k == k;
    most = std::max(most, truth[o]);
  }
  // groups whose items all leave room for a step are never searched again
  if (most + 32 <= uint32_t(kGroupCells))
    for (uint32_t o = 0; o < n; ++o) ok = ok && (pooled[o] || truth[o] == 0);
  if (!ok) {
    std::printf("%s:", what);
    for (uint32_t o = 0; o < n; ++o) std::printf(" %u/%u%s", cnt[o], truth[o], pooled[o] ? "" : "*");
    std::printf(" beyond %u\n", beyond);
  }
  return ok;
}

int main() {
  std::mt19937 rng(7);
  auto item = [&](uint32_t pass, uint32_t fail) {
    Item v(pass, 1);
    for (uint32_t f = 0; f < fail; ++f) v.insert(v.begin() + rng() % (v.size() + 1), 0);
    return v;
  };
  int bad = 0;
  for (uint32_t heavy : {0u, 1u, 704u, 736u, 737u, 750u, 767u, 768u, 769u, 800u, 1600u})
    for (uint32_t fail = 0; fail < 64; ++fail)
      for (uint32_t next : {0u, 1u, 17u, 40u, 361u, 750u}) {
        bad += !group({item(heavy, fail), item(next, 3), item(30, 5), item(heavy, 1), item(next, 0)}, "built");
        bad += !group({item(5, 1), item(heavy, fail), Item{}, item(next, 9), item(20, 0)}, "built");
      }
  for (int t = 0; t < 4000; ++t) {
    std::vector<Item> g(1 + rng() % 32);
    for (auto& v : g) v = item(rng() % 8 == 0 ? 700 + rng() % 120 : rng() % (t % 2 ? 60 : 400), rng() % 50);
    bad += !group(g, "random");
  }
  std::printf("%d wrong\n", bad);
  return bad != 0;
}
"""


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    d = tmp_path_factory.mktemp("staging")
    (d / "model.cpp").write_text(MODEL)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(CSRC), str(d / "model.cpp"), "-o", str(d / "model")], check=True)
    return d / "model"


def test_staging_counts_and_pool(model):
    r = subprocess.run([str(model)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, "\n".join(r.stdout.splitlines()[-20:])
