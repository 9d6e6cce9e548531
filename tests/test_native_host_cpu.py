"""Host-side pieces of the native sources, compiled with the system compiler and run here: protocol bookkeeping that a GPU run
only reaches after a failure."""

import os
import shutil
import subprocess

import pytest
import torch

from heavyball_b200 import ops, utils

_CSRC = os.path.join(os.path.dirname(os.path.abspath(ops.__file__)), "csrc")


def _run(tmp_path, source):
    compiler = shutil.which("g++") or shutil.which("c++")
    if compiler is None:
        pytest.skip("no C++ compiler")
    (tmp_path / "t.cpp").write_text(source)
    subprocess.run([compiler, "-std=c++17", "-O1", "-pthread", "-I", _CSRC, str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t")], check=True)
    done = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True, timeout=120)
    assert done.returncode == 0, done.stdout + done.stderr


def test_pair_teardown_accounts_for_every_load_in_flight(tmp_path):
    """Two producers fill a ring whose phases live on one barrier (one arrival announcing both CTAs' bytes, and the bytes as they
    land) while a consumer frees stages in order.  Everything stops at a random point with loads still in flight; after the
    bookkeeping of the teardown each phase that may hold a load completes exactly when its last load has landed, and no load in
    flight belongs to a phase that is not waited for."""
    _run(tmp_path, r"""
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>
#include "pair_drain.h"
struct Bar {  // an mbarrier with one expected arrival: phase ends when the arrival is there and no bytes are outstanding
  int phase = 0, pending = 1; long tx = 0;
  void settle() { if (pending == 0 && tx == 0) { ++phase; pending = 1; } }
  void expect(long b) { if (pending == 0) { puts("second arrival in a phase"); exit(1); } tx += b; --pending; settle(); }
  void count_off(long b) { tx -= b; settle(); }
};
struct Load { int fill; long bytes; };
int main() {
  std::mt19937 rng(1);
  for (int trial = 0; trial < 20000; ++trial) {
    const int stages = 1 + rng() % 6;
    std::vector<Bar> full(stages);
    std::vector<Load> flight;
    std::vector<long> bytes(64);
    for (auto& b : bytes) b = rng() % 2 ? 16384 : 32768;
    int issued[2] = {0, 0}, consumed = 0;
    const int steps = rng() % 120;
    for (int i = 0; i < steps; ++i) {
      const int what = rng() % 4;
      if (what < 2) {
        const int n = issued[what];
        if (n < 64 && n < consumed + stages) {
          if (what == 0) full[n % stages].expect(2 * bytes[n]);
          flight.push_back({n, bytes[n]});
          ++issued[what];
        }
      } else if (what == 2) {
        if (!flight.empty()) {
          const size_t k = rng() % flight.size();
          full[flight[k].fill % stages].count_off(flight[k].bytes);
          flight.erase(flight.begin() + k);
        }
      } else if (consumed < 64 && full[consumed % stages].phase > consumed / stages) {
        ++consumed;
      }
    }
    const int even = issued[0], odd = issued[1], top = even > odd ? even : odd, from = hb::pair_drain_first(even, odd, stages);
    for (const Load& l : flight)
      if (l.fill < from) { puts("a load in flight is not waited for"); return 1; }
    for (int n = from; n < top; ++n) {
      const int kind = hb::pair_fill_kind(n, even, odd);
      if (kind == hb::kFillOddOnly) full[n % stages].expect(bytes[n]);
      if (kind == hb::kFillEvenOnly) full[n % stages].count_off(bytes[n]);
      while (full[n % stages].phase <= n / stages) {  // the wait: loads keep landing meanwhile, one at a time in random order
        if (flight.empty()) { printf("stuck: fill %d of %d / %d\n", n, even, odd); return 1; }
        const size_t k = rng() % flight.size();
        full[flight[k].fill % stages].count_off(flight[k].bytes);
        flight.erase(flight.begin() + k);
      }
    }
    if (!flight.empty()) { puts("returned with a load in flight"); return 1; }
  }
  return 0;
}
""")


def test_settings_are_made_once_for_every_device(tmp_path):
    """The second device of a process gets its own, from several threads each is made once, and an error is not remembered."""
    _run(tmp_path, r"""
#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>
#include "per_device.h"
int main() {
  hb::PerDevice<int> values;
  std::atomic<int> made[3] = {};
  std::atomic<bool> wrong{false};
  auto ask = [&](int device, int status) {
    int got = -1;
    const int s = values.get(device, 0, &got, [&](int& v) { ++made[device]; v = 100 + device; return status; });
    if (s != status && s != 0) wrong = true;
    if (s == 0 && got != 100 + device) wrong = true;
    return s;
  };
  if (ask(0, 7) != 7 || ask(0, 0) != 0) { puts("an error has to come back once and be forgotten"); return 1; }
  std::vector<std::thread> threads;
  for (int t = 0; t < 8; ++t)
    threads.emplace_back([&, t] { for (int i = 0; i < 1000; ++i) ask((t + i) % 3, 0); });
  for (auto& t : threads) t.join();
  if (wrong || made[0] != 2 || made[1] != 1 || made[2] != 1) { puts("made more than once, or a wrong value"); return 1; }
  return 0;
}
""")


def test_newton_schulz_tile_choice(tmp_path):
    """Sizes at which either tile was measured to be the faster one, on 74 pairs: one wave of small tiles and its end, waves that
    pairs need more of, rows off the 128-byte lines, a main loop too short, products of several sizes."""
    _run(tmp_path, r"""
#include <cstdio>
#include <vector>
#include "ns_tiles.h"
int bad = 0;
void expect(bool pairs, std::vector<hb::NsExtent> p) {
  if (hb::ns_take_pairs(p.data(), (int)p.size(), 74) != pairs) { printf("%d x %d x %d, %d: expected %d\n", p[0].M, p[0].N, p[0].K, p[0].batch, pairs); ++bad; }
}
int main() {
  expect(false, {{512, 512, 512, 8, true}});      // 24 pair tiles, a third of the pairs
  expect(false, {{1024, 1024, 1024, 8, true}});   // 288 small tiles: one wave; 80 pair tiles: two
  expect(false, {{640, 640, 640, 10, false}});
  expect(false, {{768, 3072, 768, 2, false}});    // 288 small tiles
  expect(true, {{768, 2304, 768, 3, false}});     // 324
  expect(true, {{1024, 1024, 1024, 8, false}});   // 512
  expect(false, {{1024, 1024, 1024, 16, true}});  // two waves of small tiles, three of pairs
  expect(true, {{1024, 1024, 1024, 24, true}});   // three and four
  expect(false, {{640, 640, 640, 20, false}});
  expect(true, {{900, 900, 1300, 6, true}});      // unaligned rows
  expect(false, {{900, 900, 1300, 8, true}});     // ... but 80 pair tiles
  expect(true, {{900, 900, 1300, 3, true}});      // 108 small tiles
  expect(false, {{900, 900, 1300, 2, true}});     // 72
  expect(true, {{600, 600, 1800, 32, true}});
  expect(false, {{700, 700, 700, 8, false}});     // unaligned, but a short K
  expect(false, {{768, 768, 511, 100, false}});   // main loop too short
  expect(true, {{768, 768, 768, 48, true}, {77, 200, 77, 1, false}});
  expect(true, {{768, 768, 768, 12, true}, {768, 768, 2304, 12, true}, {768, 768, 3072, 12, true}});
  return bad;
}
""")


def test_fused_chain_chunk_sizes(tmp_path):
    """Sizes at which one chunk was measured to be clearly the fastest, for the three numbers of vectors in flight."""
    _run(tmp_path, r"""
#include <cstdio>
#include <initializer_list>
#include "chain_chunks.h"
int bad = 0;
void expect(int vectors, long long elems, int chunk) {
  const int got = hb::chain_chunk(vectors, elems);
  if (got != chunk) { printf("%d vectors, %lld elements: %d\n", vectors, elems, got); ++bad; }
}
int main() {
  for (int vectors : {1, 2, 4}) { expect(vectors, 1, 2048); expect(vectors, 600000, 2048); expect(vectors, 14000000, 8192); }
  expect(1, 1200000, 2048);
  expect(2, 4800000, 4096);
  expect(4, 1200000, 4096);
  expect(4, 4800000, 4096);
  expect(4, 7000000, 8192);
  expect(4, 9600000, 8192);
  return bad;
}
""")


@pytest.mark.gpu
@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs two GPUs")
def test_tensor_core_and_leaf_kernels_run_on_a_second_device_of_the_process():
    for dev in ("cuda:0", "cuda:1"):
        mats = [torch.randn(96, 160, device=dev) for _ in range(2)]
        out = ops.newton_schulz_batched(mats, utils.NS5_COEFFS)
        assert 0.5 < torch.linalg.svdvals(out).mean().item() < 1.5
        a = torch.randn(2, 256, 256, device=dev)
        torch.testing.assert_close(ops.matmul3(a, a), a @ a, rtol=1e-3, atol=1e-3)
        r, info = torch.empty_like(a), torch.zeros(2, dtype=torch.int32, device=dev)
        inv = torch.empty(2, 1, 128, 128, device=dev)
        ops.load().chol_inv_leaf(a @ a.mT + 256 * torch.eye(256, device=dev), r, inv, 0, 128, info)
        assert info.sum().item() == 0
        ops.check_status()


def test_tile_of_symmetric_products(tmp_path):
    """Sizes on both sides of every line of the rule, with the pairs of a B200: (batch, n, K, expected choice)."""
    cases = [(4, 1536, 64, 0), (4, 2048, 192, 0), (4, 1536, 255, 0), (4, 1536, 256, 2), (3, 2048, 511, 2), (3, 2048, 512, 1), (2, 3072, 511, 0),
             (8, 1024, 2048, 0), (2, 1536, 1023, 0), (2, 1536, 1024, 2), (1, 2048, 4095, 0), (1, 2048, 4096, 2), (1, 1024, 5504, 0),
             (300, 255, 4096, 0), (300, 256, 512, 1)]  # fmt: skip
    table = ", ".join("{%d, %d, %d, %d}" % c for c in cases)
    _run(tmp_path, r"""
#include <cstdio>
#include "gemm_rules.h"
int main() {
  const int cases[][4] = {%s};
  int wrong = 0;
  for (const auto& c : cases) {
    const int got = hb::tf32_tiles(c[1], c[1], c[2], c[0], true, 74);
    if (got != c[3]) { printf("%%d of %%d, K %%d: %%d\n", c[0], c[1], c[2], got); wrong = 1; }
  }
  return wrong || hb::tf32_tiles(2048, 2048, 256, 4, false, 74) != hb::kSmallTiles;
}
""" % table)  # fmt: skip
