"""CPU: the space bookkeeping of the pinned upload ring (thx_ring.h).

The ring stages host->device uploads; a span is reused only after its copy
has completed, so a placement that overlaps a live span would corrupt an
upload still queued on the stream.  A small C++ driver (compiled here with
g++) places and retires spans in seeded random order and checks every
placement against the live spans, including the wrap that fills the ring
exactly."""
import os
import shutil
import subprocess
import tempfile

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "theseus_b200", "csrc")

DRIVER = r"""
#include "thx_ring.h"
#include <cstdio>
#include <deque>
#include <random>
#include <utility>

static int check(thx::RingSpace &r, std::deque<std::pair<size_t, size_t>> &live, size_t need,
                 size_t cap) {
  size_t off;
  while (!r.place(need, &off)) {
    if (live.empty()) { std::printf("no placement in an empty ring\n"); return 1; }
    live.pop_front();
    r.pop();
  }
  if (off + need > cap) { std::printf("span past the end: %zu+%zu\n", off, need); return 1; }
  for (auto &s : live)
    if (off < s.first + s.second && s.first < off + need) {
      std::printf("overlap: [%zu,%zu) with live [%zu,%zu)\n", off, off + need, s.first,
                  s.first + s.second);
      return 1;
    }
  live.push_back({off, need});
  r.push(off, need);
  return 0;
}

int main() {
  // the exact-fill wrap: A[0,10) B[10,20) C[20,28), retire A, D[0,5), E[5,10)
  // fills [0,10) up to the tail B: the next span must wait for B and C
  {
    thx::RingSpace r(30);
    std::deque<std::pair<size_t, size_t>> live;
    for (size_t n : {10, 10, 8}) if (check(r, live, n, 30)) return 1;
    live.pop_front(); r.pop();
    for (size_t n : {5, 5, 10}) if (check(r, live, n, 30)) return 1;
  }
  std::mt19937_64 g(7);
  for (int trial = 0; trial < 200; ++trial) {
    const size_t cap = 64 + g() % 4096;
    thx::RingSpace r(cap);
    std::deque<std::pair<size_t, size_t>> live;
    for (int it = 0; it < 4000; ++it) {
      if (!live.empty() && g() % 3 == 0) {  // a copy completes
        live.pop_front();
        r.pop();
        continue;
      }
      const size_t need = 1 + g() % (cap / 2);
      if (check(r, live, need, cap)) return 1;
    }
  }
  std::printf("ok\n");
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="g++ not found")
def test_ring_space_never_overlaps_live_spans():
    with tempfile.TemporaryDirectory() as d:
        src = os.path.join(d, "ring.cpp")
        exe = os.path.join(d, "ring")
        with open(src, "w") as f:
            f.write(DRIVER)
        subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, src, "-o", exe], check=True)
        out = subprocess.run([exe], capture_output=True, text=True, timeout=60)
        assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr


STAGING_DRIVER = r"""
#include "thx_staging.h"
#include <atomic>
#include <condition_variable>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <functional>
#include <random>
#include <thread>

// A device whose one stream copies late: the bytes are read only after the
// call that queued them has returned.
struct Fake {
  using Stream = int;
  using Event = int;
  static constexpr int kNoSpace = 7;
  static std::mutex mu;
  static std::deque<std::function<void()>> queue;
  static std::atomic<bool> done[4096];
  static std::atomic<int> next, largest;
  static std::atomic<bool> stop;
  static int alloc(void **p, size_t n) { return (*p = std::malloc(n)) ? 0 : 1; }
  static void free(void *p) { std::free(p); }
  static void post(std::function<void()> f) { std::lock_guard<std::mutex> l(mu); queue.push_back(std::move(f)); }
  static int copy(void *dst, const void *src, size_t n, int) {
    if ((int)n > largest) largest = (int)n;
    post([=] { std::memcpy(dst, src, n); });
    return 0;
  }
  static int create(int *e) { *e = next++; return *e < 4096 ? 0 : 1; }
  static void destroy(int) {}
  static int record(int e, int) { done[e] = false; post([=] { done[e] = true; }); return 0; }
  static int wait(int e) { while (!done[e]) std::this_thread::yield(); return 0; }
  static void drain(int) { while (true) { { std::lock_guard<std::mutex> l(mu); if (queue.empty()) return; } std::this_thread::yield(); } }
  static void run() {
    while (true) {
      std::function<void()> f;
      {
        std::lock_guard<std::mutex> l(mu);
        if (!queue.empty()) f = queue.front();
      }
      if (f) {
        std::this_thread::sleep_for(std::chrono::microseconds(20));
        f();
        std::lock_guard<std::mutex> l(mu);
        queue.pop_front();
      } else if (stop) return;
      else std::this_thread::yield();
    }
  }
};
std::mutex Fake::mu;
std::deque<std::function<void()>> Fake::queue;
std::atomic<bool> Fake::done[4096];
std::atomic<int> Fake::next{0}, Fake::largest{0};
std::atomic<bool> Fake::stop{false};

int main() {
  std::thread device(Fake::run);
  int bad = 0;
  {
    // two writers at the same time: each waits in its writer for the other
    thx::StagingRing<Fake> ring;
    if (ring.init(1 << 16)) return 2;
    std::atomic<int> inside{0}, met{0};
    auto one = [&] {
      std::vector<char> dst(1000);
      ring.fill(dst.data(), 1, dst.size(), 0, [&](void *to, size_t, size_t n) {
        ++inside;
        for (int i = 0; i < 3000 && inside < 2; ++i) std::this_thread::sleep_for(std::chrono::milliseconds(1));
        if (inside == 2) ++met;
        std::memset(to, 1, n);
      });
      Fake::drain(0);
    };
    std::thread a(one), b(one);
    a.join();
    b.join();
    if (met != 2) { std::printf("the writers ran one after the other\n"); bad = 1; }
  }
  {
    // more bytes than the ring holds: in pieces of at most half of it
    thx::StagingRing<Fake> ring;
    if (ring.init(4096)) return 2;
    Fake::largest = 0;
    std::vector<uint32_t> dst(5001, 0);
    ring.fill(dst.data(), 4, dst.size(), 0, [&](void *to, size_t first, size_t n) {
      for (size_t i = 0; i < n; ++i) ((uint32_t *)to)[i] = (uint32_t)(first + i) * 2654435761u;
    });
    Fake::drain(0);
    for (size_t i = 0; i < dst.size(); ++i) bad |= dst[i] != (uint32_t)i * 2654435761u;
    if (bad || Fake::largest > 2048) { std::printf("pieces: %d bytes\n", (int)Fake::largest); bad = 1; }
  }
  {
    // many threads, spans of all sizes (queued out of their order in the ring)
    thx::StagingRing<Fake> ring;
    if (ring.init(16384)) return 2;
    std::atomic<int> wrong{0};
    std::vector<std::thread> ts;
    for (int t = 0; t < 6; ++t)
      ts.emplace_back([&, t] {
        std::mt19937 g(t);
        std::vector<std::vector<unsigned char>> dst(150), ref(150);
        for (int k = 0; k < 150; ++k) {
          const size_t n = 1 + g() % (k % 10 == 0 ? 20000 : 3000);
          ref[k].resize(n);
          dst[k].assign(n, 0);
          for (auto &c : ref[k]) c = (unsigned char)g();
          if (k & 1) ring.copy(dst[k].data(), ref[k].data(), n, 0);
          else
            ring.fill(dst[k].data(), 1, n, 0, [&](void *to, size_t first, size_t m) {
              std::memcpy(to, ref[k].data() + first, m);
              std::this_thread::sleep_for(std::chrono::microseconds(g() % 50));
            });
        }
        Fake::drain(0);
        for (int k = 0; k < 150; ++k) wrong += dst[k] != ref[k];
      });
    for (auto &t : ts) t.join();
    if (wrong) { std::printf("%d copies are wrong\n", (int)wrong); bad = 1; }
  }
  Fake::stop = true;
  device.join();
  if (!bad) std::printf("ok\n");
  return bad;
}
"""


def test_staging_ring_writes_outside_its_lock():
    """Writers on several threads run at the same time, a fill larger than the
    ring goes through it in pieces, and no span is reused before its copy."""
    with tempfile.TemporaryDirectory() as d:
        src = os.path.join(d, "staging.cpp")
        exe = os.path.join(d, "staging")
        with open(src, "w") as f:
            f.write(STAGING_DRIVER)
        subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, src, "-o", exe], check=True)
        out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
        assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr
