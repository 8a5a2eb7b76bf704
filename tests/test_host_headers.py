"""Host-side headers of the library, compiled and run as plain C++."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lbmflow_b200", "csrc")


def run_cpp(tmp_path, body, *flags):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(body)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", *flags, "-I", CSRC, str(src), "-o", str(exe)],
                   check=True)
    return subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout


@pytest.mark.parametrize("spread", [1, 40, 400])
def test_quotient_is_the_division(tmp_path, spread):
    # 4 million operand pairs with exponents within +-spread: every quotient
    # is the correctly rounded one; so are the special operands' results
    out = run_cpp(tmp_path, r"""
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <initializer_list>
#include <limits>
#include "quotient.hpp"
static uint64_t s = 88172645463325252ull;
static uint64_t next() { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; }
static double draw(int spread) {
  uint64_t m = next() & 0xfffffffffffffull;
  if (next() % 8 == 0) m |= 0xffffffffff000ull;  // mantissas close to a power of two
  if (next() % 8 == 0) m &= 0xfffull;
  const uint64_t e = uint64_t(1023 + int(next() % uint64_t(2 * spread + 1)) - spread);
  const uint64_t b = (next() & 0x8000000000000000ull) | (e << 52) | m;
  double d;
  std::memcpy(&d, &b, 8);
  return d;
}
static bool same(double a, double b) { return (a != a && b != b) || a == b; }
int main() {
  long bad = 0;
  for (int i = 0; i < 4000000; ++i) {
    const double a = draw(SPREAD), b = draw(SPREAD);
    bad += !same(lbmb::quotient(a, b, lbmb::reciprocal(b)), a / b);
  }
  const double inf = std::numeric_limits<double>::infinity(), nan = std::numeric_limits<double>::quiet_NaN();
  const double v[] = {0.0, 1.0, -3.0, 1e300, -1e300, 1e-300, inf, -inf, nan};
  for (double a : v)
    for (double b : {1.0, 3.0, 1e-30, 1e300, inf, nan}) {
      const double q = lbmb::quotient(a, b, lbmb::reciprocal(b)), t = a / b;
      // (tiny quotients: last place only)
      bad += !(same(q, t) || std::fabs(q - t) <= std::numeric_limits<double>::denorm_min());
    }
  bad += !same(lbmb::quotient(0.0, 1e-310, lbmb::reciprocal(1e-310)), 0.0);
  std::printf("%ld\n", bad);
}
""".replace("SPREAD", str(spread)))
    assert int(out) == 0


def test_graph_set_keeps_one_key_and_survives_a_failed_capture(tmp_path):
    out = run_cpp(tmp_path, r"""
#include <cstdio>
#include <stdexcept>
#include "run_graphs.hpp"
struct Key { int body, cfg; };
static int live = 0;
struct Free { void operator()(int*) const { --live; } };
static int pool[64], used = 0;
static int fail_at = -1;
static int* make(int i) {
  if (i == fail_at) throw std::runtime_error("no memory");
  ++live;
  pool[used] = used;
  return &pool[used++];
}
int main() {
  {
    lbmb::GraphSet<Key, int*, Free, 4> g;
    const bool two[4] = {true, false, true, false}, all[4] = {true, true, true, true}, none[4] = {};
    g.prepare(Key{1, 1}, two, make);
    std::printf("%d %d\n", live, g[0] && !g[1] && g[2] && !g[3]);
    int* const first = g[0];
    g.prepare(Key{1, 1}, all, make);  // the missing ones are added
    std::printf("%d %d\n", live, g[0] == first);
    g.prepare(Key{2, 1}, two, make);  // another key: none of the first is left
    std::printf("%d %d\n", live, g[0] != first && !g[1]);
    fail_at = 2;  // a later length fails after an earlier one was made
    bool thrown = false;
    try {
      g.prepare(Key{3, 1}, two, make);
    } catch (const std::runtime_error&) {
      thrown = true;
    }
    std::printf("%d %d\n", live, thrown && !g[0] && !g[2]);
    fail_at = -1;
    g.prepare(Key{2, 1}, two, make);  // a call with another key starts afresh
    std::printf("%d %d\n", live, g[0] && g[2]);
    g.prepare(Key{2, 1}, none, make);
    std::printf("%d %d\n", live, g[0] && g[2]);
    g.drop();
    std::printf("%d %d\n", live, !g[0]);
    g.prepare(Key{2, 1}, two, make);  // the same key after a drop
    std::printf("%d %d\n", live, g[0] && g[2]);
  }
  std::printf("%d 1\n", live);
}
""")
    assert out.split() == "2 1 4 1 2 1 0 1 2 1 2 1 0 1 2 1 0 1".split()


FAKE_CUDA = r"""
#pragma once
#include <atomic>
#include <cstddef>
#include <cstdlib>
using cudaError_t = int;
using cudaStream_t = void*;
using cudaEvent_t = void*;
enum { cudaSuccess = 0, cudaErrorMemoryAllocation = 2, cudaErrorUnknown = 999 };
enum { cudaHostAllocPortable = 1, cudaEventDisableTiming = 2 };
inline std::atomic<int> fake_last{0}, fake_blocks{0}, fake_events{0};
inline bool fake_no_memory = false;
inline cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  if (fake_no_memory) return fake_last = cudaErrorMemoryAllocation;
  ++fake_blocks;
  *p = std::malloc(n);
  return cudaSuccess;
}
inline cudaError_t cudaFreeHost(void* p) { --fake_blocks; std::free(p); return cudaSuccess; }
inline cudaError_t cudaGetLastError() { return fake_last.exchange(0); }
inline cudaError_t cudaSetDevice(int) { return cudaSuccess; }
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { ++fake_events; *e = nullptr; return cudaSuccess; }
inline cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
inline cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
inline cudaError_t cudaEventDestroy(cudaEvent_t) { --fake_events; return cudaSuccess; }
"""


def test_readback_chunks_threads_and_failures(tmp_path):
    # a fake of the few CUDA calls: every cell of every field once, in chunks
    # of any worker; blocks and events given back, also by a failing chunk;
    # without pinned memory an error and nothing left for the next check
    (tmp_path / "cuda_runtime.h").write_text(FAKE_CUDA)
    out = run_cpp(tmp_path, r"""
#include <cstdio>
#include <stdexcept>
#include "readback.hpp"
using lbmb::ReadField;
static void check(cudaError_t e) { if (e != cudaSuccess) throw std::runtime_error("cuda"); }
int main() {
  auto pool = lbmb::StagePool::get();
  long bad = 0;
  const int64_t slot = int64_t(lbmb::StagePool::SLOT_BYTES);
  for (int64_t n : {int64_t(1), int64_t(127), slot / 64 - 1, slot / 64, slot / 64 + 1, 5 * (slot / 64) + 77}) {
    std::vector<double> a(size_t(6 * n), -1.0), b(size_t(n), -1.0), c(size_t(n), -1.0);
    lbmb::read_fields(0, nullptr, *pool, n, {ReadField{a.data(), 6}, ReadField{b.data(), 1}, ReadField{c.data(), 1}},
                      [&](const std::vector<double*>& d, int64_t c0, int64_t c1) {
                        for (int64_t i = c0; i < c1; ++i) {
                          for (int k = 0; k < 6; ++k) d[0][6 * (i - c0) + k] = double(10 * i + k);
                          d[1][i - c0] = double(i);
                          d[2][i - c0] = double(-i);
                        }
                      },
                      check);
    for (int64_t i = 0; i < n; ++i) {
      for (int k = 0; k < 6; ++k) bad += a[size_t(6 * i + k)] != double(10 * i + k);
      bad += b[size_t(i)] != double(i) || c[size_t(i)] != double(-i);
    }
  }
  std::printf("%ld\n", bad);
  // a chunk that fails: the error arrives, the block goes back to the pool
  std::vector<double> v(static_cast<size_t>(slot));
  bool thrown = false;
  try {
    lbmb::read_fields(0, nullptr, *pool, slot, {ReadField{v.data(), 1}},
                      [&](const std::vector<double*>&, int64_t c0, int64_t) {
                        if (c0 > slot / 2) throw std::runtime_error("launch");
                      },
                      check);
  } catch (const std::runtime_error&) {
    thrown = true;
  }
  std::printf("%d %d %d\n", thrown, fake_blocks.load(), fake_events.load());
  // blocks as large as their readback needs, the two largest kept, the
  // smallest that fits taken
  {
    lbmb::StagePool::Block b[3] = {pool->take(100), pool->take(size_t(slot) * 4), pool->take(5000)};
    for (auto x : b) pool->give(x);
    auto fit = pool->take(200);
    std::printf("%d %d %d\n", fake_blocks.load(), int(fit.bytes >= 200 && fit.bytes < size_t(slot) * 4),
                int(pool->take(size_t(slot) * 4).p == b[1].p));
    pool->give(fit);
    pool->give(b[1]);
  }
  const auto held = pool->take(size_t(slot) * 4), held2 = pool->take(1);  // all in use, no other to be had
  fake_no_memory = true;
  thrown = false;
  try {
    lbmb::read_fields(0, nullptr, *pool, 8, {ReadField{v.data(), 1}},
                      [](const std::vector<double*>&, int64_t, int64_t) {}, check);
  } catch (const std::runtime_error&) {
    thrown = true;
  }
  std::printf("%d %d\n", thrown, cudaGetLastError());
  pool->give(held);
  pool->give(held2);
  pool.reset();  // the last user: the largest block stays for the next one
  fake_no_memory = false;
  std::printf("%d\n", fake_blocks.load());
  pool = lbmb::StagePool::get();
  const auto again = pool->take(size_t(slot) * 4);
  std::printf("%d\n", fake_blocks.load());
  pool->give(again);
}
""", "-pthread", "-I", str(tmp_path))
    assert out.split() == "0 1 2 0 2 1 1 1 0 1 1".split(), out
