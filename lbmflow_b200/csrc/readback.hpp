// Fields of a grid from the device into caller-owned (pageable) host arrays.
//
// A readback of n cells is PCIe plus the host's page faults and copies: the
// caller's array is usually fresh memory. The kernel that computes the field
// writes it straight into pinned slots, chunk by chunk, and a few host
// threads, each with a slot of its own, copy the finished chunks out, so the
// link, the page faults and the copies overlap. On B200 with 16 host cores,
// through a device buffer (and for the moments a zeroed host vector and a
// scatter loop) -> in this form: moments of a 128 x 128 x 160 grid (84 MB)
// 55.7 -> 7.6 ms, strain and shear rate (147 MB) 29.6 -> 10.5 ms, moments of
// a 24^3 grid 158 -> 75 us.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <exception>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

namespace lbmb {

// Pinned blocks, shared by the solvers of a process: at most KEEP of them, of at
// most SLOTS slots each, stay allocated between readbacks, and when the last
// solver goes the largest one (4 MiB at most) stays for the next. Pinning takes
// 2 to 5 ms whatever the size, which a program that makes one small solver after
// another would pay for each (moments of a 32^3 grid 1.3 ms in all). A block
// belongs to one readback at a time.
class StagePool {
 public:
  static constexpr int SLOTS = 4;
  static constexpr size_t SLOT_BYTES = size_t(1) << 20;
  static constexpr size_t KEEP = 2;
  struct Block {
    char* p = nullptr;
    size_t bytes = 0;
  };

  // The process's pool, held as long as a solver may read (never destroyed: a
  // solver may go after the statics have).
  static std::shared_ptr<StagePool> get() {
    static StagePool* const pool = new StagePool();
    static std::mutex mu;
    static std::weak_ptr<StagePool> users;
    std::lock_guard<std::mutex> lk(mu);
    std::shared_ptr<StagePool> p = users.lock();
    if (!p) users = p = std::shared_ptr<StagePool>(pool, [](StagePool* s) { s->shrink(1); });
    return p;
  }
  // a block of at least `bytes`; null when no pinned memory is left
  Block take(size_t bytes) {
    {
      std::lock_guard<std::mutex> lk(mu_);
      auto best = free_.end();
      for (auto b = free_.begin(); b != free_.end(); ++b)
        if (b->bytes >= bytes && (best == free_.end() || b->bytes < best->bytes)) best = b;
      if (best != free_.end()) {
        const Block b = *best;
        free_.erase(best);
        return b;
      }
    }
    void* p = nullptr;
    if (cudaHostAlloc(&p, bytes, cudaHostAllocPortable) == cudaSuccess) return {static_cast<char*>(p), bytes};
    cudaGetLastError();  // else the next launch check reports this failure
    return {};
  }
  void give(Block b) {
    {
      std::lock_guard<std::mutex> lk(mu_);
      free_.push_back(b);
    }
    shrink(KEEP);
  }

 private:
  // frees the smallest blocks until `keep` are left
  void shrink(size_t keep) {
    for (;;) {
      Block b;
      {
        std::lock_guard<std::mutex> lk(mu_);
        if (free_.size() <= keep) return;
        auto least = std::min_element(free_.begin(), free_.end(),
                                      [](const Block& x, const Block& y) { return x.bytes < y.bytes; });
        b = *least;
        free_.erase(least);
      }
      cudaFreeHost(b.p);
    }
  }
  std::mutex mu_;
  std::vector<Block> free_;
};

// One output of a readback: `width` consecutive values per cell.
struct ReadField {
  double* out;
  int width;
};

// Fills fields[k].out[cell * width ...] for every cell of [0, n).
// launch(dst, c0, c1): enqueue the kernel that writes cells [c0, c1), cell c's
// values of field k at dst[k][(c - c0) * width ...] (host-accessible pinned
// memory), on stream s. Called from several threads at once.
template <class Launch>
void read_fields(int device, cudaStream_t s, StagePool& pool, int64_t n, const std::vector<ReadField>& fields,
                 const Launch& launch, void (*check)(cudaError_t)) {
  size_t per_cell = 0;
  for (const ReadField& f : fields) per_cell += size_t(f.width) * sizeof(double);
  if (per_cell == 0 || n == 0) return;
  const int64_t chunk = std::max<int64_t>(128, int64_t(StagePool::SLOT_BYTES / per_cell) / 128 * 128);
  const int64_t chunks = (n + chunk - 1) / chunk;
  const int workers = int(std::min<int64_t>(
      std::min<int64_t>(chunks, StagePool::SLOTS), std::max<int64_t>(1, int64_t(std::thread::hardware_concurrency()))));
  constexpr size_t STEP = size_t(64) << 10;
  const size_t slot_bytes = (size_t(std::min(n, chunk)) * per_cell + STEP - 1) / STEP * STEP;
  struct Held {
    StagePool& pool;
    StagePool::Block b;
    ~Held() {
      if (b.p) pool.give(b);
    }
  } held{pool, pool.take(size_t(workers) * slot_bytes)};
  if (!held.b.p) check(cudaErrorMemoryAllocation);
  auto work = [&](int w) {
    char* const slot = held.b.p + size_t(w) * slot_bytes;
    check(cudaSetDevice(device));
    cudaEvent_t done = nullptr;
    check(cudaEventCreateWithFlags(&done, cudaEventDisableTiming));
    struct Ev {
      cudaEvent_t e;
      ~Ev() {
        cudaEventSynchronize(e);  // the slot is not in use when it goes back
        cudaEventDestroy(e);
      }
    } ev{done};
    std::vector<double*> dst(fields.size());
    for (int64_t c = w; c < chunks; c += workers) {
      const int64_t c0 = c * chunk, c1 = std::min(n, c0 + chunk);
      char* p = slot;
      for (size_t k = 0; k < fields.size(); ++k) {
        dst[k] = reinterpret_cast<double*>(p);
        p += size_t(c1 - c0) * size_t(fields[k].width) * sizeof(double);
      }
      launch(dst, c0, c1);
      check(cudaEventRecord(done, s));
      check(cudaEventSynchronize(done));
      for (size_t k = 0; k < fields.size(); ++k) {
        const size_t w8 = size_t(fields[k].width);
        std::memcpy(fields[k].out + size_t(c0) * w8, dst[k], size_t(c1 - c0) * w8 * sizeof(double));
      }
    }
  };
  if (workers == 1) {
    work(0);
    return;
  }
  std::vector<std::exception_ptr> err(static_cast<size_t>(workers));
  std::vector<std::thread> th;
  auto guarded = [&](int w) {
    try {
      work(w);
    } catch (...) {
      err[size_t(w)] = std::current_exception();
    }
  };
  try {
    for (int w = 1; w < workers; ++w) th.emplace_back(guarded, w);
  } catch (...) {  // no more threads: this one does the rest
    for (int w = int(th.size()) + 1; w < workers; ++w) guarded(w);
  }
  guarded(0);
  for (std::thread& t : th) t.join();
  for (const std::exception_ptr& e : err)
    if (e) std::rethrow_exception(e);
}

}  // namespace lbmb
