// What a synchronous call reads back, in page-locked host memory that its kernels write directly
// (status words only where a state is illegal or a block singular): no clearing launch and no copy
// on the stream, which for a 128 x 3 x 3 right-hand side were 10 of 44 us (the copy into pageable
// memory is staged by the CUDA driver).
#pragma once

#include <cuda_runtime_api.h>
#include <stdint.h>
#include <string.h>

#include <mutex>

struct HostWords {
  int flags;       // legal-state mask of the flow; singular block of a chemistry or block handle
  double sums[2];  // norm, totals
  unsigned long long speed;
};

// A page-locked allocation costs ~0.3 ms, so the handles of a process share one page of 63 slots,
// kept while the process lives; further handles get an allocation of their own.  The memory does
// not outlive the context it was made in (a device reset), and another allocation may then get its
// address: the page carries a stamp, and every allocation the generation it belongs to.  A handle
// of a lost generation has nothing to give back.
struct WordSlot {
  HostWords* w = nullptr;
  unsigned generation = 0;
};

class WordPool {
 public:
  bool take(WordSlot* s) {
    std::lock_guard<std::mutex> lk(mu_);
    check();
    if (!page_) {
      void* p = nullptr;
      if (cudaHostAlloc(&p, (kSlots + 1) * kStride, kFlags) != cudaSuccess) return lost();
      page_ = static_cast<char*>(p);
      used_ = 0;
      const uint64_t v = stamp();
      memcpy(page_ + kSlots * kStride, &v, sizeof v);
    }
    s->generation = generation_;
    for (int k = 0; k < kSlots; ++k) {
      if (used_ >> k & 1ULL) continue;
      used_ |= 1ULL << k;
      s->w = reinterpret_cast<HostWords*>(page_ + k * kStride);
      return true;
    }
    if (cudaHostAlloc(reinterpret_cast<void**>(&s->w), sizeof(HostWords), kFlags) != cudaSuccess)
      return lost();
    return true;
  }
  void give(WordSlot* s) {
    if (!s->w) return;
    std::lock_guard<std::mutex> lk(mu_);
    check();
    const char* const c = reinterpret_cast<const char*>(s->w);
    if (s->generation == generation_) {
      if (c >= page_ && c < page_ + kSlots * kStride) used_ &= ~(1ULL << ((c - page_) / kStride));
      else cudaFreeHost(s->w);
    }
    s->w = nullptr;
  }

 private:
  static constexpr int kSlots = 63;  // the 64th place holds the stamp
  static constexpr size_t kStride = 64;
  static constexpr unsigned kFlags = cudaHostAllocMapped | cudaHostAllocPortable;
  static_assert(sizeof(HostWords) <= kStride, "a slot holds the words");

  uint64_t stamp() const {
    return 0x9E3779B97F4A7C15ULL * (generation_ + 1) ^ reinterpret_cast<uintptr_t>(this) ^
           reinterpret_cast<uintptr_t>(page_);
  }
  static bool lost() {  // clears the failed call's error
    cudaGetLastError();
    return false;
  }
  // a page whose context is gone starts a new generation
  void check() {
    if (!page_) return;
    cudaPointerAttributes a;
    const bool host = (cudaPointerGetAttributes(&a, page_) == cudaSuccess &&
                       a.type == cudaMemoryTypeHost) || lost();
    uint64_t v = 0;
    if (host) memcpy(&v, page_ + kSlots * kStride, sizeof v);
    if (host && v == stamp()) return;
    page_ = nullptr;
    ++generation_;
  }

  std::mutex mu_;
  char* page_ = nullptr;
  unsigned long long used_ = 0;
  unsigned generation_ = 0;
};
