// fault_ahead.h -- faults in the pages of a host buffer that a device-to-host copy
// is about to fill.
//
// A copy into memory that the caller has only just allocated (numpy.empty of a
// volume) takes its page faults one by one inside the driver's copy loop, which
// then waits for the kernel to clear each page: 43 MB, 9.3 ms with 2 MB pages and
// 19.4 ms with 4 KB pages, against 2.3 ms when the pages are there.  Four threads
// that populate a quarter each take 1.4 ms (2.6), and run while the device still
// computes.  MADV_POPULATE_WRITE leaves the contents alone and does nothing to
// pages that are there; where it fails (older kernels, special mappings) the copy
// faults the pages in as before.
#pragma once
#include <cuda_runtime.h>
#include <errno.h>
#include <stdint.h>
#include <sys/mman.h>

#include <algorithm>
#include <thread>

#ifndef MADV_POPULATE_WRITE
#define MADV_POPULATE_WRITE 23
#endif

namespace tg {

class FaultAhead {
 public:
  // Below MIN_BYTES the threads cost more than they save; pinned memory has its pages.
  FaultAhead(void *host, size_t bytes) {
    if (!host || bytes < MIN_BYTES) return;
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, host) != cudaSuccess) {
      cudaGetLastError();
      return;
    }
    if (at.type != cudaMemoryTypeUnregistered) return;
    const uintptr_t lo = ((uintptr_t)host + PAGE - 1) / PAGE * PAGE, hi = ((uintptr_t)host + bytes) / PAGE * PAGE;
    if (present(lo, hi)) return;
    const uintptr_t share = ((hi - lo) / THREADS + BLOCK - 1) / BLOCK * BLOCK;
    for (int i = 0; i < THREADS; ++i) {
      const uintptr_t a = lo + i * share, b = std::min(hi, a + share);
      if (a >= b) break;
      try {
        th_[n_] = std::thread([a, b] {
          // in blocks, so that threads do not hold the address space for long at a time
          for (uintptr_t p = a; p < b; p += BLOCK)
            if (madvise(reinterpret_cast<void *>(p), std::min<size_t>(BLOCK, b - p), MADV_POPULATE_WRITE) != 0 &&
                errno != EINTR && errno != EAGAIN)
              return;
        });
        ++n_;
      } catch (...) {  // no thread or no memory for one: the copy faults the rest in
        break;
      }
    }
  }
  ~FaultAhead() { join(); }
  FaultAhead(const FaultAhead &) = delete;
  FaultAhead &operator=(const FaultAhead &) = delete;
  void join() {
    while (n_ > 0) th_[--n_].join();
  }

 private:
  // A buffer that was filled before has its pages; a few tell, and starting the threads for
  // nothing would cost a small download several percent.
  static bool present(uintptr_t lo, uintptr_t hi) {
    for (int i = 0; i < PROBES; ++i) {
      const uintptr_t page = (lo + (hi - PAGE - lo) / (PROBES - 1) * i) / PAGE * PAGE;
      unsigned char in = 0;
      if (mincore(reinterpret_cast<void *>(page), PAGE, &in) != 0 || !(in & 1)) return false;
    }
    return true;
  }
  static constexpr int THREADS = 4, PROBES = 16;
  static constexpr uintptr_t PAGE = 4096, BLOCK = 2u << 20;
  static constexpr size_t MIN_BYTES = 4u << 20;
  std::thread th_[THREADS];
  int n_ = 0;
};

}  // namespace tg
