// Pages of the callers' result arrays, faulted in while the GPU works.
//
// A result goes into an array that the caller has just allocated (numpy.zeros), so
// its pages do not exist yet and the copy back stops at every one of them: 512 MB
// take 26 ms against 5.5 ms into an array that has its pages.  The entry points
// with large results start a few threads here that make the pages
// (MADV_POPULATE_WRITE, which leaves the contents as they are) while the solve
// runs, and join them before the copy: one FLEX iteration of five orbitals,
// 64x64x1024 (840 MB of Sigma) 83 -> 58 ms; a tail-corrected FP64 chi0 of 649 MB
// 53 -> 32 ms, of 1013 MB 83 -> 50.  Above 1 GB the time varies from call to call
// and can be far longer than the copy's own faults: the same chi0 of 1297 MB 62 to
// 278 ms against 104 without, of 1622 MB 78 to 383 against 131, of 5.2 GB 464 to 2135
// against 460.  Large sets of pages that wait for their copy also take longer to copy
// into, the longer they wait (2 x 1.7 GB made a second before the copy 200 to 660 ms,
// without 122).  So every result above 1 GB is left to the copy, and so are those of
// loops of many iterations (drivers.cu).
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <cstdint>
#include <exception>

#include "common.cuh"

#ifndef MADV_POPULATE_WRITE
#define MADV_POPULATE_WRITE 23
#endif

namespace pgb {

namespace {
constexpr size_t kPrefaultMin = 32u << 20;  // 36 MB 8.9 -> 8.4 ms a call, 28 MB 2.00 -> 2.05
constexpr size_t kPrefaultMax = 1u << 30;   // the whole of the result
constexpr size_t kPerThread = 64u << 20;
constexpr size_t kMaxThreads = 4;
constexpr size_t kPiece = 1u << 20;
}  // namespace

HostPrefault::HostPrefault(void* p, size_t bytes) {
  if (!p || bytes < kPrefaultMin || bytes > kPrefaultMax) return;
  const size_t page = (size_t)sysconf(_SC_PAGESIZE);
  const uintptr_t a = ((uintptr_t)p + page - 1) / page * page, b = ((uintptr_t)p + bytes) / page * page;
  if (b <= a) return;
  const size_t n = std::min(kMaxThreads, (b - a) / kPerThread + 1);
  const size_t part = ((b - a) / n + page - 1) / page * page;
  try {
    for (uintptr_t s = a; s < b; s += part)
      threads_.emplace_back([s, part, b, page] {
        // in small pieces: each holds the address space's lock, which the calling
        // thread's own mappings wait for; a kernel without the advice, or a mapping
        // it does not apply to, leaves the faults to the copy
        const size_t piece = (kPiece + page - 1) / page * page;
        const uintptr_t e = std::min<uintptr_t>(s + part, b);
        for (uintptr_t x = s; x < e; x += piece)
          if (madvise(reinterpret_cast<void*>(x), std::min<size_t>(piece, e - x), MADV_POPULATE_WRITE) != 0) return;
      });
  } catch (const std::exception&) {
    // no thread or no memory for one: the copy takes the faults (an exception that left
    // the constructor would end the process at the threads already running)
  }
}

void HostPrefault::join() {
  for (std::thread& t : threads_) t.join();
  threads_.clear();
}

HostPrefault::~HostPrefault() { join(); }

}  // namespace pgb
