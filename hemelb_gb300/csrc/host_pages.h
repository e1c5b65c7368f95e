// Whether the pages of a host array are present, by asking the kernel (no access to them).
#pragma once
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <cstddef>
#include <cstdint>

namespace hlbg {

// True when every page of [p, p + bytes) is there, so that a write to it takes no fault.
// The first piece with a page missing ends the search.  Where the kernel does not answer,
// the pages count as missing.
inline bool pages_present(const void* p, size_t bytes) {
  const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE);
  const uintptr_t end = (uintptr_t)p + bytes;
  unsigned char there[1024];
  for (uintptr_t a = (uintptr_t)p & ~(page - 1); a < end; a += sizeof(there) * page) {
    const size_t pages = std::min<size_t>(sizeof(there), (end - a + page - 1) / page);
    if (mincore(reinterpret_cast<void*>(a), pages * page, there) != 0) return false;
    for (size_t k = 0; k < pages; ++k)
      if (!(there[k] & 1)) return false;
  }
  return true;
}

}  // namespace hlbg
