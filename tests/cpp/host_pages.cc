// pages_present (csrc/host_pages.h) on arrays whose pages are all, partly or not there.
#include "host_pages.h"

#include <cstdio>
#include <cstdlib>

#define CHECK(c)                                       \
  do {                                                 \
    if (!(c)) {                                        \
      std::fprintf(stderr, "line %d: %s\n", __LINE__, #c); \
      return 1;                                        \
    }                                                  \
  } while (0)

int main() {
  const size_t page = (size_t)sysconf(_SC_PAGESIZE), n = 2500;  // three calls of mincore
  char* p = static_cast<char*>(mmap(nullptr, n * page, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0));
  CHECK(p != MAP_FAILED);
  madvise(p, n * page, MADV_NOHUGEPAGE);  // a huge page would bring its neighbours
  using hlbg::pages_present;
  CHECK(!pages_present(p, n * page) && !pages_present(p, 1) && !pages_present(p + 1, page - 1));
  for (size_t k = 0; k < n; ++k) p[k * page] = 1;
  CHECK(pages_present(p, n * page) && pages_present(p + 8, n * page - 8) && pages_present(p, 1));
  for (size_t hole : {(size_t)0, (size_t)1023, (size_t)1024, (size_t)1300, n - 1}) {
    CHECK(madvise(p + hole * page, page, MADV_DONTNEED) == 0);
    CHECK(!pages_present(p, n * page));
    CHECK(!pages_present(p + hole * page + page - 1, 1));
    // beside the hole, and from or to the byte before and behind it
    if (hole) CHECK(pages_present(p, hole * page) && !pages_present(p, hole * page + 1));
    if (hole + 1 < n) CHECK(pages_present(p + (hole + 1) * page, (n - 1 - hole) * page));
    p[hole * page] = 1;
    CHECK(pages_present(p, n * page));
  }
  CHECK(munmap(p + (n - 1) * page, page) == 0);
  CHECK(!pages_present(p, n * page) && pages_present(p, (n - 1) * page));
  return 0;
}
