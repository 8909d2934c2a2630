// Pages of host result arrays (csrc/host_pages.h): all there when they are waited
// for, with the contents that they had, and left alone when the solve fails.
#include <sys/mman.h>

#include <cstdio>
#include <cstring>

#include "host_pages.h"

namespace {

size_t resident(unsigned char *p, size_t bytes) {
  const size_t page = (size_t)sysconf(_SC_PAGESIZE), n = bytes / page;
  std::vector<unsigned char> in(n);
  if (mincore(p, bytes, in.data()) != 0) return 0;
  size_t count = 0;
  for (unsigned char v : in) count += v & 1;
  return count * page;
}

unsigned char *fresh(size_t bytes) {
  void *p = mmap(nullptr, bytes, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
  return p == MAP_FAILED ? nullptr : static_cast<unsigned char *>(p);
}

}  // namespace

int main() {
#ifndef MADV_POPULATE_WRITE
  std::printf("OK (pages are left to the copy here)\n");
  return 0;
#else
  const size_t small = (size_t)64 << 20, large = (size_t)4 << 30;
  unsigned char *a = fresh(small), *b = fresh(large);
  if (!a || !b) return 1;
  if (madvise(a, (size_t)sysconf(_SC_PAGESIZE), MADV_POPULATE_WRITE) != 0) {
    std::printf("OK (this kernel leaves pages to the copy)\n");
    return 0;
  }
  a[12345] = 7;
  {
    fapk::HostPages pages;
    const size_t n = pages.add(a + 5, small - 9);
    pages.start();
    pages.wait(n);
  }
  const size_t page = (size_t)sysconf(_SC_PAGESIZE);
  if (resident(a, small) < small - 2 * page || a[12345] != 7) {
    std::printf("FAILED: %zu of %zu bytes are there\n", resident(a, small), small);
    return 1;
  }
  {
    fapk::HostPages pages;
    pages.add(b, large);
    pages.start();
  }  // given up at once
  if (resident(b, large) > large / 2) {
    std::printf("FAILED: %zu of %zu bytes of an array that is not written\n", resident(b, large), large);
    return 1;
  }
  std::printf("OK\n");
  return 0;
#endif
}
