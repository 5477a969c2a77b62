// map_pages (scale-dg-kernel-extraction_gb300/csrc/sdg_pages.h), compiled with g++
// by test_pages_host.py: pages it is given while another thread writes to them
// keep every write, fresh pages become resident at any alignment, and memory
// that cannot be written or is not there is left alone.
#include <atomic>
#include <cstdio>
#include <cstring>
#include <thread>
#include <vector>

#include "sdg_pages.h"

static int fail(const char* what) {
  std::printf("FAIL %s\n", what);
  return 1;
}

int main() {
  const size_t page = (size_t)sysconf(_SC_PAGESIZE), n = 64 * page;
  auto fresh = [&](int prot) {
    return static_cast<char*>(mmap(nullptr, n, prot, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0));
  };
  // a writer counts up in the first byte of every page (and in the last byte)
  char* a = fresh(PROT_READ | PROT_WRITE);
  std::vector<size_t> at;
  for (size_t k = 0; k < n; k += page) at.push_back(k);
  at.push_back(n - 1);
  std::atomic<bool> done{false};
  bool lost = false;
  std::thread writer([&] {
    for (int round = 1; round <= 20000; round++) {
      for (size_t k : at) reinterpret_cast<volatile char*>(a)[k] = (char)round;
      for (size_t k : at) lost = lost || reinterpret_cast<volatile char*>(a)[k] != (char)round;
    }
    done = true;
  });
  while (!done) sdg::map_pages(a, n);
  writer.join();
  if (lost) return fail("a write was lost");
  // fresh pages are there afterwards, at any offset
  char* b = fresh(PROT_READ | PROT_WRITE);
  sdg::map_pages(b + 17, 10 * page);
  std::vector<unsigned char> in(64);
  mincore(b, n, in.data());
  for (int k = 0; k <= 10; k++)
    if (!(in[k] & 1)) return fail("not resident");
  for (size_t k = 0; k < n; k++)
    if (b[k]) return fail("contents");
  // read-only pages, a hole, nothing
  char* c = fresh(PROT_READ);
  sdg::map_pages(c, n);
  munmap(c, n);
  sdg::map_pages(c, n);
  sdg::map_pages(b, 0);
  return 0;
}
