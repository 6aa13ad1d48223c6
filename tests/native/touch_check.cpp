// touchRange and touchEach: prints the number of bytes changed in a filled array, and
// of pages not resident in a fresh one.
#include <sys/mman.h>
#include <unistd.h>

#include <cstdio>
#include <vector>

#include "emcg_pages.h"

int main() {
  const size_t page = (size_t)sysconf(_SC_PAGESIZE);
  std::vector<unsigned char> a(100003);
  for (size_t i = 0; i < a.size(); i++)
    a[i] = (unsigned char)(7 * i + 1);
  emcg::touchRange(a.data() + 1, a.size() - 1);
  emcg::touchRange(a.data(), 0);
  emcg::touchEach(a.data() + 1, a.size() - 1, page);
  emcg::touchEach(a.data(), 0, page);
  long changed = 0, absent = 0;
  for (size_t i = 0; i < a.size(); i++)
    changed += a[i] != (unsigned char)(7 * i + 1);
  const size_t n = 9 * page;
  for (int each = 0; each < 2; each++) {
    void *m = mmap(nullptr, n, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    if (m == MAP_FAILED)
      return 1;
    char *p = static_cast<char *>(m) + page / 2;
    if (each)
      emcg::touchEach(p, n - page, page);
    else
      emcg::touchRange(p, n - page);
    unsigned char in[9];
    if (mincore(m, n, in) != 0)
      return 1;
    for (unsigned char r : in)
      absent += !(r & 1);
  }
  std::printf("%ld %ld\n", changed, absent);
  return 0;
}
