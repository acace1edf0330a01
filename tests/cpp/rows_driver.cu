// Host-only check that the row-streaming TSMTTSM reads no more of a row than its n values: the row ends at the
// end of a page, with an inaccessible page behind it (an odd row in 16-byte pairs: one element before).
#include <sys/mman.h>
#include <unistd.h>

#include <cstdio>

#include "launch.cuh"

namespace skinny {
skinny_status workspace_ensure(Workspace&, size_t, cudaStream_t) { return SKINNY_NO_MEM; }
void set_error(const std::string&) {}
void count_launch() {}
}  // namespace skinny

template <int W>
static int check(unsigned char* end) {
  int bad = 0;
  for (int vec = 0; vec < 2; vec++)
    for (int n = 1; n <= W; n++) {
      double* row = reinterpret_cast<double*>(end) - (vec ? (n + 1) / 2 * 2 : n);
      for (int x = 0; x < n; x++) row[x] = x + 1;
      double v[W];
      skinny::row_vals<double, W>(row, n, true, vec != 0, v);
      for (int x = 0; x < W; x++) bad += v[x] != (x < n ? x + 1 : 0);
      skinny::row_vals<double, W>(reinterpret_cast<const double*>(end), n, false, vec != 0, v);  // past the last row
      for (int x = 0; x < W; x++) bad += v[x] != 0;
    }
  return bad;
}

int main() {
  const size_t page = (size_t)sysconf(_SC_PAGESIZE);
  unsigned char* p = static_cast<unsigned char*>(mmap(nullptr, 2 * page, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0));
  if (p == MAP_FAILED || mprotect(p + page, page, PROT_NONE) != 0) return 2;
  const int bad = check<1>(p + page) + check<2>(p + page) + check<4>(p + page) + check<8>(p + page);
  std::printf("bad %d\n", bad);
  return bad ? 1 : 0;
}
