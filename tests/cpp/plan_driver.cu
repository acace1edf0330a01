// Host-only check of the CUDA-core TSMTTSM's plan (launch.cuh): for every type pair, Gram or not, M and N
// to 1000, several row counts and launch options, the shared memory and the workspace that the plan
// asks for cover what each group of cells (gridDim.y) of the kernel touches.  The kernel's arithmetic is
// written out here again.  Launches nothing; prints the failures and their number.
#include <cstdio>
#include <thread>
#include <vector>

#include "launch.cuh"

namespace skinny {
skinny_status workspace_ensure(Workspace&, size_t, cudaStream_t) { return SKINNY_NO_MEM; }
void set_error(const std::string&) {}
void count_launch() {}
}  // namespace skinny

using namespace skinny;

static std::atomic<int> bad{0};
static std::atomic<long> plans{0}, many{0};

template <typename T, typename Acc>
static void one(const char* name, int64_t M, int64_t N, int64_t K, int64_t lda, int64_t ldb, bool gram,
                const LaunchOpts& o) {
  DeviceInfo dev;
  dev.sms = 152;
  dev.smem_optin = 232448;
  const void* base = reinterpret_cast<const void*>(uintptr_t(4096));
  TsmttsmPlan pl;
  if (tsmttsm_plan<T, Acc>(dev, M, N, K, base, lda, base, ldb, gram, o, pl) != SKINNY_OK) return;  // refused
  plans++;
  const int64_t gm = (M + pl.tm - 1) / pl.tm, gn = (N + pl.tn - 1) / pl.tn, TE = pl.tm * pl.tn;
  const int64_t cells = gram && pl.tm == pl.tn ? gm * (gm + 1) / 2 : gm * gn;
  const int64_t groups = (cells + 255) / 256, s = sizeof(T), a = sizeof(Acc);
  const int64_t stage = (pl.rows * pl.lda_s * s + 127) / 128 * 128 + (gram ? 0 : (pl.rows * pl.ldb_s * s + 127) / 128 * 128);
  bool ok = groups == pl.groups && pl.smem + 128 <= dev.smem_optin;  // (static shared memory: a flag)
  // ring: the last row's edge cell reads up to 7 entries behind the last stage
  ok = ok && 128 + pl.stages * stage + 7 * s <= pl.smem;
  int64_t entries = 0;
  for (int64_t y = 0; y < groups; y++) {
    const int64_t G = cells - 256 * y < 256 ? cells - 256 * y : 256;
    const int64_t slots = G == 1 || G == 2 || G == 4 || G == 8 || G == 16 ? 8 : 256 / G;
    const int64_t E = G * TE;
    int64_t red = slots > 1 ? slots * E : 0;
    if (2 * E <= 256 && red < 256) red = 256;  // cross-CTA sum by slices
    ok = ok && 128 + red * a <= pl.smem;
    entries = y * pl.grid * 256 * TE + pl.grid * E;
  }
  if (groups == 1) {  // two levels of sums: the groups' sums follow the CTAs'
    entries += finish_groups<Acc>(pl.grid, (int)(cells * TE)) * cells * TE;
    ok = ok && pl.entries == cells * TE;
  } else {
    many++;
  }
  ok = ok && (size_t)(entries * a) <= pl.template partials<Acc>(pl.grid);
  // up to 64 x 64 the workspace asked for covers every plan of the width (one group of cells), and so of smaller ones
  if (M <= 64 && N <= 64 && groups == 1 && o.blocks_per_sm == 0)
    ok = ok && pl.template partials<Acc>(pl.grid) <= tsmttsm_workspace<Acc>(dev, M, N);
  if (!ok && bad++ < 20)
    std::printf("%s %lld x %lld K=%lld lda=%lld gram=%d blocks=%d rows=%d: tile %d x %d, %d groups, %d bytes\n", name,
                (long long)M, (long long)N, (long long)K, (long long)lda, gram, o.blocks_per_sm, o.rows_per_tile, pl.tm,
                pl.tn, pl.groups, pl.smem);
}

template <typename T, typename Acc>
static void walk(const char* name) {
  const LaunchOpts opts[] = {{0, 0, -1}, {1, 64, -1}, {2, 0, -1}, {2, 512, -1}};
  for (int64_t M = 1; M <= 1000; M++) {
    for (const LaunchOpts& o : opts)
      for (int64_t K : {1, 17, 1000, 1 << 18, 1 << 24})
        for (int64_t pad : {0, 1, 12}) one<T, Acc>(name, M, M, K, M + pad, M + pad, true, o);
    for (int64_t N = 1; N <= 1000; N++) one<T, Acc>(name, M, N, 1 << 18, M, N, false, opts[0]);
    for (int64_t N = 1; N <= 1000; N += 7)
      for (const LaunchOpts& o : opts)
        for (int64_t K : {17, 1000, 1 << 24}) one<T, Acc>(name, M, N, K, M + 3, N + 3, false, o);
  }
}

int main() {
  std::vector<std::thread> t;
  t.emplace_back(walk<float, float>, "f32");
  t.emplace_back(walk<double, double>, "f64");
  t.emplace_back(walk<double, dd>, "f64 dd");
  t.emplace_back(walk<c32, c32>, "c64");
  t.emplace_back(walk<c64, c64>, "c128");
  t.emplace_back(walk<c32h, c32h>, "c64 conj");
  t.emplace_back(walk<c64h, c64h>, "c128 conj");
  t.emplace_back(walk<float, double>, "f32 dd");
  t.emplace_back(walk<c32, c64>, "c64 dd");
  t.emplace_back(walk<c64, zdd>, "c128 dd");
  for (auto& x : t) x.join();
  std::printf("plans %ld with several groups %ld bad %d\n", plans.load(), many.load(), bad.load());
  return bad.load() ? 1 : 0;
}
