// Test driver (CPU only) for host paths of the product's library, one per
// argument. The kernel launchers are stubs and no device is touched: what
// would allocate device memory fails there. Exit 0 when every check holds,
// else the number of the first failed check.
#include "dgpu_host.cpp"

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <new>

namespace dgpu {
void launch_profiles(const uint8_t*, const uint32_t*, const uint32_t*, uint32_t, int, uint8_t*, uint8_t*,
                     cudaStream_t) {}
void launch_profiles_sparse(const uint8_t*, const uint32_t*, const uint32_t*, uint32_t, uint32_t, uint16_t*,
                            uint8_t*, uint32_t*, uint8_t*, cudaStream_t) {}
void launch_compare(const CompareLaunch&, cudaStream_t, cudaEvent_t*) {}
uint32_t compare_screen_chunk(uint32_t, uint32_t, uint32_t) { return 4; }
int capture_compare_graph(const CompareLaunch&, cudaStream_t, uint32_t, bool, uint32_t, cudaGraph_t*) { return 1; }
void launch_fill_f64(double*, size_t, double, cudaStream_t) {}
void launch_final_subs(const FinalSubsLaunch&, cudaStream_t) {}
void launch_align_debug(int, const uint8_t*, const uint32_t*, const uint32_t*, const uint8_t*, const uint32_t*,
                        const uint32_t*, uint32_t, KParams, int, const NwGeom&, uint8_t*, uint8_t*, uint8_t*,
                        const uint32_t*, uint32_t*, uint32_t*, cudaStream_t) {}
}  // namespace dgpu

using namespace dgpu;

// operator new throws on this thread once `left` allocations have passed
static thread_local long left = -1;
void* operator new(size_t n) {
  if (left == 0) throw std::bad_alloc();
  if (left > 0) --left;
  if (void* p = std::malloc(n ? n : 1)) return p;
  throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

static int check(int no, bool ok) {
  if (!ok) std::printf("check %d failed\n", no);
  return ok ? 0 : no;
}

// The alignment kernels' resident warps: four blocks per SM, unless their
// scratch is large and the tuning asks for fewer.
static int geometry() {
  auto warps_per_sm = [](uint32_t lmax, int band, int mismatch, int homo_gap) {
    Pool* P = new Pool;  // never freed: its buffers are not
    P->nslots = 0;
    P->kp.match = 5;
    P->kp.mismatch = mismatch;
    P->kp.gap = -8;
    P->kp.homo_gap = homo_gap;
    P->kp.band = band;
    P->kp.vectorized = 1;
    P->kp.ncol = 41;
    P->lmax = lmax;
    P->lmin = lmax - 2;
    return P->size_nw() ? -1 : P->geom.nwarps / P->sms;
  };
  dgpu_tuning t;
  for (int ctas : {1, 2, 4}) {
    for (int cls = 0; cls < 3; ++cls) {
      if (int r = check(1, dgpu_tuning_get(cls == 0 ? 150 : cls == 1 ? 500 : 3000, &t) == 0)) return r;
      t.align_ctas_per_sm = ctas;
      if (int r = check(2, dgpu_tuning_set(cls, &t) == 0)) return r;
    }
    const int full = kAlignCtasPerSm * kNwWarps, tuned = ctas * kNwWarps;
    if (int r = check(3, warps_per_sm(250, 16, -4, -8) == full)) return r;    // strip aligner
    if (int r = check(4, warps_per_sm(1550, 32, -4, -1) == full)) return r;
    if (int r = check(5, warps_per_sm(250, 16, -130, -8) == full)) return r;  // vectorized forms, 16 kB a warp
    if (int r = check(6, warps_per_sm(500, -1, -4, -8) == full)) return r;    // 0.5 MB
    if (int r = check(7, warps_per_sm(3500, -1, -4, -8) == tuned)) return r;  // 24.5 MB: 58 GB a launch slot in full
    if (int r = check(8, warps_per_sm(9000, -1, -4, -1) == tuned)) return r;  // row-major
  }
  return 0;
}

// Which launches may store directly: the pairs that all of a launch's samples
// expect together have to fit the posts.
static int direct_room() {
  Pool* P = new Pool;
  P->kp.use_kmers = 1;
  Slot* L = new Slot;
  L->P = P;
  if (int r = check(1, L->direct_fits(8, 8 * 1000) == false)) return r;  // each sample's would, all eight's do not
  if (int r = check(2, L->direct_fits(8, 8 * 300) == true)) return r;
  if (int r = check(3, L->direct_fits(1, 1000) == true)) return r;
  if (int r = check(4, L->direct_fits(kScreenSmemTasks + 1, 10) == false)) return r;
  if (int r = check(5, kPostExpect < kPostMax && L->direct_fits(2, kPostExpect) && !L->direct_fits(2, kPostExpect + 1)))
    return r;
  P->kp.lambda32 = 1;
  return check(6, L->direct_fits(1, 10) == false);
}

// A large map call fills its outputs on other threads; whatever allocation
// fails meanwhile, the call ends with an error or the exception, not with the
// program. (Here it ends where it asks for pinned memory at the latest.)
static int compare_without_memory() {
  const uint32_t n = 200000;
  dgpu_ctx* ctx = new dgpu_ctx;  // never freed: its buffers are not
  ctx->uploaded = true;
  ctx->reads.assign(n, 1u);
  ctx->total_reads = n;
  Pool& P = ctx->pool;
  P.nraw = n;
  P.kp.use_kmers = 1;
  P.kp.kmer_size = 5;
  P.lock_host.h = static_cast<uint8_t*>(std::calloc(n, 1));
  P.slots.emplace_back(new Slot);
  Slot& L = P.slot0();
  L.P = &P;
  L.ntask_cap = 1;
  L.task_stage.h = static_cast<TaskDev*>(std::calloc(1, sizeof(TaskDev)));
  std::vector<double> lam(n);
  std::vector<uint32_t> ham(n);
  std::vector<uint8_t> skipped(n);
  int threw = 0;
  for (long allowed = 0; allowed < 24; ++allowed) {
    int rc = 1;
    try {
      left = allowed;
      rc = dgpu_compare(ctx, 0, 0.42, 1, lam.data(), ham.data(), skipped.data(), nullptr);
    } catch (const std::bad_alloc&) {
      ++threw;
    }
    left = -1;
    if (int r = check(1, rc != 0)) return r;
    std::vector<uint32_t>().swap(L.task_blk0);  // as before the first call
  }
  return check(2, threw > 0);
}

int main(int argc, char** argv) {
  const std::string what = argc > 1 ? argv[1] : "";
  const int r = what == "geometry" ? geometry() : what == "direct_room" ? direct_room()
                : what == "compare_without_memory" ? compare_without_memory()
                                                   : 99;
  if (r == 0) std::printf("ok\n");
  return r;
}
