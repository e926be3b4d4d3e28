// Device buffers kept between calls on a grid: cudaMalloc and cudaFree (which
// waits for the device) took 0.2 ms of a 0.05 ms preconditioner call and
// about 1 ms of a 64^3 solve.  What is kept is bounded per buffer and over
// the process, and freed with the grid, on request, and before an allocation
// of the library is given up.
#include <atomic>
#include <set>
#include <vector>

#include "pg_common.cuh"
#include "pg_solve.cuh"

namespace pg {

namespace {
constexpr int kWordsPerBlock = 1024;  // a page of status words at a time
std::mutex g_words_m;
std::vector<int*> g_words_free;
}  // namespace

pg_status StatusWord::alloc() {
  std::lock_guard<std::mutex> l(g_words_m);
  if (g_words_free.empty()) {
    void* block = nullptr;
    if (cudaHostAlloc(&block, kWordsPerBlock * sizeof(int), cudaHostAllocMapped | cudaHostAllocPortable) !=
        cudaSuccess) {
      cudaGetLastError();
      set_error("allocation of the status words failed");
      return PG_OOM;
    }
    for (int i = 0; i < kWordsPerBlock; ++i) g_words_free.push_back(static_cast<int*>(block) + i);
  }
  void* dev = nullptr;
  PG_CUDA_TRY(cudaHostGetDevicePointer(&dev, g_words_free.back(), 0));
  h = g_words_free.back();
  p = static_cast<int*>(dev);
  g_words_free.pop_back();
  *h = 0;
  return PG_OK;
}

StatusWord::~StatusWord() {
  if (!h) return;
  std::lock_guard<std::mutex> l(g_words_m);
  g_words_free.push_back(const_cast<int*>(h));
}

namespace {

constexpr long long kScratchMost = 256ll << 20;  // one grid's scratch
constexpr long long kSolveMost = 1ll << 30;      // one grid's solve buffers
constexpr long long kKeptMost = 2ll << 30;       // all grids of the process
std::atomic<long long> g_kept{0};

// Books `bytes` more of the process's total; false if that would pass it.
bool book(long long bytes) {
  long long now = g_kept.load();
  while (now + bytes <= kKeptMost)
    if (g_kept.compare_exchange_weak(now, now + bytes)) return true;
  return false;
}

// The grids that keep something.  Never destroyed: grids may outlive the
// library's static objects.
struct Keepers {
  std::mutex m;
  std::set<const pg_grid*> grids;
};
Keepers& keepers() {
  static Keepers* k = new Keepers();
  return *k;
}

bool take(std::atomic<bool>& busy) { return !busy.exchange(true, std::memory_order_acquire); }
void give(std::atomic<bool>& busy) { busy.store(false, std::memory_order_release); }

void enlist(const pg_grid* g) {
  std::lock_guard<std::mutex> l(keepers().m);
  keepers().grids.insert(g);
}

}  // namespace

// A grid that is in use by a call (this thread's own among them) keeps what
// that call holds.
size_t release_kept() {
  size_t freed = 0;
  std::lock_guard<std::mutex> l(keepers().m);
  for (const pg_grid* g : keepers().grids) {
    if (take(g->scratch_busy)) {
      freed += g->scratch.n;
      g_kept -= (long long)g->scratch.n;
      g->scratch.release();
      give(g->scratch_busy);
    }
    if (take(g->solve_busy)) {
      freed += g->solve_kept;
      g_kept -= (long long)g->solve_kept;
      g->solve_ws.reset();
      g->solve_kept = 0;
      give(g->solve_busy);
    }
  }
  return freed;
}

pg_status ScratchLease::get(size_t bytes, unsigned char** p) {
  if (take(g_->scratch_busy)) {
    held_ = true;
    if (g_->scratch.n >= bytes) {
      *p = g_->scratch.p;
      return PG_OK;
    }
    const long long before = (long long)g_->scratch.n;
    if ((long long)bytes <= kScratchMost && book((long long)bytes - before)) {
      const pg_status s = g_->scratch.alloc(bytes);  // releases the smaller one
      if (s == PG_OK) {
        enlist(g_);
        *p = g_->scratch.p;
        return PG_OK;
      }
      g_kept -= (long long)bytes;  // not taken, and the old one is gone
    }
    held_ = false;
    give(g_->scratch_busy);
  }
  PG_TRY(own_.alloc(bytes));
  *p = own_.p;
  return PG_OK;
}

ScratchLease::~ScratchLease() {
  if (held_ || own_.p) cudaStreamSynchronize(st_);
  if (held_) give(g_->scratch_busy);
}

SolveLease::SolveLease(const pg_grid* g, cudaStream_t st) : g_(g), st_(st), held_(take(g->solve_busy)) {
  if (held_) ws_ = g_->solve_ws;
  if (!ws_) ws_ = std::shared_ptr<SolveWorkspace>(workspace_create(), workspace_destroy);
}

SolveLease::~SolveLease() {
  if (!held_) return;
  cudaStreamSynchronize(st_);
  const long long bytes = (long long)workspace_bytes(ws_.get());
  if (bytes <= kSolveMost && book(bytes - (long long)g_->solve_kept)) {
    g_->solve_ws = ws_;
    g_->solve_kept = (size_t)bytes;
    enlist(g_);
  } else {
    g_kept -= (long long)g_->solve_kept;
    g_->solve_ws.reset();
    g_->solve_kept = 0;
  }
  ws_.reset();
  give(g_->solve_busy);
}

}  // namespace pg

pg_grid::~pg_grid() {
  std::lock_guard<std::mutex> l(pg::keepers().m);
  pg::keepers().grids.erase(this);
  pg::g_kept -= (long long)scratch.n + (long long)solve_kept;
}

extern "C" long pg_release_buffers(void) { return (long)pg::release_kept(); }
