// memory.cu -- memory kept between calls: device scratch of the stage calls, one per
// context, and large host blocks handed to callers, one pool for the process.
#include <malloc.h>
#include <stdlib.h>

#include <algorithm>
#include <set>

#include "runtime.h"

namespace geye {

// the scratch of every context that has some
static std::mutex g_scratch_mu;
static std::set<ScratchArena *> g_scratch;

static void free_chunks(ScratchArena &A) {
  for (auto &c : A.chunks) cudaFree(c.p);
  A.chunks.clear();
  A.used = A.total = 0;
}

// what the current device's contexts keep and do not use; whether there was any
static bool give_back_scratch() {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess) return false;
  bool any = false;
  std::lock_guard<std::mutex> g(g_scratch_mu);
  for (ScratchArena *A : g_scratch)
    if (!A->busy && A->device == dev && !A->chunks.empty()) {
      free_chunks(*A);
      any = true;
    }
  return any;
}

cudaError_t device_malloc(void **out, size_t n) {
  cudaError_t e = cudaMalloc(out, n);
  if (e != cudaErrorMemoryAllocation) return e;
  if (give_back_scratch()) {
    cudaGetLastError();   // the first attempt's
    e = cudaMalloc(out, n);
  }
  return e;
}

static geye_status device_alloc(size_t n, void **out) {
  const cudaError_t e = device_malloc(out, n);
  if (e == cudaSuccess) return GEYE_OK;
  *out = nullptr;
  set_error(std::string("cudaMalloc: ") + cudaGetErrorString(e));
  return GEYE_ERR_NOMEM;
}

DevBuf::~DevBuf() { release(); }
void DevBuf::release() {
  if (p && !arena) cudaFree(p);
  p = nullptr;
  bytes = 0;
}
geye_status DevBuf::alloc(geye_ctx *ctx, size_t n) {
  if (n <= bytes && p) return GEYE_OK;
  release();
  if (injected(ctx, "alloc")) {
    set_error("injected allocation failure");
    return GEYE_ERR_INJECTED;
  }
  if (n == 0) n = 16;
  GEYE_TRY(arena ? arena->take(ctx, n, &p) : device_alloc(n, &p));
  bytes = n;
  return GEYE_OK;
}

void ScratchArena::release() {
  std::lock_guard<std::mutex> g(g_scratch_mu);
  free_chunks(*this);
  busy = false;
  g_scratch.erase(this);
}
geye_status ScratchArena::take(geye_ctx *ctx, size_t n, void **out) {
  if (!busy) {   // (only this context's calls change it)
    std::lock_guard<std::mutex> g(g_scratch_mu);
    busy = true;
    device = ctx->device;
    g_scratch.insert(this);
  }
  n = (n + 255) & ~size_t(255);
  if (chunks.empty() || chunks.back().bytes - used < n) {
    size_t bytes = std::max({n, want, size_t(1) << 20});
    void *p = nullptr;
    geye_status st = device_alloc(bytes, &p);
    if (st != GEYE_OK && bytes > n) {   // no room for what another call has used: what this one needs
      cudaGetLastError();
      bytes = n;
      st = device_alloc(bytes, &p);
    }
    GEYE_TRY(st);
    chunks.push_back({static_cast<char *>(p), bytes});
    used = 0;
  }
  *out = chunks.back().p + used;
  used += n;
  total += n;
  return GEYE_OK;
}
void ScratchArena::reset() {
  if (!busy) return;
  std::lock_guard<std::mutex> g(g_scratch_mu);
  want = std::max(want, total);
  if (want > kScratchKeep) want = 0;
  // one chunk that held the whole call stays; several make way for one of their sum
  if (chunks.size() > 1 || (!chunks.empty() && chunks.back().bytes > kScratchKeep)) free_chunks(*this);
  used = total = 0;
  busy = false;
}

// malloc's blocks (a C caller may free() them); the kept ones with their usable sizes
static std::mutex g_host_mu;
static std::vector<std::pair<size_t, void *>> g_host_kept;
static int g_host_refs = 0;
constexpr size_t kHostBig = 1 << 20, kHostKeep = 256ull << 20;

static void free_kept() {
  for (auto &k : g_host_kept) free(k.second);
  g_host_kept.clear();
}

void *host_alloc(size_t n) {
  n = std::max<size_t>(n, 1);
  if (n >= kHostBig) {
    std::lock_guard<std::mutex> g(g_host_mu);
    for (auto it = g_host_kept.begin(); it != g_host_kept.end(); ++it)
      if (it->first >= n && it->first / 2 <= n) {
        void *p = it->second;
        g_host_kept.erase(it);
        return p;
      }
  }
  if (void *p = malloc(n)) return p;
  std::lock_guard<std::mutex> g(g_host_mu);
  free_kept();
  return malloc(n);
}
void host_free(void *p) {
  if (!p) return;
  const size_t n = malloc_usable_size(p);
  if (n >= kHostBig) {
    std::lock_guard<std::mutex> g(g_host_mu);
    size_t kept = n;
    for (auto &k : g_host_kept) kept += k.first;
    if (g_host_refs > 0 && kept <= kHostKeep && g_host_kept.size() < 8) {
      g_host_kept.push_back({n, p});
      return;
    }
  }
  free(p);
}
void host_pool_ref(int d) {
  std::lock_guard<std::mutex> g(g_host_mu);
  g_host_refs += d;
  if (g_host_refs <= 0) free_kept();
}

}  // namespace geye
