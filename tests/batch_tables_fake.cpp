// The batch engine's host code (heat_batch_host.cpp) on a fake CUDA runtime, in
// which an asynchronous copy reads its source as late as it may: when something
// waits for it or a kernel that needs it is launched.  Every copy's source must be
// page-locked memory that is still allocated and unchanged at that point, and each
// table launch must see its own grids' entries and tensor maps.  Prints the
// violations and returns their count.

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <vector>

#include "heat_batch_internal.h"

static int violations = 0;
static void violated(const char *what) {
  ++violations;
  std::printf("%s\n", what);
}

// ---- fake runtime ---------------------------------------------------------
static std::map<char *, size_t> pinned;
struct Copy {
  char *dst;
  const char *src;
  size_t n;
  std::vector<char> then;  // the source when the copy was queued
};
static std::vector<Copy> pending;
static bool page_locked(const char *p, size_t n) {
  auto it = pinned.upper_bound(const_cast<char *>(p));
  return it != pinned.begin() && (--it, p + n <= it->first + it->second);
}
static void finish_copies() {
  for (const Copy &c : pending) {
    if (!page_locked(c.src, c.n)) {
      violated("an asynchronous copy reads pageable or released memory");
      std::memset(c.dst, 0xee, c.n);
      continue;
    }
    if (std::memcmp(c.src, c.then.data(), c.n)) violated("a copy's source changed before it was read");
    std::memcpy(c.dst, c.src, c.n);
  }
  pending.clear();
}

extern "C" {
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaMalloc(void **p, size_t n) { return *p = std::calloc(1, n), cudaSuccess; }
cudaError_t cudaFree(void *p) { return finish_copies(), std::free(p), cudaSuccess; }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) {
  *p = std::malloc(n);
  pinned[static_cast<char *>(*p)] = n;
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) {
  pinned.erase(static_cast<char *>(p));
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
  const char *c = static_cast<const char *>(s);
  pending.push_back({static_cast<char *>(d), c, n, std::vector<char>(c, c + n)});
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return finish_copies(), cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
  return *s = reinterpret_cast<cudaStream_t>(std::malloc(1)), cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { return std::free(s), cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
  return *e = reinterpret_cast<cudaEvent_t>(std::malloc(1)), cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) { return std::free(e), cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { return *d = 0, cudaSuccess; }
cudaError_t cudaGetDeviceCount(int *n) { return *n = 1, cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { return *v = 152, cudaSuccess; }
// graphs are off here
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorUnknown; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *, cudaGraph_t, unsigned long long) {
  return cudaErrorUnknown;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaErrorUnknown; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *) { return cudaErrorUnknown; }
}

// ---- the parts of the library it calls --------------------------------------
static std::vector<heat_ctx *> contexts;

namespace heat {
TuneChoice tuned_choice(int, int) { return {2, 1, 3, 2}; }
int batch_blocks_per_sm(int) { return 1; }
int fx_tiles_x(int nx) { return (nx + 30) / 32; }
int fx_tiles_y(int ny) { return (ny + 13) / 16; }
int fx_fill_chunk(long, bool) { return 2; }
int fp32c_tile_rows() { return 20; }
bool two_step_form(const heat_ctx *c) { return c->precision == HEAT_FP32C; }
int ctx_flips(const heat_ctx *, long long n) { return (int)(n & 1); }
int check_err(heat_ctx *) { return HEAT_OK; }
cudaError_t enqueue_ctx_steps(heat_ctx *, int, long long, cudaStream_t, long long *) {
  return cudaSuccess;
}
cudaError_t enqueue_one_step(heat_ctx *, int, cudaStream_t, long long *) { return cudaSuccess; }

cudaError_t launch_batch(int kind, const BatchGrid *grids, const BatchTile *tiles, int n, int, int,
                         cudaStream_t) {
  finish_copies();
  if (violations) return cudaErrorUnknown;
  const int maps = form_of_kind(kind) == kFormFx ? 4 : 7;
  for (int t = 0; t < n; ++t) {
    const BatchGrid &g = grids[tiles[t].grid];
    const heat_ctx *c = nullptr;
    for (const heat_ctx *q : contexts)
      if (q->err == g.err) c = q;
    if (!c || g.nx != c->g.nx || g.ny != c->g.ny || g.nz != c->g.nz || tiles[t].k1 >= g.nz ||
        std::memcmp(g.tmaps, c->maps, maps * sizeof(CUtensorMap)))
      return violated("a tile's grid or tensor maps are not its context's"), cudaErrorUnknown;
  }
  return cudaSuccess;
}
}  // namespace heat

static heat_ctx *context(int seed) {
  heat_ctx *c = new heat_ctx();
  c->precision = seed % 2 ? HEAT_FP32C : HEAT_FP64;
  c->g.nx = 20 + seed, c->g.ny = 30 + 2 * seed, c->g.nz = 200 + 40 * seed;
  c->err = new int(0);
  c->kq = c->precision == HEAT_FP64 ? new unsigned long long : nullptr;
  std::memset(c->maps, 1 + seed, sizeof c->maps);
  contexts.push_back(c);
  return c;
}

int main() {
  heat_batch *b = nullptr;
  if (heat_batch_create(&b, nullptr, HEAT_BATCH_NO_GRAPHS) != HEAT_OK) return 100;
  for (int q = 0; q < 8; ++q)
    if (heat_batch_add(b, context(q), 5 + 3 * q) != HEAT_OK) return 101;
  // Uneven step counts rebuild the table over and over; contexts leave and join
  // between runs, as in the server.
  for (int q = 0; q < 12; ++q) {
    long long n = 0;
    heat_batch_run(b, 3, &n);
    heat_ctx *c = contexts[q % 8];
    if (q % 3 == 2 && heat_batch_remove(b, c) == HEAT_OK) heat_batch_add(b, c, 4);
    if (q == 5) heat_batch_add(b, context(11), 9);
    if (q == 7 || q == 9) {  // one leaves with steps left, and goes
      heat_batch_remove(b, contexts.back());
      delete contexts.back();
      contexts.pop_back();
    }
  }
  heat_batch_run(b, -1, nullptr);
  heat_batch_destroy(b);
  std::printf("%d violations\n", violations);
  return violations != 0;
}
