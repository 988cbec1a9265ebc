// Readbacks of device buffers to the caller's host memory.
//
// The caller's arrays are ordinary pageable memory, often never touched before: a
// plain copy into them goes through the driver's staging buffer on one thread, which
// also takes the page faults.  Large readbacks here go through pinned chunks instead: a
// few threads each ask for chunks of the buffer in turn, and while the next chunk
// crosses the bus a thread copies its last one to the caller's memory, so bus, page
// faults and copies overlap: the 2048 x 2048 Wigner function of a mode, 32 MB into a
// fresh array, takes 2.2-2.4 ms instead of 8.1 (0.2 ms of it kernels; six threads for any
// size 2.7), the 512 x 512 one 0.30 instead of 0.40.

#include <atomic>
#include <cstring>
#include <mutex>
#include <thread>

#include "cvdv_internal.cuh"

namespace cvdv {

// The staging memory: kSlots pinned chunks, one pool per process, made at the first
// large readback and given back with the process's last context.  A readback that
// finds it in use by another thread takes the plain copy.
constexpr size_t kStageChunk = 2ull << 20;  // a huge page of the destination
constexpr int kStageThreads = 6;
constexpr int kStageSlots = 2 * kStageThreads;
constexpr size_t kStageMin = 2ull << 20;  // smaller readbacks copy directly

static std::mutex g_stageMu;  // held for a whole readback
static char* g_stage = nullptr;
static std::mutex g_contextsMu;
static int g_contexts = 0;

void host_copy_context_made() {
  std::lock_guard<std::mutex> lk(g_contextsMu);
  ++g_contexts;
}

void host_copy_context_gone() {
  std::lock_guard<std::mutex> lk(g_contextsMu);
  if (--g_contexts > 0) return;
  std::lock_guard<std::mutex> stage(g_stageMu);
  if (g_stage) cudaFreeHost(g_stage);
  g_stage = nullptr;
}

static bool pinned(const void* p) {
  cudaPointerAttributes a{};
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type != cudaMemoryTypeUnregistered;
}

// Chunk boundaries at multiples of kStageChunk of the destination's addresses, so two
// threads do not fault in the same huge page.
struct StagePlan {
  char* dst;
  const char* src;
  size_t bytes, head;  // head: bytes before the first boundary (0: none)
  size_t count() const { return (head ? 1 : 0) + (bytes - head + kStageChunk - 1) / kStageChunk; }
  void chunk(size_t i, size_t* at, size_t* len) const {
    if (head && i == 0) {
      *at = 0;
      *len = head;
      return;
    }
    *at = head + (i - (head ? 1 : 0)) * kStageChunk;
    *len = bytes - *at < kStageChunk ? bytes - *at : kStageChunk;
  }
};

// One thread's share: chunks claimed in order, two in flight.
static cudaError_t stage_worker(const StagePlan& P, int device, cudaStream_t stream, char* slots,
                                std::atomic<size_t>* next, std::atomic<bool>* failed) {
  cudaError_t e = cudaSetDevice(device);
  cudaEvent_t ev[2] = {nullptr, nullptr};
  for (int k = 0; k < 2 && e == cudaSuccess; ++k) e = cudaEventCreateWithFlags(&ev[k], cudaEventDisableTiming);
  const size_t n = P.count();
  size_t at[2], len[2] = {0, 0};
  for (int s = 0; e == cudaSuccess; s ^= 1) {
    const size_t i = failed->load() ? n : next->fetch_add(1);
    len[s] = 0;
    if (i < n) {
      P.chunk(i, &at[s], &len[s]);
      e = cudaMemcpyAsync(slots + s * kStageChunk, P.src + at[s], len[s], cudaMemcpyDeviceToHost, stream);
      if (e == cudaSuccess) e = cudaEventRecord(ev[s], stream);
      if (e != cudaSuccess) break;
    }
    const int o = s ^ 1;  // the chunk asked for before this one
    if (len[o]) {
      e = cudaEventSynchronize(ev[o]);
      if (e != cudaSuccess) break;
      memcpy(P.dst + at[o], slots + o * kStageChunk, len[o]);
    } else if (!len[s]) {
      break;
    }
  }
  if (e != cudaSuccess) {
    failed->store(true);
    cudaStreamSynchronize(stream);  // none of this thread's copies writes a slot after it leaves
  }
  for (cudaEvent_t v : ev)
    if (v) cudaEventDestroy(v);
  return e;
}

bool copy_to_host(Context* ctx, void* dst, const void* src, size_t bytes, const char* what) {
  std::unique_lock<std::mutex> stage(g_stageMu, std::defer_lock);
  bool staged = bytes >= kStageMin && std::thread::hardware_concurrency() > 2 && !pinned(dst) && stage.try_lock();
  if (staged && !g_stage && cudaHostAlloc((void**)&g_stage, kStageSlots * kStageChunk, cudaHostAllocPortable) != cudaSuccess) {
    cudaGetLastError();
    g_stage = nullptr;
    staged = false;
  }
  if (!staged)
    return cuda_ok(ctx, cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, ctx->stream), what) &&
           stream_sync(ctx, what);
  StagePlan P{(char*)dst, (const char*)src, bytes, 0};
  const size_t past = (uintptr_t)dst & (kStageChunk - 1);
  if (past) P.head = kStageChunk - past < bytes ? kStageChunk - past : bytes;
  const size_t chunks = P.count();
  int threads = (int)std::thread::hardware_concurrency() - 1;
  if (threads > kStageThreads) threads = kStageThreads;
  // (at least two chunks a thread: a thread's start costs as much as a chunk's copy)
  if ((size_t)threads > chunks / 2) threads = chunks >= 2 ? (int)(chunks / 2) : 1;
  std::atomic<size_t> next{0};
  std::atomic<bool> failed{false};
  cudaError_t err[kStageThreads] = {};
  std::thread pool[kStageThreads];
  int started = 0;
  // (a thread that cannot be started leaves its share to the others)
  for (int k = 1; k < threads; ++k) {
    try {
      pool[k] = std::thread([&, k] {
        err[k] = stage_worker(P, ctx->device, ctx->stream, g_stage + 2 * k * kStageChunk, &next, &failed);
      });
      ++started;
    } catch (...) {
      break;
    }
  }
  int current = 0;
  cudaGetDevice(&current);
  err[0] = stage_worker(P, ctx->device, ctx->stream, g_stage, &next, &failed);
  for (int k = 1; k <= started; ++k) pool[k].join();
  cudaSetDevice(current);
  for (int k = 0; k <= started; ++k)
    if (!cuda_ok(ctx, err[k], what)) return false;
  return stream_sync(ctx, what);
}

}  // namespace cvdv
