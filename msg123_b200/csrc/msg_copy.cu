// msg_copy.cu -- large device-to-host copies into ordinary (pageable) memory.
//
// The ABI hands results to host arrays that it does not own, usually fresh ones whose pages
// do not exist yet.  One thread faulting the pages in and copying through the driver's
// staging buffer moves 4 to 8 GB/s, an eighth of the link.  Here copies of kMinBytes or more
// in all are cut into pieces that several threads bring in through pinned slots of their own, two each,
// so that a piece crosses the link while the one before it is copied out.  The slots and
// streams are shared by all contexts of the process: made at the first such copy, given back
// with the last context or network; a second copy at the same time, or one on another
// device, goes the plain way.  The velocities of 1.5M cells (108 MB) took 26 ms, now 6.
#include "msg_ctx.cuh"
#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>
#include <system_error>
#include <thread>

namespace msg {

constexpr int kMaxThreads = 8, kMaxCopies = 16;
constexpr size_t kSlot = (size_t)1 << 19, kMinBytes = (size_t)4 << 20;

static struct Stage {
  std::mutex mu;               // held while the slots are in use, made or given back
  int refs = 0, device = -1;
  char *slots = nullptr;
  cudaStream_t stream[kMaxThreads] = {};
  cudaEvent_t done[kMaxThreads][2] = {};
} g_stage;

static void stage_free(Stage &s) {
  for (int t = 0; t < kMaxThreads; ++t) {
    if (s.stream[t]) cudaStreamDestroy(s.stream[t]);
    s.stream[t] = nullptr;
    for (auto &e : s.done[t]) {
      if (e) cudaEventDestroy(e);
      e = nullptr;
    }
  }
  if (s.slots) cudaFreeHost(s.slots);
  s.slots = nullptr;
  s.device = -1;
}

void stage_ref() {
  std::lock_guard<std::mutex> lk(g_stage.mu);
  ++g_stage.refs;
}
void stage_unref() {
  std::lock_guard<std::mutex> lk(g_stage.mu);
  if (--g_stage.refs == 0) stage_free(g_stage);
}

static bool stage_make(Stage &s, int device) {
  if (s.slots) return s.device == device;
  bool ok = cudaHostAlloc((void **)&s.slots, kMaxThreads * 2 * kSlot, cudaHostAllocPortable) == cudaSuccess;
  for (int t = 0; t < kMaxThreads && ok; ++t) {
    ok = cudaStreamCreateWithFlags(&s.stream[t], cudaStreamNonBlocking) == cudaSuccess;
    for (auto &e : s.done[t]) ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
  }
  s.device = device;
  if (!ok) {
    cudaGetLastError();
    stage_free(s);
  }
  return ok;
}

// Every dst (host; null: none) <- src (device), whose producers have finished.  Returns when
// all are complete.
int copy_out(const CopyOut *jobs, int n) {
  CopyOut list[kMaxCopies];
  size_t first[kMaxCopies + 1] = {0};   // pieces before each
  int m = 0;
  size_t total = 0;
  for (int k = 0; k < n; ++k) {
    if (!jobs[k].dst) continue;
    cudaPointerAttributes at;
    const bool pageable = cudaPointerGetAttributes(&at, jobs[k].dst) == cudaSuccess && at.type == cudaMemoryTypeUnregistered;
    cudaGetLastError();
    if (pageable && m < kMaxCopies) {
      list[m] = jobs[k];
      first[m + 1] = first[m] + (jobs[k].bytes + kSlot - 1) / kSlot;
      total += jobs[k].bytes;
      ++m;
    } else {
      MSG_CUDA(cudaMemcpy(jobs[k].dst, jobs[k].src, jobs[k].bytes, cudaMemcpyDeviceToHost));
    }
  }
  if (total >= kMinBytes) {
    std::unique_lock<std::mutex> lk(g_stage.mu, std::try_to_lock);
    int device = 0;
    MSG_CUDA(cudaGetDevice(&device));
    if (lk.owns_lock() && g_stage.refs > 0 && stage_make(g_stage, device)) {
      Stage &s = g_stage;
      const int nt = std::max(1, std::min<int>(kMaxThreads, (int)std::thread::hardware_concurrency() - 1));
      const size_t pieces = first[m];
      std::atomic<size_t> next(0);
      std::atomic<int> err(0);
      // a thread keeps one piece on the link and copies the one before it out
      auto work = [&](int t) {
        cudaSetDevice(device);
        size_t piece[2] = {pieces, pieces};
        cudaError_t e = cudaSuccess;
        auto place = [&](size_t p, const CopyOut *&job, size_t &o, size_t &len) {
          int k = 0;
          while (p >= first[k + 1]) ++k;
          job = &list[k];
          o = (p - first[k]) * kSlot;
          len = std::min(kSlot, job->bytes - o);
        };
        const CopyOut *job;
        size_t o, len;
        auto begin = [&](int b) {
          piece[b] = next.fetch_add(1);
          if (piece[b] >= pieces) return;
          place(piece[b], job, o, len);
          e = cudaMemcpyAsync(s.slots + (2 * t + b) * kSlot, (const char *)job->src + o, len, cudaMemcpyDeviceToHost,
                              s.stream[t]);
          if (e == cudaSuccess) e = cudaEventRecord(s.done[t][b], s.stream[t]);
        };
        begin(0);
        for (int b = 0; e == cudaSuccess && piece[b] < pieces; b ^= 1) {
          begin(b ^ 1);
          if (e == cudaSuccess) e = cudaEventSynchronize(s.done[t][b]);
          if (e != cudaSuccess) break;
          place(piece[b], job, o, len);
          memcpy((char *)job->dst + o, s.slots + (2 * t + b) * kSlot, len);
        }
        if (e != cudaSuccess) {
          cudaStreamSynchronize(s.stream[t]);   // nothing of this copy stays in flight
          int none = 0;
          err.compare_exchange_strong(none, (int)e);
        }
      };
      std::thread th[kMaxThreads];
      int made = 0;
      try {
        for (; made < nt - 1; ++made) th[made] = std::thread(work, made + 1);
      } catch (const std::system_error &) {   // as many as the system gives
      }
      work(0);
      for (int t = 0; t < made; ++t) th[t].join();
      if (err.load()) {
        set_error("copy to the host: %s", cudaGetErrorString((cudaError_t)err.load()));
        return MSG_ERR_CUDA;
      }
      return MSG_OK;
    }
  }
  for (int k = 0; k < m; ++k) MSG_CUDA(cudaMemcpy(list[k].dst, list[k].src, list[k].bytes, cudaMemcpyDeviceToHost));
  return MSG_OK;
}

int copy_out(void *dst, const void *src, size_t bytes) {
  const CopyOut job{dst, src, bytes};
  return copy_out(&job, 1);
}

}  // namespace msg
