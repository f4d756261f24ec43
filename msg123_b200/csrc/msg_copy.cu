// msg_copy.cu -- large device-to-host copies into ordinary (pageable) memory.
//
// The ABI hands results to host arrays that it does not own, usually fresh ones whose pages
// do not exist yet.  One thread faulting the pages in and copying through the driver's
// staging buffer moves 4 to 8 GB/s, an eighth of the link.  Here copies of kMinBytes or more
// in all are cut into pieces that several threads bring in through pinned slots of their own, two each,
// so that a piece crosses the link while the one before it is copied out.  The caller works
// too and waits only for pieces that another thread has taken, never for a thread: one that
// the system starts late finds nothing left (threads made and joined per copy cost a
// scheduler tick of 4 ms now and then).  Threads, slots and streams are shared by all contexts
// of the process: made at the first such copy, which pays 1.5 to 2.5 ms for them, and given back
// with the last context or network (a host that makes and drops its only context pays each
// time); a second copy at the same time, or one on another device, goes the plain way.  The
// velocities of 1.5M cells (108 MB) took 26 ms, now 6.
#include "msg_ctx.cuh"
#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstdlib>
#include <cstring>
#include <exception>
#include <memory>
#include <mutex>
#include <new>
#include <thread>
#include <sys/mman.h>

namespace msg {

constexpr int kMaxThreads = 8, kMaxCopies = 16;
constexpr size_t kSlot = (size_t)1 << 19, kMinBytes = (size_t)4 << 20, kHugePage = (size_t)2 << 20;
constexpr size_t kStageBytes = kMaxThreads * 2 * kSlot;

// One copy: its arrays cut into pieces of kSlot bytes, taken by number.
struct CopyJob {
  CopyOut list[kMaxCopies];
  size_t first[kMaxCopies + 1];   // pieces before each array
  int n = 0;
  std::atomic<size_t> next{0}, done{0};
  std::atomic<int> err{0};
  size_t pieces() const { return first[n]; }
};

struct Stage {
  int device = -1, nthreads = 1;   // the caller's among them
  char *slots = nullptr;           // [thread][2][kSlot] pinned
  cudaStream_t stream[kMaxThreads] = {};
  cudaEvent_t event[kMaxThreads][2] = {};
  std::thread thread[kMaxThreads];
  std::mutex mu;                   // job, number, stop
  std::condition_variable cv;
  std::shared_ptr<CopyJob> job;
  unsigned long long number = 0;
  bool stop = false;

  // A thread keeps one piece on the link and copies the one before it out.
  void work(CopyJob &j, int t) {
    const size_t pieces = j.pieces();
    size_t piece[2] = {pieces, pieces};
    const CopyOut *c;
    size_t o, len;
    auto place = [&](size_t p) {
      int k = 0;
      while (p >= j.first[k + 1]) ++k;
      c = &j.list[k];
      o = (p - j.first[k]) * kSlot;
      len = std::min(kSlot, c->bytes - o);
    };
    auto begin = [&](int b) {
      piece[b] = j.next.fetch_add(1);
      if (piece[b] >= pieces || j.err.load()) return;
      place(piece[b]);
      cudaError_t e = cudaMemcpyAsync(slots + (2 * t + b) * kSlot, (const char *)c->src + o, len, cudaMemcpyDeviceToHost,
                                      stream[t]);
      if (e == cudaSuccess) e = cudaEventRecord(event[t][b], stream[t]);
      if (e != cudaSuccess) j.err.store((int)e);
    };
    begin(0);
    for (int b = 0; piece[b] < pieces; b ^= 1) {
      begin(b ^ 1);
      if (!j.err.load()) {
        const cudaError_t e = cudaEventSynchronize(event[t][b]);
        if (e == cudaSuccess) {
          place(piece[b]);
          memcpy((char *)c->dst + o, slots + (2 * t + b) * kSlot, len);
        } else {
          j.err.store((int)e);
        }
      }
      if (j.err.load()) cudaStreamSynchronize(stream[t]);   // nothing of this copy stays in flight
      j.done.fetch_add(1, std::memory_order_release);
    }
  }

  bool lane(int t) {   // a thread's stream and events
    bool ok = cudaStreamCreateWithFlags(&stream[t], cudaStreamNonBlocking) == cudaSuccess;
    for (auto &e : event[t]) ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
    if (!ok) cudaGetLastError();
    return ok;
  }

  void serve(int t) {
    if (cudaSetDevice(device) != cudaSuccess || !lane(t)) return;
    unsigned long long seen = 0;
    for (;;) {
      std::shared_ptr<CopyJob> j;
      {
        std::unique_lock<std::mutex> lk(mu);
        cv.wait(lk, [&] { return stop || number != seen; });
        if (stop) return;
        seen = number;
        j = job;
      }
      if (j) work(*j, t);
    }
  }

  // Large pages where the system has them: to pin 8 MB of 4 KB pages takes 3.5 to 6.5 ms, of four
  // large ones and their first touch 1.4.  The threads make their own streams while the caller
  // copies.
  bool make(int dev) {
    device = dev;
    void *m = nullptr;
    if (posix_memalign(&m, kHugePage, kStageBytes)) return false;
    madvise(m, kStageBytes, MADV_HUGEPAGE);   // no matter if it does not take
    if (cudaHostRegister(m, kStageBytes, cudaHostRegisterPortable) != cudaSuccess) {
      cudaGetLastError();
      free(m);
      return false;
    }
    slots = (char *)m;
    if (!lane(0)) return false;
    const int want = std::max(1, std::min<int>(kMaxThreads, (int)std::thread::hardware_concurrency() - 1));
    try {
      for (; nthreads < want; ++nthreads) thread[nthreads] = std::thread(&Stage::serve, this, nthreads);
    } catch (const std::exception &) {   // as many as the system gives (no thread, no memory)
    }
    return true;
  }

  ~Stage() {
    {
      std::lock_guard<std::mutex> lk(mu);
      stop = true;
    }
    cv.notify_all();
    for (auto &t : thread)
      if (t.joinable()) t.join();
    for (int t = 0; t < kMaxThreads; ++t) {
      if (stream[t]) cudaStreamDestroy(stream[t]);
      for (auto &e : event[t])
        if (e) cudaEventDestroy(e);
    }
    if (slots) {
      cudaHostUnregister(slots);
      free(slots);
    }
  }

  void run(const std::shared_ptr<CopyJob> &j) {
    {
      std::lock_guard<std::mutex> lk(mu);
      job = j;
      ++number;
    }
    cv.notify_all();
    work(*j, 0);
    while (j->done.load(std::memory_order_acquire) < j->pieces()) std::this_thread::yield();
    std::lock_guard<std::mutex> lk(mu);
    job.reset();
  }
};

// Held while the stage is in use, made or given back; the stage itself is not a static object:
// a process that ends with contexts left leaves it, and its waiting threads, to the system.
static std::mutex g_stage_mu;
static int g_stage_refs = 0;
static Stage *g_stage = nullptr;

void stage_ref() {
  std::lock_guard<std::mutex> lk(g_stage_mu);
  ++g_stage_refs;
}
void stage_unref() {
  std::lock_guard<std::mutex> lk(g_stage_mu);
  if (--g_stage_refs == 0) {
    delete g_stage;
    g_stage = nullptr;
  }
}

// Every dst (host; null: none) <- src (device), whose producers have finished.  Returns when
// all are complete.
int copy_out(const CopyOut *jobs, int n) {
  size_t total = 0;
  bool pageable[kMaxCopies] = {};
  for (int k = 0; k < n && k < kMaxCopies; ++k) {
    if (!jobs[k].dst) continue;
    cudaPointerAttributes at;
    pageable[k] = cudaPointerGetAttributes(&at, jobs[k].dst) == cudaSuccess && at.type == cudaMemoryTypeUnregistered;
    cudaGetLastError();
    if (pageable[k]) total += jobs[k].bytes;
  }
  bool staged = false;
  if (total >= kMinBytes) {
    std::unique_lock<std::mutex> lk(g_stage_mu, std::try_to_lock);
    int device = 0;
    MSG_CUDA(cudaGetDevice(&device));
    if (lk.owns_lock() && g_stage_refs > 0) {
      if (!g_stage) {
        g_stage = new (std::nothrow) Stage();
        if (g_stage && !g_stage->make(device)) {
          delete g_stage;
          g_stage = nullptr;
        }
      }
      std::shared_ptr<CopyJob> j;
      try {
        if (g_stage && g_stage->device == device) j = std::make_shared<CopyJob>();
      } catch (const std::bad_alloc &) {
      }
      if (j) {
        j->first[0] = 0;
        for (int k = 0; k < n && k < kMaxCopies; ++k)
          if (pageable[k]) {
            j->list[j->n] = jobs[k];
            j->first[j->n + 1] = j->first[j->n] + (jobs[k].bytes + kSlot - 1) / kSlot;
            ++j->n;
          }
        g_stage->run(j);
        if (j->err.load()) {
          set_error("copy to the host: %s", cudaGetErrorString((cudaError_t)j->err.load()));
          return MSG_ERR_CUDA;
        }
        staged = true;
      }
    }
  }
  for (int k = 0; k < n; ++k)
    if (jobs[k].dst && !(staged && k < kMaxCopies && pageable[k]))
      MSG_CUDA(cudaMemcpy(jobs[k].dst, jobs[k].src, jobs[k].bytes, cudaMemcpyDeviceToHost));
  return MSG_OK;
}

int copy_out(void *dst, const void *src, size_t bytes) {
  const CopyOut job{dst, src, bytes};
  return copy_out(&job, 1);
}

}  // namespace msg
