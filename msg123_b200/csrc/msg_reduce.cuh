// msg_reduce.cuh -- second stage of the deterministic reductions inside the kernel that writes
// the partials, and the hand-over of results to the host.
#pragma once
#include "msg_common.cuh"

namespace msg {

// What a finishing kernel hands to the host: `count` results from res into pinned words, then
// the token (null word: nothing).
struct Publish {
  const double *res;
  double *host;
  int count;
  unsigned *word, token;
  __device__ __forceinline__ void operator()() const {   // one thread, all results written
    if (!word) return;
    __threadfence();
    for (int k = 0; k < count; ++k) host[k] = __ldcg(res + k);
    __threadfence_system();
    *(volatile unsigned *)word = token;
  }
};

// True in the block that arrives last of `total` (all its threads); the counter is left at 0.
__device__ __forceinline__ bool last_block(int *cnt, int total) {
  __shared__ int s_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    s_last = atomicAdd(cnt, 1) == total - 1;
    if (s_last) *cnt = 0;
  }
  __syncthreads();
  if (s_last) __threadfence();
  return s_last;
}

// Second stage by the last block of the kernel that wrote the partials (fuse), for arrays of
// at most kFuseParts: the sums of k_finish, whose thread t starts with element t; here a
// thread stands for four of its threads.
// It saves a launch (the 20 000-cell box 5.15 -> 4.3 ms) but holds every block until its
// ticket has gone round; with more blocks than the chip takes at once that costs more than
// the launch (364k cells, 1444 blocks: 9.1 against 8.6 ms).  Longer arrays therefore keep the
// separate launch, and a kernel of their own (FUSE = false): the registers of this stage
// would also halve the resident blocks of the passes that stream memory.
constexpr int kFuseParts = 512;
struct Fin {
  bool fuse;
  const double *part;
  int nparts, narr;
  double *out;
  int *cnt;
  Publish pub;
};
// MAXB: bit a set -> array a takes the maximum instead of the sum.  All 256 threads of every
// block of the grid (nblocks of them).
template <int MAXB = 0>
__device__ __forceinline__ void fin_block(const Fin &f, int nblocks) {
  if (!last_block(f.cnt, nblocks)) return;
  __shared__ double sh[256];
  const int t = threadIdx.x;
  for (int a = 0; a < f.narr; ++a) {
    const double *p = f.part + (size_t)a * f.nparts;
    const bool mx = (MAXB >> a) & 1;
    auto comb = [&](double x, double y) { return mx ? fmax(x, y) : __dadd_rn(x, y); };
    double s[4];
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      // u = 0 only: the others lie beyond kFuseParts, and their zeros add nothing
      const int i = t + 256 * v;
      s[v] = i < f.nparts ? comb(0.0, __ldcg(p + i)) : 0.0;
    }
    sh[t] = comb(comb(s[0], s[2]), comb(s[1], s[3]));
    __syncthreads();
    for (int o = 128; o >= 32; o >>= 1) {
      if (t < o) sh[t] = comb(sh[t], sh[t + o]);
      __syncthreads();
    }
    if (t < 32) {
      double r = sh[t];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) r = comb(r, __shfl_down_sync(0xffffffffu, r, o));
      if (t == 0) f.out[a] = r;
    }
    __syncthreads();
  }
  if (t == 0) f.pub();
}

// A scalar that a kernel takes from the host or from the device: the step of the line search,
// or Brown and Saad's eps of J v (calc_vecjacf, Calc_function.f90:515-621) from (v, v),
// (x, v) and |v|_1 in eps[0 .. 2].
struct Step {
  double host;
  const double *eps;
  double root;               // sqrt of the machine epsilon
  __device__ __forceinline__ double get() const {
    if (!eps) return host;
    const double l2_v = eps[0], l2_x = eps[1], l1_v = eps[2];
    const double sign = l2_x < 0.0 ? -1.0 : 1.0;
    return __ddiv_rn(__dmul_rn(__dmul_rn(sign, root), fmax(fabs(l2_x), l1_v)), l2_v);
  }
};

}  // namespace msg
