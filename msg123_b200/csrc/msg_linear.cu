// msg_linear.cu -- stencil SpMV, DILU / ILU(0) by pipelined tile sweeps, BiCGStab with
// fused dot products, deterministic reductions and scans (B200, sm_100a).
//
// SpMV and the vector updates stream the DIA arrays (d, six off-diagonals) once per
// row: 72 B/row for y = A x in FP64.  One row per thread; reductions write one
// partial per block and a fixed-order second stage (k_finish) sums them, so every
// dot product repeats bit for bit from run to run.
#include "msg_ctx.cuh"
#include <algorithm>
#include <atomic>
#include <vector>
#include <climits>
#include <cmath>
#include <cstring>
#include <thread>

namespace msg {

constexpr int kFinArr = 4;   // arrays of one second reduction stage; counters: theirs, the stage's, abserrmax's, fin_block's

struct Geo3 {
  int nx, ny, nz, nxy, N;
};
static Geo3 geo3(const msg_ctx *c) { return Geo3{c->nx, c->ny, c->nz, c->nxy, c->N}; }
static int nblk(int n) { return (n + kThreads - 1) / kThreads; }

__device__ __forceinline__ void ijk(const Geo3 &g, int i, int &ix, int &iy, int &iz) {
  iz = i / g.nxy;
  int rem = i - iz * g.nxy;
  iy = rem / g.nx;
  ix = rem - iy * g.nx;
}

// ---------------------------------------------------------------------------------
// Exclusive scan of int32 in two passes over chunks of kScanE elements: the chunks' sums,
// then every block adds up the sums before its own chunk and scans the chunk (int sums are
// the same in any order).  The last block writes the total behind the output and, in 64 bits,
// into the context's box: a sum that 32 bits do not hold is known as such.  A serial pass over the chunk sums by one thread, and a third pass to add
// them, took 7 us of the 22 us of a scan of 4.2M elements.
// ---------------------------------------------------------------------------------
constexpr int kScanT = 256, kScanU = 16, kScanE = kScanT * kScanU;

template <typename T>
__device__ __forceinline__ T scan_block_sum(T v, T *sh) {   // valid in every thread
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  T r = 0;
#pragma unroll
  for (int w = 0; w < kScanT / 32; ++w) r += sh[w];
  __syncthreads();
  return r;
}

__global__ void __launch_bounds__(kScanT) k_scan_sum(const int *__restrict__ in, int n, unsigned *bsum) {
  __shared__ unsigned sh[kScanT / 32];
  const int base = blockIdx.x * kScanE;
  unsigned v = 0;                                        // a chunk's sum is below 2^32
#pragma unroll
  for (int u = 0; u < kScanU; ++u) {
    const int i = base + u * kScanT + threadIdx.x;
    if (i < n) v += in[i];
  }
  v = scan_block_sum(v, sh);
  if (threadIdx.x == 0) bsum[blockIdx.x] = v;
}

__global__ void __launch_bounds__(kScanT) k_scan_apply(const int *__restrict__ in, int *out, int n,
                                                       const unsigned *__restrict__ bsum, const int *w1, const int *w2,
                                                       HostBox *box, unsigned token) {
  __shared__ unsigned sh[kScanT / 32];
  __shared__ unsigned long long sh64[kScanT / 32];
  __shared__ int e[kScanE + kScanE / 32];                // one pad word per 32
  const int t = threadIdx.x, base = blockIdx.x * kScanE;
  unsigned long long v = 0;
  for (int k = t; k < (int)blockIdx.x; k += kScanT) v += bsum[k];
  const unsigned long long before = scan_block_sum(v, sh64);
#pragma unroll
  for (int u = 0; u < kScanU; ++u) {
    const int k = u * kScanT + t, i = base + k;
    e[k + (k >> 5)] = i < n ? in[i] : 0;
  }
  __syncthreads();
  unsigned x[kScanU], sum = 0;
#pragma unroll
  for (int u = 0; u < kScanU; ++u) {
    const int k = t * kScanU + u;
    x[u] = sum;
    sum += e[k + (k >> 5)];
  }
  unsigned inc = sum;
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned y = __shfl_up_sync(0xffffffffu, inc, o);
    if ((t & 31) >= o) inc += y;
  }
  if ((t & 31) == 31) sh[t >> 5] = inc;
  __syncthreads();
  unsigned off = inc - sum;                              // in the chunk
  for (int w = 0; w < (t >> 5); ++w) off += sh[w];
#pragma unroll
  for (int u = 0; u < kScanU; ++u) {
    const int k = t * kScanU + u;
    e[k + (k >> 5)] = (int)((unsigned)before + off + x[u]);
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < kScanU; ++u) {
    const int k = u * kScanT + t, i = base + k;
    if (i < n) out[i] = e[k + (k >> 5)];
  }
  if (blockIdx.x == gridDim.x - 1 && t == kScanT - 1) {
    const unsigned long long total = before + (off + sum);
    out[n] = (int)total;
    if (box) {
      box->total = (long long)total;
      box->v[1] = w1 ? *w1 : 0;
      box->v[2] = w2 ? *w2 : 0;
      __threadfence_system();
      *(volatile unsigned *)&box->token = token;
    }
  }
}

// Wait until a kernel has written `token` behind its results in pinned memory: the host looks
// at the word instead of copying the results and waiting for the stream (15 us a time; this
// takes 5).
static int token_wait(msg_ctx *c, const unsigned *at, unsigned token) {
  for (unsigned it = 1;; ++it) {
    if (*(const volatile unsigned *)at == token) break;
    if ((it & 0x3f) == 0) std::this_thread::yield();   // more worker threads than cores
    if ((it & 0xfff) == 0) {   // a failed kernel never writes the token
      const cudaError_t e = cudaStreamQuery(c->stream);
      if (e == cudaSuccess && *(const volatile unsigned *)at == token) break;
      if (e != cudaErrorNotReady) {
        set_error("wait for a result: %s", e == cudaSuccess ? "none" : cudaGetErrorString(e));
        return MSG_ERR_CUDA;
      }
    }
  }
  std::atomic_thread_fence(std::memory_order_acquire);
  return MSG_OK;
}

// out[0 .. n]: exclusive scan of in[0 .. n) and, at n, the total.  got, when given, receives
// the total and the device words w1, w2 (waits for them).  A total beyond 32 bits is an error
// unless the caller takes it in `wide`; out is then of no use.
int scan_exclusive(msg_ctx *c, const int *in, int *out, int n, int *got, const int *w1, const int *w2, long long *wide) {
  const int nb = std::max(1, (n + kScanE - 1) / kScanE);
  if (nb > c->scan_cap) { set_error("scan: %d elements", n); return MSG_ERR_STATE; }
  if (nb > 1) {
    k_scan_sum<<<nb, kScanT, 0, c->stream>>>(in, n, c->scan_sums);
    MSG_CHECK_LAUNCH();
  }
  if (got) c->box_token++;
  k_scan_apply<<<nb, kScanT, 0, c->stream>>>(in, out, n, c->scan_sums, w1, w2, got ? c->box : nullptr, c->box_token);
  MSG_CHECK_LAUNCH();
  if (got) {
    int rc = token_wait(c, &c->box->token, c->box_token);
    if (rc) return rc;
    const long long total = c->box->total;
    if (wide) *wide = total;
    else if (total > INT_MAX) {
      set_error("%lld entries do not fit in 32-bit offsets", total);
      return MSG_ERR_SIZE;
    }
    got[0] = (int)total;
    if (w1) got[1] = c->box->v[1];
    if (w2) got[2] = c->box->v[2];
  }
  return MSG_OK;
}

// Scratch of the scans of up to n elements and of the second reduction stage, and the pinned
// words results reach the host in.
int scan_reserve(msg_ctx *c, int n) {
  c->scan_cap = (n + kScanE - 1) / kScanE + 1;
  MSG_CUDA(cudaMalloc(&c->scan_sums, (size_t)c->scan_cap * 4));
  // behind the reduction results in the context's pinned block
  c->box = reinterpret_cast<HostBox *>(c->hpin + kRedBlocks * 8);
  memset(c->box, 0, sizeof(HostBox));
  c->box_token = 0;
  c->res_word = reinterpret_cast<unsigned *>(c->hpin + kRedBlocks * 8 + 9);
  *c->res_word = 0;
  c->res_token = 0;
  MSG_CUDA(cudaMalloc(&c->fin_scratch, (size_t)4 * 8 * 1024 * 8));
  MSG_CUDA(cudaMalloc(&c->fin_cnt, (kFinArr + 3) * 4));
  MSG_CUDA(cudaMemsetAsync(c->fin_cnt, 0, (kFinArr + 3) * 4, c->stream));
  return MSG_OK;
}

// ---------------------------------------------------------------------------------
// Stencil SpMV y = D x + L/U x in the reference's CSR order (calc_matvec,
// Linear_solution.f90:917-951) and residual r = b - A x (calc_resi,
// Calc_simulation.f90:36-73).  Optional fused dot products into partials:
//   mode 1: (y, w1)            mode 2: (y, w1), (y, y)
// ---------------------------------------------------------------------------------
__device__ __forceinline__ double stencil_row(const Geo3 &g, int i, const double *__restrict__ d,
                                              const double *__restrict__ lu, const double *__restrict__ x) {
  int ix, iy, iz;
  ijk(g, i, ix, iy, iz);
  const size_t N = g.N;
  double t = __dmul_rn(d[i], x[i]);
  if (iz > 0) t = __dadd_rn(t, __dmul_rn(lu[0 * N + i], x[i - g.nxy]));
  if (iy > 0) t = __dadd_rn(t, __dmul_rn(lu[1 * N + i], x[i - g.nx]));
  if (ix > 0) t = __dadd_rn(t, __dmul_rn(lu[2 * N + i], x[i - 1]));
  if (ix < g.nx - 1) t = __dadd_rn(t, __dmul_rn(lu[3 * N + i], x[i + 1]));
  if (iy < g.ny - 1) t = __dadd_rn(t, __dmul_rn(lu[4 * N + i], x[i + g.nx]));
  if (iz < g.nz - 1) t = __dadd_rn(t, __dmul_rn(lu[5 * N + i], x[i + g.nxy]));
  return t;
}

template <int MODE, bool RESID, bool FUSE>
__global__ void __launch_bounds__(256) k_spmv(Geo3 g, const double *__restrict__ d, const double *__restrict__ lu,
                                              const double *__restrict__ x, const double *__restrict__ b,
                                              double *__restrict__ y, const double *__restrict__ w1,
                                              double *part, Fin fin) {
  __shared__ double sh[8];
  double a0 = 0.0, a1 = 0.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < g.N; i += gridDim.x * blockDim.x) {
    double t = stencil_row(g, i, d, lu, x);
    if (RESID) t = __dsub_rn(b[i], t);
    y[i] = t;
    if (MODE >= 1) a0 = __dadd_rn(a0, __dmul_rn(t, w1[i]));
    if (MODE >= 2) a1 = __dadd_rn(a1, __dmul_rn(t, t));
  }
  if (MODE >= 1) {
    double s = block_sum<256>(a0, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = s;
  }
  if (MODE >= 2) {
    double s = block_sum<256>(a1, sh);
    if (threadIdx.x == 0) part[gridDim.x + blockIdx.x] = s;
  }
  if (FUSE) fin_block(fin, gridDim.x);
}

int launch_spmv(msg_ctx *c, const double *x, double *y) {
  k_spmv<0, false, false><<<nblk(c->N), 256, 0, c->stream>>>(geo3(c), c->dmat, c->lu, x, nullptr, y, nullptr, nullptr, Fin{});
  MSG_CHECK_LAUNCH();
  return MSG_OK;
}

// ---------------------------------------------------------------------------------
// Vector kernels with fused reductions (fixed grid -> deterministic partials).
// ---------------------------------------------------------------------------------
// p = r + beta*(pin - omega*v)  (pin: the previous direction, p itself after the first update)
__global__ void k_bicg_p(int n, const double *pin, double *p, const double *r, const double *v, double beta,
                         double omega) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    p[i] = __dadd_rn(r[i], __dmul_rn(beta, __dsub_rn(pin[i], __dmul_rn(omega, v[i]))));
}

// Sums of NV values over groups of 256 consecutive elements, one partial per group (the order
// of block_sum): a block takes kGr groups, so a thread has that many loads in flight and one
// barrier serves them all.  One group per block, with two barriers per value, left the
// two-dot pass at a third of the copy rate.
constexpr int kGr = 4;
static int ngroups(int n) { return (n + 255) / 256; }
static int gblk(int n) { return (ngroups(n) + kGr - 1) / kGr; }
template <int NV>
__device__ __forceinline__ void group_sums(double (&v)[NV][kGr], int ng, double *part) {
  __shared__ double sh[NV][kGr][8];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int a = 0; a < NV; ++a)
#pragma unroll
      for (int k = 0; k < kGr; ++k) v[a][k] = __dadd_rn(v[a][k], __shfl_down_sync(0xffffffffu, v[a][k], o));
  if (lane == 0) {
#pragma unroll
    for (int a = 0; a < NV; ++a)
#pragma unroll
      for (int k = 0; k < kGr; ++k) sh[a][k][w] = v[a][k];
  }
  __syncthreads();
  const int t = threadIdx.x;
  if (t < NV * kGr) {
    const int a = t / kGr, k = t % kGr, g = blockIdx.x * kGr + k;
    double r = 0.0;
#pragma unroll
    for (int i = 0; i < 8; ++i) r = __dadd_rn(r, sh[a][k][i]);
    if (g < ng) part[(size_t)a * ng + g] = r;
  }
}

// A quotient of two scalars, each on the device or (null pointer) from the host: the step
// lengths of BiCGStab without a host round trip to form them.
struct Quot {
  const double *num, *den;
  double hnum;
  __device__ __forceinline__ double get() const { return __ddiv_rn(num ? *num : hnum, *den); }
};

// x = xin + a*z; r = rin - a*w; partials ||r||^2 and (r, rs).  xin null: x starts at zero
// (0 + a*z, the value the zeroed x gave, without reading it); rin: the residual before the
// update (the right-hand side itself on the first update from x = 0).
template <bool FUSE>
__global__ void __launch_bounds__(256) k_bicg_xr(int n, int ng, const double *xin, double *x, const double *rin, double *r,
                                                 const double *z, const double *w, const double *rs, Quot quot,
                                                 double *part, Fin fin) {
  const double a = quot.get();
  double v[2][kGr], zi[kGr], wi[kGr], ri[kGr], si[kGr], xi[kGr];
  const int i0 = blockIdx.x * (256 * kGr) + threadIdx.x;
#pragma unroll
  for (int k = 0; k < kGr; ++k) {
    const int i = i0 + 256 * k;
    const bool in = i < n;
    zi[k] = in ? z[i] : 0.0; wi[k] = in ? w[i] : 0.0; ri[k] = in ? rin[i] : 0.0; si[k] = in ? rs[i] : 0.0;
    xi[k] = in && xin ? xin[i] : 0.0;
  }
#pragma unroll
  for (int k = 0; k < kGr; ++k) {
    const int i = i0 + 256 * k;
    v[0][k] = v[1][k] = 0.0;
    if (i < n) {
      x[i] = __dadd_rn(xi[k], __dmul_rn(a, zi[k]));
      const double t = __dsub_rn(ri[k], __dmul_rn(a, wi[k]));
      r[i] = t;
      v[0][k] = __dmul_rn(t, t);
      v[1][k] = __dmul_rn(t, si[k]);
    }
  }
  group_sums<2>(v, ng, part);
  if (FUSE) fin_block(fin, gridDim.x);
}

// partials of (a, b)
template <bool FUSE>
__global__ void __launch_bounds__(256) k_dot(int n, int ng, const double *a, const double *b, double *part, Fin fin) {
  double v[1][kGr];
  const int i0 = blockIdx.x * (256 * kGr) + threadIdx.x;
#pragma unroll
  for (int k = 0; k < kGr; ++k) {
    const int i = i0 + 256 * k;
    v[0][k] = i < n ? __dmul_rn(a[i], b[i]) : 0.0;
  }
  group_sums<1>(v, ng, part);
  if (FUSE) fin_block(fin, gridDim.x);
}

// partials of (v, v), (x, v) and |v|_1
template <bool FUSE>
__global__ void __launch_bounds__(256) k_eps_sums(int n, int ng, const double *x, const double *y, double *part, Fin fin) {
  double v[3][kGr];
  const int i0 = blockIdx.x * (256 * kGr) + threadIdx.x;
#pragma unroll
  for (int k = 0; k < kGr; ++k) {
    const int i = i0 + 256 * k;
    const double yi = i < n ? y[i] : 0.0, xi = i < n ? x[i] : 0.0;
    v[0][k] = __dmul_rn(yi, yi);
    v[1][k] = __dmul_rn(xi, yi);
    v[2][k] = fabs(yi);
  }
  group_sums<3>(v, ng, part);
  if (FUSE) fin_block(fin, gridDim.x);
}

__global__ void k_scale(int n, double *y, double a) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) y[i] = __dmul_rn(y[i], a);
}

// check_abserrmax (Check_simulation.f90:37-91): last index wins ties.
struct ArgMax {
  double a, v;   // |value|, signed value
  int idx;
};
__device__ __forceinline__ ArgMax amax(ArgMax p, ArgMax q) {
  if (q.a > p.a || (q.a == p.a && q.idx > p.idx)) return q;
  return p;
}

// dh non-null: first forms xn = xp + 1*dh (the Newton update, the axpby it replaces, same
// rounding) and writes it, so xn is not read back.  The last block to finish reduces the
// blocks' results to res[0 .. 6]: |change|, change, cell, |value|, value, cell, any NaN.
__global__ void __launch_bounds__(256) k_abserrmax(int n, double *xn, const double *xp, const double *dh,
                                                   double *part, double *res, int *cnt, Publish pub) {
  __shared__ ArgMax s1[256], s2[256];
  __shared__ int snan[256];
  ArgMax c = {0.0, 0.0, -1}, x = {0.0, 0.0, -1};
  int nan = 0;
  const int st = gridDim.x * blockDim.x;
  for (int i0 = blockIdx.x * blockDim.x + threadIdx.x; i0 < n; i0 += 4 * st) {
    double p[4], v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = i0 + u * st;
      p[u] = i < n ? xp[i] : 0.0;
      v[u] = i < n ? (dh ? dh[i] : xn[i]) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = i0 + u * st;
      if (i < n) {
        double t = v[u];
        if (dh) {
          t = __dadd_rn(p[u], __dmul_rn(1.0, t));
          xn[i] = t;
        }
        if (t != t) nan = 1;
        const double dv = __dsub_rn(t, p[u]);
        c = amax(c, ArgMax{fabs(dv), dv, i});
        x = amax(x, ArgMax{fabs(t), t, i});
      }
    }
  }
  auto reduce = [&]() {
    s1[threadIdx.x] = c; s2[threadIdx.x] = x; snan[threadIdx.x] = nan;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
      if ((int)threadIdx.x < o) {
        s1[threadIdx.x] = amax(s1[threadIdx.x], s1[threadIdx.x + o]);
        s2[threadIdx.x] = amax(s2[threadIdx.x], s2[threadIdx.x + o]);
        snan[threadIdx.x] |= snan[threadIdx.x + o];
      }
      __syncthreads();
    }
  };
  auto put = [&](double *q) {
    q[0] = s1[0].a; q[1] = s1[0].v; q[2] = (double)s1[0].idx;
    q[3] = s2[0].a; q[4] = s2[0].v; q[5] = (double)s2[0].idx;
    q[6] = (double)snan[0];
  };
  reduce();
  if (threadIdx.x == 0) put(part + (size_t)blockIdx.x * 8);
  if (!last_block(cnt, gridDim.x)) return;
  c = x = ArgMax{0.0, 0.0, -1};
  nan = 0;
  for (int b = threadIdx.x; b < (int)gridDim.x; b += 256) {
    const double *q = part + (size_t)b * 8;
    const ArgMax cb = {__ldcg(q), __ldcg(q + 1), (int)__ldcg(q + 2)}, xb = {__ldcg(q + 3), __ldcg(q + 4), (int)__ldcg(q + 5)};
    if (cb.idx >= 0) c = amax(c, cb);
    if (xb.idx >= 0) x = amax(x, xb);
    nan |= (int)__ldcg(q + 6);
  }
  reduce();
  if (threadIdx.x == 0) {
    put(res);
    pub();
  }
}

// lam_length of run_backtr (Nonlinear_solution.f90:503-512): max(1, max_i |dh_i| / |h_i|) over
// h_i != 0.  Rounding is monotone, so the largest rounded quotient is the rounding of the
// largest exact one: each thread keeps the (numerator, denominator) pair of its largest
// exact ratio, comparing a/b with c/d through a*d against c*b exactly (the rounded product
// and its FMA error term), and divides once at the end -- the same value as dividing every
// element, without an FP64 division per cell.
__device__ __forceinline__ bool ratio_greater(double a, double b, double c, double d) {
  const double p1 = a * d, p2 = c * b;
  if (p1 != p2) return p1 > p2;
  return fma(a, d, -p1) > fma(c, b, -p2);
}
__global__ void __launch_bounds__(256) k_lamlen(int n, const double *dh, const double *hn, double *part) {
  __shared__ double s[256];
  double num = 1.0, den = 1.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double h = fabs(hn[i]), a = fabs(dh[i]);
    if (h != 0.0 && ratio_greater(a, h, num, den)) { num = a; den = h; }
  }
  const double m = __ddiv_rn(num, den);
  s[threadIdx.x] = m;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) s[threadIdx.x] = fmax(s[threadIdx.x], s[threadIdx.x + o]);
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = s[0];
}

static int fetch_partials(msg_ctx *c, int count) {
  MSG_CUDA(cudaMemcpyAsync(c->hpin, c->part, (size_t)count * 8, cudaMemcpyDeviceToHost, c->stream));
  MSG_CUDA(cudaStreamSynchronize(c->stream));
  return wave_check(c);
}

// Second reduction stage: array a is part[a*nparts .. a*nparts + nparts), summed in a fixed
// order, so every result repeats bit for bit: thread t keeps eight running sums over the
// elements t + 1024 u + 8192 k, u = 0 .. 7, combines them in a fixed tree, then the block
// reduces in a fixed tree.  Long arrays give each u a block of its own (split = 8) and the
// last block to finish combines them, the same sums: one block needed 42 us for 98 304
// partials, of which it had too few loads in flight.  When count > 0 the block that finishes
// the last array hands results to the host.
// MAXB: bit a set -> array a takes the maximum instead of the sum.
constexpr int kFinSplit = 8;
template <int MAXB>
__global__ void __launch_bounds__(1024) k_finish(const double *part, int nparts, int narr, int split, double *out,
                                                 double *scratch, int *cnt, Publish pub) {
  __shared__ double sh[1024];
  const int arr = blockIdx.x / split, t = threadIdx.x;
  const double *p = part + (size_t)arr * nparts;
  const bool mx = (MAXB >> arr) & 1;
  auto comb = [&](double x, double y) { return mx ? fmax(x, y) : __dadd_rn(x, y); };
  constexpr int U = 8;
  double a[U];
#pragma unroll
  for (int u = 0; u < U; ++u) a[u] = 0.0;
  if (split == 1) {
    for (int base = t; base < nparts; base += U * 1024) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = base + u * 1024;
        if (i < nparts) a[u] = comb(a[u], p[i]);
      }
    }
  } else {
    const int u = blockIdx.x % split;
    double s = 0.0;
    for (int base = t + u * 1024; base < nparts; base += 8 * U * 1024) {
      double x[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) x[k] = base + k * U * 1024 < nparts ? p[base + k * U * 1024] : 0.0;
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (base + k * U * 1024 < nparts) s = comb(s, x[k]);
    }
    scratch[(arr * U + u) * 1024 + t] = s;
    if (!last_block(cnt + arr, split)) return;
#pragma unroll
    for (int k = 0; k < U; ++k) a[k] = __ldcg(scratch + (arr * U + k) * 1024 + t);
  }
  sh[t] = comb(comb(comb(a[0], a[1]), comb(a[2], a[3])), comb(comb(a[4], a[5]), comb(a[6], a[7])));
  __syncthreads();
  for (int o = 512; o > 0; o >>= 1) {
    if (t < o) sh[t] = comb(sh[t], sh[t + o]);
    __syncthreads();
  }
  if (t == 0) {
    out[arr] = sh[0];
    if (pub.word) {
      __threadfence();
      const bool last = narr == 1 || atomicAdd(cnt + kFinArr, 1) == narr - 1;
      if (last) {
        if (narr > 1) cnt[kFinArr] = 0;
        pub();
      }
    }
  }
}

// The reduction results come to the host with the kernel that finishes the last of them:
// publish(c, count) in its launch, then fetch_res.
static Publish publish(msg_ctx *c, int count) {
  if (!count) return Publish{nullptr, nullptr, 0, nullptr, 0};
  return Publish{c->dres, c->hpin, count, c->res_word, ++c->res_token};
}

template <int MAXB = 0>
static int launch_finish(msg_ctx *c, int nparts, int narr, int slot, int count, int first = 0) {
  const int split = nparts > kFinSplit * 1024 ? kFinSplit : 1;
  k_finish<MAXB><<<narr * split, 1024, 0, c->stream>>>(c->part + (size_t)first * nparts, nparts, narr, split, c->dres + slot, c->fin_scratch,
                                                       c->fin_cnt, publish(c, count));
  MSG_CHECK_LAUNCH();
  return MSG_OK;
}

// Second stage of narr arrays into dres[slot ..]: by the writing kernel's last block, or, for
// long arrays, a launch after it.  Results of several stages come back with one fetch_res,
// of which the last names the count.
Fin make_fin(msg_ctx *c, int nparts, int narr, int slot, int count) {
  const bool fuse = nparts <= kFuseParts;
  return Fin{fuse, c->part, nparts, narr, c->dres + slot, c->fin_cnt + kFinArr + 2, publish(c, fuse ? count : 0)};
}
template <int MAXB>
int end_fin(msg_ctx *c, const Fin &f, int count) {
  if (f.fuse) return MSG_OK;
  return launch_finish<MAXB>(c, f.nparts, f.narr, (int)(f.out - c->dres), count);
}
template int end_fin<0>(msg_ctx *, const Fin &, int);

int fetch_res(msg_ctx *c, int count, double *out) {
  int rc = token_wait(c, c->res_word, c->res_token);
  if (rc) return rc;
  for (int a = 0; a < count; ++a) out[a] = c->hpin[a];
  return wave_check(c);
}

int finish(msg_ctx *c, int nparts, int narr, double *out) {
  int rc = launch_finish(c, nparts, narr, 0, narr);
  if (rc) return rc;
  return fetch_res(c, narr, out);
}

int finish9(msg_ctx *c, int nparts, double out[9]) {
  int rc;
  if ((rc = launch_finish(c, nparts, 4, 0, 0)) || (rc = launch_finish(c, nparts, 4, 4, 0, 4)) ||
      (rc = launch_finish(c, nparts, 1, 8, 9, 8)))
    return rc;
  return fetch_res(c, 9, out);
}

static int launch_dot(msg_ctx *c, const double *a, const double *b, int n, int slot, int count) {
  const Fin f = make_fin(c, ngroups(n), 1, slot, count);
  (f.fuse ? k_dot<true> : k_dot<false>)<<<gblk(n), 256, 0, c->stream>>>(n, ngroups(n), a, b, c->part, f);
  MSG_CHECK_LAUNCH();
  return end_fin(c, f, count);
}

int dot(msg_ctx *c, const double *a, const double *b, int n, double *out) {
  int rc = launch_dot(c, a, b, n, 0, 1);
  if (rc) return rc;
  return fetch_res(c, 1, out);
}

int launch_eps_sums(msg_ctx *c, const double *x, const double *v) {
  const int n = c->N;
  const Fin f = make_fin(c, ngroups(n), 3, kResEps, 0);
  (f.fuse ? k_eps_sums<true> : k_eps_sums<false>)<<<gblk(n), 256, 0, c->stream>>>(n, ngroups(n), x, v, c->part, f);
  MSG_CHECK_LAUNCH();
  return end_fin(c, f, 0);
}

constexpr int kResErr = 5;   // abserrmax's seven results in dres (behind the line search's five)
static int launch_abserrmax(msg_ctx *c, double *xn, const double *xp, const double *dh) {
  const int g = std::min(kRedBlocks, gblk(c->N));   // a maximum: the same whatever the grid
  k_abserrmax<<<g, 256, 0, c->stream>>>(c->N, xn, xp, dh, c->part, c->dres + kResErr, c->fin_cnt + kFinArr + 1,
                                                 publish(c, kResErr + 7));
  MSG_CHECK_LAUNCH();
  return MSG_OK;
}
static void errmax_result(const double *q, ErrMax &e) {
  e.nan = (int)q[6];
  if (!e.nan) { e.change = q[1]; e.value = q[4]; e.cell = (int)q[2] + 1; }
  else { e.change = 0.0; e.value = NAN; e.cell = 0; }
}

int abserrmax(msg_ctx *c, double *xn, const double *xp, ErrMax &e, const double *dh) {
  int rc = launch_abserrmax(c, xn, xp, dh);
  double got[kResErr + 7];
  if (rc || (rc = fetch_res(c, kResErr + 7, got))) return rc;
  errmax_result(got + kResErr, e);
  return MSG_OK;
}

// The line search's four reductions over the full step in one pass (run_backtr,
// Nonlinear_solution.f90:441-512): ||dh||^2, ||F(h + dh)||^2, the slope (s, J dh) and
// lam_length's largest ratio |dh| / |h|.  The sums use the groups and order of k_dot, so each
// has the bits of its own dot product; J dh is jv, or b - r (BiCGStab's residual from dh = 0)
// formed with the rounding of the axpby it replaces.  The maximum is exact whatever the
// grouping: one per block, in the place of its first group.
template <bool FUSE>
__global__ void __launch_bounds__(256) k_backtr_stats(int n, int ng, const double *dh, const double *hn, const double *f,
                                                      const double *s, const double *jv, const double *b,
                                                      const double *r, double *part, Fin fin) {
  __shared__ double sm[8];
  double v[3][kGr], num = 1.0, den = 1.0;
  double di[kGr], hi[kGr], fi[kGr], si[kGr], ji[kGr], bi[kGr];
  const int i0 = blockIdx.x * (256 * kGr) + threadIdx.x;
#pragma unroll
  for (int k = 0; k < kGr; ++k) {
    const int i = i0 + 256 * k;
    const bool in = i < n;
    di[k] = in ? dh[i] : 0.0; hi[k] = in ? hn[i] : 0.0; fi[k] = in ? f[i] : 0.0; si[k] = in ? s[i] : 0.0;
    ji[k] = in ? (jv ? jv[i] : r[i]) : 0.0;
    bi[k] = !in || jv ? 0.0 : b == s ? si[k] : b[i];
  }
#pragma unroll
  for (int k = 0; k < kGr; ++k) {
    v[0][k] = v[1][k] = v[2][k] = 0.0;
    if (i0 + 256 * k < n) {
      v[0][k] = __dmul_rn(di[k], di[k]);
      v[1][k] = __dmul_rn(fi[k], fi[k]);
      const double j = jv ? ji[k] : __dadd_rn(bi[k], __dmul_rn(-1.0, ji[k]));
      v[2][k] = __dmul_rn(si[k], j);
      const double h = fabs(hi[k]), a = fabs(di[k]);
      if (h != 0.0 && ratio_greater(a, h, num, den)) { num = a; den = h; }
    }
  }
  double m = __ddiv_rn(num, den);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = m;
  group_sums<3>(v, ng, part);   // its barrier covers sm
  if (threadIdx.x < kGr) {
    const int g = blockIdx.x * kGr + threadIdx.x;
    m = 0.0;
    if (threadIdx.x == 0)
      for (int w = 0; w < 8; ++w) m = fmax(m, sm[w]);
    if (g < ng) part[(size_t)3 * ng + g] = m;
  }
  if (FUSE) fin_block<8>(fin, gridDim.x);
}

int backtr_stats(msg_ctx *c, const double *dh, const double *hn, const double *f, const double *s, const double *jv,
                 const double *b, const double *r, double out[5], bool slot4) {
  const int ng = ngroups(c->N);
  if ((size_t)4 * ng > c->npart) { set_error("backtr_stats: partials buffer too small"); return MSG_ERR_STATE; }
  const Fin fin = make_fin(c, ng, 4, 0, slot4 ? 5 : 4);
  (fin.fuse ? k_backtr_stats<true> : k_backtr_stats<false>)<<<gblk(c->N), 256, 0, c->stream>>>(c->N, ng, dh, hn, f, s, jv, b, r, c->part, fin);
  MSG_CHECK_LAUNCH();
  int rc = end_fin<8>(c, fin, slot4 ? 5 : 4);
  if (rc || (rc = fetch_res(c, slot4 ? 5 : 4, out))) return rc;
  out[3] = std::fmax(1.0, out[3]);
  return MSG_OK;
}

int lam_length(msg_ctx *c, const double *dh, const double *hn, double *out) {
  k_lamlen<<<kRedBlocks, 256, 0, c->stream>>>(c->N, dh, hn, c->part);
  MSG_CHECK_LAUNCH();
  int rc = fetch_partials(c, kRedBlocks);
  if (rc) return rc;
  double m = 1.0;
  for (int b = 0; b < kRedBlocks; ++b) m = std::fmax(m, c->hpin[b]);
  *out = m;
  return MSG_OK;
}

int scale(msg_ctx *c, double *y, double a, int n) {
  k_scale<<<nblk(n), 256, 0, c->stream>>>(n, y, a);
  MSG_CHECK_LAUNCH();
  return MSG_OK;
}

// ---------------------------------------------------------------------------------
// DILU / ILU(0) (precon_dilu / solve_ilu, Linear_solution.f90:742-782, :803-855).  In
// natural order on the 7-point stencil cell (ix,iy,iz) depends on (ix-1,..), (..,iy-1,..)
// and (..,iz-1) only, so cells in any order that respects this perform exactly the
// sequential arithmetic.
//
// What bounds it is the chain of nx+ny+nz-2 dependent cells, so everything but that chain is
// kept off the threads that walk it.  A block owns a kWX x kWY tile of columns, a thread one
// column; at step s it takes its layer z = s - lx - ly.  The upper neighbour is the thread's
// own last value (a register), the west and north ones come through shared memory, one
// block barrier per step.  As many warps again copy the coefficients ahead (cp.async, eight
// neighbouring cells of a row side by side) into a ring of layers, and one warp brings in
// the columns of the tiles to the west and north.  Those cross through a slot per
// value in global memory: an empty slot holds a signalling NaN, which no arithmetic result
// is, so the value is its own flag and needs no fence; the reader empties it again for the
// next sweep.  Blocks take their tiles from a counter in an order in which a tile follows
// the two that it waits for, so they progress however many of them are resident (the last
// block sets the counter back, so nothing on the host has to follow it).  A wait is given up
// after kWLooks looks at its slot (about 1.5 s; looks, not time, so that a GPU that other
// processes share, or a debugger stops, does not end it) and reported: the sweep ends with wrong
// values, the call with an error, and the slots are emptied for the next one.
//
// 96 x 81 x 40 cells: factor 1390 -> 134 us, solve 2000 -> 214 us against a grid-wide barrier
// per plane of cells (4.6 to 6.5 us each); 20 x 20 x 50: 165 -> 40 and 195 -> 76 us against
// one block for the grid, whose scattered loads took 1.1 to 1.9 us per plane.  A step is now
// about 250 ns (the division 66 of them), a hop from tile to tile about 1 us; looking at a
// slot more than one step ahead (kWAhead) only lengthens the lag between tiles (267 us per
// solve at 4, 230 at 2, 214 at 1).
// ---------------------------------------------------------------------------------
constexpr int kWX = 16, kWY = 8, kWCols = kWX * kWY, kWThreads = 2 * kWCols + 32;
// a layer is fetched kWFetch steps ahead of the first column of its 8 x 4 group and used up
// to 7 + 3 steps after it
constexpr int kWRing = 16, kWFetch = 6, kWAhead = 1, kWPitch = 24;
constexpr unsigned long long kWEmpty = 0x7ff4a5a5a5a5a5a5ull;   // a signalling NaN
constexpr unsigned kWLooks = 1u << 22;

struct SweepArgs {
  Geo3 g;
  int tx;                        // tiles in x
  const int *order;              // tile (x + tx * y) of each ticket
  unsigned *ticket;              // 0 between sweeps
  unsigned long long *west, *north;   // slots: west[(tile * nz + z) * kWY + ly], north[.. * kWX + lx]
  int *err, *err_host;           // a wait was given up: device word, pinned word
  unsigned looks;                // of a wait
  int withhold;                  // test hook: the tile that hands nothing over (-1: none)
  const double *dmat, *lu;
  double *dd;                    // DILU diagonal (out for factor, in for solve)
  const double *b;
  double *x;
};

__device__ __forceinline__ unsigned long long ld_slot(const unsigned long long *p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_slot(unsigned long long *p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
// The value of a slot, waited for if it is still empty (v: what an earlier look found); the
// slot is left empty.
__device__ __forceinline__ double take_slot(const SweepArgs &a, unsigned long long *p, unsigned long long v, bool &dead) {
  if (v == kWEmpty && !dead) {
    for (unsigned it = 1; (v = ld_slot(p)) == kWEmpty; ++it) {
      if ((it & 1023) == 0 && (it >= a.looks || *(volatile int *)a.err)) {
        *(volatile int *)a.err = 1;
        *(volatile int *)a.err_host = 1;
        dead = true;
        break;
      }
    }
  }
  st_slot(p, kWEmpty);
  return __longlong_as_double((long long)v);
}
__device__ __forceinline__ void cp8(double *smem, const double *g) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(a), "l"(g) : "memory");
}

// values per cell in the ring, and its bytes
template <int MODE>
struct Sweep {
  static constexpr int NV = MODE == 0 ? 7 : 5;
  static constexpr int smem = kWRing * NV * kWCols * 8;
};

// MODE 0: factor (dd; the values exchanged are 1/dd); MODE 1: forward solve (x from b);
// MODE 2: backward solve (x in place), the same sweep with all three axes mirrored.
template <int MODE>
__global__ void __launch_bounds__(kWThreads) k_sweep(SweepArgs a) {
  constexpr int NV = Sweep<MODE>::NV;
  extern __shared__ double ring_mem[];
  double(*ring)[NV][kWCols] = reinterpret_cast<double(*)[NV][kWCols]>(ring_mem);
  __shared__ double ex[2][kWY + 1][kWPitch];     // step parity; row and column 0: the tiles before
  __shared__ int s_tile;
  const int t = threadIdx.x, wp = t >> 5, ln = t & 31;
  if (t == 0) s_tile = a.order[atomicInc(a.ticket, gridDim.x - 1)];   // back at 0 with the last block
  __syncthreads();
  const int tile = s_tile, bx = tile % a.tx, by = tile / a.tx;
  const int nx = a.g.nx, ny = a.g.ny, nz = a.g.nz, nxy = a.g.nxy;
  const size_t N = a.g.N;
  const int dz = MODE == 2 ? -nxy : nxy;
  // first cell of the column (gx, gy), in mirrored coordinates in MODE 2
  auto first = [&](int gx, int gy) {
    return MODE == 2 ? (nx - 1 - gx) + nx * (ny - 1 - gy) + (nz - 1) * nxy : gx + nx * gy;
  };
  const int steps = min(kWX, nx - bx * kWX) + min(kWY, ny - by * kWY) + nz - 2;
  if (wp < kWCols / 32) {
    // ---- the chain: a warp owns 8 x 4 columns
    const int lx = 8 * (wp % (kWX / 8)) + (ln & 7), ly = 4 * (wp / (kWX / 8)) + (ln >> 3);
    const int gx = bx * kWX + lx, gy = by * kWY + ly;
    const bool col = gx < nx && gy < ny, hx = gx > 0, hy = gy > 0, give = col && tile != a.withhold;
    const int layers = col ? nz : 0;
    unsigned long long *wout = lx == kWX - 1 && gx + 1 < nx && give ? a.west + ((size_t)(tile + 1) * nz) * kWY + ly : nullptr;
    unsigned long long *nout = ly == kWY - 1 && gy + 1 < ny && give ? a.north + ((size_t)(tile + a.tx) * nz) * kWX + lx : nullptr;
    const bool edge = wout || nout;
    size_t i = col ? first(gx, gy) : 0;
    int z = -lx - ly;
    double up = 0.0, q[NV];
    auto load = [&]() {
      const double *p = &ring[z & (kWRing - 1)][0][t];
#pragma unroll
      for (int k = 0; k < NV; ++k) q[k] = p[k * kWCols];
    };
    auto step = [&](const double(*in)[kWPitch], double(*out)[kWPitch]) {
      const double xw = in[ly + 1][lx], xn = in[ly][lx + 1];
      const bool on = (unsigned)z < (unsigned)layers, hz = z > 0;
      double v;
      if (MODE == 0) {
        double d = q[0];
        if (hz) d = __dsub_rn(d, __dmul_rn(__dmul_rn(q[1], up), q[4]));
        if (hy) d = __dsub_rn(d, __dmul_rn(__dmul_rn(q[2], xn), q[5]));
        if (hx) d = __dsub_rn(d, __dmul_rn(__dmul_rn(q[3], xw), q[6]));
        v = __drcp_rn(d);
        if (on) a.dd[i] = d;
      } else if (MODE == 1) {
        double r = q[0];
        if (hz) r = __dsub_rn(r, __dmul_rn(q[2], up));
        if (hy) r = __dsub_rn(r, __dmul_rn(q[3], xn));
        if (hx) r = __dsub_rn(r, __dmul_rn(q[4], xw));
        v = __ddiv_rn(r, q[1]);
        if (on) a.x[i] = v;
      } else {
        double r = 0.0;
        if (hx) r = __dadd_rn(r, __dmul_rn(q[4], xw));
        if (hy) r = __dadd_rn(r, __dmul_rn(q[3], xn));
        if (hz) r = __dadd_rn(r, __dmul_rn(q[2], up));
        v = __dsub_rn(q[0], __ddiv_rn(r, q[1]));
        if (on) a.x[i] = v;
      }
      out[ly + 1][lx + 1] = v;
      if (on) {
        up = v;
        i += dz;
        if (edge) {
          if (wout) st_slot(wout + z * kWY, (unsigned long long)__double_as_longlong(v));
          if (nout) st_slot(nout + z * kWX, (unsigned long long)__double_as_longlong(v));
        }
      }
      ++z;
      load();
      __syncthreads();
    };
    __syncthreads();
    load();
    for (int s = 0; s < steps; s += 2) {
      step(ex[1], ex[0]);
      if (s + 1 < steps) step(ex[0], ex[1]);
    }
  } else if (wp == kWCols / 32) {
    // ---- the columns of the tiles before: lanes 0 .. kWY-1 west, the next kWX north
    const bool w = ln < kWY, n = !w && ln < kWY + kWX;
    const int k = w ? ln : ln - kWY, gx = bx * kWX + (w ? 0 : k), gy = by * kWY + (w ? k : 0);
    const bool has = gx < nx && gy < ny && ((w && bx > 0) || (n && by > 0));
    const int pitch = w ? kWY : kWX;
    unsigned long long *slot = (w ? a.west : a.north) + (size_t)tile * nz * pitch + (has ? k : 0);
    const int row = w ? k + 1 : 0, cl = w ? 0 : k + 1;
    unsigned long long pre[kWAhead];
    bool dead = false;
#pragma unroll
    for (int u = 0; u < kWAhead; ++u) {
      const int z = u - k;
      pre[u] = has && z >= 0 && z < nz ? ld_slot(slot + z * pitch) : kWEmpty;
    }
    // before the barrier that step s follows: its values
    for (int s0 = 0; s0 <= steps; s0 += kWAhead) {
#pragma unroll
      for (int u = 0; u < kWAhead; ++u) {
        const int s = s0 + u, z = s - k;
        if (s <= steps) {
          if (has && z >= 0 && z < nz) ex[(s + 1) & 1][row][cl] = take_slot(a, slot + z * pitch, pre[u], dead);
          const int za = z + kWAhead;
          if (has && za >= 0 && za < nz) pre[u] = ld_slot(slot + za * pitch);
          __syncthreads();
        }
      }
    }
  } else {
    // ---- coefficients: a warp copies the 8 x 4 columns of one group (bands without a
    // neighbour hold zeros; only those read at the neighbour need it to exist)
    const int tt = t - kWCols - 32, gr = tt >> 5, wx = 8 * (gr % (kWX / 8)), wy = 4 * (gr / (kWX / 8));
    const int gx = bx * kWX + wx + (ln & 7), gy = by * kWY + wy + (ln >> 3);
    const bool hx = gx > 0, hy = gy > 0;
    const int layers = gx < nx && gy < ny ? nz : 0;
    int z = -wx - wy;
    const double *p[NV];
    const long long i0 = first(gx, gy) + (long long)z * dz;
    if (MODE == 0) {
      p[0] = a.dmat + i0;
      p[1] = a.lu + i0; p[2] = a.lu + N + i0; p[3] = a.lu + 2 * N + i0;
      p[4] = a.lu + 5 * N + i0 - nxy; p[5] = a.lu + 4 * N + i0 - nx; p[6] = a.lu + 3 * N + i0 - 1;
    } else {
      p[0] = (MODE == 1 ? a.b : a.x) + i0;
      p[1] = a.dd + i0;
      p[2] = a.lu + (MODE == 1 ? 0 : 5) * N + i0;
      p[3] = a.lu + (MODE == 1 ? 1 : 4) * N + i0;
      p[4] = a.lu + (MODE == 1 ? 2 : 3) * N + i0;
    }
    auto fetch = [&]() {
      if ((unsigned)z < (unsigned)layers) {
        double *q = &ring[z & (kWRing - 1)][0][tt];
#pragma unroll
        for (int k = 0; k < NV; ++k)
          if (MODE != 0 || k < 4 || (k == 4 && z > 0) || (k == 5 && hy) || (k == 6 && hx)) cp8(q + k * kWCols, p[k]);
      }
#pragma unroll
      for (int k = 0; k < NV; ++k) p[k] += dz;
      ++z;
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // the barrier that step s follows: the layers of steps s and s + 1 have arrived
    for (int s = 0; s < kWFetch; ++s) fetch();
    for (int s = 0; s <= steps; ++s) {
      asm volatile("cp.async.wait_group %0;" ::"n"(kWFetch - 2) : "memory");
      __syncthreads();
      fetch();
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  }
}

__global__ void k_slots_empty(size_t n, unsigned long long *p) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) p[i] = kWEmpty;
}

// All slots empty, ticket counter and error words zero; no sweep may be under way.
static int wave_reset(msg_ctx *c) {
  k_slots_empty<<<kRedBlocks, 256, 0, c->stream>>>((size_t)c->wave_tiles * c->nz * (kWX + kWY), (unsigned long long *)c->wave_slots);
  MSG_CHECK_LAUNCH();
  MSG_CUDA(cudaMemsetAsync(c->wave_ticket, 0, 8, c->stream));
  MSG_CUDA(cudaStreamSynchronize(c->stream));
  *(volatile int *)c->wave_err = 0;
  return MSG_OK;
}

// Tile order, slots, ticket counter and error words of the sweeps.
int build_wavefront(msg_ctx *c) {
  const int tx = (c->nx + kWX - 1) / kWX, ty = (c->ny + kWY - 1) / kWY, nt = tx * ty;
  std::vector<int> order;
  order.reserve(nt);
  for (int d = 0; d < tx + ty - 1; ++d)
    for (int y = std::max(0, d - tx + 1); y <= std::min(d, ty - 1); ++y) order.push_back((d - y) + tx * y);
  const size_t nslot = (size_t)nt * c->nz * (kWX + kWY);
  MSG_CUDA(cudaFuncSetAttribute(k_sweep<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, Sweep<0>::smem));
  MSG_CUDA(cudaFuncSetAttribute(k_sweep<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, Sweep<1>::smem));
  MSG_CUDA(cudaFuncSetAttribute(k_sweep<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, Sweep<2>::smem));
  MSG_CUDA(cudaMalloc(&c->wave_order, (size_t)nt * 4));
  MSG_CUDA(cudaMalloc(&c->wave_ticket, 8));      // ticket, error word
  MSG_CUDA(cudaMalloc(&c->wave_slots, nslot * 8));
  c->wave_err = reinterpret_cast<int *>(c->hpin + kRedBlocks * 8 + 8);
  *c->wave_err = 0;
  c->wave_tiles = nt;
  MSG_CUDA(cudaMemcpyAsync(c->wave_order, order.data(), (size_t)nt * 4, cudaMemcpyHostToDevice, c->stream));
  return wave_reset(c);   // and waits for the copy
}

// A sweep that gave up a wait has said so in wave_err (host memory); looked at after every
// host wait on the stream and before every sweep.  The call that finds it fails; the sweeps
// still queued end at once (they see the device word), and the next call starts clean.
int wave_check(msg_ctx *c) {
  if (!c->wave_err || !*(volatile int *)c->wave_err) return MSG_OK;
  MSG_CUDA(cudaStreamSynchronize(c->stream));
  int rc = wave_reset(c);
  if (rc) return rc;
  set_error("DILU sweep: a wait between tiles ran out");
  return MSG_ERR_CUDA;
}

template <int MODE>
static int launch_sweep(msg_ctx *c, const double *b, double *x) {
  int rc = wave_check(c);
  if (rc) return rc;
  unsigned long long *slots = (unsigned long long *)c->wave_slots;
  SweepArgs a{geo3(c), (c->nx + kWX - 1) / kWX, c->wave_order, c->wave_ticket,
              slots, slots + (size_t)c->wave_tiles * c->nz * kWY,
              (int *)c->wave_ticket + 1, c->wave_err, kWLooks, -1, c->dmat, c->lu, c->dilu_d, b, x};
  if (c->hook[MSG_HOOK_SWEEP_WITHHOLD] > 0) {
    a.withhold = c->hook[MSG_HOOK_SWEEP_WITHHOLD] - 1;
    a.looks = 1u << 12;
    c->hook[MSG_HOOK_SWEEP_WITHHOLD] = 0;
  }
  const bool refuse = hook_due(c, MSG_HOOK_SWEEP_LAUNCH);   // more shared memory than a block can have
  k_sweep<MODE><<<c->wave_tiles, kWThreads, Sweep<MODE>::smem + (refuse ? 1 << 20 : 0), c->stream>>>(a);
  MSG_CHECK_LAUNCH();
  return MSG_OK;
}

int launch_precon_dilu(msg_ctx *c) { return launch_sweep<0>(c, nullptr, nullptr); }

int launch_solve_ilu(msg_ctx *c, const double *b, double *x) {
  int rc = launch_sweep<1>(c, b, x);
  if (rc) return rc;
  return launch_sweep<2>(c, nullptr, x);
}

int apply_prec(msg_ctx *c, const double *r, double *z) {
  if (c->prm.precon_type == 0) return launch_solve_ilu(c, r, z);
  if (c->prm.ref_quirks) {
    // loop_amg of the reference returns solve_ilu at level 1 (quirk Q1) and leaves its
    // input in array_var(1)%rhs, which the line-search slope then reads (quirk Q2).
    int rc = launch_solve_ilu(c, r, z);
    if (rc) return rc;
    MSG_CUDA(cudaMemcpyAsync(c->slope_rhs, r, (size_t)c->N * 8, cudaMemcpyDeviceToDevice, c->stream));
    return MSG_OK;
  }
  return amg_apply(c, r, z);
}

// ---------------------------------------------------------------------------------
// solve_bicgs (Linear_solution.f90:234-493): right-preconditioned BiCGStab, x0 = x.
//
// The step lengths are formed on the device by the kernels that use them, so the host waits
// only for the residual norms it decides on.  With `ahead`, the Newton update's change
// (abserrmax over ahead->xn = ahead->xp + x) is taken together with the first residual norm
// when the last solve ended there, which a solve with one AMG V-cycle usually does: one wait
// fewer; a wrong guess costs the pass.
// ---------------------------------------------------------------------------------
int solve_bicgs(msg_ctx *c, double *x, bool x_zero, ErrAhead *ahead) {
  const int n = c->N;
  const Geo3 g = geo3(c);
  int rc;
  const int nb = nblk(n), ng = ngroups(n), gb = gblk(n);
  double sk = 0.0, sk0 = 1.0e20, alpha = 0.0, beta, omega = 1.0;
  bool need_dilu = (c->prm.precon_type == 0) || c->prm.ref_quirks;
  // r* (fixed during the solve), the first search direction and the residual before the
  // first update.  From x = 0 all three are b itself: nothing is copied, and x is first
  // written (not read) by the first update.
  const double *rs, *p1, *r1;
  // reduction results: (v, r*), ||r||^2 after the first update, <b, b>; behind abserrmax's
  // those of the second half
  enum { kSk2 = 0, kR1 = 1, kBB = 2, kTs = kResErr + 7, kR2 = kTs + 2 };
  if (x_zero) {
    if (need_dilu && (rc = launch_precon_dilu(c))) return rc;
    // sk = <b, b>, collected with the first residual norm
    if ((rc = launch_dot(c, c->rhs, c->rhs, n, kBB, 0))) return rc;
    rs = p1 = r1 = c->rhs;
  } else {
    // r = b - A x
    k_spmv<0, true, false><<<nb, 256, 0, c->stream>>>(g, c->dmat, c->lu, x, c->rhs, c->r, nullptr, nullptr, Fin{});
    MSG_CHECK_LAUNCH();
    if (need_dilu && (rc = launch_precon_dilu(c))) return rc;
    MSG_CUDA(cudaMemcpyAsync(c->rs, c->r, (size_t)n * 8, cudaMemcpyDeviceToDevice, c->stream));
    if ((rc = dot(c, c->r, c->rs, n, &sk))) return rc;
    rs = p1 = c->rs;
    r1 = c->r;
  }
  c->conv_flag = 0;
  double got[kR2 + 2];
  for (c->in_iter = 1; c->in_iter <= c->prm.maxinn_iter; ++c->in_iter) {
    const bool first = (c->in_iter == 1);
    const double *p = c->p;
    if (first) {
      p = p1;
    } else {
      beta = (sk / sk0) * (alpha / omega);
      k_bicg_p<<<nb, 256, 0, c->stream>>>(n, c->in_iter == 2 ? p1 : c->p, c->p, c->r, c->v, beta, omega);
      MSG_CHECK_LAUNCH();
    }
    if ((rc = apply_prec(c, p, c->z))) return rc;
    Fin f = make_fin(c, nb, 1, kSk2, 0);
    (f.fuse ? k_spmv<1, false, true> : k_spmv<1, false, false>)<<<nb, 256, 0, c->stream>>>(g, c->dmat, c->lu, c->z, nullptr, c->v, rs, c->part, f);
    MSG_CHECK_LAUNCH();
    if ((rc = end_fin(c, f, 0))) return rc;
    const bool from_bb = x_zero && first;   // sk = <b, b> is still on the device
    const bool spec = ahead && from_bb && c->one_half;
    f = make_fin(c, ng, 1, kR1, spec ? 0 : 3);
    (f.fuse ? k_bicg_xr<true> : k_bicg_xr<false>)<<<gb, 256, 0, c->stream>>>(n, ng, first && x_zero ? nullptr : x, x, first ? r1 : c->r, c->r, c->z, c->v, rs,
                                        Quot{from_bb ? c->dres + kBB : nullptr, c->dres + kSk2, sk}, c->part, f);
    MSG_CHECK_LAUNCH();
    if ((rc = end_fin(c, f, spec ? 0 : 3))) return rc;
    if (spec && (rc = launch_abserrmax(c, ahead->xn, ahead->xp, x))) return rc;
    if ((rc = fetch_res(c, spec ? kResErr + 7 : 3, got))) return rc;
    if (from_bb) sk = got[kBB];
    alpha = sk / got[kSk2];
    c->rnorm = got[kR1];
    c->conv_flag = (std::sqrt(c->rnorm / c->bnorm) <= c->errtol) ? 1 : 0;
    if (first) c->one_half = c->conv_flag;
    if (spec && c->conv_flag == 1) {
      ahead->done = true;
      errmax_result(got + kResErr, ahead->e);
    }
    if (c->conv_flag == 1) break;
    if ((rc = apply_prec(c, c->r, c->z))) return rc;
    f = make_fin(c, nb, 2, kTs, 0);
    (f.fuse ? k_spmv<2, false, true> : k_spmv<2, false, false>)<<<nb, 256, 0, c->stream>>>(g, c->dmat, c->lu, c->z, nullptr, c->t, c->r, c->part, f);
    MSG_CHECK_LAUNCH();
    if ((rc = end_fin(c, f, 0))) return rc;
    f = make_fin(c, ng, 2, kR2, kR2 + 2);
    (f.fuse ? k_bicg_xr<true> : k_bicg_xr<false>)<<<gb, 256, 0, c->stream>>>(n, ng, x, x, c->r, c->r, c->z, c->t, rs, Quot{c->dres + kTs, c->dres + kTs + 1, 0.0},
                                        c->part, f);
    MSG_CHECK_LAUNCH();
    if ((rc = end_fin(c, f, kR2 + 2)) || (rc = fetch_res(c, kR2 + 2, got))) return rc;
    omega = got[kTs] / got[kTs + 1];
    c->rnorm = got[kR2];
    c->conv_flag = (std::sqrt(c->rnorm / c->bnorm) <= c->errtol) ? 1 : 0;
    if (c->conv_flag == 1 || c->in_iter == c->prm.maxinn_iter) break;
    sk0 = sk;
    sk = got[kR2 + 1];
  }
  if (c->in_iter > c->prm.maxinn_iter) c->in_iter = c->prm.maxinn_iter;
  return MSG_OK;
}

}  // namespace msg
