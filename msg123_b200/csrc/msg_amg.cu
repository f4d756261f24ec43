// msg_amg.cu -- smoothed-aggregation AMG on the GPU: setup (strength filter, MIS-2
// aggregation, smoothed prolongation, transpose, Galerkin product) and the Jacobi
// V-cycle with a dense FP64 inverse at the coarsest level.
//
// Reference counterparts: make_amgmat / make_grapfilt / make_prolomat /
// trans_prolo2restr / make_galerkin (Make_amg_matrix.f90:20-631) and loop_amg
// (Linear_solution.f90:495-740).  The reference aggregation is a serial max-heap
// (Make_amg_matrix.f90:113-222, :633-768); here it is a deterministic distance-2
// maximal independent set computed in synchronous rounds, so the aggregates do not
// depend on thread scheduling.  Every summation order is fixed (see the Galerkin
// kernel), which makes the whole hierarchy bit-identical to the CPU oracle's.
//
// Level 1 is the context's structured Jacobian, read as bands by the V-cycle and the
// setup (its CSR image is made for the export only); levels >= 2 are CSR with the diagonal held apart, as in the
// reference's array_var(level)%{dmat,lumat}.
#include "msg_ctx.cuh"
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <vector>
#include <algorithm>
#include <climits>
#include <type_traits>

namespace cg = cooperative_groups;

namespace msg {

struct AmgLevel {
  int n = 0, nnz = 0;           // rows, off-diagonal entries
  int *rowptr = nullptr, *col = nullptr;
  double *diag = nullptr, *val = nullptr;
  // transfer to/from the next finer level (held by this, the coarser, level)
  int pnnz = 0;
  int *pptr = nullptr, *pcol = nullptr;   // P: fine rows
  double *pval = nullptr;
  int *rptr = nullptr, *rcol = nullptr;   // R = P^T: coarse rows, fine index ascending
  double *rval = nullptr;
  int *agg = nullptr;                     // aggregate of each fine row (-1: none)
  double *cinv = nullptr;                 // dense inverse (coarsest level only)
  double *x = nullptr, *b = nullptr, *r = nullptr, *x2 = nullptr;
  // mixed precision images
  float *diag_f = nullptr, *pval_f = nullptr, *rval_f = nullptr;
  __nv_bfloat16 *val_h = nullptr;
  float *xf = nullptr, *bf = nullptr, *rf = nullptr, *x2f = nullptr;
  void *pack = nullptr;                   // rows of this and the following levels for k_cycle_tail_f
};

// The mixed cycle's small levels (k_cycle_tail_f): what one launch works on, laid out by a build.
constexpr int kTailBlocks = 8, kTailMax = 16;
constexpr int kTailSlices = 192;          // of a block, over all levels
struct TailMatF {                         // byte offsets of a block's rows in shared memory; cap: room for entries
  int rp, cl, v, cap;
};
struct TailLevelF {
  int n, per;                             // per: rows of a block, a multiple of 4
  int v[2], b, d;                         // two whole iterates; the block's right-hand side and diagonal
  TailMatF R, P;
  const int *rowptr, *col;                // null at a dense last level
  const __nv_bfloat16 *val;
  const float *diag;
  const int *rptr, *rcol, *pptr, *pcol;   // R: to this level from the one before; P: to this level from the one after
  const float *rval, *pval;
};
struct TailHead {                         // of a block: its slices' first words (-1: no room) and widths, over all levels
  int words, sl0[kTailMax], off[kTailSlices], wid[kTailSlices];
  int base[2 * kTailMax], in[2 * kTailMax];   // R, P: first entry copied (a multiple of 8); whether the rows fit
};
struct TailArgsF {
  int nl, sweeps, pool, words;            // slices: offset in shared memory, room (words of a block)
  float w;
  TailHead *head;                         // by block, as are the slices behind them
  uint32_t *slices;
  const double *cinv;                     // dense inverse of the last level, or null
  const float *b;                         // of the first level, as is x
  float *x;
  int shared;                             // bytes in all
  TailLevelF lv[kTailMax];
};

struct AmgState {
  std::vector<AmgLevel> lv;
  int *col0 = nullptr;           // level-1 CSR columns, 0-based (export)
  int mis_dia = 0, mis_csr = 0;  // largest grids of the cooperative MIS-2 kernels
  double *r0 = nullptr, *t0 = nullptr;   // level-1 V-cycle work vectors
  float *x0f = nullptr, *t0f = nullptr, *r0f = nullptr;   // level-1 FP32 work vectors (precision = 1)
  float *b0f = nullptr;                                   // FP32 rounding of the cycle's right-hand side
  // Device arena for everything one hierarchy build allocates: the levels grow from the
  // bottom, reset at each rebuild; what only the building of one level needs (strength
  // flags, MIS-2 words, products) grows from the top, reset after the level.  Rebuilds never
  // go to the allocator; a build that outgrows the arena takes the rest from the
  // stream-ordered pool and the arena is enlarged before the next build.
  char *arena = nullptr;
  size_t arena_cap = 0, arena_used = 0, arena_tmp = 0, arena_spill = 0;
  bool tail_set = false;                  // shared-memory limit of k_cycle_tail_f raised
  int tail_level = -1;                    // its first level, -1 none
  TailArgsF tail;
};

static AmgState *S(msg_ctx *c) { return reinterpret_cast<AmgState *>(c->amg); }
static int nb(int n) { return (n + kThreads - 1) / kThreads; }

// ---------------------------------------------------------------------------------
// Hierarchy build.  Level 1 is read in its DIA form: six bands, and the strong ones of a
// cell as six bits of a byte, so a pass of the aggregation reads bytes of the stencil
// neighbours instead of row bounds, columns, flags and 8-byte tuples.  The coarser levels
// are CSR; `scol` is their column array with -1 at the weak entries.  They are small, so
// their passes are laid out for latency: eight lanes per row where a row is reduced, a warp
// per row where its entries are matched with each other.
// ---------------------------------------------------------------------------------
struct Bands {   // level 1
  int nx, ny, nz, nxy, N;
  const double *d, *lu;
  int y0 = 0, z0 = 0;   // first row and layer of a launch over tiles (level1_tiles)
};
__device__ __forceinline__ int band_off(const Bands &g, int d) {
  return d == 0 ? -g.nxy : d == 1 ? -g.nx : d == 2 ? -1 : d == 3 ? 1 : d == 4 ? g.nx : g.nxy;
}

// ---------------------------------------------------------------------------------
// Strength filter (make_grapfilt, Make_amg_matrix.f90:67-111):
//   strong(i,k) <=> lu_k^2 > |d_i d_j theta^2| and d_i d_j lu_k > 0
//   tdm_i = d_i + sum of the weak lu_k in CSR order
// ---------------------------------------------------------------------------------
__device__ __forceinline__ bool strong_entry(double di, double dj, double lu, double th2) {
  const double ddmat = __dmul_rn(di, dj);
  return __dmul_rn(lu, lu) > fabs(__dmul_rn(ddmat, th2)) && __dmul_rn(ddmat, lu) > 0.0;
}
// 3D grid of 32 x 8 tiles: mask byte and starting state of each cell.
__global__ void k_strength_dia(Bands g, double th2, unsigned char *msk, unsigned char *st) {
  const int ix = blockIdx.x * 32 + threadIdx.x, iy = g.y0 + blockIdx.y * 8 + threadIdx.y, iz = g.z0 + blockIdx.z;
  if (ix >= g.nx || iy >= g.ny) return;
  const size_t N = g.N;
  const int i = ix + g.nx * (iy + g.ny * iz);
  const bool has[6] = {iz > 0, iy > 0, ix > 0, ix < g.nx - 1, iy < g.ny - 1, iz < g.nz - 1};
  const double di = g.d[i];
  unsigned m = 0;
#pragma unroll
  for (int d = 0; d < 6; ++d)
    if (has[d] && strong_entry(di, g.d[i + band_off(g, d)], g.lu[d * N + i], th2)) m |= 1u << d;
  msk[i] = (unsigned char)m;
  st[i] = m ? 1 : 0;
}
// A warp per row.
__global__ void __launch_bounds__(128) k_strength_csr(int n, const int *__restrict__ rowptr, const int *__restrict__ col,
                                                      const double *__restrict__ val, const double *__restrict__ diag,
                                                      double th2, int *scol, unsigned char *st, double *tdm) {
  const int i = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (i >= n) return;
  const int b = rowptr[i], e = rowptr[i + 1];
  const double di = diag[i];
  double t = di;
  bool any = false;
  for (int k0 = b; k0 < e; k0 += 32) {
    const int k = k0 + lane;
    double lu = 0.0;
    bool s = false;
    if (k < e) {
      const int j = col[k];
      lu = val[k];
      s = strong_entry(di, diag[j], lu, th2);
      scol[k] = s ? j : -1;
    }
    any |= s;
    for (unsigned w = __ballot_sync(0xffffffffu, k < e && !s); w; w &= w - 1)
      t = __dadd_rn(t, __shfl_sync(0xffffffffu, lu, __ffs(w) - 1));
  }
  any = __any_sync(0xffffffffu, any);
  if (lane == 0) { tdm[i] = t; st[i] = any ? 1 : 0; }
}

// ---------------------------------------------------------------------------------
// MIS-2 in synchronous rounds.  Tuple = state(2 bits) | hash priority(30) | index(32);
// state 0 = decided non-root or no strong link (never wins), 1 = undecided, 2 = root.  A round
// takes the largest tuple of each node's strong neighbourhood (itself included) and the
// largest of those over the neighbourhood again; an undecided node that finds itself becomes
// a root, one that finds a root drops out.
//
// All rounds run in one cooperative launch, a grid barrier between the two halves of a
// round, and end with the first round that leaves nothing undecided.  The first half keeps
// only whose tuple won (level 1: direction and state in a byte; CSR: index and state in a
// word); the second makes the tuple again from the index, cheaper than 8-byte gathers.
// ---------------------------------------------------------------------------------
__device__ __forceinline__ unsigned mis_hash(unsigned x, unsigned lev) {
  x ^= 0x9e3779b9u * (lev + 1u);
  x ^= x >> 16; x *= 0x7feb352dU; x ^= x >> 15; x *= 0x846ca68bU; x ^= x >> 16;
  return x;
}
__device__ __forceinline__ unsigned long long mis_tuple(int state, int i, int lev) {
  if (state == 0) return 0ull;
  return ((unsigned long long)state << 62) | ((unsigned long long)(mis_hash((unsigned)i, (unsigned)lev) & 0x3fffffffu) << 32) |
         (unsigned long long)(unsigned)i;
}
// few, large blocks: a barrier of the grid costs with the number of blocks; a level of at most
// kMisSmall rows runs in one cluster, whose barrier is the hardware's
constexpr int kMisSmall = 1 << 14, kMisCluster = 8;
constexpr int kMisRounds = 64, kMisBlock = 512;
constexpr unsigned kMisFinal = 1u << 29;   // CSR word: state in the two top bits, this, index (below 2^29)

__device__ __forceinline__ void mis_decide(int i, unsigned long long t, unsigned char *st, bool &und) {
  if ((unsigned)(t & 0xffffffffull) == (unsigned)i) st[i] = 2;
  else if ((t >> 62) == 2ull) st[i] = 0;
  else und = true;
}
// undecided nodes of the round, one atomic per warp
__device__ __forceinline__ void mis_count(bool und, int *cnt) {
  const unsigned b = __ballot_sync(0xffffffffu, und);
  if ((threadIdx.x & 31) == 0 && b) atomicAdd(cnt, __popc(b));
}

// Four neighbouring cells per thread (the byte arrays are padded to a multiple of four): one
// load passes over four that are done.
__global__ void __launch_bounds__(kMisBlock) k_mis_dia(Bands g, const unsigned char *__restrict__ msk, unsigned char *st,
                                                       unsigned char *w1, int lev, int *cnt) {
  const int nth = gridDim.x * blockDim.x, t0 = blockIdx.x * blockDim.x + threadIdx.x;
  const int nq = (g.N + 3) / 4, nq32 = (nq + 31) & ~31;
  for (int round = 0; round < kMisRounds; ++round) {
    for (int t = t0; t < nq; t += nth) {
      unsigned w = round > 0 ? reinterpret_cast<unsigned *>(w1)[t] : 0u;
      if ((w & 0x80808080u) == 0x80808080u) continue;
      const unsigned m4 = reinterpret_cast<const unsigned *>(msk)[t], s4 = reinterpret_cast<unsigned *>(st)[t];
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        const int i = 4 * t + v;
        if (i < g.N && !(w >> (8 * v) & 128u)) {
          const unsigned m = m4 >> (8 * v) & 255u;
          const int s = s4 >> (8 * v) & 255u;
          unsigned code = 6, ws = s;   // itself
          bool fin = s != 1;
          if (m) {
            unsigned long long best = mis_tuple(s, i, lev);
#pragma unroll
            for (int d = 0; d < 6; ++d)
              if (m >> d & 1) {
                const int j = i + band_off(g, d), sj = st[j];
                const unsigned long long u = mis_tuple(sj, j, lev);
                if (u > best) { best = u; code = d; ws = sj; }
                fin = fin && sj != 1;
              }
          }
          w = (w & ~(255u << (8 * v))) | (code | ws << 3 | (fin ? 128u : 0u)) << (8 * v);
        }
      }
      reinterpret_cast<unsigned *>(w1)[t] = w;
    }
    cg::this_grid().sync();
    for (int t = t0; t < nq32; t += nth) {
      int open = 0;
      const unsigned s4 = t < nq ? reinterpret_cast<unsigned *>(st)[t] : 0u;
      if (s4 & 0x01010101u) {   // state 1 is the only odd one
        const unsigned m4 = reinterpret_cast<const unsigned *>(msk)[t];
        auto tup = [&](int j) {
          const unsigned w = w1[j], code = w & 7u;
          return mis_tuple(w >> 3 & 3u, code == 6 ? j : j + band_off(g, code), lev);
        };
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          const int i = 4 * t + v;
          if (i < g.N && (s4 >> (8 * v) & 1u)) {
            const unsigned m = m4 >> (8 * v) & 255u;
            unsigned long long best = tup(i);
#pragma unroll
            for (int d = 0; d < 6; ++d)
              if (m >> d & 1) {
                const unsigned long long u = tup(i + band_off(g, d));
                if (u > best) best = u;
              }
            bool und = false;
            mis_decide(i, best, st, und);
            open += und;
          }
        }
      }
      open = (int)__reduce_add_sync(0xffffffffu, (unsigned)open);
      if ((threadIdx.x & 31) == 0 && open) atomicAdd(cnt + round, open);
    }
    cg::this_grid().sync();
    if (*(volatile int *)(cnt + round) == 0) break;
  }
}

// eight lanes of a row: the largest of their values, in all of them
__device__ __forceinline__ unsigned long long max8(unsigned long long v) {
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) {
    const unsigned long long w = __shfl_xor_sync(0xffffffffu, v, o);
    if (w > v) v = w;
  }
  return v;
}
__device__ __forceinline__ unsigned long long max4(unsigned long long v) {
#pragma unroll
  for (int o = 2; o > 0; o >>= 1) {
    const unsigned long long w = __shfl_xor_sync(0xffffffffu, v, o);
    if (w > v) v = w;
  }
  return v;
}
// Four lanes per row, each with four entries in flight: the passes wait for the chain row
// bounds -> column -> word.
template <bool CLUSTER>
__global__ void __launch_bounds__(kMisBlock) k_mis_csr(int n, const int *__restrict__ rowptr, const int *__restrict__ scol,
                                                       unsigned char *st, unsigned *w1, int lev, int *cnt) {
  auto sync_all = [] {
    if (CLUSTER) cg::this_cluster().sync();
    else cg::this_grid().sync();
  };
  const int q = threadIdx.x & 3;
  const int nrow = (gridDim.x * blockDim.x) >> 2, r0 = (blockIdx.x * blockDim.x + threadIdx.x) >> 2;
  const int n8 = (n + 7) & ~7;   // all eight rows of a warp stay in the loop
  // fn of the lane's strong neighbours in row i
  auto each = [&](int i, auto word, auto fn) {
    const int e = rowptr[i + 1];
    for (int k = rowptr[i] + q; k < e; k += 16) {
      int j[4];
      unsigned w[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) j[u] = k + 4 * u < e ? scol[k + 4 * u] : -1;
#pragma unroll
      for (int u = 0; u < 4; ++u) w[u] = j[u] >= 0 ? word(j[u]) : 0u;
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (j[u] >= 0) fn(j[u], w[u]);
    }
  };
  for (int round = 0; round < kMisRounds; ++round) {
    for (int i = r0; i < n8; i += nrow) {
      unsigned long long best = 0ull;
      const bool todo = i < n && (round == 0 || !(w1[i] & kMisFinal));
      if (!__any_sync(0xffffffffu, todo)) continue;
      bool open = false;   // something undecided in the neighbourhood
      if (todo) {
        if (q == 0) {
          const int si = st[i];
          best = mis_tuple(si, i, lev);
          open = si == 1;
        }
        each(i, [&](int j) { return (unsigned)st[j]; },
             [&](int j, unsigned sj) {
               const unsigned long long v = mis_tuple((int)sj, j, lev);
               if (v > best) best = v;
               open = open || sj == 1;
             });
      }
      best = max4(best);
      const bool fin = !(__ballot_sync(0xffffffffu, open) >> (threadIdx.x & 28) & 0xfu);
      if (todo && q == 0)
        w1[i] = (unsigned)(best >> 62) << 30 | (fin ? kMisFinal : 0u) | (unsigned)(best & (kMisFinal - 1u));
    }
    sync_all();
    for (int i = r0; i < n8; i += nrow) {
      unsigned long long best = 0ull;
      const bool open = i < n && st[i] == 1;
      if (!__any_sync(0xffffffffu, open)) continue;
      auto tup = [&](unsigned w) { return mis_tuple(w >> 30, (int)(w & (kMisFinal - 1u)), lev); };
      if (open) {
        if (q == 0) best = tup(w1[i]);
        each(i, [&](int j) { return w1[j]; },
             [&](int, unsigned w) {
               const unsigned long long v = tup(w);
               if (v > best) best = v;
             });
      }
      best = max4(best);
      bool und = false;
      if (open && q == 0) mis_decide(i, best, st, und);
      mis_count(und, cnt + round);
    }
    sync_all();
    if (*(volatile int *)(cnt + round) == 0) break;
  }
}

__global__ void k_root_flag(int n, const unsigned char *st, int *flag) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) flag[i] = (st[i] == 2);
}

// pass A: roots keep their id; others join the best root among strong neighbours
__global__ void k_agg_a_dia(Bands g, const unsigned char *__restrict__ msk, const unsigned char *__restrict__ st,
                            const int *__restrict__ aggid, int *agg2, int lev) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= g.N) return;
  if (st[i] == 2) { agg2[i] = aggid[i]; return; }
  const unsigned m = msk[i];
  unsigned long long best = 0;
  int bj = -1;
#pragma unroll
  for (int d = 0; d < 6; ++d)
    if (m >> d & 1) {
      const int j = i + band_off(g, d);
      if (st[j] == 2) {
        const unsigned long long v = mis_tuple(1, j, lev);
        if (v > best) { best = v; bj = j; }
      }
    }
  agg2[i] = bj >= 0 ? aggid[bj] : -1;
}
// pass B: unassigned rows join the best already-assigned strong neighbour
__global__ void k_agg_b_dia(Bands g, const unsigned char *__restrict__ msk, const int *__restrict__ agg2, int *agg,
                            int lev) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= g.N) return;
  int a = agg2[i];
  if (a < 0) {
    const unsigned m = msk[i];
    unsigned long long best = 0;
    int bj = -1;
#pragma unroll
    for (int d = 0; d < 6; ++d)
      if (m >> d & 1) {
        const int j = i + band_off(g, d);
        if (agg2[j] >= 0) {
          const unsigned long long v = mis_tuple(1, j, lev);
          if (v > best) { best = v; bj = j; }
        }
      }
    a = bj >= 0 ? agg2[bj] : -1;
  }
  agg[i] = a;
}
// Passes A (ROOTS) and B of a CSR level, eight lanes per row.
template <bool ROOTS>
__global__ void __launch_bounds__(256) k_agg_csr(int n, const int *__restrict__ rowptr, const int *__restrict__ scol,
                                                 const unsigned char *__restrict__ st, const int *__restrict__ in,
                                                 int *out, int lev) {
  const int q = threadIdx.x & 7, i = (blockIdx.x * blockDim.x + threadIdx.x) >> 3;
  unsigned long long best = 0;
  bool own = true;
  if (i < n) {
    own = ROOTS ? st[i] == 2 : in[i] >= 0;
    if (!own)
      for (int k = rowptr[i] + q; k < rowptr[i + 1]; k += 8) {
        const int j = scol[k];
        if (j >= 0 && (ROOTS ? st[j] == 2 : in[j] >= 0)) {
          const unsigned long long v = mis_tuple(1, j, lev);
          if (v > best) best = v;
        }
      }
  }
  best = max8(best);
  if (i < n && q == 0) out[i] = own ? in[i] : best ? in[(unsigned)(best & 0xffffffffull)] : -1;
}

// ---------------------------------------------------------------------------------
// Smoothed prolongation (make_prolomat, Make_amg_matrix.f90:224-371):
//   columns in first-appearance order over the strong neighbours (CSR order), then
//   the row's own aggregate; values v = -sum lu over strong j of that aggregate,
//   v = v*omega/tdm, own += 1 - omega.
// The fill pass also counts the entries of each column (the rows of R).
// ---------------------------------------------------------------------------------
constexpr int kPRowMax = 96;   // longer prolongation rows stop the coarsening (CPU oracle: same rule)
template <bool FILL>
__global__ void k_p_dia(Bands g, const unsigned char *__restrict__ msk, const int *__restrict__ agg, double om,
                        int *cnt, const int *__restrict__ pptr, int *pcol, double *pval, int *rcnt) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= g.N) return;
  const size_t N = g.N;
  const unsigned m = msk[i];
  const int own = agg[i];
  if (!m) {   // no strong neighbour: in no aggregate
    if (!FILL) cnt[i] = 0;
    return;
  }
  int J[7];
  unsigned first = 0;
#pragma unroll
  for (int d = 0; d < 7; ++d) {
    J[d] = d < 6 ? (m >> d & 1 ? agg[i + band_off(g, d)] : -1) : own;
    bool f = J[d] >= 0;
#pragma unroll
    for (int e = 0; e < d; ++e) f = f && J[e] != J[d];
    first |= (unsigned)f << d;
  }
  if (!FILL) { cnt[i] = __popc(first); return; }
  double lu[6], t = g.d[i];
  {
    const int iz = i / g.nxy, rem = i - iz * g.nxy, iy = rem / g.nx, ix = rem - iy * g.nx;
    const bool has[6] = {iz > 0, iy > 0, ix > 0, ix < g.nx - 1, iy < g.ny - 1, iz < g.nz - 1};
#pragma unroll
    for (int d = 0; d < 6; ++d) {
      lu[d] = has[d] ? g.lu[d * N + i] : 0.0;
      if (has[d] && !(m >> d & 1)) t = __dadd_rn(t, lu[d]);
    }
  }
  int o = pptr[i];
#pragma unroll
  for (int d = 0; d < 7; ++d)
    if (first >> d & 1) {
      double v = 0.0;
#pragma unroll
      for (int e = 0; e < 6; ++e)
        if (e >= d && J[e] == J[d]) v = __dsub_rn(v, lu[e]);
      v = __ddiv_rn(__dmul_rn(v, om), t);
      if (J[d] == own) v = __dsub_rn(__dadd_rn(v, 1.0), om);
      pcol[o] = J[d];
      pval[o] = v;
      ++o;
      atomicAdd(&rcnt[J[d]], 1);
    }
}

// A warp per row of a CSR level: the aggregates of the strong neighbours in entry order (and
// the own one last) as a list in shared memory; an entry whose aggregate stands nowhere
// before it opens a column, and adds up the values of the entries that match it, in order.
// Rows hold at most kHashMax off-diagonals (longer Galerkin rows stop the coarsening); a list
// of that length would leave a quarter of the warps in flight, so rows beyond kPShort entries
// are collected by the count pass and go through a launch of their own (LONG).
constexpr int kHashMax = 700, kPShort = 64;
template <bool FILL, bool LONG>
__global__ void __launch_bounds__(128) k_p_csr(int n, const int *__restrict__ rowptr, const int *__restrict__ scol,
                                               const double *__restrict__ val, const int *__restrict__ agg,
                                               const double *__restrict__ tdm, double om, int *cnt, int *overflow,
                                               int *longrows, int *nlong, const int *__restrict__ pptr, int *pcol,
                                               double *pval, int *rcnt) {
  constexpr int CAP = (LONG ? kHashMax : kPShort) + 4;
  __shared__ int sj[4][CAP];
  __shared__ double sv[4][FILL ? CAP : 1];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, nr = LONG ? *nlong : n;
  int *J = sj[w];
  double *V = sv[w];
  for (int rid = blockIdx.x * 4 + w; rid < nr; rid += gridDim.x * 4) {
    const int i = LONG ? longrows[rid] : rid, b = rowptr[i], e = rowptr[i + 1], own = agg[i];
    if (!LONG && e - b > kPShort) {
      if (!FILL && lane == 0) longrows[atomicAdd(nlong, 1)] = i;
      continue;
    }
    int m = 0;
    for (int k0 = b; k0 < e; k0 += 32) {
      const int k = k0 + lane, j = k < e ? scol[k] : -1, a = j >= 0 ? agg[j] : -1;
      const unsigned bal = __ballot_sync(0xffffffffu, a >= 0);
      if (a >= 0) {
        const int pos = m + __popc(bal & ((1u << lane) - 1u));
        J[pos] = a;
        if (FILL) V[pos] = val[k];
      }
      m += __popc(bal);
    }
    const int len = m + (own >= 0 ? 1 : 0);
    if (own >= 0 && lane == 0) J[m] = own;
    __syncwarp();
    int cols = 0;
    for (int t0 = 0; t0 < len; t0 += 32) {
      const int t = t0 + lane;
      bool f = t < len;
      const int a = f ? J[t] : -1;
      for (int u = 0; u < t && f; ++u) f = J[u] != a;
      const unsigned bal = __ballot_sync(0xffffffffu, f);
      if (FILL && f) {
        double v = 0.0;
        for (int u = t; u < m; ++u)
          if (J[u] == a) v = __dsub_rn(v, V[u]);
        v = __ddiv_rn(__dmul_rn(v, om), tdm[i]);
        if (a == own) v = __dsub_rn(__dadd_rn(v, 1.0), om);
        const int o = pptr[i] + cols + __popc(bal & ((1u << lane) - 1u));
        pcol[o] = a;
        pval[o] = v;
        atomicAdd(&rcnt[a], 1);
      }
      cols += __popc(bal);
    }
    if (!FILL && lane == 0) {
      cnt[i] = min(cols, kPRowMax);
      if (cols > kPRowMax) atomicExch(overflow, 1);
    }
    __syncwarp();
  }
}

// R = P^T: the entries fill their counted rows in any order, each with its row beside it; an
// entry's place in the row is then the number of smaller fine indexes there (keys are
// unique), a thread per entry reading a row of a few cached words.
__global__ void k_r_fill(int nf, const int *pptr, const int *pcol, const double *pval, const int *rptr, int *fill,
                         int *trow, int *tcol, double *tval) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nf) return;
  for (int q = pptr[i]; q < pptr[i + 1]; ++q) {
    int J = pcol[q];
    int pos = rptr[J] + atomicAdd(&fill[J], 1);
    trow[pos] = J;
    tcol[pos] = i;
    tval[pos] = pval[q];
  }
}
__global__ void k_r_rank(int nnz, const int *__restrict__ rptr, const int *__restrict__ trow,
                         const int *__restrict__ tcol, const double *__restrict__ tval, int *rcol, double *rval,
                         float *rval_f) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= nnz) return;
  const int J = trow[e], b = rptr[J], end = rptr[J + 1], key = tcol[e];
  int o = b;
  for (int u = b; u < end; ++u) o += tcol[u] < key;
  const double v = tval[e];
  rcol[o] = key;
  rval[o] = v;
  if (rval_f) rval_f[o] = (float)v;
}

// ---------------------------------------------------------------------------------
// Row-wise sparse product C = A*B with deterministic accumulation: A's entries of a
// row are visited in order (its diagonal first when given), and the products that fall on
// one column are added in that order, the order the CPU oracle uses.
//
// A row's number of products is known from the row lengths alone, so its result goes to a
// place of that size (`start`, a scan of the product counts) and its length beside it; no
// pass counts distinct columns first.  Only where the products are more than 32-bit offsets
// or the memory hold (with every neighbour strong there are 28 per fine cell on 3 columns) does a
// first pass over the rows find the lengths, and the places are exact.  A*P is read back through start and length as it
// stands; the Galerkin operator, which stays, is then copied together, ascending columns,
// diagonal apart (1.0 if absent).  More than kHashMax distinct columns set *overflow, and the
// caller stops coarsening at that level.
// ---------------------------------------------------------------------------------
constexpr int kShort = 64;   // products of a short row

struct Spg {
  const int *ap, *ac;            // A: rows, columns
  const double *av, *adiag;      // values, diagonal (null: none)
  const int *bs, *bl, *bc;       // B: row starts, lengths (null: bs[j + 1] - bs[j]), columns
  const double *bv;
  int split;                     // C's diagonal goes to cdiag and rows are sorted
  const int *cnt, *start;        // products and place of each row of C
  int *len, *ccol;               // ccol null: lengths only
  double *cval, *cdiag;
  __device__ __forceinline__ int blen(int j) const { return bl ? bl[j] : bs[j + 1] - bs[j]; }
};

// Products of each row, eight lanes per row.
__global__ void __launch_bounds__(256) k_spg_bound(int n, Spg s, int *cnt) {
  const int q = threadIdx.x & 7, i = (blockIdx.x * blockDim.x + threadIdx.x) >> 3;
  int m = 0;
  if (i < n) {
    if (s.adiag && q == 0) m = s.blen(i);
    for (int k = s.ap[i] + q; k < s.ap[i + 1]; k += 8) m += s.blen(s.ac[k]);
  }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) m += __shfl_xor_sync(0xffffffffu, m, o);
  if (i < n && q == 0) cnt[i] = m;
}

// A warp per row.  The lanes take an entry of A each (its B row's bounds), then a product each
// (its entry by bisection of the entries' prefix sums), so a window of 32 products is loaded
// together whatever the row lengths, the next one ahead of the current one's additions.
// The window's columns are entered in a hash table together; its values are then added entry
// by entry: B's rows hold unique columns, so within one entry a slot receives at most one
// addition.
// T: table slots.  T = kTabShort handles rows 0 .. *nrows of at most kShort products and
// appends the others to `next`; the larger tables walk a list of rows and pass on to `next`
// those whose columns fill more than three quarters of the table; the largest reports them.
// (A list per row in which each product looks for its column took 1.5 times as long on rows
// of 40 to 60 products and 6 times on rows of 500.)  The short table's kernel spills 4 bytes at
// its 40 registers.
constexpr int kTabShort = 128, kTabMid = 256, kTabMax = 1024;
template <int T>
struct SpgShape {
  static constexpr int warps = T == kTabMax ? 3 : 4;
};
template <int T>
__global__ void __launch_bounds__(32 * SpgShape<T>::warps) k_spg_row(Spg s, int n, const int *__restrict__ nrows,
                                                                     const int *__restrict__ rows, int *next,
                                                                     int *nnext, int *overflow) {
  constexpr int W = SpgShape<T>::warps, kCols = T == kTabMax ? kHashMax : T == kTabShort ? T : T * 3 / 4;
  constexpr unsigned mask = T - 1;
  __shared__ __align__(16) int hk[W][T + 4];
  __shared__ double hv[W][T];
  __shared__ unsigned short comp[W][T];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int *K = hk[w];
  double *V = hv[w];
  const int nr = rows ? *nrows : n;
  for (int rid = blockIdx.x * W + w; rid < nr; rid += gridDim.x * W) {
    const int row = rows ? rows[rid] : rid, o = s.start[row];
    if (T == kTabShort && s.cnt[row] > kShort) {
      if (lane == 0) next[atomicAdd(nnext, 1)] = row;
      continue;
    }
#pragma unroll
    for (int t = lane; t < T; t += 32) { K[t] = -1; V[t] = 0.0; }
    __syncwarp();
    const int a0 = s.ap[row], a1 = s.ap[row + 1];
    int fresh = 0;   // columns this lane opened
    bool full = false;
    for (int k0 = a0 - (s.adiag ? 1 : 0); k0 < a1 && !full; k0 += 32) {
      const int k = k0 + lane;
      int j = row, b0 = 0, len = 0;
      double coef = 0.0;
      if (k < a1) {
        if (k >= a0) { j = s.ac[k]; coef = s.av[k]; }
        else coef = s.adiag[row];
        b0 = s.bs[j];
        len = s.blen(j);
      }
      int inc = len;
#pragma unroll
      for (int p = 1; p < 32; p <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, inc, p);
        if (lane >= p) inc += y;
      }
      const int tot = __shfl_sync(0xffffffffu, inc, 31), rel = b0 - (inc - len);   // product t at rel + t
      // window of product t0 + lane: entry, column, value
      auto load = [&](int t0, int &e, int &c, double &v) {
        const int t = t0 + lane;
        e = 0;   // entries that end at or before product t
#pragma unroll
        for (int p = 16; p > 0; p >>= 1)
          if (__shfl_sync(0xffffffffu, inc, e + p - 1) <= t) e += p;
        const int at = __shfl_sync(0xffffffffu, rel, e) + t;
        const double cf = __shfl_sync(0xffffffffu, coef, e);
        c = -1;
        v = 0.0;
        if (t < tot) {
          c = s.bc[at];
          v = __dmul_rn(cf, s.bv[at]);
        } else {
          e = 32;
        }
      };
      int e, c;
      double v;
      if (tot > 0) load(0, e, c, v);
      for (int t0 = 0; t0 < tot; t0 += 32) {
        int e1 = 32, c1 = -1;
        double v1 = 0.0;
        if (t0 + 32 < tot) load(t0 + 32, e1, c1, v1);
        unsigned slot = 0;
        if (c >= 0) {
          slot = ((unsigned)c * 2654435761u) >> 20 & mask;
          for (int probe = 0; probe < T; ++probe) {
            const int cur = atomicCAS(&K[slot], -1, c);
            if (cur == -1 || cur == c) { fresh += cur == -1; break; }
            slot = (slot + 1) & mask;
          }
        }
        // entry by entry, in order
        for (int q = __shfl_sync(0xffffffffu, e, 0);; ) {
          if (e == q) V[slot] = __dadd_rn(V[slot], v);
          __syncwarp();
          const unsigned later = __ballot_sync(0xffffffffu, e > q && e < 32);
          if (!later) break;
          q = __shfl_sync(0xffffffffu, e, __ffs(later) - 1);
        }
        e = e1; c = c1; v = v1;
        if (T != kTabShort) {
          full = __reduce_add_sync(0xffffffffu, fresh) > kCols;
          if (full) break;
        }
      }
    }
    if (T != kTabShort && full) {
      if (lane == 0) {
        s.len[row] = 0;
        if (T == kTabMax) atomicExch(overflow, 1);
        else next[atomicAdd(nnext, 1)] = row;
      }
      __syncwarp();
      continue;
    }
    // compact: the u-th occupied slot's number to comp[u], its key to K[u] (u is at most the
    // slot's own number, and a slot is read before a later one writes below it)
    int u = 0;
    bool hasd = false;
    for (int base = 0; base < T; base += 32) {
      const int t = base + lane, key = K[t];
      const bool diag = s.split && key == row, occ = key >= 0 && !diag;
      const unsigned bal = __ballot_sync(0xffffffffu, occ);
      if (occ) {
        const int pos = u + __popc(bal & ((1u << lane) - 1));
        comp[w][pos] = (unsigned short)t;
        K[pos] = key;
      }
      if (diag) { s.cdiag[row] = V[t]; hasd = true; }
      u += __popc(bal);
      __syncwarp();
    }
    hasd = __any_sync(0xffffffffu, hasd);
    if (s.split && !hasd && lane == 0) s.cdiag[row] = 1.0;
    if (lane < 4) K[u + lane] = 0x7fffffff;   // the rank loop reads four at a time
    __syncwarp();
    // rank sort by column
    for (int t = lane; t < (s.ccol ? u : 0); t += 32) {
      const int key = K[t];
      int rank = t;
      if (s.split) {
        rank = 0;
        for (int q = 0; q < u; q += 4) {
          const int4 k4 = *reinterpret_cast<const int4 *>(K + q);
          rank += (k4.x < key) + (k4.y < key) + (k4.z < key) + (k4.w < key);
        }
      }
      s.ccol[o + rank] = key;
      s.cval[o + rank] = V[comp[w][t]];
    }
    if (lane == 0) s.len[row] = u;
    __syncwarp();
  }
}

// A*P on level 1: a thread per cell walks its bands (diagonal first) and the prolongation
// rows behind them (0 to 3 entries, most one or none) and keeps the columns it has met in
// shared memory (8 to 10 where there are any; as an unrolled search through registers this
// took twice as long); the rare row of more than kTU columns works in its place in memory, or,
// where only the length is wanted (COUNT), looks back through the products before.
constexpr int kTU = 12, kApT = 128;
__global__ void k_ap_bound_dia(Bands g, const int *__restrict__ pptr, int *cnt) {
  const int ix = blockIdx.x * 32 + threadIdx.x, iy = g.y0 + blockIdx.y * 8 + threadIdx.y, iz = g.z0 + blockIdx.z;
  if (ix >= g.nx || iy >= g.ny) return;
  const int i = ix + g.nx * (iy + g.ny * iz);
  const bool has[6] = {iz > 0, iy > 0, ix > 0, ix < g.nx - 1, iy < g.ny - 1, iz < g.nz - 1};
  int m = pptr[i + 1] - pptr[i];
#pragma unroll
  for (int d = 0; d < 6; ++d)
    if (has[d]) {
      const int j = i + band_off(g, d);
      m += pptr[j + 1] - pptr[j];
    }
  cnt[i] = m;
}
template <bool COUNT>
__global__ void __launch_bounds__(kApT) k_ap_dia(Bands g, const int *__restrict__ pptr, const int *__restrict__ pcol,
                                                 const double *__restrict__ pval, const int *__restrict__ start,
                                                 int *len, int *ccol, double *cval) {
  __shared__ int uc[kTU][kApT];
  __shared__ double uv[kTU][kApT];
  const int ix = blockIdx.x * 32 + threadIdx.x, iy = g.y0 + blockIdx.y * (kApT / 32) + threadIdx.y, iz = g.z0 + blockIdx.z;
  if (ix >= g.nx || iy >= g.ny) return;
  const int tt = threadIdx.y * 32 + threadIdx.x;
  const size_t N = g.N;
  const int i = ix + g.nx * (iy + g.ny * iz);
  const bool has[7] = {true, iz > 0, iy > 0, ix > 0, ix < g.nx - 1, iy < g.ny - 1, iz < g.nz - 1};
  int q0[7], q1[7], fc[7], any = 0;
  double fv[7];
  // bounds and first entry of the seven prolongation rows, all loads in flight together
#pragma unroll
  for (int e = 0; e < 7; ++e) {
    const int j = e == 0 ? i : i + band_off(g, e - 1);
    q0[e] = has[e] ? pptr[j] : 0;
    q1[e] = has[e] ? pptr[j + 1] : 0;
    any |= q1[e] - q0[e];
  }
  if (!any) { len[i] = 0; return; }
#pragma unroll
  for (int e = 0; e < 7; ++e) {
    fc[e] = q0[e] < q1[e] ? pcol[q0[e]] : -1;
    fv[e] = q0[e] < q1[e] ? __dmul_rn(e == 0 ? g.d[i] : g.lu[(e - 1) * N + i], pval[q0[e]]) : 0.0;
  }
  const int o = COUNT ? 0 : start[i];
  int u = 0;
  // entry q of prolongation row e
  auto add = [&](int cc, double p, int e, int q) {
    const int m = min(u, kTU);
    for (int t = 0; t < m; ++t)
      if (uc[t][tt] == cc) { uv[t][tt] = __dadd_rn(uv[t][tt], p); return; }
    if constexpr (COUNT) {
      if (u >= kTU) {
#pragma unroll
        for (int f = 0; f < 7; ++f)
          if (f <= e)
            for (int k = q0[f], end = f == e ? q : q1[f]; k < end; ++k)
              if (pcol[k] == cc) return;
      }
    } else {
      for (int t = kTU; t < u; ++t)
        if (ccol[o + t] == cc) { cval[o + t] = __dadd_rn(cval[o + t], p); return; }
    }
    if (u < kTU) { uc[u][tt] = cc; uv[u][tt] = p; }
    else if (!COUNT) { ccol[o + u] = cc; cval[o + u] = p; }
    ++u;
  };
#pragma unroll
  for (int e = 0; e < 7; ++e) {
    if (fc[e] < 0) continue;
    add(fc[e], fv[e], e, q0[e]);
    if (q0[e] + 1 < q1[e]) {
      const double coef = e == 0 ? g.d[i] : g.lu[(e - 1) * N + i];
      for (int q = q0[e] + 1; q < q1[e]; ++q) add(pcol[q], __dmul_rn(coef, pval[q]), e, q);
    }
  }
  len[i] = u;
  if constexpr (!COUNT)
    for (int t = 0; t < min(u, kTU); ++t) { ccol[o + t] = uc[t][tt]; cval[o + t] = uv[t][tt]; }
}

// The Galerkin rows copied together, eight lanes per row, and their FP32 / BF16 images.
__global__ void __launch_bounds__(256) k_spg_pack(int n, const int *__restrict__ start, const int *__restrict__ ptr,
                                                  const int *__restrict__ tcol, const double *__restrict__ tval,
                                                  const double *__restrict__ diag, int *col, double *val,
                                                  __nv_bfloat16 *val_h, float *diag_f) {
  const int q = threadIdx.x & 7, i = (blockIdx.x * blockDim.x + threadIdx.x) >> 3;
  if (i >= n) return;
  const int s = start[i], o = ptr[i], m = ptr[i + 1] - o;
  for (int k = q; k < m; k += 8) {
    const double v = tval[s + k];
    col[o + k] = tcol[s + k];
    val[o + k] = v;
    if (val_h) val_h[o + k] = __double2bfloat16(v);
  }
  if (q == 0 && diag_f) diag_f[i] = (float)diag[i];
}

// ---------------------------------------------------------------------------------
// Dense Gauss-Jordan inverse (partial pivoting, ties to the smallest row), one
// cooperative grid; matrix M is n x 2n row-major in global memory.
// ---------------------------------------------------------------------------------
__global__ void k_dense_fill(int n, const int *rowptr, const int *col, const double *val, const double *diag,
                             double *M) {
  int i = blockIdx.x;
  int w = 2 * n;
  for (int c = threadIdx.x; c < w; c += blockDim.x) M[(size_t)i * w + c] = (c == n + i) ? 1.0 : 0.0;
  __syncthreads();
  if (threadIdx.x == 0) {
    M[(size_t)i * w + i] = diag[i];
    for (int k = rowptr[i]; k < rowptr[i + 1]; ++k) M[(size_t)i * w + col[k]] = val[k];
  }
}

template <bool COOP, int NT>
__global__ void __launch_bounds__(NT) k_gj(int n, double *M, int *piv_out) {
  struct Sync {
    __device__ void operator()() const {
      if (COOP) cg::this_grid().sync();
      else __syncthreads();
    }
  } sync_all;
  __shared__ double sa[NT];
  __shared__ int si[NT];
  const int w = 2 * n;
  const int tid = blockIdx.x * blockDim.x + threadIdx.x, nth = gridDim.x * blockDim.x;
  for (int p = 0; p < n; ++p) {
    // pivot search by block 0
    if (blockIdx.x == 0) {
      double best = -1.0; int bi = n;
      for (int r = p + threadIdx.x; r < n; r += blockDim.x) {
        double v = fabs(M[(size_t)r * w + p]);
        if (v > best || (v == best && r < bi)) { best = v; bi = r; }
      }
      sa[threadIdx.x] = best; si[threadIdx.x] = bi;
      __syncthreads();
      for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) {
          double v = sa[threadIdx.x + o]; int r = si[threadIdx.x + o];
          if (v > sa[threadIdx.x] || (v == sa[threadIdx.x] && r < si[threadIdx.x])) { sa[threadIdx.x] = v; si[threadIdx.x] = r; }
        }
        __syncthreads();
      }
      if (threadIdx.x == 0) *piv_out = si[0];
    }
    sync_all();
    int piv = *(volatile int *)piv_out;
    // swap rows p and piv, then scale row p
    if (piv != p)
      for (int c = tid; c < w; c += nth) {
        double t = M[(size_t)p * w + c];
        M[(size_t)p * w + c] = M[(size_t)piv * w + c];
        M[(size_t)piv * w + c] = t;
      }
    sync_all();
    double pinv = __ddiv_rn(1.0, ((volatile double *)M)[(size_t)p * w + p]);
    sync_all();
    for (int c = tid; c < w; c += nth) M[(size_t)p * w + c] = __dmul_rn(M[(size_t)p * w + c], pinv);
    sync_all();
    // eliminate column p from every other row; the factor is read before the row
    // changes (column p included: a_rp - f*a_pp, as the sequential loop computes it)
    {
      const int lane = threadIdx.x & 31;
      const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
      const double *prow = M + (size_t)p * w;
      for (int r = gw; r < n; r += nw) {
        if (r == p) continue;
        double *rrow = M + (size_t)r * w;
        double f = rrow[p];
        __syncwarp();
        if (f == 0.0) continue;
        for (int cc = lane; cc < w; cc += 32) rrow[cc] = __dsub_rn(rrow[cc], __dmul_rn(f, prow[cc]));
        __syncwarp();
      }
    }
    sync_all();
  }
}

// The same inverse for n <= 128 with the matrix in the registers of one block: thread
// (tr, tc) of 16 x 32 holds the elements (tr + 16 i, tc + 32 j).  The identity half is never
// stored: its column of the row that becomes pivot p is still a unit vector then, so it takes
// the place of column p, which no later step reads (perm keeps which row's it is); every
// element sees the operations of the augmented elimination in the same order.  Per pivot:
// column p and the two rows to swap through shared memory, three barriers, and 2 n^2 FP64
// operations on one SM (512 cycles at n = 128).  The augmented matrix in global memory took
// 0.50 ms at 76 rows and 0.84 ms at 128, six barriers and a read and a write of 2 n^2 values
// from L2 per pivot; in registers 0.066 ms at 60 rows and 0.35 at 128 with a branch around
// each row, 0.055 and 0.26 with all rows updated alike (a row whose factor is zero keeps its
// bits by selection) and the two rows that change places mended after.
constexpr int kGjReg = 128;
template <int NB>
__global__ void __launch_bounds__(512) k_gj_reg(int n, const int *__restrict__ rowptr, const int *__restrict__ col,
                                                 const double *__restrict__ val, const double *__restrict__ diag,
                                                 const double *__restrict__ dense, double *inv) {
  __shared__ double scol[2][kGjReg], srow[2][kGjReg], spiv[2][kGjReg];
  __shared__ int perm[kGjReg], s_piv;
  __shared__ double s_pinv;
  const int tc = threadIdx.x & 31, tr = threadIdx.x >> 5;
  constexpr int NR = 2 * NB;
  double m[NR][NB];
#pragma unroll
  for (int i = 0; i < NR; ++i)
#pragma unroll
    for (int j = 0; j < NB; ++j) {
      const int r = tr + 16 * i, c = tc + 32 * j;
      m[i][j] = dense && r < n && c < n ? dense[(size_t)r * n + c] : 0.0;
    }
  if (!dense) {   // CSR rows with the diagonal apart
#pragma unroll
    for (int i = 0; i < NR; ++i) {
      const int r = tr + 16 * i;
      if (r < n) {
        for (int k = rowptr[r]; k < rowptr[r + 1]; ++k) {
          const int c = col[k];
          const double v = val[k];
#pragma unroll
          for (int j = 0; j < NB; ++j)
            if (tc + 32 * j == c) m[i][j] = v;
        }
#pragma unroll
        for (int j = 0; j < NB; ++j)
          if (tc + 32 * j == r) m[i][j] = diag[r];
      }
    }
  }
  if (threadIdx.x < kGjReg) perm[threadIdx.x] = threadIdx.x;
#pragma unroll
  for (int pb = 0; pb < NB; ++pb)   // unrolled, so that m is never indexed by a variable
  for (int p = 32 * pb; p < min(n, 32 * pb + 32); ++p) {
    double *sc = scol[p & 1], *sr = srow[p & 1], *sp = spiv[p & 1];
    if (tc == (p & 31)) {
#pragma unroll
      for (int i = 0; i < NR; ++i) sc[tr + 16 * i] = m[i][pb];
    }
    __syncthreads();
    // one warp finds the pivot: largest magnitude (its bits, which order as the values do; a
    // NaN does not count), ties to the lowest row
    if (tr == 0) {
      unsigned long long key = 0;   // the top bit is set where there is a candidate
      int row = n;
#pragma unroll
      for (int i = 0; i < NB; ++i) {
        const int r = tc + 32 * i;
        const unsigned long long v = (unsigned long long)__double_as_longlong(fabs(sc[r]));
        const unsigned long long u = r >= p && r < n && v <= 0x7ff0000000000000ull ? v | 0x8000000000000000ull : 0ull;
        row = u > key ? r : row;
        key = u > key ? u : key;
      }
      const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
      const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
      const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
      row = (int)__reduce_min_sync(0xffffffffu, hi == mh && lo == ml ? (unsigned)row : (unsigned)n);
      if (row == n) row = p;   // a column of NaN
      if (tc == 0) {
        s_piv = row;
        s_pinv = __ddiv_rn(1.0, sc[row]);
        const int q = perm[p];
        perm[p] = perm[row];
        perm[row] = q;
      }
    }
    __syncthreads();
    const int piv = s_piv;
    if (tr == (p & 15) || tr == (piv & 15)) {   // the same in all lanes of the warp
#pragma unroll
      for (int i = 0; i < NR; ++i) {
        const int r = tr + 16 * i;
#pragma unroll
        for (int j = 0; j < NB; ++j) {
          if (r == p) sr[tc + 32 * j] = m[i][j];
          if (r == piv) sp[tc + 32 * j] = m[i][j];
        }
      }
    }
    __syncthreads();
    const double pinv = s_pinv;
    // only the block column pb holds column p, whose place the identity's column takes
    const bool mine = tc == (p & 31);
    double prow[NB];
#pragma unroll
    for (int j = 0; j < NB; ++j) prow[j] = __dmul_rn(j == pb && mine ? 1.0 : sp[tc + 32 * j], pinv);
    // all rows alike, without branches between them; the two rows that change places after
#pragma unroll
    for (int i = 0; i < NR; ++i) {
      const double f = sc[tr + 16 * i];
      if (mine) m[i][pb] = 0.0;
#pragma unroll
      for (int j = 0; j < NB; ++j) {
        const double v = __dsub_rn(m[i][j], __dmul_rn(f, prow[j]));
        m[i][j] = f != 0.0 ? v : m[i][j];
      }
    }
    if (tr == (p & 15) || tr == (piv & 15)) {   // the same in all lanes of the warp
      const double f = sc[p];
#pragma unroll
      for (int i = 0; i < NR; ++i) {
        const int r = tr + 16 * i;
#pragma unroll
        for (int j = 0; j < NB; ++j) {
          const double o = j == pb && mine ? 0.0 : sr[tc + 32 * j];
          if (r == p) m[i][j] = prow[j];
          else if (r == piv) m[i][j] = f != 0.0 ? __dsub_rn(o, __dmul_rn(f, prow[j])) : o;
        }
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < NR; ++i)
#pragma unroll
    for (int j = 0; j < NB; ++j) {
      const int r = tr + 16 * i, c = tc + 32 * j;
      if (r < n && c < n) inv[(size_t)r * n + perm[c]] = m[i][j];
    }
}
static int launch_gj_reg(int n, const int *rowptr, const int *col, const double *val, const double *diag,
                         const double *dense, double *inv, cudaStream_t s) {
  if (n <= 32) k_gj_reg<1><<<1, 512, 0, s>>>(n, rowptr, col, val, diag, dense, inv);
  else if (n <= 64) k_gj_reg<2><<<1, 512, 0, s>>>(n, rowptr, col, val, diag, dense, inv);
  else if (n <= 96) k_gj_reg<3><<<1, 512, 0, s>>>(n, rowptr, col, val, diag, dense, inv);
  else k_gj_reg<4><<<1, 512, 0, s>>>(n, rowptr, col, val, diag, dense, inv);
  MSG_CHECK_LAUNCH();
  return MSG_OK;
}

// [A | I] from a dense row-major matrix
__global__ void k_dense_fill_rm(int n, const double *a, double *M) {
  int i = blockIdx.x;
  int w = 2 * n;
  for (int c = threadIdx.x; c < w; c += blockDim.x)
    M[(size_t)i * w + c] = (c < n) ? a[(size_t)i * n + c] : ((c == n + i) ? 1.0 : 0.0);
}

__global__ void k_dense_extract(int n, const double *M, double *inv) {
  int i = blockIdx.x;
  for (int j = threadIdx.x; j < n; j += blockDim.x) inv[(size_t)i * n + j] = M[(size_t)i * 2 * n + n + j];
}

// ---------------------------------------------------------------------------------
// V-cycle kernels (loop_amg restated as a Jacobi-smoothed V-cycle)
// ---------------------------------------------------------------------------------
struct Dia {
  int nx, ny, nz, nxy, N;
  const double *d, *lu;
};

__device__ __forceinline__ double dia_row(const Dia &A, int i, const double *x) {
  int iz = i / A.nxy, rem = i - iz * A.nxy, iy = rem / A.nx, ix = rem - iy * A.nx;
  const size_t N = A.N;
  double t = __dmul_rn(A.d[i], x[i]);
  if (iz > 0) t = __dadd_rn(t, __dmul_rn(A.lu[0 * N + i], x[i - A.nxy]));
  if (iy > 0) t = __dadd_rn(t, __dmul_rn(A.lu[1 * N + i], x[i - A.nx]));
  if (ix > 0) t = __dadd_rn(t, __dmul_rn(A.lu[2 * N + i], x[i - 1]));
  if (ix < A.nx - 1) t = __dadd_rn(t, __dmul_rn(A.lu[3 * N + i], x[i + 1]));
  if (iy < A.ny - 1) t = __dadd_rn(t, __dmul_rn(A.lu[4 * N + i], x[i + A.nx]));
  if (iz < A.nz - 1) t = __dadd_rn(t, __dmul_rn(A.lu[5 * N + i], x[i + A.nxy]));
  return t;
}

__device__ __forceinline__ double csr_row(int i, const int *rp, const int *cl, const double *v, const double *d,
                                          const double *x) {
  double t = __dmul_rn(d[i], x[i]);
  for (int k = rp[i]; k < rp[i + 1]; ++k) t = __dadd_rn(t, __dmul_rn(v[k], x[cl[k]]));
  return t;
}

// first sweep from x = 0: r = b exactly, x = 0 + w*b/d
__global__ void k_jac_first(int n, const double *b, const double *d, double w, double *x) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    x[i] = __ddiv_rn(__dmul_rn(w, b[i]), d[i]);
}
__global__ void k_jac_dia(Dia A, const double *b, double w, const double *x, double *y) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < A.N; i += gridDim.x * blockDim.x) {
    double r = __dsub_rn(b[i], dia_row(A, i, x));
    y[i] = __dadd_rn(x[i], __ddiv_rn(__dmul_rn(w, r), A.d[i]));
  }
}
__global__ void k_jac_csr(int n, const int *rp, const int *cl, const double *v, const double *d, const double *b,
                          double w, const double *x, double *y) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    double r = __dsub_rn(b[i], csr_row(i, rp, cl, v, d, x));
    y[i] = __dadd_rn(x[i], __ddiv_rn(__dmul_rn(w, r), d[i]));
  }
}
__global__ void k_res_dia(Dia A, const double *b, const double *x, double *r) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < A.N; i += gridDim.x * blockDim.x)
    r[i] = __dsub_rn(b[i], dia_row(A, i, x));
}
__global__ void k_res_csr(int n, const int *rp, const int *cl, const double *v, const double *d, const double *b,
                          const double *x, double *r) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    r[i] = __dsub_rn(b[i], csr_row(i, rp, cl, v, d, x));
}
// b_c = R r  (sum in R row order)
__global__ void k_restrict(int nc, const int *rp, const int *rc, const double *rv, const double *r, double *bc) {
  for (int I = blockIdx.x * blockDim.x + threadIdx.x; I < nc; I += gridDim.x * blockDim.x) {
    double s = 0.0;
    for (int q = rp[I]; q < rp[I + 1]; ++q) s = __dadd_rn(s, __dmul_rn(rv[q], r[rc[q]]));
    bc[I] = s;
  }
}
// x += P xc (sum in P row order)
__global__ void k_prolong(int nf, const int *pp, const int *pc, const double *pv, const double *xc, double *x) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nf; i += gridDim.x * blockDim.x) {
    double s = 0.0;
    for (int q = pp[i]; q < pp[i + 1]; ++q) s = __dadd_rn(s, __dmul_rn(pv[q], xc[pc[q]]));
    x[i] = __dadd_rn(x[i], s);
  }
}
// x = Cinv b, each row summed in column order
__global__ void k_gemv(int n, const double *Ci, const double *b, double *x) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double s = 0.0;
  for (int j = 0; j < n; ++j) s = __dadd_rn(s, __dmul_rn(Ci[(size_t)i * n + j], b[j]));
  x[i] = s;
}


// ---------------------------------------------------------------------------------
// Mixed-precision V-cycle (precision = 1): FP32 vectors, FP32 level-1 operator and
// transfer weights, BF16 off-diagonals and FP32 diagonal on the coarse levels, FP64
// dense inverse at the coarsest level.  The Krylov recurrences stay FP64: the input r
// is read as double and the output z written as double.
// ---------------------------------------------------------------------------------
struct Dia32 {
  int nx, ny, nz, nxy, N;
  const float *d, *lu;
};


// Row i of the FP32 level-1 operator (DIA: diagonal, then the up, north, west, east, south
// and down off-diagonals) times x, with the cell's grid coordinates given by a 3D launch (x
// from the thread, y from the block's y, the layer from the block's z): no integer
// division per cell.
__device__ __forceinline__ float dia_row3_f(const Dia32 &A, int i, int ix, int iy, int iz, const float *x) {
  const size_t N = A.N;
  float t = A.d[i] * x[i];
  if (iz > 0) t += A.lu[0 * N + i] * x[i - A.nxy];
  if (iy > 0) t += A.lu[1 * N + i] * x[i - A.nx];
  if (ix > 0) t += A.lu[2 * N + i] * x[i - 1];
  if (ix < A.nx - 1) t += A.lu[3 * N + i] * x[i + 1];
  if (iy < A.ny - 1) t += A.lu[4 * N + i] * x[i + A.nx];
  if (iz < A.nz - 1) t += A.lu[5 * N + i] * x[i + A.nxy];
  return t;
}
// Fine-level Jacobi sweep (y = x + w (b - A x) / d) and residual (b - A x) over a 3D grid
// of (32, B/32) thread blocks.
template <typename TY>
__global__ void k_jac_dia3(Dia32 A, const float *__restrict__ b, float w, const float *__restrict__ x, TY *y) {
  const int ix = blockIdx.x * 32 + threadIdx.x, iy = blockIdx.y * blockDim.y + threadIdx.y, iz = blockIdx.z;
  if (ix >= A.nx || iy >= A.ny) return;
  const int i = ix + A.nx * (iy + A.ny * iz);
  float r = b[i] - dia_row3_f(A, i, ix, iy, iz, x);
  y[i] = (TY)(x[i] + (w * r) / A.d[i]);
}
__global__ void k_res_dia3(Dia32 A, const float *__restrict__ b, const float *__restrict__ x, float *r) {
  const int ix = blockIdx.x * 32 + threadIdx.x, iy = blockIdx.y * blockDim.y + threadIdx.y, iz = blockIdx.z;
  if (ix >= A.nx || iy >= A.ny) return;
  const int i = ix + A.nx * (iy + A.ny * iz);
  r[i] = b[i] - dia_row3_f(A, i, ix, iy, iz, x);
}

template <typename TB>
__global__ void k_jac_first_f(int n, const TB *b, const float *d, float w, float *x) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    x[i] = (w * (float)b[i]) / d[i];
}
// First fine-level sweep from x = 0; also stores the FP32 rounding of the FP64 right-hand
// side, which every later fine sweep of the cycle reads instead of rounding b again (the
// same values, half the bytes).
// Four elements per thread, all loads issued before the stores: 48 B in flight per thread
// instead of 12, which the one-element form lacked to cover the HBM latency (138 us at
// 25.2M cells, 3.6 TB/s).  Launch with grid4(n, block).
__global__ void k_jac_first_b(int n, const double *__restrict__ b, const float *__restrict__ d, float w,
                              float *__restrict__ x, float *__restrict__ bf) {
  const int st = gridDim.x * blockDim.x;
  for (int i0 = blockIdx.x * blockDim.x + threadIdx.x; i0 < n; i0 += 4 * st) {
    double bv[4];
    float dv[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = i0 + u * st;
      bv[u] = i < n ? b[i] : 0.0;
      dv[u] = i < n ? d[i] : 1.f;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = i0 + u * st;
      if (i < n) {
        const float bi = (float)bv[u];
        bf[i] = bi;
        x[i] = (w * bi) / dv[u];
      }
    }
  }
}
static int grid4(long long n, int block) { return (int)std::max(1LL, (n + 4LL * block - 1) / (4LL * block)); }
__global__ void k_b2f(int n, const double *b, float *bf) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) bf[i] = (float)b[i];
}
// Coarse levels: four lanes per row (lane q takes entries q, q+4, ... of the row; quad
// shuffle sum).  Each lane issues the column and value loads of four of its entries before
// it gathers x for any of them, and the four gathers before it adds: one memory round trip
// per four entries instead of one per entry (a row of 16 entries is one round trip).  The
// products of a lane are added in entry order.  Every lane reaches the shuffles.
__device__ __forceinline__ float ldf(const float *p) { return *p; }
__device__ __forceinline__ float ldf(const __nv_bfloat16 *p) { return __bfloat162float(*p); }
// Two rows per quad: the quad walks rows 2Q and 2Q+1 together (column and value loads of
// both rows, then the gathers of both), so a warp keeps sixteen rows' loads in flight
// (4% off the mixed V-cycle at 25.2M cells against one row per quad).  Launch with
// grid2r(n): four threads per two rows.
template <typename TV>
__device__ __forceinline__ void csr_off_h4x2(int i0, int q, int n, const int *rp, const int *cl, const TV *v,
                                             const float *x, float &t0, float &t1, int k0 = 0) {
  float s[2] = {0.f, 0.f};
  int k[2], e[2];
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const bool live = i0 + r < n;
    k[r] = live ? rp[i0 + r] - k0 + q : 0;
    e[r] = live ? rp[i0 + r + 1] - k0 : 0;
  }
  while (k[0] < e[0] || k[1] < e[1]) {
    int c[2][4];
    float a[2][4], xv[2][4];
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int kk = k[r] + 4 * u;
        c[r][u] = kk < e[r] ? cl[kk] : -1;
        a[r][u] = kk < e[r] ? ldf(v + kk) : 0.f;
      }
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int u = 0; u < 4; ++u) xv[r][u] = c[r][u] >= 0 ? x[c[r][u]] : 0.f;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (c[r][u] >= 0) s[r] += a[r][u] * xv[r][u];
      k[r] += 16;
    }
  }
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    s[r] += __shfl_xor_sync(0xffffffffu, s[r], 1);
    s[r] += __shfl_xor_sync(0xffffffffu, s[r], 2);
  }
  t0 = s[0];
  t1 = s[1];
}
__global__ void k_jac_csr_h(int n, const int *rp, const int *cl, const __nv_bfloat16 *v, const float *d,
                            const float *b, float w, const float *x, float *y) {
  const long long gt = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int i0 = (int)(gt >> 2) * 2, q = (int)(gt & 3);
  const int i = i0 + (q & 1);        // lanes 0 and 1 of the quad finish rows i0 and i0 + 1
  const bool own = q < 2 && i < n;
  float bi = 0.f, di = 1.f, xi = 0.f;
  if (own) { bi = b[i]; di = d[i]; xi = x[i]; }   // in flight during the row walk
  float o0, o1;
  csr_off_h4x2(i0, q, n, rp, cl, v, x, o0, o1);
  if (own) {
    const float off = q ? o1 : o0;
    const float r = bi - (di * xi + off);
    y[i] = xi + (w * r) / di;
  }
}
__global__ void k_res_csr_h(int n, const int *rp, const int *cl, const __nv_bfloat16 *v, const float *d,
                            const float *b, const float *x, float *r) {
  const long long gt = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int i0 = (int)(gt >> 2) * 2, q = (int)(gt & 3);
  const int i = i0 + (q & 1);
  const bool own = q < 2 && i < n;
  float bi = 0.f, di = 0.f, xi = 0.f;
  if (own) { bi = b[i]; di = d[i]; xi = x[i]; }
  float o0, o1;
  csr_off_h4x2(i0, q, n, rp, cl, v, x, o0, o1);
  if (own) r[i] = bi - (di * xi + (q ? o1 : o0));
}
// 4 threads per two rows
static int grid2r(int n) { return (int)((((long long)n + 1) / 2 * 4 + kThreads - 1) / kThreads); }

// Block-streamed CSR passes of the mixed V-cycle's coarse levels and transfers (the
// CSR-stream scheme of Greathouse and Daga, "Efficient sparse matrix-vector multiplication
// on GPUs using the CSR storage format", SC 2014).  A block owns kSR consecutive rows,
// whose entries are one contiguous range of the CSR arrays: the block walks that range in
// chunks of kSC entries with consecutive threads on consecutive entries (column and value
// loads coalesced, four entries per thread issued before their gathers), parks the
// products in shared memory, and each thread then adds its own row's products in entry
// order.  Rows of any length are handled by the chunk loop.
constexpr int kSR = 128, kSC = 2048, kSU = 4;
enum { kCsrJacobi = 0, kCsrResidual = 1, kCsrRowSum = 2, kCsrAddTo = 3 };
// OP kCsrJacobi: y_i = x_i + w (b_i - d_i x_i - sum_k v_k x_{c_k}) / d_i
// OP kCsrResidual: y_i = b_i - d_i x_i - sum_k v_k x_{c_k}
// OP kCsrRowSum: y_i = sum_k v_k x_{c_k}               (restriction, R = P^T)
// OP kCsrAddTo: y_i = y_i + sum_k v_k x_{c_k}          (prolongation, x += P x_c)
template <int OP, typename TV>
__global__ void __launch_bounds__(kSR) k_csr_stream(int n, const int *__restrict__ rp, const int *__restrict__ cl,
                                                    const TV *__restrict__ v, const float *__restrict__ d,
                                                    const float *__restrict__ b, float w, const float *__restrict__ x,
                                                    float *y) {
  __shared__ float prod[kSC];
  const int t = threadIdx.x;
  const int i0 = blockIdx.x * kSR, i = i0 + t;
  const bool own = i < n;
  const int beg = rp[i0], end = rp[min(i0 + kSR, n)];
  int rb = 0, re = 0;
  float bi = 0.f, di = 1.f, xi = 0.f;
  if (own) {
    rb = rp[i];
    re = rp[i + 1];
    if (OP == kCsrJacobi || OP == kCsrResidual) { bi = b[i]; di = d[i]; xi = x[i]; }
    if (OP == kCsrAddTo) xi = y[i];
  }
  float s = 0.f;
  for (int c0 = beg; c0 < end; c0 += kSC) {
    const int c1 = min(c0 + kSC, end);
    for (int k = c0 + t; k < c1; k += kSR * kSU) {
      int cc[kSU];
      float a[kSU], xv[kSU];
#pragma unroll
      for (int u = 0; u < kSU; ++u) {
        const int kk = k + u * kSR;
        cc[u] = kk < c1 ? cl[kk] : -1;
        a[u] = kk < c1 ? ldf(v + kk) : 0.f;
      }
#pragma unroll
      for (int u = 0; u < kSU; ++u) xv[u] = cc[u] >= 0 ? x[cc[u]] : 0.f;
#pragma unroll
      for (int u = 0; u < kSU; ++u)
        if (cc[u] >= 0) prod[k + u * kSR - c0] = a[u] * xv[u];
    }
    __syncthreads();
    const int lo = max(rb, c0), hi = min(re, c1);
    for (int k = lo; k < hi; ++k) s += prod[k - c0];
    __syncthreads();
  }
  if (!own) return;
  if (OP == kCsrJacobi) y[i] = xi + (w * (bi - (di * xi + s))) / di;
  else if (OP == kCsrResidual) y[i] = bi - (di * xi + s);
  else if (OP == kCsrRowSum) y[i] = s;
  else y[i] = xi + s;
}
static int gridS(int n) { return (n + kSR - 1) / kSR; }
// Restriction b_c = R r: a coarse row gathers from every fine row its aggregate's
// smoothed prolongation reaches (tens of entries), so it is split over four lanes like the
// coarse-level smoother.  Launch with grid2r(nc).
__global__ void k_restrict_f(int nc, const int *rp, const int *rc, const float *rv, const float *r, float *bc) {
  const long long gt = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int I0 = (int)(gt >> 2) * 2, q = (int)(gt & 3);
  float t0, t1;
  csr_off_h4x2(I0, q, nc, rp, rc, rv, r, t0, t1);
  const int I = I0 + (q & 1);
  if (q < 2 && I < nc) bc[I] = q ? t1 : t0;
}
// Prolongation x += P x_c, a thread per fine row, four rows per thread (rows i0 + u*stride):
// the row bounds, the own values, the first entry of each row and its gather are issued for
// all four rows before any sum (prolongation rows hold 0 to 3 entries, most one or none);
// the rest of a row continues the same in-order sum.  Launch with grid4(nf, block).
__device__ __forceinline__ float csr_row_from(float s, int beg, int end, const int *cl, const float *val,
                                              const float *x) {
  for (int k = beg; k < end; k += 4) {
    int c[4];
    float a[4], xv[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int kk = k + u;
      c[u] = kk < end ? cl[kk] : -1;
      a[u] = kk < end ? val[kk] : 0.f;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) xv[u] = c[u] >= 0 ? x[c[u]] : 0.f;
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (c[u] >= 0) s += a[u] * xv[u];
  }
  return s;
}
__global__ void k_prolong_f(int nf, const int *__restrict__ pp, const int *__restrict__ pc,
                            const float *__restrict__ pv, const float *__restrict__ xc, float *x) {
  const int st = gridDim.x * blockDim.x;
  for (int i0 = blockIdx.x * blockDim.x + threadIdx.x; i0 < nf; i0 += 4 * st) {
    int beg[4], end[4], c[4];
    float a[4], g[4], xi[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = i0 + u * st;
      const bool live = i < nf;
      beg[u] = live ? pp[i] : 0;
      end[u] = live ? pp[i + 1] : 0;
      xi[u] = live ? x[i] : 0.f;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      c[u] = beg[u] < end[u] ? pc[beg[u]] : -1;
      a[u] = beg[u] < end[u] ? pv[beg[u]] : 0.f;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) g[u] = c[u] >= 0 ? xc[c[u]] : 0.f;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = i0 + u * st;
      if (i < nf) {
        float s = 0.f;
        if (c[u] >= 0) s += a[u] * g[u];
        if (beg[u] + 1 < end[u]) s = csr_row_from(s, beg[u] + 1, end[u], pc, pv, xc);
        x[i] = xi[u] + s;
      }
    }
  }
}
// One coarse-level CSR pass.  Measured per pass at 25.2M cells (levels of 2.78M rows x 14
// entries, 204k x 44, 22k x 48, ...): the block-streamed kernel takes 94.6 us per Jacobi
// sweep of the 2.78M-row level against 107.4 for four lanes per row, and 49.6 against 59.4
// for the restriction onto it (5.7 entries per row), but is slower on the short, dense
// levels (28.1 against 24.4 us at 204k rows, 16.1 against 7.8 at 22k) and for the
// prolongation rows (0.6 to 3 entries; 148 against 125 us on the fine grid).  So: long
// levels of short rows stream, the rest runs four lanes per row, prolongation a thread
// per row.
template <int OP, typename TV>
static void csr_pass(int n, int nnz, const int *rp, const int *cl, const TV *v, const float *d, const float *b,
                     float w, const float *x, float *y, cudaStream_t s) {
  const bool stream = OP != kCsrAddTo && n >= (1 << 19) && (long long)nnz <= 24LL * n;
  if (stream) {
    k_csr_stream<OP, TV><<<gridS(n), kSR, 0, s>>>(n, rp, cl, v, d, b, w, x, y);
  } else if constexpr (OP == kCsrJacobi) {
    k_jac_csr_h<<<grid2r(n), kThreads, 0, s>>>(n, rp, cl, v, d, b, w, x, y);
  } else if constexpr (OP == kCsrResidual) {
    k_res_csr_h<<<grid2r(n), kThreads, 0, s>>>(n, rp, cl, v, d, b, x, y);
  } else if constexpr (OP == kCsrRowSum) {
    k_restrict_f<<<grid2r(n), kThreads, 0, s>>>(n, rp, cl, v, x, y);
  } else {
    k_prolong_f<<<grid4(n, kThreads), kThreads, 0, s>>>(n, rp, cl, v, x, y);
  }
}
// coarsest level: FP64 dense inverse applied to a float right-hand side, one warp per
// row (coalesced row reads, fixed shuffle tree).  Launch with n warps; a warp's row index
// is the same in all its lanes, so a warp past the end leaves as a whole.
__global__ void k_gemv_mixed(int n, const double *Ci, const float *b, float *x) {
  const int row = (int)(((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (row >= n) return;
  double s = 0.0;
  for (int j = lane; j < n; j += 32) s += Ci[(size_t)row * n + j] * (double)b[j];
#pragma unroll
  for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) x[row] = (float)s;
}
__global__ void k_d2f(int n, const double *a, float *b) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) b[i] = (float)a[i];
}
__global__ void k_f2d(int n, const float *a, double *b) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) b[i] = (double)a[i];
}

// ---------------------------------------------------------------------------------
// The small levels of a V-cycle in one launch: one cluster of blocks walks down from the
// first level of at most kTailRows rows and back up, its barrier (a fraction of a
// microsecond) between the passes that are launches of 4 us each otherwise.  Every row is
// computed as by the kernels of the larger levels, in the same order.  (A persistent grid
// over the whole chip, whose barrier costs as much as a launch, had not paid.)  Of the FP64
// launch's 1024 threads the registers are 32, and the compiler spills 60 bytes.
// ---------------------------------------------------------------------------------
// A dense coarsest level beyond kTailDense rows wants the whole chip's bandwidth.
constexpr int kTailRows = 8192, kTailDense = 512, kTailThreads = 1024, kTailThreadsF = 512;
struct TailLevel {
  int n;
  const int *rowptr, *col;
  const double *val, *diag;
  const int *rptr, *rcol, *pptr, *pcol;   // to this level from the one before, and back
  const double *rval, *pval;
  double *x, *b, *r, *x2;
};
struct TailArgs {
  int nl, sweeps;
  double w;
  const double *cinv;                     // dense inverse of the last level, or null
  TailLevel lv[kTailMax];
};

// FP64 rows: eight lanes share a row's loads and products and add the products in entry order
// (every lane the same sum).  Ends together in all lanes of the warp.
template <typename F>
__device__ __forceinline__ double ordered_sum8(double t, int beg, int end, F product) {
  const int q = threadIdx.x & 7;
  while (__any_sync(0xffffffffu, beg < end)) {
    const double p = beg + q < end ? product(beg + q) : 0.0;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const double v = __shfl_sync(0xffffffffu, p, u, 8);
      if (beg + u < end) t = __dadd_rn(t, v);
    }
    beg += 8;
  }
  return t;
}

__global__ void __launch_bounds__(kTailThreads) k_cycle_tail(TailArgs a) {
  const int nt = kTailBlocks * kTailThreads, t = blockIdx.x * kTailThreads + threadIdx.x;
  auto sync_all = [] { cg::this_cluster().sync(); };
  auto first = [&](const TailLevel &L, double *x) {   // from x = 0
    for (int i = t; i < L.n; i += nt) x[i] = __ddiv_rn(__dmul_rn(a.w, L.b[i]), L.diag[i]);
    sync_all();
  };
  // y = x + w (b - A x) / d, or (RES) y = b - A x
  auto pass = [&](const TailLevel &L, const double *x, double *y, bool res) {
    for (int i0 = 0; i0 < L.n; i0 += nt / 8) {
      const int i = i0 + (t >> 3);
      const bool live = i < L.n;
      const double di = live ? L.diag[i] : 1.0, xi = live ? x[i] : 0.0;
      const double s = ordered_sum8(__dmul_rn(di, xi), live ? L.rowptr[i] : 0, live ? L.rowptr[i + 1] : 0,
                                    [&](int k) { return __dmul_rn(L.val[k], x[L.col[k]]); });
      if (live && (t & 7) == 0) {
        const double r = __dsub_rn(L.b[i], s);
        y[i] = res ? r : __dadd_rn(xi, __ddiv_rn(__dmul_rn(a.w, r), di));
      }
    }
    sync_all();
  };
  auto restrict_to = [&](const TailLevel &C, const double *r) {
    for (int i0 = 0; i0 < C.n; i0 += nt / 8) {
      const int i = i0 + (t >> 3);
      const bool live = i < C.n;
      const double s = ordered_sum8(0.0, live ? C.rptr[i] : 0, live ? C.rptr[i + 1] : 0,
                                    [&](int k) { return __dmul_rn(C.rval[k], r[C.rcol[k]]); });
      if (live && (t & 7) == 0) C.b[i] = s;
    }
    sync_all();
  };
  auto prolong = [&](const TailLevel &C, int nf, double *x) {
    for (int i = t; i < nf; i += nt) {
      double s = 0.0;
      for (int k = C.pptr[i], e = C.pptr[i + 1]; k < e; ++k) s = __dadd_rn(s, __dmul_rn(C.pval[k], C.x[C.pcol[k]]));
      x[i] = __dadd_rn(x[i], s);
    }
    sync_all();
  };
  const int sw = a.sweeps;
  // where the iterate lies: sweeps alternate between two buffers and end in x
  auto start = [&](const TailLevel &L, double *&cur, double *&oth) {
    cur = sw > 0 ? L.x2 : L.x;            // 2 sw - 1 sweeps
    oth = cur == L.x ? L.x2 : L.x;
  };
  auto smooth = [&](const TailLevel &L, double *&cur, double *&oth, int k) {
    for (; k > 0; --k) {
      pass(L, cur, oth, false);
      double *q = cur;
      cur = oth;
      oth = q;
    }
  };
  auto pre = [&](const TailLevel &L, double *&cur, double *&oth) {
    start(L, cur, oth);
    if (sw == 0) {
      for (int i = t; i < L.n; i += nt) cur[i] = 0.0;
      sync_all();
    } else {
      first(L, cur);
      smooth(L, cur, oth, sw - 1);
    }
  };
  double *cur, *oth;
  for (int l = 0; l + 1 < a.nl; ++l) {
    const TailLevel &L = a.lv[l];
    pre(L, cur, oth);
    pass(L, cur, L.r, true);
    restrict_to(a.lv[l + 1], L.r);
  }
  {
    const TailLevel &L = a.lv[a.nl - 1];
    if (a.cinv) {
      for (int i0 = 0; i0 < L.n; i0 += nt / 8) {
        const int i = i0 + (t >> 3);
        const bool live = i < L.n;
        const double s = ordered_sum8(0.0, 0, live ? L.n : 0, [&](int j) { return __dmul_rn(a.cinv[(size_t)i * L.n + j], L.b[j]); });
        if (live && (t & 7) == 0) L.x[i] = s;
      }
      sync_all();
    } else {
      pre(L, cur, oth);
      smooth(L, cur, oth, sw);
    }
  }
  for (int l = a.nl - 2; l >= 0; --l) {
    const TailLevel &L = a.lv[l];
    start(L, cur, oth);
    if (sw > 0 && sw % 2 == 0) { double *q = cur; cur = oth; oth = q; }   // after sw - 1 sweeps
    prolong(a.lv[l + 1], L.n, cur);
    smooth(L, cur, oth, sw);
  }
}

// The same of the mixed cycle, out of shared memory: every block keeps the iterates whole, the
// lanes that finish a row storing it into all blocks' copies, and the operator rows that it
// computes.  A pass is bounded by the shared memory's loads, so an off-diagonal is one word
// (column and BF16 value), laid out by slices of sixteen rows, a warp's, in the order in which
// the lanes take them (without bank conflicts): a load of it and one of x per entry.  Rows of
// the transfers, used once, are copied as they are; what does not fit is read from memory.
// The build lays the slices out, so that a launch copies them as they are (laid out by each
// launch: 8 us more at 3507 rows).  A whole cycle against the passes out of L2: 113 -> 92 us on
// 64 x 57 x 33 cells (1270 rows at the first small level), 141 -> 114 on 113 x 87 x 37 (3507),
// 422 -> 379 on 256 x 256 x 64 (3880).  What is left is latency: 1.2 us a pass of a small
// level, most of it the barrier, the rows' store and the control that every warp walks; so 512
// threads (1024 take 2 us more a cycle, 256 6 us more).
constexpr int kTailShared = 222 * 1024;   // of a block's 227 KB
// bytes from src (16-byte aligned, in an allocation of a multiple of 256 bytes), by NT threads
template <int NT>
__device__ __forceinline__ void tail_fetch(char *dst, const void *src, int bytes, int i) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  for (int o = i * 16; o < bytes; o += NT * 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + o), "l"((const char *)src + o) : "memory");
}

__device__ __forceinline__ int tail_row(const TailLevelF &L, int rank) { return min(L.n, rank * L.per); }

// What k_cycle_tail_f's block of the same number will copy: extents of its rows of the
// transfers, slices of its operators' rows (as wide as the longest row wants, in steps of
// two; the first that find no room and all behind them are left to memory).
__global__ void __launch_bounds__(kTailThreads) k_tail_pack(const __grid_constant__ TailArgsF a) {
  __shared__ TailLevelF lv[kTailMax];     // a copy: constants under a variable index answer slowly
  __shared__ TailHead h;
  const int t = threadIdx.x, rank = blockIdx.x, lane = t & 31, warp = t >> 5, q = t & 3, nl = a.nl;
#pragma unroll
  for (int l = 0; l < kTailMax; ++l)
    if (t == 16 * l && l < nl) lv[l] = a.lv[l];
  __syncthreads();
  int nsl = 0;
  for (int l = 0; l < nl; ++l) {
    const TailLevelF &L = lv[l];
    if (t == 0) h.sl0[l] = nsl;
    if (!L.rowptr) continue;
    const int r0 = tail_row(L, rank), nr = tail_row(L, rank + 1) - r0, ns = (nr + 15) / 16;
    for (int s = warp; s < ns; s += kTailThreads / 32) {
      const int j = s * 16 + (lane & 15);
      const int len = j < nr ? L.rowptr[r0 + j + 1] - L.rowptr[r0 + j] : 0;
      const int w = (__reduce_max_sync(0xffffffffu, (len + 3) / 4) + 1) & ~1;
      if (lane == 0) h.wid[nsl + s] = w;
    }
    nsl += ns;
  }
  if (warp == kTailThreads / 32 - 1 && lane < 2 * nl) {
    const TailLevelF &L = lv[lane >> 1];
    const TailMatF &m = lane & 1 ? L.P : L.R;
    const int *rp = lane & 1 ? L.pptr : L.rptr;
    const int r0 = tail_row(L, rank), nr = tail_row(L, rank + 1) - r0;
    bool fits = m.cap > 0 && nr > 0;      // r0 is a multiple of 4 where there are rows
    int b = 0;
    if (fits) {
      b = rp[r0] & ~7;
      fits = rp[r0 + nr] - b <= m.cap;
    }
    h.base[lane] = b;
    h.in[lane] = fits;
  }
  __syncthreads();
  if (warp == 0) {
    int run = 0, words = 0;
    for (int s0 = 0; s0 < nsl; s0 += 32) {
      const int w = s0 + lane < nsl ? h.wid[s0 + lane] * 64 : 0;
      int e = w;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, e, o);
        if (lane >= o) e += v;
      }
      const bool fits = run + e <= a.words;
      if (s0 + lane < nsl) h.off[s0 + lane] = fits ? run + e - w : -1;
      words = max(words, (int)__reduce_max_sync(0xffffffffu, fits ? run + e : 0));
      run += __shfl_sync(0xffffffffu, e, 31);
    }
    if (lane == 0) h.words = words;
  }
  __syncthreads();
  for (int i = t; i < (int)(sizeof(TailHead) / 4); i += kTailThreads)
    reinterpret_cast<int *>(a.head + rank)[i] = reinterpret_cast<const int *>(&h)[i];
  uint32_t *out = a.slices + (size_t)rank * a.words;
  for (int l = 0; l < nl; ++l) {
    const TailLevelF &L = lv[l];
    if (!L.rowptr) continue;
    const int r0 = tail_row(L, rank), nr = tail_row(L, rank + 1) - r0;
    const uint32_t pad = (uint32_t)((L.n + 1) & ~1) << 16;
    for (int s = warp; s * 16 < nr; s += kTailThreads / 32) {
      const int o = h.off[h.sl0[l] + s], w = h.wid[h.sl0[l] + s], j = s * 16 + (lane >> 2) * 2;
      if (o < 0) continue;
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        int k = 0, e = 0;
        if (j + r < nr) { k = L.rowptr[r0 + j + r] + q; e = L.rowptr[r0 + j + r + 1]; }
        for (int u = 0; u < w; ++u) {
          const int kk = k + 4 * u;
          out[o + (2 * u + r) * 32 + lane] = kk < e ? (uint32_t)L.col[kk] << 16 | __bfloat16_as_ushort(L.val[kk]) : pad;
        }
      }
    }
  }
}

__global__ void __launch_bounds__(kTailThreadsF) k_cycle_tail_f(const __grid_constant__ TailArgsF a) {
  extern __shared__ __align__(16) char sm[];
  __shared__ TailLevelF lv[kTailMax];     // a copy: constants under a variable index answer slowly
  __shared__ TailHead h;
  auto cl = cg::this_cluster();
  const int t = threadIdx.x, rank = (int)cl.block_rank(), lane = t & 31, warp = t >> 5, q = t & 3, nl = a.nl, sw = a.sweeps;
  auto vec = [&](int o) { return reinterpret_cast<float *>(sm + o); };
  auto first_row = [&](const TailLevelF &L) { return tail_row(L, rank); };
  auto own_rows = [&](const TailLevelF &L) { return tail_row(L, rank + 1) - tail_row(L, rank); };
  for (int i = t; i < (int)(sizeof(TailHead) / 4); i += kTailThreadsF)
    reinterpret_cast<int *>(&h)[i] = reinterpret_cast<const int *>(a.head + rank)[i];
#pragma unroll
  for (int l = 0; l < kTailMax; ++l)
    if (t == 16 * l && l < nl) lv[l] = a.lv[l];
  __syncthreads();
  const int *off = h.off, *wid = h.wid, *sl0 = h.sl0, *base = h.base, *in = h.in;
  // ---- everything on its way: slices, transfers and diagonals, the first sweep
  uint32_t *pool = reinterpret_cast<uint32_t *>(sm + a.pool);
  tail_fetch<kTailThreadsF>(sm + a.pool, a.slices + (size_t)rank * a.words, h.words * 4, t);
  for (int k = warp; k < 3 * nl; k += kTailThreadsF / 32) {
    const int l = k / 3, m = k % 3;
    const TailLevelF &L = lv[l];
    const int r0 = first_row(L), nr = own_rows(L);
    if (m == 2) {
      if (L.diag) tail_fetch<32>(sm + L.d, L.diag + r0, nr * 4, lane);
    } else if (in[2 * l + m]) {
      const TailMatF &M = m ? L.P : L.R;
      const int *rp = m ? L.pptr : L.rptr, b = base[2 * l + m], n = rp[r0 + nr] - b;
      tail_fetch<32>(sm + M.rp, rp + r0, (nr + 1) * 4, lane);
      tail_fetch<32>(sm + M.cl, (m ? L.pcol : L.rcol) + b, n * 4, lane);
      tail_fetch<32>(sm + M.v, (m ? L.pval : L.rval) + b, n * 4, lane);
    }
  }
  if (t < 2 * nl) vec(lv[t >> 1].v[t & 1])[(lv[t >> 1].n + 1) & ~1] = 0.f;   // what the padding multiplies
  const bool dense0 = a.cinv && nl == 1;
  {                                       // the first level's right-hand side and first sweep, whole in every block
    const TailLevelF &L = lv[0];
    const int r0 = first_row(L), nr = own_rows(L);
    const int n = L.n;
    const float *d = L.diag;
    float *lb = vec(L.b), *x = vec(L.v[0]);
    for (int i0 = t; i0 < n; i0 += 4 * kTailThreadsF) {
      float b[4], di[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int i = i0 + u * kTailThreadsF;
        b[u] = i < n ? a.b[i] : 0.f;
        di[u] = i < n && !dense0 ? d[i] : 1.f;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int i = i0 + u * kTailThreadsF;
        if (i >= r0 && i < r0 + nr) lb[i - r0] = b[u];
        if (i < n) x[i] = dense0 ? b[u] : sw > 0 ? (a.w * b[u]) / di[u] : 0.f;
      }
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  cl.sync();                              // also: every block's shared memory exists
  // ---- passes, one at a time: smoothing from v[k & 1] to the other, k = 0 .. sw - 2 on the
  // way down and .. 2 sw - 2 on the way up, r in the iterate that is free
  enum { kSmooth, kResidual, kRestrict, kProlong, kDense };
  bool up = false, out = false;
  for (int l = 0, k = 0, res = 0; l >= 0;) {
    const TailLevelF &L = lv[l];
    const bool last = l == nl - 1;
    int kind, lw = l;                     // lw: the level whose rows are computed
    if (!up && last && a.cinv) kind = kDense;
    else if (up && res) kind = kProlong;
    else if (k < (up || last ? 2 * sw - 1 : sw - 1)) kind = kSmooth;
    else if (up || last) {                // level finished: prolong to the one before
      up = true;
      res = 1;
      k = max(sw - 1, 0);
      --l;
      continue;
    } else kind = res ? kRestrict : kResidual;
    if (kind == kRestrict) lw = l + 1;
    const TailLevelF &W = lv[lw];
    const int r0 = first_row(W), nr = own_rows(W), cur = L.v[k & 1], oth = L.v[~k & 1];
    out = kind == kSmooth && l == 0 && (up || last) && k == 2 * sw - 2;   // the cycle's last pass
    // rows j and j + 1 (r0, j even; copies end on a pair) to every block, two blocks a lane
    auto put = [&](int o, int j, float y) {
      const float2 y2 = make_float2(__shfl_sync(0xffffffffu, y, 0, 4), __shfl_sync(0xffffffffu, y, 1, 4));
      if (j >= nr) return;
      float2 *dst = reinterpret_cast<float2 *>(vec(o) + r0 + j);
      *cl.map_shared_rank(dst, 2 * q) = y2;
      *cl.map_shared_rank(dst, 2 * q + 1) = y2;
    };
    if (kind <= kResidual) {              // y = x + w (b - A x) / d, or b - A x
      const float *x = vec(cur), *xr = x + r0, *b = vec(W.b), *d = vec(W.d);
      for (int s = warp; s * 16 < nr; s += kTailThreadsF / 32) {
        const int j = s * 16 + (lane >> 2) * 2, i = j + (q & 1), o = off[sl0[l] + s], w = wid[sl0[l] + s];
        float bi = 0.f, di = 1.f, xi = 0.f, s0 = 0.f, s1 = 0.f;
        if (i < nr) { bi = b[i]; di = d[i]; xi = xr[i]; }
        if (o >= 0) {
          const uint32_t *p = pool + o + lane;
#pragma unroll 2
          for (int u = 0; u < w; u += 2, p += 128) {
            const uint32_t e0 = p[0], f0 = p[32], e1 = p[64], f1 = p[96];
            const float xe0 = x[e0 >> 16], xf0 = x[f0 >> 16], xe1 = x[e1 >> 16], xf1 = x[f1 >> 16];
            s0 += __uint_as_float(e0 << 16) * xe0;
            s1 += __uint_as_float(f0 << 16) * xf0;
            s0 += __uint_as_float(e1 << 16) * xe1;
            s1 += __uint_as_float(f1 << 16) * xf1;
          }
          s0 += __shfl_xor_sync(0xffffffffu, s0, 1);
          s1 += __shfl_xor_sync(0xffffffffu, s1, 1);
          s0 += __shfl_xor_sync(0xffffffffu, s0, 2);
          s1 += __shfl_xor_sync(0xffffffffu, s1, 2);
        } else {
          csr_off_h4x2(j, q, nr, W.rowptr + r0, W.col, W.val, x, s0, s1);
        }
        const float r = bi - (di * xi + ((q & 1) ? s1 : s0));
        const float y = i >= nr ? 0.f : kind == kResidual ? r : xi + (a.w * r) / di;
        if (!out) put(oth, j, y);
        else if (q < 2 && i < nr) a.x[r0 + i] = y;
      }
      if (kind == kSmooth) ++k;
      else res = 1;
    } else if (kind == kRestrict) {       // b = R r and the first sweep from it; a dense level: b itself
      const float *x = vec(oth), *d = vec(W.d);
      float *b = vec(W.b);
      const bool dense = a.cinv && lw == nl - 1;
      for (int s = warp; s * 16 < nr; s += kTailThreadsF / 32) {
        const int j = s * 16 + (lane >> 2) * 2, i = j + (q & 1);
        float s0, s1;
        if (in[2 * lw])
          csr_off_h4x2(j, q, nr, reinterpret_cast<const int *>(sm + W.R.rp), reinterpret_cast<const int *>(sm + W.R.cl),
                       vec(W.R.v), x, s0, s1, base[2 * lw]);
        else csr_off_h4x2(j, q, nr, W.rptr + r0, W.rcol, W.rval, x, s0, s1);
        float y = (q & 1) ? s1 : s0;
        if (i >= nr) y = 0.f;
        else {
          if (q < 2) b[i] = y;
          if (!dense) y = sw > 0 ? (a.w * y) / d[i] : 0.f;
        }
        put(W.v[0], j, y);
      }
      l = lw;
      k = res = 0;
    } else if (kind == kProlong) {        // x += P x of the level after
      const float *xc = vec(lv[l + 1].v[(a.cinv && l == nl - 2) || sw > 0]);   // 2 sw - 1 sweeps change buffers
      const int mk = 2 * l + 1, b0 = base[mk];
      const int *srp = reinterpret_cast<const int *>(sm + L.P.rp), *sc = reinterpret_cast<const int *>(sm + L.P.cl);
      float *x = vec(cur) + r0;
      for (int j = t; j < nr; j += kTailThreadsF) {
        const float s = in[mk] ? csr_row_from(0.f, srp[j] - b0, srp[j + 1] - b0, sc, vec(L.P.v), xc)
                               : csr_row_from(0.f, L.pptr[r0 + j], L.pptr[r0 + j + 1], L.pcol, L.pval, xc);
        const float y = x[j] + s;
#pragma unroll
        for (int w = 0; w < kTailBlocks; ++w) *cl.map_shared_rank(x + j, w) = y;
      }
      res = 0;
    } else {                              // dense: b whole in v[0], x to v[1]
      const int n = L.n, per = (n + kTailBlocks - 1) / kTailBlocks;
      const int d0 = min(n, rank * per), d1 = min(n, d0 + per);
      const float *b = vec(L.v[0]);
      for (int i = d0 + warp; i < d1; i += kTailThreadsF / 32) {
        const double *Ci = a.cinv + (size_t)i * n;
        double s = 0.0;
#pragma unroll 4
        for (int j = lane; j < n; j += 32) s += Ci[j] * (double)b[j];
#pragma unroll
        for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane < kTailBlocks) *cl.map_shared_rank(vec(L.v[1]) + i, lane) = (float)s;
      }
      up = true;
      res = 1;
      k = max(sw - 1, 0);
      --l;
    }
    if (out) break;
    cl.sync();
  }
  if (!out) {                             // no sweeps, or the dense level alone
    const TailLevelF &L = lv[0];
    const float *x = vec(L.v[dense0 || sw > 0]) + first_row(L);
    for (int j = t; j < own_rows(L); j += kTailThreadsF) a.x[first_row(L) + j] = x[j];
  }
}

__global__ void k_col0(int nnz, const int *offrow1, int *col0) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < nnz) col0[k] = offrow1[k] - 1;
}

// ---------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------
// Allocation of one hierarchy build: from the arena, else (arena full, or a test wants it) from
// the pool.
static bool in_arena(const msg_ctx *c, size_t bytes) {
  const AmgState *A = S(const_cast<msg_ctx *>(c));
  return A->arena && !c->hook[MSG_HOOK_AMG_ALLOC] && A->arena_used + A->arena_tmp + bytes <= A->arena_cap;
}
static int from_pool(msg_ctx *c, void **p, size_t bytes) {
  const bool armed = c->hook[MSG_HOOK_AMG_ALLOC] > 0, refuse = hook_due(c, MSG_HOOK_AMG_ALLOC);   // more than any device has
  MSG_CUDA(cudaMallocAsync(p, refuse ? (size_t)1 << 60 : bytes, c->stream));
  if (!armed) S(c)->arena_spill += bytes;
  return MSG_OK;
}
template <typename T>
static int halloc(msg_ctx *c, T **p, size_t n) {
  AmgState *A = S(c);
  const size_t bytes = ((n ? n : 1) * sizeof(T) + 255) & ~(size_t)255;
  if (in_arena(c, bytes)) {
    *p = reinterpret_cast<T *>(A->arena + A->arena_used);
    A->arena_used += bytes;
    return MSG_OK;
  }
  void *q = nullptr;
  int rc = from_pool(c, &q, bytes);
  if (!rc) *p = reinterpret_cast<T *>(q);
  return rc;
}

// Temporaries of one level's building, given back together (stream order: the next level's
// kernels may take the memory over).
struct Temps {
  static constexpr int kMax = 32;         // a level takes up to 27
  msg_ctx *c;
  void *pool[kMax];
  int n = 0;
  explicit Temps(msg_ctx *ctx) : c(ctx) {}
  ~Temps() {
    S(c)->arena_tmp = 0;
    for (int k = 0; k < n; ++k) cudaFreeAsync(pool[k], c->stream);
  }
  template <typename T>
  int get(T **p, size_t count) {
    AmgState *A = S(c);
    const size_t bytes = ((count ? count : 1) * sizeof(T) + 255) & ~(size_t)255;
    if (in_arena(c, bytes)) {
      A->arena_tmp += bytes;
      *p = reinterpret_cast<T *>(A->arena + A->arena_cap - A->arena_tmp);
      return MSG_OK;
    }
    if (n == kMax) { set_error("AMG build: more than %d temporaries", kMax); return MSG_ERR_STATE; }
    int rc = from_pool(c, &pool[n], bytes);
    if (!rc) *p = reinterpret_cast<T *>(pool[n++]);
    return rc;
  }
  // columns and values of n entries, together or not at all
  int entries(int **col, double **val, size_t count) {
    char *b = nullptr;
    const size_t v = (count * 8 + 255) & ~(size_t)255;
    int rc = get(&b, v + count * 4);
    if (!rc) { *val = reinterpret_cast<double *>(b); *col = reinterpret_cast<int *>(b + v); }
    return rc;
  }
};

// Release a pointer from halloc: arena memory is reclaimed at the next reset.
static void hfree(AmgState *A, void *q, cudaStream_t s) {
  if (!q) return;
  const char *b = reinterpret_cast<const char *>(q);
  if (A->arena && b >= A->arena && b < A->arena + A->arena_cap) return;
  cudaFreeAsync(q, s);
}

static void free_level(AmgState *A, AmgLevel &L, cudaStream_t s) {
  void *p[] = {L.rowptr, L.col, L.diag, L.val, L.pptr, L.pcol, L.pval, L.rptr, L.rcol, L.rval, L.agg, L.cinv,
               L.x, L.b, L.r, L.x2, L.diag_f, L.pval_f, L.rval_f, L.val_h, L.xf, L.bf, L.rf, L.x2f, L.pack};
  for (void *q : p) hfree(A, q, s);
  L = AmgLevel();
}

// A level on its way: given back unless it gets its place in the hierarchy.
struct NewLevel : AmgLevel {
  msg_ctx *c;
  explicit NewLevel(msg_ctx *ctx) : c(ctx) {}
  ~NewLevel() { free_level(S(c), *this, c->stream); }
  void keep() {
    S(c)->lv.push_back(*this);
    static_cast<AmgLevel &>(*this) = AmgLevel();
  }
};

template <typename T>
static int dalloc(msg_ctx *c, T **p, size_t n) {
  MSG_CUDA(cudaMallocAsync((void **)p, (n ? n : 1) * sizeof(T), c->stream));
  return MSG_OK;
}

// Places and memory of C's rows: of the products' size (their counts in g.cnt), or, when that is
// too much, of the size that `lengths` finds (into g.len).
template <typename F>
static int spgemm_places(msg_ctx *c, Temps &tmp, int n, Spg &g, F lengths) {
  int rc, got[1], *start = nullptr;
  long long total = 0;
  if ((rc = tmp.get(&start, n + 1)) || (rc = tmp.get(&g.len, n))) return rc;
  g.start = start;
  if ((rc = scan_exclusive(c, g.cnt, start, n, got, nullptr, nullptr, &total))) return rc;
  const long long most = c->hook[MSG_HOOK_AMG_PRODUCTS] > 0 ? c->hook[MSG_HOOK_AMG_PRODUCTS] : INT_MAX;
  if (total <= most && !tmp.entries(&g.ccol, &g.cval, total)) return MSG_OK;
  if ((rc = lengths()) || (rc = scan_exclusive(c, g.len, start, n, got))) return rc;
  return tmp.entries(&g.ccol, &g.cval, got[0]);
}

// C = A*B; long rows through the larger tables.  *ovf: device word set when a row has too many
// columns.
static int spgemm_rows(msg_ctx *c, Temps &tmp, int n, Spg &g, int *cnt, int *ovf) {
  cudaStream_t s = c->stream;
  int rc, *longrows = nullptr, *biggest = nullptr, *nl = nullptr;
  k_spg_bound<<<(8 * (long long)n + 255) / 256, 256, 0, s>>>(n, g, cnt);
  MSG_CHECK_LAUNCH();
  g.cnt = cnt;
  if ((rc = tmp.get(&longrows, n)) || (rc = tmp.get(&biggest, n)) || (rc = tmp.get(&nl, 2))) return rc;
  auto rows = [&]() -> int {
    MSG_CUDA(cudaMemsetAsync(nl, 0, 8, s));
    k_spg_row<kTabShort><<<(n + 3) / 4, 128, 0, s>>>(g, n, nullptr, nullptr, longrows, nl, nullptr);
    MSG_CHECK_LAUNCH();
    // the counts of the long rows stay on the device: grids that fill the chip walk them
    k_spg_row<kTabMid><<<std::min((n + 3) / 4, 12 * kNumSM), 128, 0, s>>>(g, n, nl, longrows, biggest, nl + 1, nullptr);
    MSG_CHECK_LAUNCH();
    k_spg_row<kTabMax><<<std::min((n + 2) / 3, 4 * kNumSM), 96, 0, s>>>(g, n, nl + 1, biggest, nullptr, nullptr, ovf);
    MSG_CHECK_LAUNCH();
    return MSG_OK;
  };
  if ((rc = spgemm_places(c, tmp, n, g, rows))) return rc;
  return rows();
}

// A pass over level 1 in blocks of 32 x `rows` cells of a layer; more launches where the rows or
// the layers are more than a grid has blocks in y or z.
template <typename F>
static int level1_tiles(const Bands &g, int rows, F launch) {
  constexpr int kMaxYZ = 65535;
  const int by = (g.ny + rows - 1) / rows;
  for (int z = 0; z < g.nz; z += kMaxYZ)
    for (int y = 0; y < by; y += kMaxYZ) {
      Bands part = g;
      part.y0 = y * rows;
      part.z0 = z;
      launch(dim3((g.nx + 31) / 32, std::min(by - y, kMaxYZ), std::min(g.nz - z, kMaxYZ)), dim3(32, rows), part);
      MSG_CHECK_LAUNCH();
    }
  return MSG_OK;
}

// Build level lv+1 from level lv; returns 1 when a coarser level was made, 0 otherwise.
static int coarsen(msg_ctx *c, AmgState *A, int lv, int *made) {
  *made = 0;
  const AmgLevel F = A->lv[lv];
  const int n = F.n, n8 = (int)((8 * (long long)n + 255) / 256);
  const bool dia = lv == 0;
  int rc, got[2];
  cudaStream_t s = c->stream;
  Temps tmp(c);
  const Bands g{c->nx, c->ny, c->nz, c->nxy, c->N, c->dmat, c->lu};
  const double th = (double)c->prm.amg_theta, th2 = th * th, om = (double)c->prm.jac_omega;
  unsigned char *msk = nullptr, *st = nullptr, *w1b = nullptr;
  int *scol = nullptr, *cnt = nullptr, *aggid = nullptr, *agg2 = nullptr, *words = nullptr;
  unsigned *w1 = nullptr;
  double *tdm = nullptr;
  if ((rc = tmp.get(&st, n + 3)) || (rc = tmp.get(&cnt, n)) || (rc = tmp.get(&aggid, n + 1)) || (rc = tmp.get(&agg2, n)) ||
      (rc = tmp.get(&words, kMisRounds + 3)))
    return rc;
  // too long: prolongation row, product row; rows beyond kPShort entries
  int *ovf_p = words + kMisRounds, *ovf = ovf_p + 1, *npl = ovf + 1, *prow = nullptr;
  MSG_CUDA(cudaMemsetAsync(words, 0, (kMisRounds + 3) * 4, s));
  // strength and aggregates
  if (dia) {
    if ((rc = tmp.get(&msk, n + 3)) || (rc = tmp.get(&w1b, n + 3))) return rc;
    if ((rc = level1_tiles(g, 8, [&](dim3 tg, dim3 tb, const Bands &part) { k_strength_dia<<<tg, tb, 0, s>>>(part, th2, msk, st); }))) return rc;
  } else {
    if ((rc = tmp.get(&scol, F.nnz)) || (rc = tmp.get(&w1, n)) || (rc = tmp.get(&tdm, n)) || (rc = tmp.get(&prow, n)))
      return rc;
    k_strength_csr<<<(n + 3) / 4, 128, 0, s>>>(n, F.rowptr, F.col, F.val, F.diag, th2, scol, st, tdm);
    MSG_CHECK_LAUNCH();
  }
  {
    int l = lv;
    Bands gb = g;
    if (dia) {
      void *args[] = {&gb, &msk, &st, &w1b, &l, &words};
      MSG_CUDA(cudaLaunchCooperativeKernel((void *)k_mis_dia, std::min((n + 4 * kMisBlock - 1) / (4 * kMisBlock), A->mis_dia), kMisBlock, args, 0, s));
    } else {
      int nn = n, *rp = F.rowptr;
      void *args[] = {&nn, &rp, &scol, &st, &w1, &l, &words};
      if (n <= kMisSmall) {
        cudaLaunchAttribute at;
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = kMisCluster; at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cudaLaunchConfig_t cf = {};
        cf.gridDim = dim3(kMisCluster); cf.blockDim = dim3(kMisBlock); cf.stream = s; cf.attrs = &at; cf.numAttrs = 1;
        MSG_CUDA(cudaLaunchKernelExC(&cf, (const void *)k_mis_csr<true>, args));
      } else {
        const int g = (int)std::min((4 * (long long)n + kMisBlock - 1) / kMisBlock, (long long)A->mis_csr);
        MSG_CUDA(cudaLaunchCooperativeKernel((void *)k_mis_csr<false>, g, kMisBlock, args, 0, s));
      }
    }
    __atomic_fetch_add(&g_launches, 1LL, __ATOMIC_RELAXED);
  }
  k_root_flag<<<nb(n), kThreads, 0, s>>>(n, st, cnt);
  MSG_CHECK_LAUNCH();
  if ((rc = scan_exclusive(c, cnt, aggid, n, got))) return rc;
  const int nc = got[0];
  if (nc == 0 || nc >= n) return MSG_OK;
  NewLevel C(c);
  C.n = nc;
  if ((rc = halloc(c, &C.agg, n))) return rc;
  if (dia) {
    k_agg_a_dia<<<nb(n), kThreads, 0, s>>>(g, msk, st, aggid, agg2, lv);
    MSG_CHECK_LAUNCH();
    k_agg_b_dia<<<nb(n), kThreads, 0, s>>>(g, msk, agg2, C.agg, lv);
  } else {
    k_agg_csr<true><<<n8, 256, 0, s>>>(n, F.rowptr, scol, st, aggid, agg2, lv);
    MSG_CHECK_LAUNCH();
    k_agg_csr<false><<<n8, 256, 0, s>>>(n, F.rowptr, scol, st, agg2, C.agg, lv);
  }
  MSG_CHECK_LAUNCH();
  // P
  auto p_rows = [&](auto fill, int *rcnt) -> int {
    constexpr bool FILL = decltype(fill)::value;
    k_p_csr<FILL, false><<<(n + 3) / 4, 128, 0, s>>>(n, F.rowptr, scol, F.val, C.agg, tdm, om, cnt, ovf_p, prow, npl,
                                                    C.pptr, C.pcol, C.pval, rcnt);
    MSG_CHECK_LAUNCH();
    k_p_csr<FILL, true><<<std::min((n + 3) / 4, 2 * kNumSM), 128, 0, s>>>(n, F.rowptr, scol, F.val, C.agg, tdm, om, cnt,
                                                                         ovf_p, prow, npl, C.pptr, C.pcol, C.pval, rcnt);
    return MSG_OK;
  };
  if (dia) k_p_dia<false><<<nb(n), kThreads, 0, s>>>(g, msk, C.agg, om, cnt, nullptr, nullptr, nullptr, nullptr);
  else if ((rc = p_rows(std::false_type(), nullptr))) return rc;
  MSG_CHECK_LAUNCH();
  if ((rc = halloc(c, &C.pptr, n + 1))) return rc;
  if ((rc = scan_exclusive(c, cnt, C.pptr, n, got, ovf_p))) return rc;
  if (got[1]) return MSG_OK;              // a row beyond kPRowMax
  const int pnnz = got[0];
  C.pnnz = pnnz;
  if ((rc = halloc(c, &C.pcol, pnnz)) || (rc = halloc(c, &C.pval, pnnz))) return rc;
  int *rcnt = nullptr;
  if ((rc = tmp.get(&rcnt, nc))) return rc;
  MSG_CUDA(cudaMemsetAsync(rcnt, 0, (size_t)nc * 4, s));
  if (dia) k_p_dia<true><<<nb(n), kThreads, 0, s>>>(g, msk, C.agg, om, nullptr, C.pptr, C.pcol, C.pval, rcnt);
  else if ((rc = p_rows(std::true_type(), rcnt))) return rc;
  MSG_CHECK_LAUNCH();
  // R = P^T
  if ((rc = halloc(c, &C.rptr, nc + 1))) return rc;
  if ((rc = scan_exclusive(c, rcnt, C.rptr, nc, nullptr))) return rc;
  if ((rc = halloc(c, &C.rcol, pnnz)) || (rc = halloc(c, &C.rval, pnnz))) return rc;
  MSG_CUDA(cudaMemsetAsync(rcnt, 0, (size_t)nc * 4, s));
  int *trow = nullptr, *tcol = nullptr;
  double *tval = nullptr;
  if ((rc = tmp.get(&trow, pnnz)) || (rc = tmp.get(&tcol, pnnz)) || (rc = tmp.get(&tval, pnnz))) return rc;
  if (c->prm.precision == 1 && ((rc = halloc(c, &C.pval_f, pnnz)) || (rc = halloc(c, &C.rval_f, pnnz)))) return rc;
  k_r_fill<<<nb(n), kThreads, 0, s>>>(n, C.pptr, C.pcol, C.pval, C.rptr, rcnt, trow, tcol, tval);
  MSG_CHECK_LAUNCH();
  k_r_rank<<<nb(pnnz), kThreads, 0, s>>>(pnnz, C.rptr, trow, tcol, tval, C.rcol, C.rval, C.rval_f);
  MSG_CHECK_LAUNCH();
  // AP = A*P (diagonal first)
  Spg ap{F.rowptr, F.col, F.val, F.diag, C.pptr, nullptr, C.pcol, C.pval, 0};
  if (dia) {
    if ((rc = level1_tiles(g, 8, [&](dim3 tg, dim3 tb, const Bands &part) { k_ap_bound_dia<<<tg, tb, 0, s>>>(part, C.pptr, cnt); }))) return rc;
    ap.cnt = cnt;
    auto rows = [&](auto count) -> int {
      return level1_tiles(g, kApT / 32, [&](dim3 tg, dim3 tb, const Bands &part) {
        k_ap_dia<decltype(count)::value><<<tg, tb, 0, s>>>(part, C.pptr, C.pcol, C.pval, ap.start, ap.len, ap.ccol, ap.cval);
      });
    };
    if ((rc = spgemm_places(c, tmp, n, ap, [&] { return rows(std::true_type()); })) || (rc = rows(std::false_type()))) return rc;
  } else if ((rc = spgemm_rows(c, tmp, n, ap, cnt, ovf))) {
    return rc;
  }
  // A_c = R * AP, diagonal split off
  if ((rc = halloc(c, &C.diag, nc)) || (rc = halloc(c, &C.rowptr, nc + 1))) return rc;
  Spg ra{C.rptr, C.rcol, C.rval, nullptr, ap.start, ap.len, ap.ccol, ap.cval, 1};
  ra.cdiag = C.diag;
  if ((rc = spgemm_rows(c, tmp, nc, ra, cnt, ovf))) return rc;
  if ((rc = scan_exclusive(c, ra.len, C.rowptr, nc, got, ovf))) return rc;
  if (got[1]) return MSG_OK;              // a row beyond kHashMax
  C.nnz = got[0];
  if ((rc = halloc(c, &C.col, C.nnz)) || (rc = halloc(c, &C.val, C.nnz))) return rc;
  if (c->prm.precision == 1) {
    if ((rc = halloc(c, &C.val_h, C.nnz)) || (rc = halloc(c, &C.diag_f, nc)) || (rc = halloc(c, &C.xf, nc)) ||
        (rc = halloc(c, &C.bf, nc)) || (rc = halloc(c, &C.rf, nc)) || (rc = halloc(c, &C.x2f, nc)))
      return rc;
    k_d2f<<<std::max(1, std::min(nb(pnnz), kRedBlocks * 4)), kThreads, 0, s>>>(pnnz, C.pval, C.pval_f);
    MSG_CHECK_LAUNCH();
  } else if ((rc = halloc(c, &C.x, nc)) || (rc = halloc(c, &C.b, nc)) || (rc = halloc(c, &C.r, nc)) ||
             (rc = halloc(c, &C.x2, nc))) {
    return rc;
  }
  k_spg_pack<<<(8 * (long long)nc + 255) / 256, 256, 0, s>>>(nc, ra.start, C.rowptr, ra.ccol, ra.cval, C.diag, C.col,
                                                            C.val, C.val_h, C.diag_f);
  MSG_CHECK_LAUNCH();
  C.keep();
  *made = 1;
  return MSG_OK;
}

static int dense_inverse(msg_ctx *c, AmgLevel &L) {
  int n = L.n, rc;
  cudaStream_t s = c->stream;
  double *M = nullptr;
  int *piv = nullptr;
  if (n <= kGjReg) {
    if ((rc = halloc(c, &L.cinv, (size_t)n * n))) return rc;
    return launch_gj_reg(n, L.rowptr, L.col, L.val, L.diag, nullptr, L.cinv, s);
  }
  Temps tmp(c);
  if ((rc = tmp.get(&M, (size_t)n * 2 * n)) || (rc = tmp.get(&piv, 1))) return rc;
  if ((rc = halloc(c, &L.cinv, (size_t)n * n))) return rc;
  k_dense_fill<<<n, 256, 0, s>>>(n, L.rowptr, L.col, L.val, L.diag, M);
  MSG_CHECK_LAUNCH();
  if (n <= 1024) {
    // one block: __syncthreads between the phases of a pivot step
    k_gj<false, 1024><<<1, 1024, 0, s>>>(n, M, piv);
    MSG_CHECK_LAUNCH();
  } else {
    int per_sm = 0, sms = 0;
    MSG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_gj<true, 256>, 256, 0));
    MSG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device));
    int grid = std::max(1, std::min(sms * std::max(per_sm, 1), (n * 2 * n + 255) / 256));
    void *args[] = {&n, &M, &piv};
    MSG_CUDA(cudaLaunchCooperativeKernel((void *)k_gj<true, 256>, grid, 256, args, 0, s));
    __atomic_fetch_add(&g_launches, 1LL, __ATOMIC_RELAXED);
  }
  k_dense_extract<<<n, 256, 0, s>>>(n, M, L.cinv);
  MSG_CHECK_LAUNCH();
  return MSG_OK;
}

void amg_free(msg_ctx *c) {
  AmgState *A = S(c);
  if (!A) return;
  cudaStream_t s = c->stream;
  for (size_t l = 1; l < A->lv.size(); ++l) free_level(A, A->lv[l], s);
  A->lv.clear();
  void *p[] = {A->col0, A->r0, A->t0, A->x0f, A->t0f, A->r0f, A->b0f};
  for (void *q : p) if (q) cudaFreeAsync(q, s);
  cudaStreamSynchronize(s);
  if (A->arena) cudaFree(A->arena);
  delete A;
  c->amg = nullptr;
}

// Per-cell bytes of the arena reserved when a context is made: a build of the block and
// ensemble workloads takes 150 to 200 B per fine cell at its peak, the first coarsening
// (levels and transfer operators end at 55 to 80); a build that outgrows the reservation
// spills to the pool and the arena is enlarged at the next build.
constexpr size_t kArenaPerCell = 288;

static int amg_state(msg_ctx *c);

// Reserve the hierarchy's arena while the context is made, so that the first rebuilds of a
// run allocate nothing: a multi-GB cudaMalloc inside a later rebuild took 50-150 ms more on
// some machines than on others.
int amg_reserve(msg_ctx *c) {
  int rc;
  if ((rc = amg_state(c))) return rc;
  AmgState *A = S(c);
  if (A->arena) return MSG_OK;
  const size_t cap = (kArenaPerCell * (size_t)c->N + ((size_t)1 << 20) - 1) & ~(((size_t)1 << 20) - 1);
  if (cudaMalloc((void **)&A->arena, cap) == cudaSuccess) A->arena_cap = cap;
  else { A->arena = nullptr; A->arena_cap = 0; cudaGetLastError(); }   // the builds use the pool
  return MSG_OK;
}

static int amg_state(msg_ctx *c) {
  int rc;
  AmgState *A = S(c);
  cudaStream_t s = c->stream;
  if (!A) {
    A = new AmgState();
    c->amg = A;
    if ((rc = dalloc(c, &A->col0, c->nnz))) return rc;
    if ((rc = dalloc(c, &A->r0, c->N))) return rc;
    if ((rc = dalloc(c, &A->t0, c->N))) return rc;
    if (c->prm.precision == 1) {
      if ((rc = dalloc(c, &A->x0f, c->N))) return rc;
      if ((rc = dalloc(c, &A->t0f, c->N))) return rc;
      if ((rc = dalloc(c, &A->r0f, c->N))) return rc;
      if ((rc = dalloc(c, &A->b0f, c->N))) return rc;
    }
    int sms = 0, per = 0;
    MSG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device));
    MSG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_mis_dia, kMisBlock, 0));
    A->mis_dia = sms * std::max(per, 1);
    MSG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_mis_csr<false>, kMisBlock, 0));
    A->mis_csr = sms * std::max(per, 1);
    k_col0<<<nb(c->nnz), kThreads, 0, s>>>(c->nnz, c->offrow, A->col0);
    MSG_CHECK_LAUNCH();
  }
  return MSG_OK;
}

template <typename K, typename Args>
static int tail_launch(msg_ctx *c, K kernel, const Args &a, int threads, int shared) {
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = kTailBlocks; at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cudaLaunchConfig_t cf = {};
  cf.gridDim = dim3(kTailBlocks); cf.blockDim = dim3(threads); cf.dynamicSmemBytes = shared;
  cf.stream = c->stream; cf.attrs = &at; cf.numAttrs = 1;
  MSG_CUDA(cudaLaunchKernelEx(&cf, kernel, a));
  __atomic_fetch_add(&g_launches, 1LL, __ATOMIC_RELAXED);
  return MSG_OK;
}
// Levels l .. of a V-cycle from their right-hand side to their correction, when they are
// small; *done is left 0 when they are not.
static bool tail_takes(const AmgState *A, int l) {
  return A->lv[l].n <= kTailRows && (int)A->lv.size() - l <= kTailMax && A->lv.back().n <= kTailDense;
}
// Lays the small levels out for k_cycle_tail_f at the end of a build.
static int tail_setup(msg_ctx *c) {
  AmgState *A = S(c);
  int l = 1, rc;
  while (l < (int)A->lv.size() && !tail_takes(A, l)) ++l;
  if (c->prm.precision != 1 || l >= (int)A->lv.size()) return MSG_OK;
  TailArgsF &a = A->tail;
  const int nl = a.nl = (int)A->lv.size() - l;
  a.cinv = A->lv.back().cinv;
  a.b = A->lv[l].bf;
  a.x = A->lv[l].xf;
  int used = 0, slices = 0;
  auto place = [&](size_t bytes) {
    const int o = used;
    used += (int)((bytes + 15) & ~(size_t)15);
    return o;
  };
  size_t words = 0;
  for (int k = 0; k < nl; ++k) {
    const AmgLevel &L = A->lv[l + k], *N = k + 1 < nl ? &A->lv[l + k + 1] : nullptr;
    const bool dense = a.cinv && !N;
    TailLevelF &q = a.lv[k];
    q.n = L.n;
    q.per = ((L.n + kTailBlocks - 1) / kTailBlocks + 3) & ~3;
    q.rowptr = dense ? nullptr : L.rowptr; q.col = L.col; q.val = L.val_h; q.diag = L.diag_f;
    q.rptr = L.rptr; q.rcol = L.rcol; q.rval = L.rval_f;
    q.pptr = N ? N->pptr : nullptr; q.pcol = N ? N->pcol : nullptr; q.pval = N ? N->pval_f : nullptr;
    for (int v = 0; v < 2; ++v) q.v[v] = place(((size_t)L.n + 2) * 4);
    q.b = place((size_t)q.per * 4);
    q.d = place((size_t)q.per * 4);
    slices += (q.per + 15) / 16;
    // a slice's rows are padded to its longest and blocks differ: 2.2 words per entry
    if (!dense) words += (size_t)L.nnz / kTailBlocks * 11 / 5 + 512;
  }
  if (used > kTailShared || slices > kTailSlices) return MSG_OK;
  a.words = (int)std::min(words, (size_t)(kTailShared - used) / 4) & ~3;
  a.pool = place((size_t)a.words * 4);
  // transfers while there is room: an even share of the entries and half as many
  auto hold = [&](TailMatF &m, int per, int nnz) {
    const int cap = (nnz / kTailBlocks / 2 * 3 + 64 + 7) & ~7, before = used;
    m.rp = place((size_t)(per + 1) * 4);
    m.cl = place((size_t)cap * 4);
    m.v = place((size_t)cap * 4);
    m.cap = used <= kTailShared ? cap : 0;
    if (!m.cap) used = before;
  };
  for (int k = 0; k < nl; ++k) {
    a.lv[k].R.cap = a.lv[k].P.cap = 0;
    if (k > 0) hold(a.lv[k].R, a.lv[k].per, A->lv[l + k].pnnz);
    if (k + 1 < nl) hold(a.lv[k].P, a.lv[k].per, A->lv[l + k + 1].pnnz);
  }
  a.shared = used;
  char *pack = nullptr;
  if ((rc = halloc(c, &pack, kTailBlocks * (sizeof(TailHead) + (size_t)a.words * 4)))) return rc;
  A->lv[l].pack = pack;
  a.head = reinterpret_cast<TailHead *>(pack);
  a.slices = reinterpret_cast<uint32_t *>(pack + kTailBlocks * sizeof(TailHead));
  if (!A->tail_set) {
    MSG_CUDA(cudaFuncSetAttribute(k_cycle_tail_f, cudaFuncAttributeMaxDynamicSharedMemorySize, kTailShared));
    A->tail_set = true;
  }
  k_tail_pack<<<kTailBlocks, kTailThreads, 0, c->stream>>>(a);
  MSG_CHECK_LAUNCH();
  A->tail_level = l;
  return MSG_OK;
}

static void drop_levels(msg_ctx *c) {
  AmgState *A = S(c);
  for (size_t l = 1; l < A->lv.size(); ++l) free_level(A, A->lv[l], c->stream);
  A->lv.clear();
  A->tail_level = -1;
  c->amg_nlevel = 0;
}

static int build_levels(msg_ctx *c) {
  int rc;
  AmgState *A = S(c);
  cudaStream_t s = c->stream;
  // reset the arena; enlarge it first when the previous build did not fit
  if (A->arena_spill) {
    const size_t need = A->arena_cap + A->arena_spill;   // what did not fit beside a full arena
    if (A->arena) {
      MSG_CUDA(cudaStreamSynchronize(s));
      cudaFree(A->arena);
      A->arena = nullptr;
      A->arena_cap = 0;
    }
    const size_t cap = ((need + need / 4) + ((size_t)1 << 20) - 1) & ~(((size_t)1 << 20) - 1);
    if (cudaMalloc((void **)&A->arena, cap) == cudaSuccess) A->arena_cap = cap;
    else { A->arena = nullptr; cudaGetLastError(); }   // keep using the pool
  }
  A->arena_used = A->arena_tmp = 0;
  A->arena_spill = 0;
  AmgLevel L0;
  L0.n = c->N; L0.nnz = c->nnz; L0.rowptr = c->offind; L0.col = A->col0; L0.diag = c->dmat;
  A->lv.push_back(L0);
  int maxlev = std::min(std::max(c->prm.amg_nlevel, 2), 16);
  while ((int)A->lv.size() < maxlev && A->lv.back().n > c->prm.amg_coarse_max) {
    int made = 0;
    if ((rc = coarsen(c, A, (int)A->lv.size() - 1, &made))) return rc;
    if (!made) break;
  }
  if (A->lv.size() > 1 && A->lv.back().n <= std::max(c->prm.amg_coarse_max, 1)) {
    if ((rc = dense_inverse(c, A->lv.back()))) return rc;
  }
  return tail_setup(c);
}

// A build that fails leaves no hierarchy: amg_apply refuses to run and the next assembly builds
// again, whatever amg_lag says.
int amg_setup(msg_ctx *c) {
  int rc;
  if ((rc = amg_state(c))) return rc;
  drop_levels(c);
  if ((rc = build_levels(c))) drop_levels(c);
  else c->amg_nlevel = (int)S(c)->lv.size();
  return rc;
}

static int cycle_tail(msg_ctx *c, int l, int *done) {
  AmgState *A = S(c);
  *done = 0;
  if (c->hook[MSG_HOOK_CYCLE_LAUNCHES] || !tail_takes(A, l)) return MSG_OK;
  TailArgs a;
  a.nl = (int)A->lv.size() - l;
  a.sweeps = std::max(c->prm.amg_sweeps, 0);
  a.w = (double)c->prm.smooth_omega;
  a.cinv = A->lv.back().cinv;
  for (int k = 0; k < a.nl; ++k) {
    const AmgLevel &L = A->lv[l + k];
    a.lv[k] = {L.n, L.rowptr, L.col, L.val, L.diag, L.rptr, L.rcol, L.pptr, L.pcol, L.rval, L.pval, L.x, L.b, L.r, L.x2};
  }
  *done = 1;
  return tail_launch(c, k_cycle_tail, a, kTailThreads, 0);
}
static int cycle_tail_f(msg_ctx *c, int l, int *done) {
  AmgState *A = S(c);
  *done = l == A->tail_level && !c->hook[MSG_HOOK_CYCLE_LAUNCHES];
  if (!*done) return MSG_OK;
  A->tail.sweeps = std::max(c->prm.amg_sweeps, 0);
  A->tail.w = c->prm.smooth_omega;
  return tail_launch(c, k_cycle_tail_f, A->tail, kTailThreadsF, A->tail.shared);
}

// One V-cycle z = M^-1 r (x = 0 start, amg_sweeps Jacobi sweeps before and after).
static int vcycle(msg_ctx *c, int l, const double *b, double *x) {
  AmgState *A = S(c);
  AmgLevel &L = A->lv[l];
  cudaStream_t s = c->stream;
  const int n = L.n, sw = std::max(c->prm.amg_sweeps, 0);
  const double w = (double)c->prm.smooth_omega;
  const int g = nb(n);
  const bool last = (l == (int)A->lv.size() - 1);
  if (l > 0) {
    int done = 0, rc = cycle_tail(c, l, &done);
    if (rc || done) return rc;
  }
  if (last && L.cinv) {
    k_gemv<<<nb(n), kThreads, 0, s>>>(n, L.cinv, b, x);
    MSG_CHECK_LAUNCH();
    return MSG_OK;
  }
  Dia D{c->nx, c->ny, c->nz, c->nxy, c->N, c->dmat, c->lu};
  const int bs = (l == 0 && c->blk_smooth > 0) ? c->blk_smooth : kThreads;
  const int gs = (n + bs - 1) / bs;
  double *r = (l == 0) ? A->r0 : L.r;
  double *tmp = (l == 0) ? A->t0 : L.x2;
  auto sweep = [&](const double *xin, double *xout) {
    if (l == 0) k_jac_dia<<<gs, bs, 0, s>>>(D, b, w, xin, xout);
    else k_jac_csr<<<g, kThreads, 0, s>>>(n, L.rowptr, L.col, L.val, L.diag, b, w, xin, xout);
  };
  // pre-smoothing: the current iterate alternates between x and tmp, so that every
  // sweep reads one buffer and writes the other; total sweeps 2*sw end in x.
  double *cur = x, *oth = tmp;
  if (sw == 0) {
    MSG_CUDA(cudaMemsetAsync(x, 0, (size_t)n * 8, s));
  } else {
    if (sw % 2 == 0) { cur = tmp; oth = x; }
    k_jac_first<<<gs, bs, 0, s>>>(n, b, l == 0 ? c->dmat : L.diag, w, cur);
    MSG_CHECK_LAUNCH();
    for (int k = 1; k < sw; ++k) {
      sweep(cur, oth);
      MSG_CHECK_LAUNCH();
      std::swap(cur, oth);
    }
  }
  if (!last) {
    AmgLevel &C = A->lv[l + 1];
    if (l == 0) k_res_dia<<<gs, bs, 0, s>>>(D, b, cur, r);
    else k_res_csr<<<g, kThreads, 0, s>>>(n, L.rowptr, L.col, L.val, L.diag, b, cur, r);
    MSG_CHECK_LAUNCH();
    k_restrict<<<std::min(nb(C.n), kRedBlocks * 4), kThreads, 0, s>>>(C.n, C.rptr, C.rcol, C.rval, r, C.b);
    MSG_CHECK_LAUNCH();
    int rc = vcycle(c, l + 1, C.b, C.x);
    if (rc) return rc;
    k_prolong<<<gs, bs, 0, s>>>(n, C.pptr, C.pcol, C.pval, C.x, cur);
    MSG_CHECK_LAUNCH();
  }
  for (int k = 0; k < sw; ++k) {
    sweep(cur, oth);
    MSG_CHECK_LAUNCH();
    std::swap(cur, oth);
  }
  if (cur != x) MSG_CUDA(cudaMemcpyAsync(x, cur, (size_t)n * 8, cudaMemcpyDeviceToDevice, s));
  return MSG_OK;
}


// Mixed-precision V-cycle on levels >= 1 (float vectors).
static int vcycle_f(msg_ctx *c, int l, const float *b, float *x) {
  AmgState *A = S(c);
  AmgLevel &L = A->lv[l];
  cudaStream_t s = c->stream;
  const int n = L.n, sw = std::max(c->prm.amg_sweeps, 0);
  const float w = c->prm.smooth_omega;
  const int g = nb(n);
  const bool last = (l == (int)A->lv.size() - 1);
  {
    int done = 0, rc = cycle_tail_f(c, l, &done);
    if (rc || done) return rc;
  }
  if (last && L.cinv) {
    k_gemv_mixed<<<(int)(((long long)n * 32 + kThreads - 1) / kThreads), kThreads, 0, s>>>(n, L.cinv, b, x);
    MSG_CHECK_LAUNCH();
    return MSG_OK;
  }
  float *cur = x, *oth = L.x2f;
  if (sw == 0) {
    MSG_CUDA(cudaMemsetAsync(x, 0, (size_t)n * 4, s));
  } else {
    if (sw % 2 == 0) { cur = L.x2f; oth = x; }
    k_jac_first_f<float><<<g, kThreads, 0, s>>>(n, b, L.diag_f, w, cur);
    MSG_CHECK_LAUNCH();
    for (int k = 1; k < sw; ++k) {
      csr_pass<kCsrJacobi>(n, L.nnz, L.rowptr, L.col, L.val_h, L.diag_f, b, w, cur, oth, s);
      MSG_CHECK_LAUNCH();
      std::swap(cur, oth);
    }
  }
  if (!last) {
    AmgLevel &C = A->lv[l + 1];
    csr_pass<kCsrResidual>(n, L.nnz, L.rowptr, L.col, L.val_h, L.diag_f, b, 0.f, cur, L.rf, s);
    MSG_CHECK_LAUNCH();
    csr_pass<kCsrRowSum>(C.n, C.pnnz, C.rptr, C.rcol, C.rval_f, nullptr, nullptr, 0.f, L.rf, C.bf, s);
    MSG_CHECK_LAUNCH();
    int rc = vcycle_f(c, l + 1, C.bf, C.xf);
    if (rc) return rc;
    csr_pass<kCsrAddTo>(n, C.pnnz, C.pptr, C.pcol, C.pval_f, nullptr, nullptr, 0.f, C.xf, cur, s);
    MSG_CHECK_LAUNCH();
  }
  for (int k = 0; k < sw; ++k) {
    csr_pass<kCsrJacobi>(n, L.nnz, L.rowptr, L.col, L.val_h, L.diag_f, b, w, cur, oth, s);
    MSG_CHECK_LAUNCH();
    std::swap(cur, oth);
  }
  if (cur != x) MSG_CUDA(cudaMemcpyAsync(x, cur, (size_t)n * 4, cudaMemcpyDeviceToDevice, s));
  return MSG_OK;
}

// Level 1 of the mixed V-cycle: r (FP64 Krylov vector) in, z (FP64) out.
static int vcycle_mixed(msg_ctx *c, const double *b, double *z) {
  AmgState *A = S(c);
  cudaStream_t s = c->stream;
  const int n = c->N, sw = std::max(c->prm.amg_sweeps, 0);
  const float w = c->prm.smooth_omega;
  Dia32 D{c->nx, c->ny, c->nz, c->nxy, c->N, c->dmat_f, c->lu_f};
  const bool single = (A->lv.size() == 1);
  const int bs = c->blk_smooth > 0 ? c->blk_smooth : kThreads;
  const int gs = (n + bs - 1) / bs;
  // stencil sweeps: 3D grid, 32 cells of a row per warp, bs / 32 rows per block
  const int by = std::max(bs / 32, 1);
  const dim3 b3(32, by), g3((c->nx + 31) / 32, (c->ny + by - 1) / by, c->nz);
  float *cur = A->x0f, *oth = A->t0f, *bf = A->b0f;
  if (sw == 0) {
    MSG_CUDA(cudaMemsetAsync(cur, 0, (size_t)n * 4, s));
    k_b2f<<<gs, bs, 0, s>>>(n, b, bf);
    MSG_CHECK_LAUNCH();
  } else {
    k_jac_first_b<<<grid4(n, bs), bs, 0, s>>>(n, b, c->dmat_f, w, cur, bf);
    MSG_CHECK_LAUNCH();
    for (int k = 1; k < sw; ++k) {
      k_jac_dia3<float><<<g3, b3, 0, s>>>(D, bf, w, cur, oth);
      MSG_CHECK_LAUNCH();
      std::swap(cur, oth);
    }
  }
  if (!single) {
    AmgLevel &C = A->lv[1];
    k_res_dia3<<<g3, b3, 0, s>>>(D, bf, cur, A->r0f);
    MSG_CHECK_LAUNCH();
    csr_pass<kCsrRowSum>(C.n, C.pnnz, C.rptr, C.rcol, C.rval_f, nullptr, nullptr, 0.f, A->r0f, C.bf, s);
    MSG_CHECK_LAUNCH();
    int rc = vcycle_f(c, 1, C.bf, C.xf);
    if (rc) return rc;
    csr_pass<kCsrAddTo>(n, C.pnnz, C.pptr, C.pcol, C.pval_f, nullptr, nullptr, 0.f, C.xf, cur, s);
    MSG_CHECK_LAUNCH();
  }
  for (int k = 0; k < sw; ++k) {
    if (k == sw - 1) {   // the last sweep writes the FP64 output
      k_jac_dia3<double><<<g3, b3, 0, s>>>(D, bf, w, cur, z);
      MSG_CHECK_LAUNCH();
      return MSG_OK;
    }
    k_jac_dia3<float><<<g3, b3, 0, s>>>(D, bf, w, cur, oth);
    MSG_CHECK_LAUNCH();
    std::swap(cur, oth);
  }
  k_f2d<<<gs, bs, 0, s>>>(n, cur, z);
  MSG_CHECK_LAUNCH();
  return MSG_OK;
}

int amg_apply(msg_ctx *c, const double *r, double *z) {
  if (!S(c) || S(c)->lv.empty()) { set_error("AMG hierarchy not built"); return MSG_ERR_STATE; }
  if (c->prm.precision == 1) return vcycle_mixed(c, r, z);
  return vcycle(c, 0, r, z);
}

}  // namespace msg


// ---------------------------------------------------------------------------------
// Allocation-free dense inverse.
//
// Some callers cannot call cudaMalloc: a Fortran host that hands over device arrays it
// already owns (CUDA Fortran or OpenACC data regions) while its own allocator holds the
// device heap, or a solver step that runs under a fixed device-memory budget where an
// allocation could fail or stall mid-step.  msg_gpu_dense_inverse_noalloc serves them:
// it takes the caller's device buffers and keeps its Gauss-Jordan workspace (the
// augmented [A | I] block and the pivot slot) in the file-scope array below, sized for
// n <= kNoAllocMaxN.  Every GPU that loads this library holds that array (about 4 MiB)
// until the process exits.
// ---------------------------------------------------------------------------------
constexpr int kNoAllocMaxN = 512;
static __device__ __align__(256) double g_noalloc_gj[(size_t)2 * kNoAllocMaxN * kNoAllocMaxN + 32];

// In host code g_noalloc_gj names a host-side stand-in, not device memory: the device
// address comes from cudaGetSymbolAddress with the caller's device current.  It is looked
// up again on every call rather than cached: after a cudaDeviceReset the runtime builds a
// new primary context and reloads this module, and the array may then sit elsewhere, so
// an address kept from before the reset would point into freed memory.  The lookup is a
// host-side table search (the module is loaded by the first call), far cheaper than the
// three kernels it precedes.
static int noalloc_scratch(double **out) {
  void *p = nullptr;
  cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_gj);
  if (e != cudaSuccess || !p) {
    ::msg::set_error("dense_inverse_noalloc: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
    return MSG_ERR_CUDA;
  }
  *out = static_cast<double *>(p);
  return MSG_OK;
}

// Hierarchy export for structural tests (levels are 0-based; level 0 is the Jacobian).
using namespace msg;
extern "C" {
// Dense FP64 inverse by Gauss-Jordan with partial pivoting: the coarsest-level
// solve of the AMG V-cycle, on host arrays (row-major n x n).
MSG_API int msg_gpu_dense_inverse(int32_t n, const double *a, double *inv) {
  if (n < 1 || !a || !inv) { set_error("dense_inverse: bad arguments"); return MSG_ERR_ARG; }
  double *da = nullptr, *M = nullptr, *dinv = nullptr;
  int *piv = nullptr;
  const size_t nn = (size_t)n * n;
  MSG_CUDA(cudaMalloc(&da, nn * 8));
  if (n <= kGjReg) {
    MSG_CUDA(cudaMalloc(&dinv, nn * 8));
    MSG_CUDA(cudaMemcpy(da, a, nn * 8, cudaMemcpyHostToDevice));
    int rc = launch_gj_reg(n, nullptr, nullptr, nullptr, nullptr, da, dinv, 0);
    if (!rc) MSG_CUDA(cudaMemcpy(inv, dinv, nn * 8, cudaMemcpyDeviceToHost));
    cudaFree(da); cudaFree(dinv);
    return rc;
  }
  MSG_CUDA(cudaMalloc(&M, 2 * nn * 8));
  MSG_CUDA(cudaMalloc(&dinv, nn * 8));
  MSG_CUDA(cudaMalloc(&piv, 4));
  MSG_CUDA(cudaMemcpy(da, a, nn * 8, cudaMemcpyHostToDevice));
  k_dense_fill_rm<<<n, 256>>>(n, da, M);
  MSG_CHECK_LAUNCH();
  if (n <= 1024) {
    k_gj<false, 1024><<<1, 1024>>>(n, M, piv);
    MSG_CHECK_LAUNCH();
  } else {
    int dev = 0, per_sm = 0, sms = 0;
    MSG_CUDA(cudaGetDevice(&dev));
    MSG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_gj<true, 256>, 256, 0));
    MSG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    int grid = std::max(1, std::min(sms * std::max(per_sm, 1), (int)((2 * nn + 255) / 256)));
    int nn32 = n;
    void *args[] = {&nn32, &M, &piv};
    MSG_CUDA(cudaLaunchCooperativeKernel((void *)k_gj<true, 256>, grid, 256, args, 0, 0));
    __atomic_fetch_add(&g_launches, 1LL, __ATOMIC_RELAXED);
  }
  k_dense_extract<<<n, 256>>>(n, M, dinv);
  MSG_CHECK_LAUNCH();
  MSG_CUDA(cudaMemcpy(inv, dinv, nn * 8, cudaMemcpyDeviceToHost));
  cudaFree(da); cudaFree(M); cudaFree(dinv); cudaFree(piv);
  return MSG_OK;
}

// Same result as msg_gpu_dense_inverse, bit for bit, without any allocation: a_dev and
// inv_dev are device arrays (row-major n x n) owned by the caller; the work runs on
// `stream` (NULL: the legacy default stream) and is complete when that stream is.
// Each call looks up the scratch address (cudaGetSymbolAddress) with the current device;
// the first call on a device also loads this module there, so make that first call
// before any stream capture.  All calls share one workspace per device, so calls that
// overlap on the GPU race; each call writes the whole [A | I] block and the pivot slot
// before reading them, so nothing needs to start at zero.  A singular input is not
// detected: a zero pivot gives inf/NaN entries and the call still returns MSG_OK (the
// work is queued, not awaited, so no status can come back from the device).
MSG_API int msg_gpu_dense_inverse_noalloc(int32_t n, const double *a_dev, double *inv_dev, void *stream) {
  if (n < 1 || n > kNoAllocMaxN) {
    set_error("dense_inverse_noalloc: n = %d outside 1..%d (workspace limit)", (int)n, kNoAllocMaxN);
    return MSG_ERR_SIZE;
  }
  if (!a_dev || !inv_dev) { set_error("dense_inverse_noalloc: null device pointer"); return MSG_ERR_ARG; }
  double *M = nullptr;
  int rc = noalloc_scratch(&M);
  if (rc) return rc;
  int *piv = reinterpret_cast<int *>(M + (size_t)2 * kNoAllocMaxN * kNoAllocMaxN);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  k_dense_fill_rm<<<n, 256, 0, s>>>(n, a_dev, M);
  MSG_CHECK_LAUNCH();
  k_gj<false, 1024><<<1, 1024, 0, s>>>(n, M, piv);
  MSG_CHECK_LAUNCH();
  k_dense_extract<<<n, 256, 0, s>>>(n, M, inv_dev);
  MSG_CHECK_LAUNCH();
  return MSG_OK;
}

MSG_API int msg_gpu_amg_nlevel(msg_ctx_t *c) {
  return (c && S(c)) ? (int)S(c)->lv.size() : 0;
}
MSG_API int msg_gpu_amg_level_sizes(msg_ctx_t *c, int32_t lv, int32_t *n, int32_t *nnz, int32_t *pnnz) {
  if (!c || !S(c) || lv < 0 || lv >= (int)S(c)->lv.size()) return MSG_ERR_ARG;
  AmgLevel &L = S(c)->lv[lv];
  *n = L.n; *nnz = L.nnz; *pnnz = L.pnnz;
  return MSG_OK;
}
MSG_API int msg_gpu_amg_level(msg_ctx_t *c, int32_t lv, int32_t *offind, int32_t *offrow, double *dmat,
                              double *lumat, int32_t *pindex, int32_t *poffrow, double *pval, int32_t *agg) {
  if (!c || !S(c) || lv < 0 || lv >= (int)S(c)->lv.size()) return MSG_ERR_ARG;
  MSG_CUDA(cudaStreamSynchronize(c->stream));
  AmgLevel &L = S(c)->lv[lv];
  if (offind) MSG_CUDA(cudaMemcpy(offind, L.rowptr, (size_t)(L.n + 1) * 4, cudaMemcpyDeviceToHost));
  if (offrow) MSG_CUDA(cudaMemcpy(offrow, L.col, (size_t)L.nnz * 4, cudaMemcpyDeviceToHost));
  if (dmat) MSG_CUDA(cudaMemcpy(dmat, L.diag, (size_t)L.n * 8, cudaMemcpyDeviceToHost));
  if (lumat && lv == 0) {   // the Jacobian's bands in CSR order
    int rc = launch_dia_to_csr(c, csr_scratch(c));
    if (rc) return rc;
    MSG_CUDA(cudaStreamSynchronize(c->stream));
    MSG_CUDA(cudaMemcpy(lumat, csr_scratch(c), (size_t)L.nnz * 8, cudaMemcpyDeviceToHost));
  } else if (lumat) {
    MSG_CUDA(cudaMemcpy(lumat, L.val, (size_t)L.nnz * 8, cudaMemcpyDeviceToHost));
  }
  if (lv > 0) {
    int nf = S(c)->lv[lv - 1].n;
    if (pindex) MSG_CUDA(cudaMemcpy(pindex, L.pptr, (size_t)(nf + 1) * 4, cudaMemcpyDeviceToHost));
    if (poffrow) MSG_CUDA(cudaMemcpy(poffrow, L.pcol, (size_t)L.pnnz * 4, cudaMemcpyDeviceToHost));
    if (pval) MSG_CUDA(cudaMemcpy(pval, L.pval, (size_t)L.pnnz * 8, cudaMemcpyDeviceToHost));
    if (agg) MSG_CUDA(cudaMemcpy(agg, L.agg, (size_t)nf * 4, cudaMemcpyDeviceToHost));
  }
  return MSG_OK;
}
}
