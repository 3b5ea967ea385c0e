// MIC(0)-preconditioned CG on a general sparse symmetric matrix given in CSR
// form: the call shape of robertbridson::PCGSolver<double>::solve
// (libWetCloth/Core/PCGSolver/PCGSolver.h:260-308), which the reference calls
// on assembled SparseMatrix objects (the implicit viscosity solve,
// Core/Viscosity.cpp:112-116; the pressure system re-solved with MIC(0)).
//
// Everything numeric runs on the GPU:
//   * structure: the factor's columns are the upper parts of the matrix rows
//     (factor_modified_incomplete_cholesky0 copies them, PCGSolver.h:106-117),
//     their transpose lists for each column the earlier columns that update
//     it;
//   * the factorisation, one launch: a thread per column waits for the earlier
//     columns that update it and gathers their eliminations in ascending
//     column order, with the reference's dropped-entry rule ("missing",
//     modification 0.97) and its pivot test (ratio 0.25), so every entry sees
//     the reference's sequence of subtractions (PCGSolver.h:142-204);
//   * the triangular solves, one launch each: a thread per row waits for the
//     rows it depends on and subtracts their terms in the order solve_lower /
//     solve_lower_transpose_in_place apply them (:211-239);
//   * the PCG iteration of PCGSolver::solve with its infinity-norm stop, tested
//     on the device; the host looks at it every kCheck iterations (launches
//     after the stop return at once).
// Rows are handed out to blocks by an atomic ticket in the order of the
// dependencies (ascending, or descending for the backward solve), so whatever
// a row waits for belongs to a block that started earlier or to its own.  Every
// wait is bounded: it ends when no row of the launch has got on for some millions
// of rounds (Patience), however long the chain of rows before it is.
// Products and sums are rounded separately (_rn intrinsics), as the
// reference's compiled code evaluates them.  Dot products are deterministic
// block reductions; their summation order is not Eigen's, so the iterates
// agree with the reference's to rounding, not bit for bit.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/wetcloth_gpu.h"
#include "wcg_context.h"
#include "wcg_scan.cuh"

namespace wcg {
namespace {

constexpr double kOmega = 0.97;     // modification parameter (PCGSolver.h:100)
constexpr double kMinRatio = 0.25;  // min_diagonal_ratio (:101)
constexpr int kThreads = 256;
constexpr int kDotBlocks = 296;     // 2 per SM of a B200
constexpr int kCheck = 8;           // iterations per look at the stop test
constexpr long long kOneAlloc = 8 << 20;  // entries up to which a solve allocates once

inline unsigned nblocks(long long n) { return (unsigned)((n + kThreads - 1) / kThreads); }

struct Mem {
  void* p = nullptr;
  ~Mem() {
    if (p) cudaFree(p);
  }
  cudaError_t alloc(size_t bytes) { return cudaMalloc(&p, bytes ? bytes : 16); }
  template <typename T>
  T* as() const { return (T*)p; }
};

#define CSR_TRY(x)                       \
  do {                                   \
    cudaError_t e_ = (x);                \
    if (e_ != cudaSuccess) return e_;    \
  } while (0)

// rows (whose bounds the host has checked) must list strictly ascending columns in
// [0, n); counts the upper entries of each row (the factor's column) and takes the
// diagonal
__global__ void k_csr_rows(int n, const int* __restrict__ rowstart, const int* __restrict__ col,
                           const double* __restrict__ val, int* __restrict__ ucount,
                           double* __restrict__ adiag, int* bad) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int s = rowstart[i], e = rowstart[i + 1];
  int prev = -1, cnt = 0;
  double d = 0.0;
  for (int p = s; p < e; ++p) {
    const int c = col[p];
    if (c < 0 || c >= n || c <= prev) atomicExch(bad, 1);
    prev = c;
    if (c > i) ++cnt;
    else if (c == i) d = val[p];
  }
  ucount[i] = cnt;
  adiag[i] = d;
}

// factor column k = the entries of row k right of the diagonal, in row order
__global__ void k_csr_upper(int n, const int* __restrict__ rowstart, const int* __restrict__ col,
                            const double* __restrict__ val, const int* __restrict__ ustart,
                            int* __restrict__ urow, double* __restrict__ uval,
                            int* __restrict__ tcount) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  int q = ustart[k];
  for (int p = rowstart[k]; p < rowstart[k + 1]; ++p) {
    const int c = col[p];
    if (c <= k) continue;
    urow[q] = c;
    uval[q] = val[p];
    ++q;
    atomicAdd(&tcount[c], 1);
  }
}

// for each column j: the earlier columns k holding row j, with the position
// of that entry
__global__ void k_csr_transpose(int n, const int* __restrict__ ustart,
                                const int* __restrict__ urow, const int* __restrict__ tstart,
                                int* __restrict__ tcur, int* __restrict__ tk,
                                int* __restrict__ tp) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  for (int p = ustart[k]; p < ustart[k + 1]; ++p) {
    const int j = urow[p];
    const int q = tstart[j] + atomicAdd(&tcur[j], 1);
    tk[q] = k;
    tp[q] = p;
  }
}

// ascending column order inside each transpose list (insertion sort)
__global__ void k_csr_sort_transpose(int n, const int* __restrict__ tstart, int* __restrict__ tk,
                                     int* __restrict__ tp) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const int s = tstart[j], e = tstart[j + 1];
  for (int a = s + 1; a < e; ++a) {
    const int k = tk[a], p = tp[a];
    int b = a - 1;
    while (b >= s && tk[b] > k) {
      tk[b + 1] = tk[b];
      tp[b + 1] = tp[b];
      --b;
    }
    tk[b + 1] = k;
    tp[b + 1] = p;
  }
}

typedef unsigned long long u64;

__device__ inline void ld_words(const u64* p, u64& a, u64& b) {
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(a) : "l"(p));
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(b) : "l"(p + 1));
}
__device__ inline void st_word(u64* p, u64 v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v));
}
__device__ inline int ld_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ inline void st_release(int* p, int v) {
  asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ inline int ld_relaxed(const int* p) {
  int v;
  asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// How long a warp waits.  The last rows of a long chain are resident from the
// start and idle until the chain reaches them (a band of 24 over 60 000 rows:
// seconds), so a wait does not end after a number of its own rounds but once the
// whole launch has stood still for that long: every elimination of the
// factorisation and every finished row of a solve adds to `progress`, and a warp
// that idles looks there every kLook rounds.  What may pass between two additions
// is the walk over one row's entries (two rows' in an elimination), at a few
// rounds each: the limit has room for the longest.  A warp that gives up sets
// `err`, and all others follow.  (The additions cost 0.5 of 34 ms on a 40^3 grid;
// a clock read in every round that got on, to add less often, 1.5.)
constexpr long long kMaxRounds = 1ll << 22;  // a third of a second at the least
constexpr int kLook = 1024;

struct Patience {
  int* progress;
  int* err;
  long long limit;
  long long idle = 0;
  int round = 0, seen = 0;
  __device__ Patience(int* progress_, int* err_, int longest_row)
      : progress(progress_), err(err_), limit(kMaxRounds + 16ll * longest_row) {}
  // a round without progress of the warp's own (all its lanes call): true once
  // the wait is over
  __device__ bool over() {
    if (++round & (kLook - 1)) return false;
    int p = 0, e = 0;
    if ((threadIdx.x & 31) == 0) {
      p = ld_relaxed(progress);
      e = ld_relaxed(err);
    }
    p = __shfl_sync(0xffffffffu, p, 0);
    if (__shfl_sync(0xffffffffu, e, 0)) return true;
    idle = p == seen ? idle + kLook : 0;
    seen = p;
    if (idle <= limit) return false;
    if ((threadIdx.x & 31) == 0) atomicExch(err, 1);
    return true;
  }
};

// The eliminations of column k (finished) in column j: mult is the entry of
// row j in column k, d the running pivot of column j.
__device__ inline double eliminate(int j, int k, double mult, double d,
                                   const int* __restrict__ rowstart,
                                   const int* __restrict__ col, const int* __restrict__ ustart,
                                   const int* __restrict__ urow, double* uval) {
  double missing = 0.0;
  int a = ustart[k];
  const int ek = ustart[k + 1];
  const int ej = ustart[j + 1];
  // dropped entries above the diagonal of column j: rows of column k below
  // j that row j of the matrix does not hold
  int b = rowstart[j];
  const int eb = rowstart[j + 1];
  while (a < ek && urow[a] < j) {
    while (b < eb) {
      const int c = col[b];
      if (c < urow[a]) {
        ++b;
      } else if (c == urow[a]) {
        break;
      } else {
        missing = __dadd_rn(missing, __ldcg(uval + a));
        break;
      }
    }
    ++a;
  }
  if (a < ek && urow[a] == j) d = __dsub_rn(d, __dmul_rn(mult, __ldcg(uval + a)));
  ++a;
  // entries below the diagonal of column j, or dropped into missing
  int bb = ustart[j];
  while (a < ek && bb < ej) {
    if (urow[bb] < urow[a]) {
      ++bb;
    } else if (urow[bb] == urow[a]) {
      uval[bb] = __dsub_rn(uval[bb], __dmul_rn(mult, __ldcg(uval + a)));
      ++a;
      ++bb;
    } else {
      missing = __dadd_rn(missing, __ldcg(uval + a));
      ++a;
    }
  }
  while (a < ek) {
    missing = __dadd_rn(missing, __ldcg(uval + a));
    ++a;
  }
  return __dsub_rn(d, __dmul_rn(__dmul_rn(kOmega, mult), missing));
}

// factor_modified_incomplete_cholesky0 (PCGSolver.h:142-204): column j applies
// the eliminations of the earlier columns k that hold row j in ascending k (the
// order in which the reference's column loop reaches j), each once column k is
// finished (ready[k] = 1), then takes its pivot and scales itself.
__global__ void __launch_bounds__(kThreads)
    k_csr_factor(int n, int* ticket, const int* __restrict__ rowstart,
                 const int* __restrict__ col, const int* __restrict__ ustart,
                 const int* __restrict__ urow, double* uval, const int* __restrict__ tstart,
                 const int* __restrict__ tk, const int* __restrict__ tp,
                 const double* __restrict__ adiag, double* __restrict__ invdiag, int* ready,
                 int* progress, int* err, int longest_row) {
  __shared__ int s_block;
  if (threadIdx.x == 0) s_block = atomicAdd(ticket, 1);
  __syncthreads();
  const int j = s_block * kThreads + threadIdx.x;
  bool fin = j >= n;
  int q = fin ? 0 : tstart[j];
  const int eq = fin ? 0 : tstart[j + 1];
  double d = fin ? 0.0 : adiag[j];
  Patience wait(progress, err, longest_row);
  // lanes of a warp may depend on one another: every round lets each lane do
  // what it can, so the lanes that are ready go on
  while (__any_sync(0xffffffffu, !fin)) {
    bool moved = false;
    if (!fin) {
      if (q < eq) {
        const int k = tk[q];
        if (adiag[k] == 0.0) {  // null row/column: skipped (:144)
          ++q;
          moved = true;
        } else if (ld_acquire(ready + k)) {
          d = eliminate(j, k, __ldcg(uval + tp[q]), d, rowstart, col, ustart, urow, uval);
          atomicAdd(progress, 1);
          ++q;
          moved = true;
        }
      } else {
        double inv = d;
        if (adiag[j] != 0.0) {
          const double piv = d < __dmul_rn(kMinRatio, adiag[j]) ? adiag[j] : d;
          inv = __ddiv_rn(1.0, __dsqrt_rn(piv));
          for (int p = ustart[j]; p < ustart[j + 1]; ++p) uval[p] = __dmul_rn(uval[p], inv);
        }
        invdiag[j] = inv;
        __threadfence();
        st_release(ready + j, 1);
        fin = true;
        moved = true;
      }
    }
    if (!__any_sync(0xffffffffu, moved) && wait.over()) fin = true;
  }
}

// scalar slots (doubles); SC_DONE holds an int: 1 converged, 2 iteration limit,
// 3 a wait gave up
enum : int { SC_RHO = 0, SC_RES, SC_ITER, SC_DONE, SC_ALPHA, SC_BETA, SC_TOL, SC_MAXIT, kNumSc };

// solve_lower (PCGSolver.h:211-222, LOWER) or solve_lower_transpose_in_place
// (:226-239): a thread per row, rows ascending or descending.  A row's terms
// are subtracted in list order, four at a time, once the rows they name have
// published their values: as two tagged words (tag << 32 | 32 data bits) each,
// in shared memory for rows of the same block and in `words` for all others.
// Bound by the chain of dependent rows: a hop inside the block costs a pass
// over shared memory, one between blocks a round trip to L2, so the block is as
// large as it can be.  The former launch per level took 2.5-3 us a level (two
// solves over 118 levels of a 40^3 grid: 0.7 ms of a 1 ms iteration).
constexpr int kTriThreads = 1024;
template <bool LOWER>
__global__ void __launch_bounds__(kTriThreads, 1)
    k_csr_tri(int n, int* ticket, int ticket_base, unsigned tag, const int* __restrict__ start,
              const int* __restrict__ dep, const int* __restrict__ pos,
              const double* __restrict__ uval, const double* __restrict__ invdiag,
              const double* in, double* out, u64* words, const double* __restrict__ sc,
              int* progress, int* err, int longest_row) {
  __shared__ u64 sw[2 * kTriThreads];
  __shared__ int s_block;
  constexpr unsigned full = 0xffffffffu;
  if (threadIdx.x == 0) s_block = atomicAdd(ticket, 1) - ticket_base;
  if (*(const int*)(sc + SC_DONE)) return;  // set by an earlier launch: uniform
  sw[2 * threadIdx.x] = sw[2 * threadIdx.x + 1] = 0ull;
  __syncthreads();
  const int lo = s_block * kTriThreads;
  const int idx = lo + threadIdx.x;
  const int row = LOWER ? idx : n - 1 - idx;
  bool fin = idx >= n;
  int q = fin ? 0 : start[row];
  const int e = fin ? 0 : start[row + 1];
  double acc = fin ? 0.0 : in[row];
  const double inv = fin ? 0.0 : invdiag[row];
  int src[4];       // >= 0: slot in this block, < 0: -1 - row
  double u[4], val[4];
  int cnt = 0;
  unsigned pend = 0, near = 0;
  volatile u64* const vs = sw;
  auto next_terms = [&]() {
    cnt = min(4, e - q);
    pend = (1u << cnt) - 1u;
    near = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      src[j] = 0;
      u[j] = val[j] = 0.0;
      if (j < cnt) {
        const int k = dep[q + j];
        const int at = (LOWER ? k : n - 1 - k) - lo;
        src[j] = at >= 0 ? at : -1 - k;
        if (at >= 0) near |= 1u << j;
        u[j] = uval[LOWER ? pos[q + j] : q + j];
      }
    }
  };
  if (!fin) next_terms();
  Patience wait(progress, err, longest_row);
  while (!__all_sync(full, fin)) {
    bool moved = false;
    // terms from other blocks, all loads in flight at once
    if (!fin && (pend & ~near)) {
      u64 w0[4], w1[4];
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if ((pend & ~near) >> j & 1) ld_words(words + 2ll * (-1 - src[j]), w0[j], w1[j]);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (((pend & ~near) >> j & 1) && (unsigned)(w0[j] >> 32) == tag &&
            (unsigned)(w1[j] >> 32) == tag) {
          val[j] = __longlong_as_double((long long)((w1[j] << 32) | (w0[j] & 0xffffffffull)));
          pend &= ~(1u << j);
          moved = true;
        }
    }
    // terms from this block, for as long as any lane of the warp gets on
    bool again;
    do {
      bool step = false;
      if (!fin) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if ((pend & near) >> j & 1) {
            const u64 w0 = vs[2 * src[j]], w1 = vs[2 * src[j] + 1];
            if ((unsigned)(w0 >> 32) == tag && (unsigned)(w1 >> 32) == tag) {
              val[j] = __longlong_as_double((long long)((w1 << 32) | (w0 & 0xffffffffull)));
              pend &= ~(1u << j);
              step = true;
            }
          }
        if (!pend) {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (j < cnt) acc = __dsub_rn(acc, __dmul_rn(u[j], val[j]));
          q += cnt;
          step = true;
          if (q < e) {
            next_terms();
          } else {
            const double y = __dmul_rn(acc, inv);
            const u64 b = (u64)__double_as_longlong(y);
            const u64 w0 = ((u64)tag << 32) | (b & 0xffffffffull);
            const u64 w1 = ((u64)tag << 32) | (b >> 32);
            vs[2 * threadIdx.x] = w0;
            vs[2 * threadIdx.x + 1] = w1;
            st_word(words + 2ll * row, w0);
            st_word(words + 2ll * row + 1, w1);
            out[row] = y;
            atomicAdd(progress, 1);
            fin = true;
          }
        }
      }
      again = __any_sync(full, step);
      moved = moved || again;
    } while (again);
    if (!__any_sync(full, moved) && wait.over()) fin = true;
  }
}

// sum (or maximum, NaN first) over a block of kThreads
__device__ inline double block_reduce(double v, double* sm, bool is_max) {
  sm[threadIdx.x] = v;
  __syncthreads();
  for (int s = kThreads / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) {
      const double a = sm[threadIdx.x], o = sm[threadIdx.x + s];
      sm[threadIdx.x] = is_max ? ((o > a || o != o) ? o : a) : __dadd_rn(a, o);
    }
    __syncthreads();
  }
  const double r = sm[0];
  __syncthreads();
  return r;
}

// Writes this block's partial; true in the last block, with the reduction of
// all partials in block order by thread, then the block tree (deterministic).
__device__ inline bool grid_reduce(double v, double* part, int* ctr, double* sm, bool is_max,
                                   double* out) {
  __shared__ int s_last;
  const double b = block_reduce(v, sm, is_max);
  if (threadIdx.x == 0) {
    part[blockIdx.x] = b;
    __threadfence();
    s_last = atomicAdd(ctr, 1) == (int)gridDim.x - 1;
    if (s_last) {
      atomicExch(ctr, 0);
      __threadfence();
    }
  }
  __syncthreads();
  if (!s_last) return false;
  double acc = 0.0;
  for (int i = threadIdx.x; i < (int)gridDim.x; i += kThreads) {
    const double o = __ldcg(part + i);
    acc = is_max ? ((o > acc || o != o) ? o : acc) : __dadd_rn(acc, o);
  }
  *out = block_reduce(acc, sm, is_max);
  return true;
}

// z = A s (multiply(FixedSparseMatrix, x, result), SparseMatrix.h:299-320);
// the last block: alpha = rho / s.z
__global__ void __launch_bounds__(kThreads)
    k_csr_spmv(int n, const int* __restrict__ rowstart, const int* __restrict__ col,
               const double* __restrict__ val, const double* __restrict__ s,
               double* __restrict__ z, double* sc, double* part, int* ctr) {
  __shared__ double sm[kThreads];
  if (*(const int*)(sc + SC_DONE)) return;
  double dot = 0.0;
  for (int i = blockIdx.x * kThreads + threadIdx.x; i < n; i += gridDim.x * kThreads) {
    double acc = 0.0;
    for (int p = rowstart[i]; p < rowstart[i + 1]; ++p)
      acc = __dadd_rn(acc, __dmul_rn(val[p], s[col[p]]));
    z[i] = acc;
    dot = __dadd_rn(dot, __dmul_rn(s[i], acc));
  }
  double sz;
  if (grid_reduce(dot, part, ctr, sm, false, &sz) && threadIdx.x == 0)
    sc[SC_ALPHA] = __ddiv_rn(sc[SC_RHO], sz);
}

// result += s * alpha;  r += z * (-alpha)  (BLAS::add_scaled, BLASWrapper.h:
// 52-56); the last block: the stop test on max |r|.  x null: max |r| alone.
__global__ void __launch_bounds__(kThreads)
    k_csr_update_xr(int n, const double* __restrict__ s, const double* __restrict__ z,
                    double* __restrict__ x, double* __restrict__ r, double* sc, double* part,
                    int* ctr) {
  __shared__ double sm[kThreads];
  if (*(const int*)(sc + SC_DONE)) return;
  const double alpha = sc[SC_ALPHA];
  double m = 0.0;
  for (int i = blockIdx.x * kThreads + threadIdx.x; i < n; i += gridDim.x * kThreads) {
    double rv = r[i];
    if (x) {
      x[i] = __dadd_rn(x[i], __dmul_rn(s[i], alpha));
      rv = __dadd_rn(rv, __dmul_rn(z[i], -alpha));
      r[i] = rv;
    }
    const double v = fabs(rv);
    m = (v > m || v != v) ? v : m;  // NaN propagates
  }
  double res;
  if (grid_reduce(m, part, ctr, sm, true, &res) && threadIdx.x == 0) {
    sc[SC_RES] = res;
    if (x) {
      sc[SC_ITER] += 1.0;
      if (res <= sc[SC_TOL]) *(int*)(sc + SC_DONE) = 1;
      else if (sc[SC_ITER] >= sc[SC_MAXIT]) *(int*)(sc + SC_DONE) = 2;
    }
  }
}

// the last block: rho_new = z.r, beta = rho_new / rho (init: rho alone), and the
// end of the solve where a wait of the factorisation or of a triangular solve
// before it gave up
__global__ void __launch_bounds__(kThreads)
    k_csr_dot(int n, const double* __restrict__ z, const double* __restrict__ r, double* sc,
              double* part, int* ctr, const int* __restrict__ err, int init) {
  __shared__ double sm[kThreads];
  if (*(const int*)(sc + SC_DONE)) return;
  double acc = 0.0;
  for (int i = blockIdx.x * kThreads + threadIdx.x; i < n; i += gridDim.x * kThreads)
    acc = __dadd_rn(acc, __dmul_rn(z[i], r[i]));
  double rho;
  if (grid_reduce(acc, part, ctr, sm, false, &rho) && threadIdx.x == 0) {
    if (!init) sc[SC_BETA] = __ddiv_rn(rho, sc[SC_RHO]);
    sc[SC_RHO] = rho;
    if (*err) *(int*)(sc + SC_DONE) = 3;
  }
}

// s = z + s * beta
__global__ void __launch_bounds__(kThreads)
    k_csr_direction(int n, const double* __restrict__ z, double* __restrict__ s,
                    const double* __restrict__ sc) {
  if (*(const int*)(sc + SC_DONE)) return;
  const double beta = sc[SC_BETA];
  for (int i = blockIdx.x * kThreads + threadIdx.x; i < n; i += gridDim.x * kThreads)
    s[i] = __dadd_rn(z[i], __dmul_rn(s[i], beta));
}

struct Solver {
  int n = 0;
  cudaStream_t st = nullptr;
  int *rowstart, *col, *ustart, *urow, *tstart, *tk, *tp, *ctl;
  double *val, *adiag, *invdiag, *uval, *x, *r, *z, *s, *part, *sc;
  u64* words;
  unsigned tag = 0;   // of the last triangular solve
  int tickets = 0;    // handed out by the triangular solves so far
  int longest = 0;    // entries of the longest row

  // ctl: 0 malformed matrix, 1 wait given up, 2 reduction count, 3 ticket of
  // the triangular solves, 4 ticket of the factorisation, 5 progress of the rows
  void precondition(const double* in, double* out) {
    const int nb = (n + kTriThreads - 1) / kTriThreads;
    k_csr_tri<true><<<nb, kTriThreads, 0, st>>>(n, ctl + 3, tickets, ++tag, tstart, tk, tp, uval,
                                                invdiag, in, out, words, sc, ctl + 5, ctl + 1,
                                                longest);
    tickets += nb;
    k_csr_tri<false><<<nb, kTriThreads, 0, st>>>(n, ctl + 3, tickets, ++tag, ustart, urow, nullptr,
                                                 uval, invdiag, out, out, words, sc, ctl + 5,
                                                 ctl + 1, longest);
    tickets += nb;
  }
  unsigned grid() const { return std::min(nblocks(n), (unsigned)kDotBlocks); }
  cudaError_t read(double* out, int slot, int k) {
    CSR_TRY(cudaMemcpyAsync(out, sc + slot, k * sizeof(double), cudaMemcpyDeviceToHost, st));
    return cudaStreamSynchronize(st);
  }
};

// 0: converged, 1: not converged (iteration limit or rho 0/NaN), 2: bad matrix,
// 3: a wait gave up
cudaError_t csr_solve(const int* h_rowstart, const int* h_col, const double* h_val, int n,
                      const double* h_rhs, double* h_x, double tolerance_factor, int maxiter,
                      double* residual_out, int* iters_out, int* outcome) {
  Solver S;
  S.n = n;
  CSR_TRY(cudaStreamCreateWithFlags(&S.st, cudaStreamNonBlocking));
  struct StreamGuard {
    cudaStream_t s;
    ~StreamGuard() { cudaStreamDestroy(s); }
  } guard{S.st};
  cudaStream_t st = S.st;
  const long long nnz = (long long)h_rowstart[n] - h_rowstart[0];
  // One allocation, or two for more than kOneAlloc entries: the factor's columns
  // hold the entries right of the diagonal, whose number comes from the device.  (A
  // second allocation, its release and the wait cost 0.7 of 35 ms at 0.45M entries;
  // the room for all entries at most 160 MB.)
  const size_t vb = (size_t)n * sizeof(double), ib = (size_t)(n + 1) * sizeof(int);
  const size_t scan_b = (size_t)((n + 1 + kScanTile - 1) / kScanTile + 1) * sizeof(int);
  Mem mem, factor;
  size_t total = 0;
  auto place = [&](size_t bytes) {
    const size_t at = total;
    total += (bytes + 255) & ~(size_t)255;
    return at;
  };
  const size_t o_rs = place(ib), o_col = place(nnz * sizeof(int)),
               o_val = place(nnz * sizeof(double));
  const size_t o_us = place(ib), o_ts = place(ib);
  const size_t o_ad = place(vb), o_id = place(vb);
  const size_t o_x = place(vb), o_r = place(vb), o_z = place(vb), o_s = place(vb);
  const size_t o_part = place(kDotBlocks * sizeof(double)), o_tmp = place(scan_b);
  struct FactorPlace {
    size_t uval, urow, tk, tp;
  };
  auto place_factor = [&](size_t k) {
    return FactorPlace{place(k * sizeof(double)), place(k * sizeof(int)), place(k * sizeof(int)),
                       place(k * sizeof(int))};
  };
  FactorPlace fp{};
  if (nnz <= kOneAlloc) fp = place_factor(nnz);
  // zeroed: counters, the ready flags, the scalars, and the words of the
  // triangular solves (16 bytes a row), whose place the transpose counts and cursors
  // have first (4 (n + 1) bytes each)
  const size_t wb = 2 * (size_t)n * sizeof(u64);
  const size_t o_zero = total;
  const size_t o_ctl = place(8 * sizeof(int)), o_rdy = place(ib);
  const size_t o_sc = place(kNumSc * sizeof(double)), o_w = place(wb);
  CSR_TRY(mem.alloc(total));
  unsigned char* const m = mem.as<unsigned char>();
  S.rowstart = (int*)(m + o_rs);
  S.col = (int*)(m + o_col);
  S.val = (double*)(m + o_val);
  S.ustart = (int*)(m + o_us);
  S.tstart = (int*)(m + o_ts);
  S.adiag = (double*)(m + o_ad);
  S.invdiag = (double*)(m + o_id);
  S.x = (double*)(m + o_x);
  S.r = (double*)(m + o_r);
  S.z = (double*)(m + o_z);
  S.s = (double*)(m + o_s);
  S.part = (double*)(m + o_part);
  S.ctl = (int*)(m + o_ctl);
  S.words = (u64*)(m + o_w);
  S.sc = (double*)(m + o_sc);
  int* const tmp = (int*)(m + o_tmp);
  int* const tcount = (int*)(m + o_w);
  int* const tcur = tcount + n + 1;
  int* const ready = (int*)(m + o_rdy);
  CSR_TRY(cudaMemsetAsync(m + o_zero, 0, total - o_zero, st));
  // rowstart relative to its first entry
  std::vector<int> rs(h_rowstart, h_rowstart + n + 1);
  const int base = rs[0];
  for (int& v : rs) v -= base;
  for (int i = 0; i < n; ++i) S.longest = std::max(S.longest, rs[i + 1] - rs[i]);
  CSR_TRY(cudaMemcpyAsync(S.rowstart, rs.data(), ib, cudaMemcpyHostToDevice, st));
  CSR_TRY(cudaMemcpyAsync(S.col, h_col + base, nnz * sizeof(int), cudaMemcpyHostToDevice, st));
  CSR_TRY(cudaMemcpyAsync(S.val, h_val + base, nnz * sizeof(double), cudaMemcpyHostToDevice, st));
  // the upper counts of the rows go to tstart's place until they are scanned
  int* const ucount = S.tstart;
  k_csr_rows<<<nblocks(n), kThreads, 0, st>>>(n, S.rowstart, S.col, S.val, ucount, S.adiag, S.ctl);
  // factor columns: the upper parts of the rows
  exclusive_scan<int, int>(ucount, n, S.ustart, tmp, S.ustart + n, st);
  int hctl[2] = {0, 0}, nu = 0;
  CSR_TRY(cudaMemcpyAsync(hctl, S.ctl, sizeof(int), cudaMemcpyDeviceToHost, st));
  if (nnz > kOneAlloc)
    CSR_TRY(cudaMemcpyAsync(&nu, S.ustart + n, sizeof(int), cudaMemcpyDeviceToHost, st));
  CSR_TRY(cudaStreamSynchronize(st));
  if (hctl[0]) {
    *outcome = 2;
    return cudaSuccess;
  }
  unsigned char* f = m;
  if (nnz > kOneAlloc) {
    total = 0;
    fp = place_factor(nu);
    CSR_TRY(factor.alloc(total));
    f = factor.as<unsigned char>();
  }
  S.uval = (double*)(f + fp.uval);
  S.urow = (int*)(f + fp.urow);
  S.tk = (int*)(f + fp.tk);
  S.tp = (int*)(f + fp.tp);
  // their entries and their transpose
  k_csr_upper<<<nblocks(n), kThreads, 0, st>>>(n, S.rowstart, S.col, S.val, S.ustart, S.urow,
                                               S.uval, tcount);
  exclusive_scan<int, int>(tcount, n, S.tstart, tmp, S.tstart + n, st);
  k_csr_transpose<<<nblocks(n), kThreads, 0, st>>>(n, S.ustart, S.urow, S.tstart, tcur, S.tk, S.tp);
  k_csr_sort_transpose<<<nblocks(n), kThreads, 0, st>>>(n, S.tstart, S.tk, S.tp);
  CSR_TRY(cudaMemsetAsync(S.words, 0, wb, st));
  CSR_TRY(cudaGetLastError());

  // PCG
  CSR_TRY(cudaMemsetAsync(S.x, 0, vb, st));
  CSR_TRY(cudaMemcpyAsync(S.r, h_rhs, vb, cudaMemcpyHostToDevice, st));
  int iters = 0;
  bool ok = false;
  double res = 0.0;
  k_csr_update_xr<<<S.grid(), kThreads, 0, st>>>(n, nullptr, nullptr, nullptr, S.r, S.sc, S.part,
                                                 S.ctl + 2);
  CSR_TRY(S.read(&res, SC_RES, 1));
  if (res < 1e-30) {
    ok = true;
  } else {
    const double tf = tolerance_factor < 1e-30 ? 1e-30 : tolerance_factor;
    const double lim[2] = {tf * res, (double)maxiter};  // SC_TOL, SC_MAXIT
    CSR_TRY(cudaMemcpyAsync(S.sc + SC_TOL, lim, sizeof(lim), cudaMemcpyHostToDevice, st));
    k_csr_factor<<<nblocks(n), kThreads, 0, st>>>(n, S.ctl + 4, S.rowstart, S.col, S.ustart, S.urow,
                                                  S.uval, S.tstart, S.tk, S.tp, S.adiag, S.invdiag,
                                                  ready, S.ctl + 5, S.ctl + 1, S.longest);
    S.precondition(S.r, S.z);
    k_csr_dot<<<S.grid(), kThreads, 0, st>>>(n, S.z, S.r, S.sc, S.part, S.ctl + 2, S.ctl + 1, 1);
    CSR_TRY(cudaGetLastError());
    double h0[4];
    CSR_TRY(S.read(h0, SC_RHO, 4));  // rho, residual, iterations, done
    const double rho = h0[0];
    int done0;
    std::memcpy(&done0, &h0[3], sizeof(done0));
    if (!done0 && !(rho == 0.0 || rho != rho) && maxiter > 0) {
      CSR_TRY(cudaMemcpyAsync(S.s, S.z, vb, cudaMemcpyDeviceToDevice, st));
      for (;;) {
        for (int k = 0; k < kCheck; ++k) {
          k_csr_spmv<<<S.grid(), kThreads, 0, st>>>(n, S.rowstart, S.col, S.val, S.s, S.z, S.sc,
                                                    S.part, S.ctl + 2);
          k_csr_update_xr<<<S.grid(), kThreads, 0, st>>>(n, S.s, S.z, S.x, S.r, S.sc, S.part,
                                                         S.ctl + 2);
          S.precondition(S.r, S.z);
          k_csr_dot<<<S.grid(), kThreads, 0, st>>>(n, S.z, S.r, S.sc, S.part, S.ctl + 2, S.ctl + 1,
                                                   0);
          k_csr_direction<<<S.grid(), kThreads, 0, st>>>(n, S.z, S.s, S.sc);
        }
        CSR_TRY(cudaGetLastError());
        double h[3];
        CSR_TRY(S.read(h, SC_RES, 3));  // residual, iterations, done
        int done;
        std::memcpy(&done, &h[2], sizeof(done));
        res = h[0];
        iters = (int)h[1];
        if (done) {
          ok = done == 1;
          break;
        }
      }
    }
  }
  CSR_TRY(cudaMemcpyAsync(hctl, S.ctl, 2 * sizeof(int), cudaMemcpyDeviceToHost, st));
  CSR_TRY(cudaMemcpyAsync(h_x, S.x, vb, cudaMemcpyDeviceToHost, st));
  CSR_TRY(cudaStreamSynchronize(st));
  CSR_TRY(cudaGetLastError());
  *residual_out = res;
  *iters_out = iters;
  *outcome = hctl[1] ? 3 : (ok ? 0 : 1);
  return cudaSuccess;
}

}  // namespace
}  // namespace wcg

extern "C" int wcg_pcg_solve_csr(const int* rowstart, const int* col, const double* val, int n,
                                 const double* rhs, double* x, double tolerance_factor,
                                 int max_iterations, double* residual_out, int* iterations_out) {
  if (n < 0) return wcg::set_last_error(WCG_ERR_ARG, "wcg_pcg_solve_csr: negative size");
  if (n > 0 && (!rowstart || !col || !val || !rhs || !x))
    return wcg::set_last_error(WCG_ERR_ARG, "wcg_pcg_solve_csr: null array");
  if (!residual_out || !iterations_out)
    return wcg::set_last_error(WCG_ERR_ARG, "wcg_pcg_solve_csr: null output");
  if (max_iterations < 0)
    return wcg::set_last_error(WCG_ERR_ARG, "wcg_pcg_solve_csr: negative iteration limit");
  *residual_out = 0.0;
  *iterations_out = 0;
  if (n == 0) return WCG_OK;
  // no row may reach outside [rowstart[0], rowstart[n]): the kernels read what it names
  for (int i = 0; i < n; ++i)
    if (rowstart[i + 1] < rowstart[i])
      return wcg::set_last_error(WCG_ERR_ARG, "wcg_pcg_solve_csr: rowstart decreases");
  int outcome = 0;
  const cudaError_t e = wcg::csr_solve(rowstart, col, val, n, rhs, x, tolerance_factor,
                                       max_iterations, residual_out, iterations_out, &outcome);
  if (e != cudaSuccess)
    return wcg::set_last_error(WCG_ERR_CUDA, std::string("wcg_pcg_solve_csr: ") +
                                                 cudaGetErrorString(e));
  if (outcome == 2)
    return wcg::set_last_error(WCG_ERR_ARG,
                               "wcg_pcg_solve_csr: rows must hold strictly ascending columns "
                               "in [0, n)");
  if (outcome == 3)
    return wcg::set_last_error(WCG_ERR_DEVICE,
                               "wcg_pcg_solve_csr: a row reached its wait limit");
  if (outcome == 1)
    return wcg::set_last_error(WCG_ERR_NOT_CONVERGED,
                               "wcg_pcg_solve_csr: iteration limit reached or rho was 0/NaN");
  return WCG_OK;
}
