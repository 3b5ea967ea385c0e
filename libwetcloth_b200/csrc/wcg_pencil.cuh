// MIC(0)-PCG in the skewed pencil layout.
//
// The pressure unknowns of one solve (the bounding box of the DOF cells) are
// copied once into a layout built for the triangular sweeps.  One grid axis is
// the stream axis s (the longest extent of the box); the other two (a, c) are
// cut into patches of 16 x 16 lines.  Line (al, cl) of a patch is skewed by
// d = al + cl rows: cell (s, a, c) sits at row t = s + d of its patch, and
// element (patch, t, line) is stored at ((patch * R + t) * 256 + line) with
// line = al + 16 cl and R = Ls + 30 rows.  Rows outside a line's range and
// lines outside the box hold zeros.
//
// In this layout every MIC(0) hyperplane dependency is one row back (one row
// forward for the backward sweep):
//   (s-1, a, c): row t-1 of the same line
//   (s, a-1, c): row t-1 of line - 1
//   (s, a, c-1): row t-1 of line - 16
// so a CTA takes a patch, one warp per strip of 32 lines, and every strip walks
// its rows with contiguous loads and stores.  The factor is stored interleaved
// per cell {1/sqrt(d'), S_s, S_a, S_c} so a sweep reads it with one vector load.
// Values crossing a patch edge go through a global buffer of tagged 64-bit
// words, (epoch << 32 | 32 data bits), one word per 32 bits of payload: the
// consumer re-reads its word until the tag equals the launch's epoch, so no
// fence or flag is needed and a patch waits only for the rows it reads.
// Patches are handed out by an atomic ticket in wave order (PAi + PCi), so a
// patch's upstream patches always started before it.
//
// The arithmetic is that of the tile sweeps in wcg_pcg.cuh (restating
// robertbridson's factor_modified_incomplete_cholesky0 / solve_lower /
// solve_lower_transpose_in_place, libWetCloth/Core/PCGSolver/PCGSolver.h:
// 97-239): per DOF j, d_j = A_jj - sum over the three lower neighbours k of
// [L^2 + omega L miss], L = A(k, j) / sqrt(d_k'), miss = the other two upper
// couplings of k over sqrt(d_k'); forward y_j = (r_j - sum S_k y_k) / sqrt(d_j');
// backward z_j = (y_j - sum S_j z_k) / sqrt(d_j').  The lower neighbours are
// taken in the order c, a, s (z, y, x when s is x).
#pragma once

#include <cuda_runtime.h>

#include "wcg_common.cuh"
#include "wcg_context.h"
#include "wcg_pcg.cuh"

namespace wcg {

constexpr int kPatch = 16;                    // lines per patch edge
constexpr int kPatchLines = kPatch * kPatch;
constexpr int kPlBlocks = 592;                // streaming kernels: 4 x 148 SMs
// the fused SpMV in FP32 (32 registers): 8 resident CTAs per SM, so twice the
// loads in flight of the other streaming kernels
constexpr int kPlSpmvBlocks32 = 1184;
static_assert(kRedThreads == kPatchLines, "streaming kernels walk one row per block");

__host__ __device__ inline long long pl_index(const PencilGeom& G, long long p, int t, int l) {
  return (p * G.R + t) * kPatchLines + l;
}

// ---- tagged edge words -----------------------------------------------------------
typedef unsigned long long u64;

__device__ inline u64 ld_relaxed_u64(const u64* p) {
  u64 v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p));
  return v;
}

__device__ inline void st_relaxed_u64(u64* p, u64 v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v));
}

template <typename R>
struct TagWords;
template <>
struct TagWords<float> {
  static constexpr int W = 1;
  __device__ static void pack(float v, unsigned tag, u64* w) {
    w[0] = ((u64)tag << 32) | (u64)__float_as_uint(v);
  }
  __device__ static float unpack(const u64* w) { return __uint_as_float((unsigned)w[0]); }
};
template <>
struct TagWords<double> {
  static constexpr int W = 2;
  __device__ static void pack(double v, unsigned tag, u64* w) {
    const u64 b = (u64)__double_as_longlong(v);
    w[0] = ((u64)tag << 32) | (b & 0xffffffffull);
    w[1] = ((u64)tag << 32) | (b >> 32);
  }
  __device__ static double unpack(const u64* w) {
    return __longlong_as_double((long long)((w[1] << 32) | (w[0] & 0xffffffffull)));
  }
};

__device__ inline unsigned smem_u32(const void* p) {
  return (unsigned)__cvta_generic_to_shared(p);
}

// Values a strip stages per cell: factor A_d, A_s, A_a, A_c; forward r, q (with
// the update), coef x4; backward y, r, coef x4.
__host__ __device__ constexpr int sweep_slot(int mode) { return mode == 0 ? 4 : 6; }

// Words of the edge buffer: entry (patch that writes, face, row, line), EW
// words each.  face 0: towards the next patch along a (line k = cl), face 1:
// along c (line k = al); row = the row of the strip that takes the word.
__host__ __device__ inline long long edge_rows(const PencilGeom& G) { return G.Ls + 15; }
__device__ inline long long edge_word(const PencilGeom& G, long long p, int face, int row, int k,
                                      int EW) {
  return (((p * 2 + face) * edge_rows(G) + row) * kPatch + k) * EW;
}

// The MIC(0) factor of a cell, interleaved: {1/sqrt(d'), S_s, S_a, S_c}.
__device__ inline void ld_coef_shared(const float* p, float* c) {
  const float4 t = *reinterpret_cast<const float4*>(p);
  c[0] = t.x; c[1] = t.y; c[2] = t.z; c[3] = t.w;
}
__device__ inline void ld_coef_shared(const double* p, double* c) {
  const double2 a = reinterpret_cast<const double2*>(p)[0];
  const double2 b = reinterpret_cast<const double2*>(p)[1];
  c[0] = a.x; c[1] = a.y; c[2] = b.x; c[3] = b.y;
}
__device__ inline void st_coef(float* p, float a, float b, float c, float d) {
  *reinterpret_cast<float4*>(p) = make_float4(a, b, c, d);
}
__device__ inline void st_coef(double* p, double a, double b, double c, double d) {
  reinterpret_cast<double2*>(p)[0] = make_double2(a, b);
  reinterpret_cast<double2*>(p)[1] = make_double2(c, d);
}

template <typename R>
struct PencilSweepArgs {
  PencilGeom G;
  const int* order;   // patches in wave order
  int* ticket;
  int ticket_base;    // tickets already handed out this solve
  unsigned epoch;     // tag of this launch's edge words
  u64* edge;
  // factorisation input
  const R* AD;
  const R* AS;
  const R* AA;
  const R* AC;
  R* coef;      // factor: 4 per cell {1/sqrt(d'), S_s, S_a, S_c}
  // sweeps
  const R* in;  // forward: r; backward: y
  R* out;       // forward: y; backward: z
  R* r;         // forward (update): r updated in place; backward: r for z.r
  const R* q;   // forward (update)
  double* sc;            // device scalars (the last CTA of a reducing sweep writes them)
  double* part;  // per-patch partial: forward max|r|, backward z.r
  R omega, min_ratio;
  int* err;
  int* done_ctr;         // with part: the last CTA reduces the partials (forward with
                         // update: max|r| and the stop test; backward: z.r and beta)
  int red_init;          // backward: the first z.r of a solve (beta = 0)
  int npart;             // partials (patches)
  long long spin_limit;  // polls of an edge word before the wait gives up
  int stale_patch;       // failure-path test: this patch waits for a tag nothing
                         // writes (-1: none)
};

// MODE: kFactor, kForward, kBackward.  UPD: the forward sweep first applies
// r -= alpha q (and reports max|r|); the matching x += alpha s is applied by
// the next SpMV (k_pl_spmv_s) or, after the last iteration, by k_pl_axpy.
//
// A patch is one CTA of 8 strip warps and 2 receiver warps.  Strip w holds the
// 32 lines cl = 2w and 2w + 1 (lane = al + 16 (cl & 1)) and walks its own rows
// v = 0 .. Ls + 15 (row t = v + 2w of the patch) without any CTA barrier:
//   * its row data is copied D rows ahead into a shared-memory ring that only
//     this warp uses (cp.async, 16 bytes per lane);
//   * the a-neighbour and the c-neighbour inside the strip come by shuffle of
//     the previous row's outputs;
//   * the c-neighbour in strip w - 1 and the values from the patches upstream
//     along a and c come as tagged 64-bit words (tag << 32 | 32 data bits) in
//     the strip's inbox in shared memory.  Strip w - 1 writes the c words of
//     row v - 1 of its own count; the receivers write the rest.
// Words across a patch face go through a global buffer (tag: the launch's
// epoch).  The receivers (one warp for the a-face, one for the c-face, two
// lanes per line: even and odd rows) poll it, up to 8 rows per lane in flight,
// and move what has arrived into the inboxes, so a strip never waits for a
// round trip to L2 of its own.  An inbox slot is reused once the strip has
// published that it took the word (s_prog).  Every wait is bounded.
//
// The backward sweep is the same walk mirrored: patches, strips, lanes and
// rows counted from the other end.
//
// Bound: the chain of Ls + NA + NC rows that the last cell waits for, then the
// bytes of a row (forward 8, backward 7 values per cell).  The former CTA of
// one warp per two lines of c, all eight meeting at a barrier in every row and
// every face lane polling its own word in L2, took per launch 426 us at 256^3
// in FP32 (in clusters of 9 along c) where this takes 270; in FP64 287 / 161 us
// for the half box at 128^3, 105 / 62 us for the dam break at 64^3, 62 / 39 us
// at 16^3 (all with the events around each launch).
//
// The body takes the launch's CTA count (nblocks) as an argument so a launch
// over several solves (k_pencil_sweep_batch) can run it per solve.
constexpr int kStrips = kPatchLines / 32;
constexpr int kPencilThreads = kPatchLines + 64;  // strips, then two receiver warps
constexpr int kInC = 16;   // inbox rows of c words (16 per row)
constexpr int kInA = 32;   // inbox rows of a words (2 per row)
constexpr int kRecv = 8;   // rows a receiver lane polls at once
constexpr long long kInboxPolls = 1ll << 24;  // bound of a wait in shared memory

template <typename R>
struct SweepStages {
  static constexpr int D = sizeof(R) == 4 ? 16 : 8;
};
__host__ __device__ constexpr int sweep_words(int mode, size_t rbytes) {
  return (mode == 0 ? 2 : 1) * (int)(rbytes / 4);  // 64-bit words per edge entry
}
template <typename R>
__host__ __device__ constexpr size_t sweep_ring_bytes(int mode) {
  return (size_t)kStrips * SweepStages<R>::D * sweep_slot(mode) * 32 * sizeof(R);
}
template <typename R>
__host__ __device__ constexpr size_t sweep_dyn_smem(int mode) {
  return sweep_ring_bytes<R>(mode) +
         (size_t)kStrips * (kInC * 16 + kInA * 2) * sweep_words(mode, sizeof(R)) * 8;
}

__device__ inline void cp_async16(unsigned dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ inline void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ inline void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
// EW tagged words of one entry (each 64-bit word is read and written whole and
// carries its own tag)
template <int EW>
__device__ inline void ld_words_shared(unsigned addr, u64* w) {
  if (EW == 1) {
    asm volatile("ld.volatile.shared.u64 %0, [%1];" : "=l"(w[0]) : "r"(addr) : "memory");
  } else {
#pragma unroll
    for (int k = 0; k < EW; k += 2)
      asm volatile("ld.volatile.shared.v2.u64 {%0, %1}, [%2];"
                   : "=l"(w[k]), "=l"(w[k + 1])
                   : "r"(addr + 8 * k)
                   : "memory");
  }
}
template <int EW>
__device__ inline void st_words_shared(unsigned addr, const u64* w) {
  if (EW == 1) {
    asm volatile("st.volatile.shared.u64 [%0], %1;" ::"r"(addr), "l"(w[0]) : "memory");
  } else {
#pragma unroll
    for (int k = 0; k < EW; k += 2)
      asm volatile("st.volatile.shared.v2.u64 [%0], {%1, %2};" ::"r"(addr + 8 * k), "l"(w[k]),
                   "l"(w[k + 1])
                   : "memory");
  }
}
template <int EW>
__device__ inline bool words_tagged(const u64* w, unsigned tag) {
  bool ok = true;
#pragma unroll
  for (int k = 0; k < EW; ++k) ok = ok && (unsigned)(w[k] >> 32) == tag;
  return ok;
}
__device__ inline int ld_volatile_int(unsigned addr) {
  int v;
  asm volatile("ld.volatile.shared.s32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}
__device__ inline void st_volatile_int(unsigned addr, int v) {
  asm volatile("st.volatile.shared.s32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

template <typename R, int MODE, bool UPD>
__device__ __forceinline__ void pencil_sweep_run(const PencilSweepArgs<R>& A, int nblocks) {
  constexpr bool BWD = MODE == kBackward;
  constexpr int PW = MODE == kFactor ? 2 : 1;  // values sent across an edge
  constexpr int TW = TagWords<R>::W;
  constexpr int EW = PW * TW;
  static_assert(kFactor == 0 && kForward == 1 && kBackward == 2, "mode numbering");
  constexpr int D = SweepStages<R>::D;
  constexpr int NF = sweep_slot(MODE);
  constexpr bool TWO = MODE == kBackward || UPD;  // two vectors per row
  constexpr int SLOT = NF * 32;                   // Reals per staged strip row
  constexpr unsigned full = 0xffffffffu;
  __shared__ int s_ticket;
  __shared__ int s_prog[kStrips];
  __shared__ double red[kPatchLines];
  extern __shared__ __align__(128) unsigned char dsm[];  // strip rings, then the inboxes
  const PencilGeom& G = A.G;
  const int tid = threadIdx.x;
  const int lane = tid & 31, w = tid >> 5;
  // one ticket per patch, taken even by a launch that returns at once, so the
  // counter stays in step with the host's base
  if (tid == 0) s_ticket = atomicAdd(A.ticket, 1) - A.ticket_base;
  if (*(const int*)(A.sc + S_DONE)) return;  // set by an earlier launch: uniform
  constexpr int INBOX = (kInC * 16 + kInA * 2) * EW;  // words per strip
  {
    u64* ib = reinterpret_cast<u64*>(dsm + sweep_ring_bytes<R>(MODE));
    for (int i = tid; i < kStrips * INBOX; i += kPencilThreads) ib[i] = 0ull;
    if (tid < kStrips) s_prog[tid] = 0;
  }
  __syncthreads();
  const int tk = s_ticket;
  bool run = true;
  if (tk < 0 || tk >= (int)G.npatch) {
    if (tid == 0) record_error(A.err, kErrIndex);
    run = false;
  }
  double rmax = 0, dsum = 0;
  int p = 0;
  if (run) {
    p = BWD ? A.order[(int)G.npatch - 1 - tk] : A.order[tk];
    const int PAi = p % G.nPA, PCi = p / G.nPA;
    const int Ls = G.Ls;
    const int NV = Ls + kPatch;            // rows of a strip
    const int na = Ls + 1, nc = Ls + 15;   // rows that take a-face and c-face words
    // patches upstream (their words come in) and downstream
    const int up_a = BWD ? (PAi + 1 < G.nPA ? p + 1 : -1) : (PAi > 0 ? p - 1 : -1);
    const int up_c = BWD ? (PCi + 1 < G.nPC ? p + G.nPA : -1) : (PCi > 0 ? p - G.nPA : -1);
    const bool pub_a = BWD ? PAi > 0 : PAi + 1 < G.nPA;
    const bool pub_c = BWD ? PCi > 0 : PCi + 1 < G.nPC;
    const unsigned inbox0 = smem_u32(dsm + sweep_ring_bytes<R>(MODE));
    const unsigned prog0 = smem_u32(s_prog);
    const unsigned ep = A.epoch;
    if (w >= kStrips) {
      // ---- receivers ----
      const bool cface = w == kStrips + 1;
      const int up = cface ? up_c : up_a;
      if (up >= 0) {
        // the tag this patch waits for: the launch's, except on the patch a
        // failure-path test marks, whose waits then run into their limit
        const unsigned want = p == A.stale_patch ? (ep ^ 0x80000000u) : ep;
        const int k = lane & 15;                     // line of the face
        const int strip = cface ? 0 : k >> 1;
        const int rows = cface ? nc : na;
        const unsigned box = inbox0 + (unsigned)(strip * INBOX) * 8u +
                             (cface ? (unsigned)(k * EW) * 8u
                                    : (unsigned)((kInC * 16 + (k & 1)) * EW) * 8u);
        const int depth = cface ? kInC : kInA;
        const unsigned pitch = (cface ? 16u : 2u) * EW * 8u;
        const unsigned prog = prog0 + 4u * strip;
        const u64* src = A.edge + edge_word(G, up, cface ? 1 : 0, 0, k, EW);
        int v = lane >> 4;  // this lane's next row; rows of one parity
        long long idle = 0;
        bool gave_up = false;
        while (__any_sync(full, v < rows)) {
          const int room = ld_volatile_int(prog) + depth;  // rows below it may be written
          // a lane that saw nothing new polls one row, else kRecv rows
          const int most = idle > 0 ? 1 : kRecv;
          u64 wd[kRecv][EW];
          bool mine[kRecv];
#pragma unroll
          for (int j = 0; j < kRecv; ++j) {
            const int vj = v + 2 * j;
            mine[j] = j < most && vj < rows && vj < room;
            if (mine[j]) {
#pragma unroll
              for (int q = 0; q < EW; ++q)
                wd[j][q] = ld_relaxed_u64(src + (long long)vj * (16 * EW) + q);
            }
          }
          int got = 0;
          bool open = true;
#pragma unroll
          for (int j = 0; j < kRecv; ++j) {
            const int vj = v + 2 * j;
            if (mine[j] && gave_up) {
#pragma unroll
              for (int q = 0; q < EW; ++q) wd[j][q] = (u64)want << 32;
            }
            open = open && mine[j] && words_tagged<EW>(wd[j], want);
            if (open) {
              u64 o[EW];
#pragma unroll
              for (int q = 0; q < EW; ++q)
                o[q] = ((u64)(unsigned)(vj + 1) << 32) | (wd[j][q] & 0xffffffffull);
              st_words_shared<EW>(box + (unsigned)(vj & (depth - 1)) * pitch, o);
              got = j + 1;
            }
          }
          v += 2 * got;
          if (got > 0) {
            idle = 0;
          } else if (v < rows && v < room) {
            if (++idle > A.spin_limit && !gave_up) {
              record_error(A.err, kErrWaitTimeout);
              gave_up = true;
            }
          } else if (v < rows && ++idle > kInboxPolls) {
            // the strip no longer takes words (its own wait gave up)
            record_error(A.err, kErrWaitTimeout);
            v = rows;
          }
        }
      }
    } else {
      // ---- strips ----
      // mirrored for the backward sweep: strip w walks the physical strip 7 - w
      // and lane l the physical lane 31 - l, rows from the end
      const int pl = BWD ? 31 - lane : lane;
      const int ps = BWD ? kStrips - 1 - w : w;
      const long long pbase = (long long)p * G.R * kPatchLines + 32 * ps;
      const int t0 = BWD ? G.R - 1 - 2 * w : 2 * w;
      constexpr int RS = BWD ? -kPatchLines : kPatchLines;  // element step per row
      const long long row0 = pbase + (long long)t0 * kPatchLines;
      R* const ring = reinterpret_cast<R*>(dsm) + (size_t)w * D * SLOT;
      const unsigned ring0 = smem_u32(ring);
      // copies of one row: 16 bytes per lane and pass
      constexpr int RW = 32 * sizeof(R);  // bytes of one strip row
      constexpr int PR = RW / 16;         // lanes that copy one array's row
      auto issue = [&](int v) {
        if (v < NV) {
          const long long e = row0 + (long long)v * RS;
          const unsigned dst = ring0 + (unsigned)(v & (D - 1)) * (SLOT * (unsigned)sizeof(R));
          if (MODE == kFactor) {
            const R* a4[4] = {A.AD, A.AS, A.AA, A.AC};
#pragma unroll
            for (int i = 0; i < 4 * PR / 32; ++i) {
              const int c = lane + 32 * i;
              const int arr = c / PR, off = c % PR;
              const R* s = arr == 0 ? a4[0] : (arr == 1 ? a4[1] : (arr == 2 ? a4[2] : a4[3]));
              cp_async16(dst + arr * RW + off * 16,
                         reinterpret_cast<const unsigned char*>(s + e) + off * 16);
            }
          } else {
            // the vectors (one or two rows), then the factor (four rows' worth)
            const R* v1 = MODE == kForward ? A.q : A.r;
            if (lane < (TWO ? 2 : 1) * PR) {
              const R* s = lane < PR ? A.in : v1;
              const int off = lane % PR;
              cp_async16(dst + (lane / PR) * RW + off * 16,
                         reinterpret_cast<const unsigned char*>(s + e) + off * 16);
            }
#pragma unroll
            for (int i = 0; i < PR * 4 / 32; ++i)
              cp_async16(dst + 2 * RW + (lane + 32 * i) * 16,
                         reinterpret_cast<const unsigned char*>(A.coef + 4 * e) +
                             (lane + 32 * i) * 16);
          }
        }
        cp_async_commit();
      };
      for (int j = 0; j < D; ++j) issue(j);

      // the words this lane takes: lanes 0..15 the c-face, 16 and 17 the
      // a-face lines 2w and 2w + 1
      const bool has_c = w > 0 || up_c >= 0, has_a = up_a >= 0;
      const int vlim = lane < 16 ? (has_c ? nc : 0) : (lane < 18 && has_a ? na : 0);
      const unsigned box = inbox0 + (unsigned)(w * INBOX) * 8u;
      const unsigned wsrc =
          lane < 16 ? box + (unsigned)(lane * EW) * 8u
                    : box + (unsigned)((kInC * 16 + (lane & 1)) * EW) * 8u;
      const int wmask = lane < 16 ? kInC - 1 : kInA - 1;
      const unsigned wpitch = (lane < 16 ? 16u : 2u) * EW * 8u;
      // outgoing: lanes 16..31 the c words of row v - 1 of the next strip (or
      // of the patch downstream), lanes 15 and 31 the a-face words of row v - 15
      const bool to_box = w + 1 < kStrips;
      const bool put_c = lane >= 16 && (to_box || pub_c);
      const bool put_a = (lane & 15) == 15 && pub_a;
      const unsigned obox = inbox0 + (unsigned)((w + 1) * INBOX) * 8u +
                            (unsigned)((lane & 15) * EW) * 8u;
      u64* const gc = A.edge + edge_word(G, p, 1, 0, lane & 15, EW);
      u64* const ga = A.edge + edge_word(G, p, 0, 0, 2 * w + (lane >> 4), EW);
      const unsigned prog = prog0 + 4u * w;
      const R al_r = (MODE == kForward && UPD) ? (R)A.sc[S_ALPHA] : R(0);
      const R omega = A.omega, min_ratio = A.min_ratio;
      const long long eb = row0 + pl;
      R* const pcoef = MODE == kFactor ? A.coef + 4 * eb : nullptr;
      R* const o_out = MODE == kFactor ? nullptr : A.out + eb;
      R* const o_r = (MODE == kForward && UPD) ? A.r + eb : nullptr;
      R carry[PW], prev_a[PW], prev_c[PW], f[NF];
#pragma unroll
      for (int k = 0; k < PW; ++k) carry[k] = prev_a[k] = prev_c[k] = R(0);
      R rm = 0;
      bool gave_up = false;
      u64 wd[EW];
      auto load_row = [&](int v) {
        const R* S = ring + (size_t)(v & (D - 1)) * SLOT;
        if (MODE == kFactor) {
#pragma unroll
          for (int k = 0; k < 4; ++k) f[k] = S[32 * k + pl];
        } else {
          f[0] = S[pl];
          if (TWO) f[NF - 1] = S[32 + pl];
          ld_coef_shared(S + 64 + 4 * pl, f + 1);
        }
      };
      cp_async_wait<D - 1>();
      __syncwarp();
      load_row(0);
      ld_words_shared<EW>(wsrc, wd);
      int room = kInC;  // rows the next strip's inbox can take
#pragma unroll 2
      for (int v = 0; v < NV; ++v) {
        // this row's incoming words
        {
          const bool need = v < vlim;
          const unsigned tag = (unsigned)(v + 1);
          bool ok = !need || words_tagged<EW>(wd, tag);
          if (!__all_sync(full, ok)) {
            long long it = 0;
            while (!__all_sync(full, ok) && !gave_up) {
              if (!ok) {
                ld_words_shared<EW>(wsrc + (unsigned)(v & wmask) * wpitch, wd);
                ok = words_tagged<EW>(wd, tag);
              }
              if (++it > kInboxPolls) {
                if (lane == 0) record_error(A.err, kErrWaitTimeout);
                gave_up = true;
              }
            }
          }
        }
        R in_a[PW], in_c[PW];
        {
          R word[PW];
#pragma unroll
          for (int k = 0; k < PW; ++k) {
            word[k] = v < vlim ? TagWords<R>::unpack(wd + k * TW) : R(0);
            const R wa = __shfl_sync(full, word[k], 16 + (lane >> 4));
            const R sa = __shfl_up_sync(full, prev_a[k], 1);
            const R sc = __shfl_up_sync(full, prev_c[k], 16);
            in_a[k] = (lane & 15) == 0 ? wa : sa;
            in_c[k] = lane < 16 ? word[k] : sc;
          }
        }
        // the next row's words, read early; taken once their tag is right
        ld_words_shared<EW>(wsrc + (unsigned)((v + 1) & wmask) * wpitch, wd);
        if ((v & 3) == 3 && lane == 0) st_volatile_int(prog, v + 1);
        const long long off = (long long)v * RS;
        R out_s[PW], out_a[PW], out_c[PW];
        if (MODE == kFactor) {
          const R ad = f[0];
          R d = ad;
          R iv = R(0);
          if (ad != R(0)) {
            d = d - in_c[0] * in_c[0];
            d = d - (omega * in_c[0]) * in_c[PW - 1];
            d = d - in_a[0] * in_a[0];
            d = d - (omega * in_a[0]) * in_a[PW - 1];
            d = d - carry[0] * carry[0];
            d = d - (omega * carry[0]) * carry[PW - 1];
            const R piv = d < min_ratio * ad ? ad : d;
            iv = R(1) / sqrt(piv);
          }
          const R ss = f[1] * iv, sa = f[2] * iv, scv = f[3] * iv;
          st_coef(pcoef + 4 * off, iv, ss, sa, scv);
          out_s[0] = ss; out_s[PW - 1] = sa + scv;
          out_a[0] = sa; out_a[PW - 1] = ss + scv;
          out_c[0] = scv; out_c[PW - 1] = ss + sa;
        } else if (MODE == kForward) {
          R rv = f[0];
          if (UPD) {
            rv = rv - al_r * f[NF - 1];
            o_r[off] = rv;
            const R av = fabs(rv);
            rm = av > rm ? av : rm;
          }
          R vv = rv;
          vv -= in_c[0];
          vv -= in_a[0];
          vv -= carry[0];
          const R y = vv * f[1];
          o_out[off] = y;
          out_s[0] = f[2] * y;
          out_a[0] = f[3] * y;
          out_c[0] = f[NF - 2] * y;
        } else {
          R vv = f[0];
          vv -= f[2] * carry[0];
          vv -= f[3] * in_a[0];
          vv -= f[NF - 2] * in_c[0];
          const R z = vv * f[1];
          o_out[off] = z;
          dsum += (double)z * (double)f[NF - 1];
          out_s[0] = out_a[0] = out_c[0] = z;
        }
        // c words of row v - 1 downstream
        if (to_box) {
          if (v >= room + 1) {
            // the next strip has to take a row first
            long long it = 0;
            const unsigned np = prog0 + 4u * (w + 1);
            do {
              room = ld_volatile_int(np) + kInC;
              if (++it > kInboxPolls) {
                if (lane == 0) record_error(A.err, kErrWaitTimeout);
                gave_up = true;
                room = 1 << 30;
              }
            } while (v >= room + 1);
          }
          if (put_c && v > 0) {
            u64 o[EW];
#pragma unroll
            for (int k = 0; k < PW; ++k) TagWords<R>::pack(out_c[k], (unsigned)v, o + k * TW);
            st_words_shared<EW>(obox + (unsigned)((v - 1) & (kInC - 1)) * (16u * EW * 8u), o);
          }
        } else if (put_c && v > 0) {
          u64 o[EW];
#pragma unroll
          for (int k = 0; k < PW; ++k) TagWords<R>::pack(out_c[k], ep, o + k * TW);
#pragma unroll
          for (int k = 0; k < EW; ++k)
            st_relaxed_u64(gc + (long long)(v - 1) * (16 * EW) + k, o[k]);
        }
        if (put_a && v >= kPatch - 1) {
          u64 o[EW];
#pragma unroll
          for (int k = 0; k < PW; ++k) TagWords<R>::pack(out_a[k], ep, o + k * TW);
#pragma unroll
          for (int k = 0; k < EW; ++k)
            st_relaxed_u64(ga + (long long)(v - (kPatch - 1)) * (16 * EW) + k, o[k]);
        }
#pragma unroll
        for (int k = 0; k < PW; ++k) {
          prev_a[k] = out_a[k];
          prev_c[k] = out_c[k];
          carry[k] = out_s[k];
        }
        // every lane has read row v (the shuffles above follow its loads), so
        // its slot takes row v + D
        __syncwarp();
        issue(v + D);
        cp_async_wait<D - 1>();
        __syncwarp();
        if (v + 1 < NV) load_row(v + 1);
      }
      if (lane == 0) st_volatile_int(prog, 1 << 29);  // nothing waits for this strip any more
      cp_async_wait<0>();
      rmax = (double)rm;
    }
  }
  // partials, summed in line order whatever the direction
  if (A.part && ((MODE == kForward && UPD) || MODE == kBackward)) {
    const int line = BWD ? kPatchLines - 1 - tid : tid;
    if (tid < kPatchLines) red[line] = MODE == kForward ? rmax : dsum;
    __syncthreads();
    if (MODE == kForward) {
      const double m = tree_max(red);
      if (tid == 0 && run) A.part[p] = m;
    } else {
      const double sm = tree_sum(red);
      if (tid == 0 && run) A.part[p] = sm;
    }
    // every CTA counts, running or not; the last one reduces the partials
    if (A.done_ctr && last_block(A.done_ctr, nblocks)) {
      if (MODE == kForward)
        red_conv_body(A.part, A.npart, A.sc, red);
      else
        red_beta_body(A.part, A.npart, A.sc, red, A.red_init);
    }
  }
}

template <typename R, int MODE, bool UPD>
__global__ void __launch_bounds__(kPencilThreads, 1)
    k_pencil_sweep(const PencilSweepArgs<R> A) {
  pencil_sweep_run<R, MODE, UPD>(A, (int)gridDim.x);
}

// The solve of block b in a launch over several solves: first[] holds each
// solve's first block (first[n] = the grid), so b lies in [first[s],
// first[s + 1]).
__device__ inline int batch_solve_of(const int* __restrict__ first, int n, int b) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (__ldg(first + mid) <= b) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// One sweep launch over several solves (the shared solve of a batch of
// scenes): solve s owns first[s + 1] - first[s] CTAs (its patches) and its
// arguments come from tab[s].  Launch k of a chunk advances each solve's
// edge-word epoch by k and its ticket base by k launches of its patches, as k
// separate launches would.
template <typename R, int MODE, bool UPD>
__global__ void __launch_bounds__(kPencilThreads, 1)
    k_pencil_sweep_batch(const PencilSweepArgs<R>* __restrict__ tab, const int* __restrict__ first,
                         int nsolve, int k) {
  const int s = batch_solve_of(first, nsolve, (int)blockIdx.x);
  PencilSweepArgs<R> A = tab[s];
  const int nb = __ldg(first + s + 1) - __ldg(first + s);
  A.epoch += (unsigned)k;
  A.ticket_base += k * nb;
  pencil_sweep_run<R, MODE, UPD>(A, nb);
}

// x += alpha s (the update of the last PCG iteration, which no SpMV follows)
template <typename R>
__global__ void k_pl_axpy(long long len, const double* __restrict__ sc, const R* __restrict__ s,
                          R* __restrict__ x) {
  const R al = (R)sc[S_ALPHA];
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < len;
       e += (long long)gridDim.x * blockDim.x)
    x[e] = x[e] + al * s[e];
}

// ---- streaming kernels over the pencil layout --------------------------------
// Element e -> (patch, row, line) and the cell's position in the box.
struct PlCell {
  long long p;
  int t, l, al, cl, PAi, PCi, s;
  bool live;
};

// Cell of line l in row `row` (= patch * R + t) of the layout; 32-bit math
// (npatch * R stays far below 2^31).
__device__ inline PlCell pl_cell(const PencilGeom& G, int row, int l) {
  PlCell c;
  const int p = row / G.R;
  c.p = p;
  c.t = row - p * G.R;
  c.l = l;
  c.al = l & (kPatch - 1);
  c.cl = l / kPatch;
  c.PAi = p % G.nPA;
  c.PCi = p / G.nPA;
  c.s = c.t - c.al - c.cl;
  c.live = c.s >= 0 && c.s < G.Ls && c.PAi * kPatch + c.al < G.NA &&
           c.PCi * kPatch + c.cl < G.NC;
  return c;
}

// Indices of the six neighbours of a live cell (-1 where the box ends).
struct PlNbr {
  long long ms, ps, ma, pa, mc, pc;
};

__device__ inline PlNbr pl_nbr(const PencilGeom& G, const PlCell& c, long long e) {
  PlNbr n;
  n.ms = c.s > 0 ? e - kPatchLines : -1;
  n.ps = c.s + 1 < G.Ls ? e + kPatchLines : -1;
  if (c.al > 0) n.ma = e - kPatchLines - 1;
  else n.ma = c.PAi > 0 ? pl_index(G, c.p - 1, c.t + kPatch - 1, c.l + kPatch - 1) : -1;
  if (c.al < kPatch - 1) n.pa = e + kPatchLines + 1;
  else n.pa = c.PAi + 1 < G.nPA ? pl_index(G, c.p + 1, c.t - (kPatch - 1), c.l - (kPatch - 1)) : -1;
  if (c.cl > 0) n.mc = e - kPatchLines - kPatch;
  else n.mc = c.PCi > 0 ? pl_index(G, c.p - G.nPA, c.t + kPatch - 1,
                                    c.l + kPatch * (kPatch - 1)) : -1;
  if (c.cl < kPatch - 1) n.pc = e + kPatchLines + kPatch;
  else n.pc = c.PCi + 1 < G.nPC ? pl_index(G, c.p + G.nPA, c.t - (kPatch - 1),
                                            c.l - kPatch * (kPatch - 1)) : -1;
  return n;
}

// s_new = z + beta s_old (at all 7 stencil points), q = A s_new,
// partial[block] = sum s_new.q.  Row order of the reference's sorted row for
// interior cells: -c, -a, -s, diagonal, +s, +a, +c.
//
// The previous iteration's x += alpha s_old is applied here too (alpha is
// still the previous iteration's when this kernel runs; 0 before the first).
//
// Block bid of nblk: the arithmetic of k_pl_spmv_s (below) for one solve of a
// launch over several solves (k_pl_spmv_batch).
template <typename R>
__device__ __forceinline__ void pl_spmv_run(
    const PencilGeom& G, const R* __restrict__ AD, const R* __restrict__ AS,
    const R* __restrict__ AA, const R* __restrict__ AC, const R* __restrict__ z,
    const R* __restrict__ sold, R* __restrict__ snew, R* __restrict__ q, R* __restrict__ x,
    double* __restrict__ sc, double* __restrict__ partial, int* __restrict__ done_ctr, int bid,
    int nblk) {
  __shared__ double sm[kRedThreads];
  if (*(const int*)(sc + S_DONE)) return;
  const R be = (R)sc[S_BETA];
  const R al = (R)sc[S_ALPHA];
  double acc = 0;
  const int nrow = (int)(G.npatch * G.R);
  for (int row = bid; row < nrow; row += nblk) {
    const long long e = (long long)row * kPatchLines + threadIdx.x;
    const PlCell c = pl_cell(G, row, threadIdx.x);
    if (!c.live) continue;
    const PlNbr n = pl_nbr(G, c, e);
    R r = 0;
    if (n.mc >= 0) r += AC[n.mc] * (z[n.mc] + be * sold[n.mc]);
    if (n.ma >= 0) r += AA[n.ma] * (z[n.ma] + be * sold[n.ma]);
    if (n.ms >= 0) r += AS[n.ms] * (z[n.ms] + be * sold[n.ms]);
    const R so = sold[e];
    x[e] = x[e] + al * so;
    const R sn = z[e] + be * so;
    r += AD[e] * sn;
    if (n.ps >= 0) r += AS[e] * (z[n.ps] + be * sold[n.ps]);
    if (n.pa >= 0) r += AA[e] * (z[n.pa] + be * sold[n.pa]);
    if (n.pc >= 0) r += AC[e] * (z[n.pc] + be * sold[n.pc]);
    snew[e] = sn;
    q[e] = r;
    acc += (double)sn * (double)r;
  }
  acc = block_sum<double>(acc, sm);
  if (threadIdx.x == 0) partial[bid] = acc;
  // the last block: alpha = rho / s.q (k_red_alpha's body)
  if (done_ctr && last_block(done_ctr, nblk)) red_alpha_body(partial, nblk, sc, sm);
}

// (written out rather than through pl_spmv_run: the launch alone ran about
// 10 % slower through the shared body)
template <typename R>
__global__ void __launch_bounds__(kRedThreads, sizeof(R) == 4 ? 8 : 4)
    k_pl_spmv_s(PencilGeom G, const R* __restrict__ AD, const R* __restrict__ AS,
                const R* __restrict__ AA, const R* __restrict__ AC, const R* __restrict__ z,
                const R* __restrict__ sold, R* __restrict__ snew, R* __restrict__ q,
                R* __restrict__ x, double* __restrict__ sc,
                double* __restrict__ partial, int* __restrict__ done_ctr) {
  __shared__ double sm[kRedThreads];
  if (*(const int*)(sc + S_DONE)) return;
  const R be = (R)sc[S_BETA];
  const R al = (R)sc[S_ALPHA];
  double acc = 0;
  const int nrow = (int)(G.npatch * G.R);
  for (int row = blockIdx.x; row < nrow; row += gridDim.x) {
    const long long e = (long long)row * kPatchLines + threadIdx.x;
    const PlCell c = pl_cell(G, row, threadIdx.x);
    if (!c.live) continue;
    const PlNbr n = pl_nbr(G, c, e);
    R r = 0;
    if (n.mc >= 0) r += AC[n.mc] * (z[n.mc] + be * sold[n.mc]);
    if (n.ma >= 0) r += AA[n.ma] * (z[n.ma] + be * sold[n.ma]);
    if (n.ms >= 0) r += AS[n.ms] * (z[n.ms] + be * sold[n.ms]);
    const R so = sold[e];
    x[e] = x[e] + al * so;
    const R sn = z[e] + be * so;
    r += AD[e] * sn;
    if (n.ps >= 0) r += AS[e] * (z[n.ps] + be * sold[n.ps]);
    if (n.pa >= 0) r += AA[e] * (z[n.pa] + be * sold[n.pa]);
    if (n.pc >= 0) r += AC[e] * (z[n.pc] + be * sold[n.pc]);
    snew[e] = sn;
    q[e] = r;
    acc += (double)sn * (double)r;
  }
  acc = block_sum<double>(acc, sm);
  if (threadIdx.x == 0) partial[blockIdx.x] = acc;
  // the last block: alpha = rho / s.q (k_red_alpha's body)
  if (done_ctr && last_block(done_ctr, (int)gridDim.x))
    red_alpha_body(partial, (int)gridDim.x, sc, sm);
}

// Blocks of k_pl_spmv_s for a layout: about four rows per block, at most the
// resident capacity (kPlSpmvBlocks32).  The partial sums of s.q follow the
// block count, so a solve alone and in a launch over several solves use this
// same count and give the same bits.
__host__ __device__ inline int pl_spmv_blocks(const PencilGeom& G) {
  const long long nrow = G.npatch * G.R;
  const long long b = (nrow + 3) / 4;
  return (int)(b < 1 ? 1 : (b > kPlSpmvBlocks32 ? kPlSpmvBlocks32 : b));
}

// One SpMV launch over several solves: solve s owns first[s + 1] - first[s]
// blocks; iteration it of a chunk takes s_old / s_new from s0 / s1 by the
// solve's iteration parity.
template <typename R>
struct PlSpmvArgs {
  PencilGeom G;
  const R* AD;
  const R* AS;
  const R* AA;
  const R* AC;
  const R* z;
  R* s0;
  R* s1;
  R* q;
  R* x;
  double* sc;
  double* part;
  int* done_ctr;
  int parity;  // iterations the solve ran before the chunk, mod 2
};

template <typename R>
__global__ void __launch_bounds__(kRedThreads, sizeof(R) == 4 ? 6 : 3)
    k_pl_spmv_batch(const PlSpmvArgs<R>* __restrict__ tab, const int* __restrict__ first,
                    int nsolve, int it) {
  const int s = batch_solve_of(first, nsolve, (int)blockIdx.x);
  const PlSpmvArgs<R>& a = tab[s];
  const int b0 = __ldg(first + s);
  const bool odd = ((a.parity + it) & 1) != 0;
  pl_spmv_run<R>(a.G, a.AD, a.AS, a.AA, a.AC, a.z, odd ? a.s1 : a.s0, odd ? a.s0 : a.s1, a.q,
                 a.x, a.sc, a.part, a.done_ctr, (int)blockIdx.x - b0, __ldg(first + s + 1) - b0);
}

// status[6 s + j] = sc_s[S_RES + j] (residual, beta, tolerance, iteration,
// iteration limit, done) for each solve of a chunk
__global__ void k_pl_batch_status(double* const* __restrict__ scs, int nsolve,
                                  double* __restrict__ status) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < 6 * nsolve) status[i] = __ldcg(scs[i / 6] + S_RES + i % 6);
}

// k_pl_spmv_s's arithmetic, streamed: block (patch p, chunk k) walks rows
// [t0, t1) of one patch in order, one thread per line.  s_new of rows t - 1,
// t and t + 1 sits in a ring of three shared-memory rows and the couplings
// A_s, A_a, A_c of row t - 1 in a second ring, so every in-patch neighbour
// (one row back or ahead, the same line, line -+1 or line -+16) is read from
// shared memory and each value is loaded from global memory once; only the
// neighbours across a patch face (lines at a = 0 / 15, c = 0 / 15) are read
// from global memory as k_pl_spmv_s reads them.  Terms are summed in the same
// order as k_pl_spmv_s, missing neighbours skipped.  partial[block] = s_new.q
// over the chunk (blocks ordered patch-major, then chunk).
template <typename R>
__global__ void __launch_bounds__(kRedThreads)
    k_pl_spmv_stream(PencilGeom G, int rows_per_chunk, int nchunk, const R* __restrict__ AD,
                     const R* __restrict__ AS, const R* __restrict__ AA,
                     const R* __restrict__ AC, const R* __restrict__ z,
                     const R* __restrict__ sold, R* __restrict__ snew, R* __restrict__ q,
                     R* __restrict__ x, const double* __restrict__ sc,
                     double* __restrict__ partial) {
  __shared__ R ring[3][kPatchLines];
  __shared__ R cs[2][kPatchLines], ca[2][kPatchLines], cc[2][kPatchLines];
  __shared__ double sm[kRedThreads];
  if (*(const int*)(sc + S_DONE)) return;
  const R be = (R)sc[S_BETA];
  const R al = (R)sc[S_ALPHA];
  const int l = threadIdx.x;
  const int p = blockIdx.x / nchunk;
  const int k = blockIdx.x - p * nchunk;
  const int t0 = k * rows_per_chunk;
  const int t1 = min(G.R, t0 + rows_per_chunk);
  double acc = 0;
  if (t0 < t1) {
    const long long base = (long long)p * G.R * kPatchLines + l;
    // s_new and the couplings of row t0 - 1 (zero before the first row)
    if (t0 > 0) {
      const long long e = base + (long long)(t0 - 1) * kPatchLines;
      ring[(t0 + 2) % 3][l] = z[e] + be * sold[e];
      cs[(t0 + 1) & 1][l] = AS[e];
      ca[(t0 + 1) & 1][l] = AA[e];
      cc[(t0 + 1) & 1][l] = AC[e];
    } else {
      ring[2][l] = R(0);
      cs[1][l] = ca[1][l] = cc[1][l] = R(0);
    }
    // row t's own values and row t + 1's z, s_old, held one row ahead in
    // registers so the loads of the next row overlap this row's work
    long long e0 = base + (long long)t0 * kPatchLines;
    R nz = z[e0], ns = sold[e0];
    ring[t0 % 3][l] = nz + be * ns;
    R ad = AD[e0], as = AS[e0], aa = AA[e0], ac = AC[e0], so = ns, xv = x[e0];
    if (t0 + 1 < G.R) {
      nz = z[e0 + kPatchLines];
      ns = sold[e0 + kPatchLines];
    }
    for (int t = t0; t < t1; ++t) {
      const long long e = base + (long long)t * kPatchLines;
      if (t + 1 < G.R) ring[(t + 1) % 3][l] = nz + be * ns;
      cs[t & 1][l] = as;
      ca[t & 1][l] = aa;
      cc[t & 1][l] = ac;
      const R ns1 = ns;
      // prefetch: row t + 1's own values, row t + 2's z and s_old
      R ad_n = 0, as_n = 0, aa_n = 0, ac_n = 0, xv_n = 0;
      if (t + 1 < t1) {
        ad_n = AD[e + kPatchLines];
        as_n = AS[e + kPatchLines];
        aa_n = AA[e + kPatchLines];
        ac_n = AC[e + kPatchLines];
        xv_n = x[e + kPatchLines];
        if (t + 2 < G.R) {
          nz = z[e + 2 * kPatchLines];
          ns = sold[e + 2 * kPatchLines];
        }
      }
      __syncthreads();
      const PlCell c = pl_cell(G, p * G.R + t, l);
      if (c.live) {
        const R* sm1 = ring[(t + 2) % 3];
        const R* s0 = ring[t % 3];
        const R* sp1 = ring[(t + 1) % 3];
        const int pr = (t + 1) & 1;  // coupling ring slot of row t - 1
        R r = 0;
        // -c
        if (c.cl > 0) {
          r += cc[pr][l - kPatch] * sm1[l - kPatch];
        } else if (c.PCi > 0) {
          const long long n = pl_index(G, p - G.nPA, t + kPatch - 1, l + kPatch * (kPatch - 1));
          r += AC[n] * (z[n] + be * sold[n]);
        }
        // -a
        if (c.al > 0) {
          r += ca[pr][l - 1] * sm1[l - 1];
        } else if (c.PAi > 0) {
          const long long n = pl_index(G, p - 1, t + kPatch - 1, l + kPatch - 1);
          r += AA[n] * (z[n] + be * sold[n]);
        }
        // -s
        if (c.s > 0) r += cs[pr][l] * sm1[l];
        x[e] = xv + al * so;
        const R sn = s0[l];
        r += ad * sn;
        // +s
        if (c.s + 1 < G.Ls) r += as * sp1[l];
        // +a
        if (c.al < kPatch - 1) {
          r += aa * sp1[l + 1];
        } else if (c.PAi + 1 < G.nPA) {
          const long long n = pl_index(G, p + 1, t - (kPatch - 1), l - (kPatch - 1));
          r += aa * (z[n] + be * sold[n]);
        }
        // +c
        if (c.cl < kPatch - 1) {
          r += ac * sp1[l + kPatch];
        } else if (c.PCi + 1 < G.nPC) {
          const long long n = pl_index(G, p + G.nPA, t - (kPatch - 1), l - kPatch * (kPatch - 1));
          r += ac * (z[n] + be * sold[n]);
        }
        snew[e] = sn;
        q[e] = r;
        acc += (double)sn * (double)r;
      }
      ad = ad_n;
      as = as_n;
      aa = aa_n;
      ac = ac_n;
      xv = xv_n;
      so = ns1;
      __syncthreads();
    }
  }
  acc = block_sum<double>(acc, sm);
  if (threadIdx.x == 0) partial[blockIdx.x] = acc;
}

// FP64 residual r64 = b - A x64 with the coefficients promoted; partial max|r64|
template <typename R>
__global__ void __launch_bounds__(kRedThreads)
    k_pl_residual64(PencilGeom G, const R* __restrict__ AD, const R* __restrict__ AS,
                    const R* __restrict__ AA, const R* __restrict__ AC,
                    const R* __restrict__ b, const double* __restrict__ x,
                    double* __restrict__ r, double* __restrict__ partial) {
  __shared__ double sm[kRedThreads];
  double m = 0;
  const int nrow = (int)(G.npatch * G.R);
  for (int row = blockIdx.x; row < nrow; row += gridDim.x) {
    const long long e = (long long)row * kPatchLines + threadIdx.x;
    const PlCell c = pl_cell(G, row, threadIdx.x);
    if (!c.live) continue;
    const PlNbr n = pl_nbr(G, c, e);
    double acc = (double)AD[e] * x[e];
    if (n.ms >= 0) acc += (double)AS[n.ms] * x[n.ms];
    if (n.ma >= 0) acc += (double)AA[n.ma] * x[n.ma];
    if (n.mc >= 0) acc += (double)AC[n.mc] * x[n.mc];
    if (n.ps >= 0) acc += (double)AS[e] * x[n.ps];
    if (n.pa >= 0) acc += (double)AA[e] * x[n.pa];
    if (n.pc >= 0) acc += (double)AC[e] * x[n.pc];
    const double rv = (double)b[e] - acc;
    r[e] = rv;
    const double av = fabs(rv);
    m = av > m ? av : m;
  }
  m = block_max<double>(m, sm);
  if (threadIdx.x == 0) partial[blockIdx.x] = m;
}

// r32 = r64 / res, x32 = 0 (inner solve of one refinement)
template <typename R>
__global__ void k_pl_demote(long long len, const double* __restrict__ r64,
                            const double* __restrict__ sc, R* __restrict__ r,
                            R* __restrict__ x) {
  const double scale = 1.0 / sc[0];
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < len;
       e += (long long)gridDim.x * blockDim.x) {
    r[e] = (R)(r64[e] * scale);
    x[e] = R(0);
  }
}

// x64 += x32 * res
template <typename R>
__global__ void k_pl_accumulate(long long len, const R* __restrict__ x,
                                const double* __restrict__ sc, double* __restrict__ x64) {
  const double s = sc[0];
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < len;
       e += (long long)gridDim.x * blockDim.x)
    x64[e] += (double)x[e] * s;
}

// r64 = b (promoted)
template <typename R>
__global__ void k_pl_promote(long long len, const R* __restrict__ b, double* __restrict__ o) {
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < len;
       e += (long long)gridDim.x * blockDim.x)
    o[e] = (double)b[e];
}

// The DOF box: block-reduced min/max of the DOF cell coordinates into
// bbox[0..5] (min x,y,z, max x,y,z) and the DOF count into partial[block].
__global__ void __launch_bounds__(kRedThreads)
    k_dof_box(GridDesc g, const int* __restrict__ active_list, long long nent,
              const unsigned char* __restrict__ dof, int* __restrict__ bbox,
              double* __restrict__ partial) {
  __shared__ int smn[3][kRedThreads / 32], smx[3][kRedThreads / 32];
  __shared__ double sm[kRedThreads];
  int mn[3] = {1 << 30, 1 << 30, 1 << 30}, mx[3] = {-1, -1, -1};
  double cnt = 0;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < nent;
       e += (long long)gridDim.x * blockDim.x) {
    const long long n = active_node(active_list, e);
    if (!(dof[n] & 1)) continue;
    int I, J, K;
    node_ijk(g, n, I, J, K);
    const int v[3] = {I, J, K};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      mn[a] = v[a] < mn[a] ? v[a] : mn[a];
      mx[a] = v[a] > mx[a] ? v[a] : mx[a];
    }
    cnt += 1.0;
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const int wmn = __reduce_min_sync(0xffffffffu, mn[a]);
    const int wmx = __reduce_max_sync(0xffffffffu, mx[a]);
    if (lane == 0) { smn[a][wid] = wmn; smx[a][wid] = wmx; }
  }
  cnt = block_sum<double>(cnt, sm);  // contains __syncthreads
  if (threadIdx.x == 0) {
    partial[blockIdx.x] = cnt;
    for (int a = 0; a < 3; ++a) {
      int bmn = 1 << 30, bmx = -1;
      for (int w = 0; w < kRedThreads / 32; ++w) {
        bmn = smn[a][w] < bmn ? smn[a][w] : bmn;
        bmx = smx[a][w] > bmx ? smx[a][w] : bmx;
      }
      if (bmx >= 0) {
        atomicMin(bbox + a, bmn);
        atomicMax(bbox + 3 + a, bmx);
      }
    }
  }
}

// Gather the assembled system into the pencil layout.  Couplings are kept
// only between two DOF cells (the reference's matrix has no other entries).
template <typename R>
__global__ void __launch_bounds__(kRedThreads)
    k_pl_gather(PencilGeom G, GridDesc g, const unsigned char* __restrict__ active,
                const unsigned char* __restrict__ dof, const R* __restrict__ F,
                long long fs, R* __restrict__ AD, R* __restrict__ AS, R* __restrict__ AA,
                R* __restrict__ AC, R* __restrict__ B) {
  const int nrow = (int)(G.npatch * G.R);
  for (int row = blockIdx.x; row < nrow; row += gridDim.x) {
    const long long e = (long long)row * kPatchLines + threadIdx.x;
    const PlCell c = pl_cell(G, row, threadIdx.x);
    R ad = 0, as = 0, aa = 0, ac = 0, bv = 0;
    if (c.live) {
      int P[3];
      P[G.ax_s] = G.lo[G.ax_s] + c.s;
      P[G.ax_a] = G.lo[G.ax_a] + c.PAi * kPatch + c.al;
      P[G.ax_c] = G.lo[G.ax_c] + c.PCi * kPatch + c.cl;
      if (in_grid(g, P[0], P[1], P[2]) && active[bucket_of(g, P[0], P[1], P[2])]) {
        const long long n = node_linear(g, P[0], P[1], P[2]);
        if (dof[n] & 1) {
          ad = F[G_ADIAG * fs + n];
          bv = F[G_B * fs + n];
          const int axes[3] = {G.ax_s, G.ax_a, G.ax_c};
          R cpl[3];
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            int Q[3] = {P[0], P[1], P[2]};
            Q[axes[k]] += 1;
            cpl[k] = R(0);
            if (in_grid(g, Q[0], Q[1], Q[2]) && active[bucket_of(g, Q[0], Q[1], Q[2])] &&
                (dof[node_linear(g, Q[0], Q[1], Q[2])] & 1))
              cpl[k] = F[(G_AX + axes[k]) * fs + n];
          }
          as = cpl[0]; aa = cpl[1]; ac = cpl[2];
        }
      }
    }
    AD[e] = ad; AS[e] = as; AA[e] = aa; AC[e] = ac; B[e] = bv;
  }
}

// pressure of every active node from the pencil solution (0 off the DOFs)
template <typename R>
__global__ void k_pl_scatter_pressure(PencilGeom G, GridDesc g, const int* __restrict__ active_list,
                                      long long nent, const unsigned char* __restrict__ dof,
                                      const R* __restrict__ x32, const double* __restrict__ x64,
                                      R* __restrict__ p) {
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < nent;
       e += (long long)gridDim.x * blockDim.x) {
    const long long n = active_node(active_list, e);
    R v = R(0);
    if (dof[n] & 1) {
      int P[3];
      node_ijk(g, n, P[0], P[1], P[2]);
      const int s = P[G.ax_s] - G.lo[G.ax_s];
      const int a = P[G.ax_a] - G.lo[G.ax_a];
      const int c = P[G.ax_c] - G.lo[G.ax_c];
      const int PAi = a / kPatch, al = a - PAi * kPatch;
      const int PCi = c / kPatch, cl = c - PCi * kPatch;
      const long long idx = pl_index(G, (long long)PCi * G.nPA + PAi, s + al + cl, al + kPatch * cl);
      v = x64 ? (R)x64[idx] : x32[idx];
    }
    p[n] = v;
  }
}

}  // namespace wcg
