// MIC(0)-PCG in the skewed pencil layout.
//
// The pressure unknowns of one solve (the bounding box of the DOF cells) are
// copied once into a layout built for the triangular sweeps.  One grid axis is
// the stream axis s (the longest extent of the box); the other two (a, c) are
// cut into patches of 16 x 16 lines, a patch into 8 strips of 16 x 2 lines.
// A lane takes the cells of its line in pairs along s, one pair per step.  Line
// (al, cl) is skewed by al + (cl & 1) steps within its strip w = cl / 2: cell
// (s, a, c) is element b = s & 1 of the pair at step v = s / 2 + al + (cl & 1),
// stored at (((patch * 8 + w) * R + v) * 32 + lane) * 2 + b with lane = al +
// 16 (cl & 1) and R = (Ls + 1) / 2 + 16 steps, rounded up to a whole chunk of 2.
// Pairs outside a line's range and lines outside the box hold zeros.
//
// In this layout every MIC(0) dependency of a pair is one step back (one step
// forward for the backward sweep) or inside the pair:
//   (s-1, a, c): the pair itself, or step v-1 of the same lane
//   (s, a-1, c): step v-1 of lane - 1 (step v+15 of lane + 15 of the patch below)
//   (s, a, c-1): step v-1 of lane - 16, or step v+1 of lane + 16 of the strip
//                before (of the last strip of the patch before along c)
// so a warp takes a strip, a CTA a group of consecutive strips along c (a patch in
// FP32, half of one in FP64), and every strip reads and writes one contiguous run
// of memory.  The factor lies step by step too, four rows of 64 per step:
// 1/sqrt(d'), S_s, S_a, S_c.
// Values crossing a patch edge along a, or along c the edge of a group that is not
// in the same cluster, go through a global buffer of tagged 64-bit words,
// (epoch << 32 | 32 data bits), one word per 32 bits of payload: the consumer
// re-reads its word until the tag equals the launch's epoch, so no fence or flag is
// needed and a strip waits only for the words of its next step.
// Groups, or clusters of them, are handed out by an atomic ticket in wave order
// (column along a + cluster along c), so whatever is upstream of one always
// started before it.
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
constexpr int kStrips = kPatchLines / 32;     // strips of 32 lines per patch
constexpr int kChunk = 2;                     // steps a strip stages at a time
constexpr int kPlBlocks = 592;                // streaming kernels: 4 x 148 SMs
static_assert(kRedThreads == kPatchLines, "streaming kernels walk one row per block");

// element of line (al, cl) of patch p at stream position s
__host__ __device__ inline long long pl_index(const PencilGeom& G, long long p, int s, int al,
                                              int cl) {
  const long long step = (p * kStrips + (cl >> 1)) * G.R + ((s >> 1) + al + (cl & 1));
  return step * 64 + 2 * (al + 16 * (cl & 1)) + (s & 1);
}

// a lane's pair of cells
template <typename R>
struct Pair;
template <>
struct Pair<float> {
  using T = float2;
};
template <>
struct Pair<double> {
  using T = double2;
};

// Strips of a sweep CTA.  FP32: a whole patch.  FP64: half a patch, since eight
// FP64 strips keep one SM's issue slots and shared memory busy (per sweep launch
// in groups of 8 / 4: 178 / 149 us for the half box at 128^3, 65 / 52 us for the
// dam break at 64^3; FP32 at 256^3 211 / 260 us, 12 and more warps per SM).
template <typename R>
__host__ __device__ constexpr int sweep_group() {
  return sizeof(R) == 4 ? kStrips : kStrips / 2;
}
template <typename R>
__host__ __device__ constexpr int sweep_threads() {
  return sweep_group<R>() * 32 + 64;  // strips, then two receiver warps
}
// groups of strips in a column of patches, and over the whole box
template <typename R>
__host__ __device__ inline int pl_groups(const PencilGeom& G) {
  return G.nPC * (kStrips / sweep_group<R>());
}
template <typename R>
__host__ __device__ inline int pl_units(const PencilGeom& G) {
  return G.nPA * pl_groups<R>(G);
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

// Words of the edge buffer, EW words per entry.  a-face: entry (patch that
// writes, step, line cl of the sweep); c-face: (group that writes, step, line
// al).  step = the step of the strip that wrote it (the strip that takes it does
// so 15 steps earlier in its own count along a, one along c).
__host__ __device__ inline long long edge_words(const PencilGeom& G, int units, int EW) {
  return (G.npatch + units) * G.R * kPatch * EW;
}
__device__ inline long long edge_a(const PencilGeom& G, long long p, int step, int k, int EW) {
  return ((p * G.R + step) * kPatch + k) * EW;
}
__device__ inline long long edge_c(const PencilGeom& G, long long unit, int step, int k, int EW) {
  return (((G.npatch + unit) * G.R + step) * kPatch + k) * EW;
}

template <typename R>
struct PencilSweepArgs {
  PencilGeom G;
  const int* order;   // clusters in wave order: column + nPA * cluster of the column
  int* ticket;
  int ticket_base;    // tickets already handed out this solve
  unsigned epoch;     // tag of this launch's edge words
  u64* edge;
  // factorisation input
  const R* AD;
  const R* AS;
  const R* AA;
  const R* AC;
  R* coef;      // factor: 4 rows of 64 per step, 1/sqrt(d'), S_s, S_a, S_c
  // sweeps
  const R* in;  // forward: r; backward: y
  R* out;       // forward: y; backward: z
  R* r;         // forward (update): r updated in place; backward: r for z.r
  const R* q;   // forward (update)
  double* sc;            // device scalars (the last CTA of a reducing sweep writes them)
  double* part;  // per-group partial: forward max|r|, backward z.r
  R omega, min_ratio;
  int* err;
  int* done_ctr;         // with part: the last CTA reduces the partials (forward with
                         // update: max|r| and the stop test; backward: z.r and beta)
  int red_init;          // backward: the first z.r of a solve (beta = 0)
  int npart;             // partials (groups)
  long long spin_limit;  // polls of an edge word before the wait gives up
  int box_polls;         // and of a word or a count in shared memory (inbox_polls)
  int stale_patch;       // failure-path test: this patch waits for a tag nothing
                         // writes (-1: none)
};

// MODE: kFactor, kForward, kBackward.  UPD: the forward sweep first applies
// r -= alpha q (and reports max|r|); the matching x += alpha s is applied by
// the next SpMV (k_pl_spmv_s) or, after the last iteration, by k_pl_axpy.
//
// The strips of one column of patches (all c, one a) form a chain.  A CTA takes
// a group of consecutive strips of it, one warp each, with two receiver warps; the
// CTAs of a thread-block cluster take consecutive groups.  A strip walks its R
// steps (two cells of every line each) without any CTA barrier:
//   * its cells are copied a few chunks ahead into a shared-memory ring that
//     only this warp uses (cp.async, 16 bytes per lane: a chunk is contiguous);
//   * the a-neighbour and the c-neighbour inside the strip come by shuffle of
//     the previous step's outputs;
//   * the c-neighbour in the strip before and the values of the column before
//     along a come as tagged 64-bit words (tag << 32 | 32 data bits) in the
//     strip's inbox in shared memory.  The strip before writes the c words of
//     step v - 1 of its own count, through the cluster's shared memory where it
//     is in the CTA before; the receivers write the rest.  A step's words are
//     read a step ahead and read again only where they were not there yet.
// Words to the next column, and along c out of a cluster, go through a global
// buffer (tag: the launch's epoch).  The receivers (one warp for the a-face, one for the c-face, two
// lanes per line: even and odd steps) poll it, up to 4 steps per lane in flight,
// and move what has arrived into the inboxes, so a strip never waits for a
// round trip to L2 of its own.  An inbox slot is reused once the strip has
// published that it took the word (s_prog).  Every wait is bounded.
//
// The backward sweep is the same walk mirrored: patches, strips, lanes and
// rows counted from the other end.
//
// Bound: the chain of Ls / 2 + NA + NC steps that the last cell waits for, then
// the bytes of a step (forward 8, backward 7 values per cell).  A step takes
// about 500 cycles of a warp in FP32 and 900 in FP64, some 85 and 155 instructions
// of one warp at 6.1 and 5.7 cycles each: the fixed latency of dependent
// instructions takes 1.9 of those, branches 1.2 and 0.9, loads of either memory 0.9
// and 1.3 (counters at 192^3 and 128^3; DRAM at 12 and 10 %).  So a step is kept to
// two cells per lane: with single cells a row took 320-400 and 450-500 and a hop between
// strips 1500.  Per launch (the events around it included), one CTA barrier per
// row and every face lane polling L2 / one-cell strips / this: 256^3 half box in
// FP32 426 / 270 / 213 us; FP64 half box at 128^3 287 / 161 / 138, dam break at
// 64^3 105 / 62 / 53, at 16^3 62 / 39 / 34.
//
// The body takes the launch's CTA count (nblocks) as an argument so a launch
// over several solves (k_pencil_sweep_batch) can run it per solve.
constexpr int kInA = 16;   // inbox steps of a entries (2 per step)
// inbox steps of c entries (16 per step): as many as shared memory has room for,
// so that a strip seldom has to look whether the next one took some
template <typename R>
__host__ __device__ constexpr int sweep_inc() {
  return sizeof(R) == 4 ? 16 : 8;
}
constexpr int kRecv = 4;   // steps a receiver lane polls at once

// chunks of a strip in flight or in use (96 KB a CTA in FP32, one CTA per SM; 72 KB
// in FP64, two)
template <typename R>
struct SweepSlots {
  static constexpr int N = sizeof(R) == 4 ? 4 : 3;
};
__host__ __device__ constexpr int sweep_words(int mode, size_t rbytes) {
  return 2 * (mode == 0 ? 2 : 1) * (int)(rbytes / 4);  // 64-bit words per edge entry
}
template <typename R>
__host__ __device__ constexpr size_t sweep_ring_bytes(int mode) {
  return (size_t)sweep_group<R>() * SweepSlots<R>::N * sweep_slot(mode) * kChunk * 64 * sizeof(R);
}
template <typename R>
__host__ __device__ constexpr size_t sweep_dyn_smem(int mode) {
  return sweep_ring_bytes<R>(mode) +
         (size_t)sweep_group<R>() * (sweep_inc<R>() * 16 + kInA * 2) * sweep_words(mode, sizeof(R)) * 8;
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
// the same from the lanes with on != 0 alone, to shared (32-bit address) or
// global memory (predicated: the lanes of a strip never part)
template <int EW>
__device__ inline void st_words_shared_if(int on, unsigned addr, const u64* w) {
#pragma unroll
  for (int k = 0; k < EW; k += 2)
    asm volatile(
        "{\n .reg .pred q;\n setp.ne.s32 q, %3, 0;\n @q st.volatile.shared.v2.u64 [%0], {%1, %2};\n}" ::
            "r"(addr + 8 * k), "l"(w[k]), "l"(w[k + 1]), "r"(on)
        : "memory");
}
template <int EW>
__device__ inline void st_words_global_if(int on, u64* p, const u64* w) {
#pragma unroll
  for (int k = 0; k < EW; k += 2)
    asm volatile(
        "{\n .reg .pred q;\n setp.ne.s32 q, %3, 0;\n @q st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};\n}" ::
            "l"(p + k), "l"(w[k]), "l"(w[k + 1]), "r"(on)
        : "memory");
}
// nonzero where a tag of the entry is not `tag`
template <int EW>
__device__ inline unsigned words_off(const u64* w, unsigned tag) {
  unsigned off = 0;
#pragma unroll
  for (int k = 0; k < EW; ++k) off |= (unsigned)(w[k] >> 32) ^ tag;
  return off;
}
// the value's bits under a mask of all ones or zeros, and (a & m) | b
__device__ inline float keep(float v, unsigned m) { return __uint_as_float(__float_as_uint(v) & m); }
__device__ inline double keep(double v, unsigned m) {
  return __hiloint2double(__double2hiint(v) & (int)m, __double2loint(v) & (int)m);
}
__device__ inline float merge(float a, unsigned m, float b) {
  return __uint_as_float((__float_as_uint(a) & m) | __float_as_uint(b));
}
__device__ inline double merge(double a, unsigned m, double b) {
  return __hiloint2double((__double2hiint(a) & (int)m) | __double2hiint(b),
                          (__double2loint(a) & (int)m) | __double2loint(b));
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

// thread-block clusters
__device__ inline int cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return (int)r;
}
// every thread of every CTA of the cluster; orders the shared memory each CTA
// wrote before it against the accesses after it
__device__ inline void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n"
               "barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// address of the same shared variable in CTA `rank` of the cluster
__device__ inline unsigned cluster_map(unsigned local, int rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"((unsigned)rank));
  return r;
}
__device__ inline int ld_cluster_int(unsigned addr) {
  int v;
  asm volatile("ld.relaxed.cluster.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}
template <int EW>
__device__ inline void st_words_cluster_if(int on, unsigned addr, const u64* w) {
#pragma unroll
  for (int k = 0; k < EW; ++k)
    asm volatile(
        "{\n .reg .pred q;\n setp.ne.s32 q, %2, 0;\n"
        " @q st.relaxed.cluster.shared::cluster.u64 [%0], %1;\n}" ::"r"(addr + 8 * k),
        "l"(w[k]), "r"(on)
        : "memory");
}

template <typename R, int MODE, bool UPD, int CL>
__device__ __forceinline__ void pencil_sweep_run(const PencilSweepArgs<R>& A, int nblocks) {
  constexpr bool BWD = MODE == kBackward;
  constexpr int PW = MODE == kFactor ? 2 : 1;  // values sent across an edge
  constexpr int TW = TagWords<R>::W;
  constexpr int EW = 2 * PW * TW;              // words of an entry: both cells
  static_assert(kFactor == 0 && kForward == 1 && kBackward == 2, "mode numbering");
  constexpr int NS = SweepSlots<R>::N;
  constexpr int NF = sweep_slot(MODE);
  constexpr bool TWO = MODE == kBackward || UPD;  // two vectors per row
  constexpr int SLOT = NF * kChunk * 64;          // Reals per staged chunk
  using P2 = typename Pair<R>::T;
  constexpr unsigned full = 0xffffffffu;
  __shared__ int s_ticket;
  constexpr int kGroup = sweep_group<R>();
  __shared__ int s_prog[kGroup];
  __shared__ double red[kRedThreads];
  extern __shared__ __align__(128) unsigned char dsm[];  // strip rings, then the inboxes
  const PencilGeom& G = A.G;
  const int tid = threadIdx.x;
  const int lane = tid & 31, w = tid >> 5;
  const int rank = CL > 1 ? cluster_rank() : 0;
  // one ticket per cluster, taken even by a launch that returns at once, so the
  // counter stays in step with the host's base
  if (tid == 0 && rank == 0) s_ticket = atomicAdd(A.ticket, 1) - A.ticket_base;
  // set by an earlier launch, so uniform: the whole cluster returns before any
  // access to another CTA
  if (*(const int*)(A.sc + S_DONE)) return;
  constexpr int kPencilThreads = sweep_threads<R>();
  constexpr int kInC = sweep_inc<R>();
  constexpr int INBOX = (kInC * 16 + kInA * 2) * EW;  // words per strip
  {
    u64* ib = reinterpret_cast<u64*>(dsm + sweep_ring_bytes<R>(MODE));
    for (int i = tid; i < kGroup * INBOX; i += kPencilThreads) ib[i] = 0ull;
    if (tid < kGroup) s_prog[tid] = 0;
  }
  if (CL > 1) cluster_sync();
  else __syncthreads();
  const int tk = CL > 1 ? ld_cluster_int(cluster_map(smem_u32(&s_ticket), 0)) : s_ticket;
  const int ngroup = pl_groups<R>(G), ncl = (ngroup + CL - 1) / CL;
  bool run = true;
  if (tk < 0 || tk >= G.nPA * ncl) {
    if (tid == 0) record_error(A.err, kErrIndex);
    run = false;
  }
  double rmax = 0, dsum = 0;
  int col = 0, grp = 0;  // column along a and group along c, in sweep order
  if (run) {
    const int unit = A.order[tk];
    col = unit % G.nPA;
    grp = unit / G.nPA * CL + rank;
    run = grp < ngroup;  // the last cluster of a column may reach past its end
  }
  if (run) {
    const int NV = G.R;
    const int na = NV - 15, nc = NV - 1;   // steps that take a-face and c-face words
    const int S0 = grp * kGroup;           // first strip of the group in its column
    const int PCs = S0 / kStrips;          // its patch along c, in sweep order
    const int p = BWD ? (G.nPC - 1 - PCs) * G.nPA + (G.nPA - 1 - col) : PCs * G.nPA + col;
    // upstream: the column before (same strips) and the group before; the groups
    // of a cluster reach one another through shared memory
    const bool up_a = col > 0, dn_a = col + 1 < G.nPA;
    const bool up_c = grp > 0, dn_c = grp + 1 < ngroup;
    const bool up_near = CL > 1 && rank > 0, dn_near = CL > 1 && dn_c && rank + 1 < CL;
    const long long unit_id = (long long)grp * G.nPA + col;
    const unsigned inbox0 = smem_u32(dsm + sweep_ring_bytes<R>(MODE));
    const unsigned prog0 = smem_u32(s_prog);
    const unsigned ep = A.epoch;
    if (w >= kGroup) {
      // ---- receivers ----
      const bool cface = w == kGroup + 1;
      if (cface ? up_c && !up_near : up_a) {
        // the tag this patch waits for: the launch's, except on the patch a
        // failure-path test marks, whose waits then run into their limit
        const unsigned want = p == A.stale_patch ? (ep ^ 0x80000000u) : ep;
        // lanes per line: steps v, v + nl, ... each
        const int lines = cface ? 16 : 2 * kGroup;
        const int nl = 32 / lines;
        const int k = lane % lines;                  // line of the face
        const int strip = cface ? 0 : k >> 1;
        const int rows = cface ? nc : na;
        const unsigned box = inbox0 + (unsigned)(strip * INBOX) * 8u +
                             (cface ? (unsigned)(k * EW) * 8u
                                    : (unsigned)((kInC * 16 + (k & 1)) * EW) * 8u);
        const int depth = cface ? kInC : kInA;
        const unsigned pitch = (cface ? 16u : 2u) * EW * 8u;
        const unsigned prog = prog0 + 4u * strip;
        const long long up_p = BWD ? p + 1 : p - 1;
        const u64* src = A.edge + (cface ? edge_c(G, unit_id - G.nPA, 1, k, EW)
                                         : edge_a(G, up_p, 15, 2 * (S0 % kStrips) + k, EW));
        int v = lane / lines;  // this lane's next step
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
            const int vj = v + nl * j;
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
            const int vj = v + nl * j;
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
          v += nl * got;
          if (got > 0) {
            idle = 0;
          } else if (v < rows && v < room) {
            if (++idle > A.spin_limit && !gave_up) {
              record_error(A.err, kErrWaitTimeout);
              gave_up = true;
            }
          } else if (v < rows && ++idle > A.box_polls) {
            // the strip no longer takes words (its own wait gave up)
            record_error(A.err, kErrWaitTimeout);
            v = rows;
          }
        }
      }
    } else {
      // ---- strips ----
      // mirrored for the backward sweep: strips, lanes, steps and the cells of a
      // pair from the end
      const int pl = BWD ? 31 - lane : lane;
      const int sp = (S0 + w) % kStrips;  // strip of the patch, in sweep order
      const int ps = BWD ? kStrips - 1 - sp : sp;
      const long long strip0 = ((long long)p * kStrips + ps) * NV * 64;  // its first element
      constexpr int RS = BWD ? -64 : 64;                                 // element step per step
      R* const ring = reinterpret_cast<R*>(dsm) + (size_t)w * NS * SLOT;
      // Copies of one chunk, 16 bytes per lane and pass.  Slot layout: the
      // arrays one after the other, each kChunk steps in memory order (the
      // backward sweep takes them from the last).
      constexpr int AB = kChunk * 64 * sizeof(R);  // bytes of one array's chunk
      const long long e00 = strip0 + (BWD ? (long long)(NV - kChunk) * 64 : 0);
      const unsigned char *g0, *g1, *g2, *g3;
      if (MODE == kFactor) {
        g0 = reinterpret_cast<const unsigned char*>(A.AD + e00) + lane * 16;
        g1 = reinterpret_cast<const unsigned char*>(A.AS + e00) + lane * 16;
        g2 = reinterpret_cast<const unsigned char*>(A.AA + e00) + lane * 16;
        g3 = reinterpret_cast<const unsigned char*>(A.AC + e00) + lane * 16;
      } else {
        g0 = reinterpret_cast<const unsigned char*>(A.in + e00) + lane * 16;
        g1 = reinterpret_cast<const unsigned char*>((MODE == kForward ? A.q : A.r) + e00) + lane * 16;
        g2 = reinterpret_cast<const unsigned char*>(A.coef + 4 * e00) + lane * 16;
        g3 = nullptr;
      }
      int left = NV / kChunk;  // chunks still to copy
      auto issue = [&](unsigned dst) {
        if (left > 0) {
          auto copy = [&](unsigned at, const unsigned char* g, int nbytes) {
#pragma unroll
            for (int i = 0; i < nbytes / 512; ++i) cp_async16(dst + at + i * 512, g + i * 512);
          };
          constexpr int CS = BWD ? -AB : AB;
          copy(0, g0, AB);
          g0 += CS;
          if (MODE == kFactor || TWO) {
            copy(AB, g1, AB);
            g1 += CS;
          }
          copy(2 * AB, g2, MODE == kFactor ? AB : 4 * AB);
          g2 += MODE == kFactor ? CS : 4 * CS;
          if (MODE == kFactor) {
            copy(3 * AB, g3, AB);
            g3 += CS;
          }
          --left;
        }
        cp_async_commit();
      };
      const unsigned ring0 = smem_u32(ring) + lane * 16;
      constexpr unsigned SB = SLOT * (unsigned)sizeof(R);
#pragma unroll
      for (int k = 0; k < NS; ++k) issue(ring0 + k * SB);

      // the entries this lane takes: lanes 0..15 the c-face, lanes 0 and 16 the
      // a-face lines of the strip (the others read along)
      const int lim_c = (w > 0 || up_c) && lane < 16 ? nc : 0;
      const int lim_a = up_a && (lane & 15) == 0 ? na : 0;
      u64* const box = reinterpret_cast<u64*>(dsm + sweep_ring_bytes<R>(MODE)) + w * INBOX;
      const unsigned csrc = smem_u32(box + (lane & 15) * EW);
      const unsigned asrc = smem_u32(box + (kInC * 16 + (lane >> 4)) * EW);
      constexpr unsigned CP = 16u * EW * 8u, AP = 2u * EW * 8u;  // bytes of an inbox step
      // outgoing: lanes 16..31 the c entries of step v - 1 of the next strip (in
      // this CTA, in the next one of the cluster, or beyond it), lanes 15 and 31
      // the a-face entries
      const bool last = w + 1 == kGroup;
      const bool to_box = !last || dn_near;
      const int put_c = lane >= 16 && (!last || dn_c);
      const int put_a = (lane & 15) == 15 && dn_a;
      const unsigned obox0 = smem_u32(box + (last ? -(kGroup - 1) : 1) * INBOX + (lane & 15) * EW);
      const unsigned obox = CL > 1 && last && dn_near ? cluster_map(obox0, rank + 1) : obox0;
      // lanes that take the shuffled value along c and along a
      const unsigned from_c = lane < 16 ? 0u : ~0u, from_a = (lane & 15) == 0 ? 0u : ~0u;
      u64* gc = A.edge + edge_c(G, unit_id, 0, lane & 15, EW);
      u64* ga = A.edge + edge_a(G, p, 0, 2 * sp + (lane >> 4), EW);
      const unsigned prog = prog0 + 4u * w;
      const R al_r = (MODE == kForward && UPD) ? (R)A.sc[S_ALPHA] : R(0);
      const R omega = A.omega, min_ratio = A.min_ratio;
      const long long eb = strip0 + (BWD ? (long long)(NV - 1) * 64 : 0) + 2 * pl;
      R* pcoef = MODE == kFactor ? A.coef + 4 * strip0 + 2 * pl : nullptr;
      R* o_out = MODE == kFactor ? nullptr : A.out + eb;
      R* o_r = (MODE == kForward && UPD) ? A.r + eb : nullptr;
      // prev_*: the previous step's outputs, [cell][value]; cells in sweep order
      R carry[PW], prev_a[2][PW], prev_c[2][PW];
#pragma unroll
      for (int k = 0; k < PW; ++k)
        carry[k] = prev_a[0][k] = prev_a[1][k] = prev_c[0][k] = prev_c[1][k] = R(0);
      R rm = 0;
      bool gave_up = false;
      // a step's values, cells in sweep order (the backward sweep takes the
      // second cell of a pair first)
      auto load_step = [&](int slot, int j, R (&f)[2][NF]) {
        const R* S = ring + slot * SLOT;
        const int at = (BWD ? kChunk - 1 - j : j) * 64 + 2 * pl;
        constexpr int B0 = BWD ? 1 : 0, B1 = BWD ? 0 : 1;
        auto pair = [&](int off, int k) {
          const P2 t = *reinterpret_cast<const P2*>(S + off);
          f[B0][k] = t.x;
          f[B1][k] = t.y;
        };
        pair(at, 0);
        if (MODE == kFactor) {
#pragma unroll
          for (int k = 1; k < 4; ++k) pair(k * kChunk * 64 + at, k);
        } else {
          if (TWO) pair(kChunk * 64 + at, NF - 1);
          const int ac = 2 * kChunk * 64 + (BWD ? kChunk - 1 - j : j) * 256 + 2 * pl;
#pragma unroll
          for (int k = 0; k < 4; ++k) pair(ac + 64 * k, 1 + k);
        }
      };
      u64 wc[EW], wa[EW];
      auto load_words = [&](int v) {
        ld_words_shared<EW>(csrc + (unsigned)(v & (kInC - 1)) * CP, wc);
        ld_words_shared<EW>(asrc + (unsigned)(v & (kInA - 1)) * AP, wa);
      };
      auto step = [&](int v, const R (&f)[2][NF], unsigned oc, int j) __attribute__((always_inline)) {
        // all ones where the lane takes an entry of this step
        const unsigned mc = (unsigned)((v - lim_c) >> 31), ma = (unsigned)((v - lim_a) >> 31);
        const unsigned tag = (unsigned)(v + 1);
        unsigned off = (words_off<EW>(wc, tag) & mc) | (words_off<EW>(wa, tag) & ma);
        if (__any_sync(full, off != 0)) {
          int it = 0;
          do {
            load_words(v);
            off = (words_off<EW>(wc, tag) & mc) | (words_off<EW>(wa, tag) & ma);
            if (++it > A.box_polls) {
              if (lane == 0) record_error(A.err, kErrWaitTimeout);
              gave_up = true;
            }
          } while (__any_sync(full, off != 0) && !gave_up);
        }
        R in_a[2][PW], in_c[2][PW];
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
          for (int k = 0; k < PW; ++k) {
            const R sa = __shfl_up_sync(full, prev_a[b][k], 1);
            const R sc = __shfl_up_sync(full, prev_c[b][k], 16);
            in_a[b][k] = merge(sa, from_a, keep(TagWords<R>::unpack(wa + (b * PW + k) * TW), ma));
            in_c[b][k] = merge(sc, from_c, keep(TagWords<R>::unpack(wc + (b * PW + k) * TW), mc));
          }
        // the next step's words, read early; taken once their tag is right
        load_words(v + 1);
        P2 o2, r2;       // in memory order
        R cf[2][4];      // the factor's coefficients
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          R out_s[PW], out_a[PW], out_c[PW];
          if (MODE == kFactor) {
            const R ad = f[b][0];
            R d = ad;
            R iv = R(0);
            if (ad != R(0)) {
              d = d - in_c[b][0] * in_c[b][0];
              d = d - (omega * in_c[b][0]) * in_c[b][PW - 1];
              d = d - in_a[b][0] * in_a[b][0];
              d = d - (omega * in_a[b][0]) * in_a[b][PW - 1];
              d = d - carry[0] * carry[0];
              d = d - (omega * carry[0]) * carry[PW - 1];
              const R piv = d < min_ratio * ad ? ad : d;
              iv = R(1) / sqrt(piv);
            }
            const R ss = f[b][1] * iv, sa = f[b][2] * iv, scv = f[b][3] * iv;
            cf[b][0] = iv; cf[b][1] = ss; cf[b][2] = sa; cf[b][3] = scv;
            out_s[0] = ss; out_s[PW - 1] = sa + scv;
            out_a[0] = sa; out_a[PW - 1] = ss + scv;
            out_c[0] = scv; out_c[PW - 1] = ss + sa;
          } else if (MODE == kForward) {
            R rv = f[b][0];
            if (UPD) {
              rv = rv - al_r * f[b][NF - 1];
              if (b == 0) r2.x = rv;
              else r2.y = rv;
              const R av = fabs(rv);
              rm = av > rm ? av : rm;
            }
            R vv = rv;
            vv -= in_c[b][0];
            vv -= in_a[b][0];
            vv -= carry[0];
            const R y = vv * f[b][1];
            if (b == 0) o2.x = y;
            else o2.y = y;
            out_s[0] = f[b][2] * y;
            out_a[0] = f[b][3] * y;
            out_c[0] = f[b][NF - 2] * y;
          } else {
            R vv = f[b][0];
            vv -= f[b][2] * carry[0];
            vv -= f[b][3] * in_a[b][0];
            vv -= f[b][NF - 2] * in_c[b][0];
            const R z = vv * f[b][1];
            if (b == 0) o2.y = z;
            else o2.x = z;
            dsum += (double)z * (double)f[b][NF - 1];
            out_s[0] = out_a[0] = out_c[0] = z;
          }
#pragma unroll
          for (int k = 0; k < PW; ++k) {
            prev_a[b][k] = out_a[k];
            prev_c[b][k] = out_c[k];
            carry[k] = out_s[k];
          }
        }
        u64 o[EW];
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
          for (int k = 0; k < PW; ++k)
            TagWords<R>::pack(prev_c[b][k], to_box ? (unsigned)v : ep, o + (b * PW + k) * TW);
        if (!last) st_words_shared_if<EW>(put_c, oc, o);
        else if (CL > 1 && dn_near) st_words_cluster_if<EW>(put_c, oc, o);
        else st_words_global_if<EW>(put_c, gc + j * (16 * EW), o);
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
          for (int k = 0; k < PW; ++k)
            TagWords<R>::pack(prev_a[b][k], ep, o + (b * PW + k) * TW);
        st_words_global_if<EW>(put_a, ga + j * (16 * EW), o);
        if (MODE == kFactor) {
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            P2 t;
            t.x = cf[0][k];
            t.y = cf[1][k];
            *reinterpret_cast<P2*>(pcoef + j * 256 + 64 * k) = t;
          }
        } else {
          *reinterpret_cast<P2*>(o_out + j * RS) = o2;
        }
        if (MODE == kForward && UPD) *reinterpret_cast<P2*>(o_r + j * RS) = r2;
      };
      int slot = 0;
      R f0[2][NF], f1[2][NF];
      cp_async_wait<NS - 1>();
      __syncwarp();
      load_step(0, 0, f0);
      load_words(0);
      const unsigned next_prog = last ? (CL > 1 && dn_near ? cluster_map(prog0, rank + 1) : prog)
                                      : prog0 + 4u * (w + 1);
      auto look = [&]() {
        return CL > 1 && last && dn_near ? ld_cluster_int(next_prog) : ld_volatile_int(next_prog);
      };
      int taken = 0;  // steps the next strip had taken when last looked at
      for (int v0 = 0; v0 < NV; v0 += 2) {
        load_step(slot, 1, f1);
        if (to_box && v0 >= taken + kInC && !gave_up) {
          // the next strip has to take its steps first
          int it = 0;
          while (v0 >= (taken = look()) + kInC) {
            if (++it > A.box_polls) {
              if (lane == 0) record_error(A.err, kErrWaitTimeout);
              gave_up = true;
              break;
            }
          }
        }
        // the c entries go to steps v0 - 1 and v0 of the next strip's inbox
        // (step -1: the last slot with tag 0, which nothing takes), or to steps
        // v0 and v0 + 1 of the patch's own face
        step(v0, f0, obox + (unsigned)((v0 - 1) & (kInC - 1)) * CP, 0);
        // every lane holds this chunk's values: its slot takes a later one
        __syncwarp();
        issue(ring0 + slot * SB);
        slot = slot + 1 == NS ? 0 : slot + 1;
        taken = look();
        cp_async_wait<NS - 1>();
        __syncwarp();
        if (v0 + 2 < NV) load_step(slot, 0, f0);
        step(v0 + 1, f1, obox + (unsigned)(v0 & (kInC - 1)) * CP, 1);
        st_volatile_int(prog, v0 + 2);  // (every lane the same)
        gc += 2 * 16 * EW;
        ga += 2 * 16 * EW;
        if (MODE == kFactor) pcoef += 2 * 256;
        else o_out += 2 * RS;
        if (MODE == kForward && UPD) o_r += 2 * RS;
      }
      if (lane == 0) st_volatile_int(prog, 1 << 29);  // nothing waits for this strip any more
      cp_async_wait<0>();
      rmax = (double)rm;
    }
  }
  // partials, summed in line order whatever the direction
  if (A.part && ((MODE == kForward && UPD) || MODE == kBackward)) {
    constexpr int NL = kGroup * 32;
    for (int i = tid; i < kRedThreads; i += kPencilThreads) red[i] = 0;
    __syncthreads();
    if (tid < NL) red[BWD ? NL - 1 - tid : tid] = MODE == kForward ? rmax : dsum;
    const int at = (BWD ? ngroup - 1 - grp : grp) * G.nPA + (BWD ? G.nPA - 1 - col : col);
    if (MODE == kForward) {
      const double m = tree_max(red);
      if (tid == 0 && run) A.part[at] = m;
    } else {
      const double sm = tree_sum(red);
      if (tid == 0 && run) A.part[at] = sm;
    }
    // every CTA counts, running or not; the last one reduces the partials
    if (A.done_ctr && last_block(A.done_ctr, nblocks)) {
      if (MODE == kForward)
        red_conv_body(A.part, A.npart, A.sc, red);
      else
        red_beta_body(A.part, A.npart, A.sc, red, A.red_init);
    }
  }
  // no CTA leaves while another may write to its inbox or look at its progress
  if (CL > 1) cluster_sync();
}

template <typename R, int MODE, bool UPD, int CL>
__global__ void __launch_bounds__(sweep_threads<R>(), 1)
    k_pencil_sweep(const PencilSweepArgs<R> A) {
  pencil_sweep_run<R, MODE, UPD, CL>(A, (int)gridDim.x);
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
// scenes): solve s owns first[s + 1] - first[s] CTAs (whole clusters) and its
// arguments come from tab[s].  Launch k of a chunk advances each solve's
// edge-word epoch by k and its ticket base by k launches of its clusters, as k
// separate launches would.
template <typename R, int MODE, bool UPD, int CL>
__global__ void __launch_bounds__(sweep_threads<R>(), 1)
    k_pencil_sweep_batch(const PencilSweepArgs<R>* __restrict__ tab, const int* __restrict__ first,
                         int nsolve, int k) {
  const int s = batch_solve_of(first, nsolve, (int)blockIdx.x);
  PencilSweepArgs<R> A = tab[s];
  const int nb = __ldg(first + s + 1) - __ldg(first + s);
  A.epoch += (unsigned)k;
  A.ticket_base += k * (nb / CL);
  pencil_sweep_run<R, MODE, UPD, CL>(A, nb);
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
// Element e -> (patch, strip, step, lane, cell) and the position in the box.
struct PlCell {
  int p, w, al, cl, PAi, PCi, s;
  bool live;
};

__device__ inline PlCell pl_cell(const PencilGeom& G, long long e) {
  PlCell c;
  const int row = (int)(e >> 6), lane = (int)(e >> 1) & 31;  // npatch * 8 * R far below 2^31
  const int strip = row / G.R;
  const int v = row - strip * G.R;
  c.p = strip / kStrips;
  c.w = strip - c.p * kStrips;
  c.al = lane & (kPatch - 1);
  c.cl = 2 * c.w + (lane >> 4);
  c.PAi = c.p % G.nPA;
  c.PCi = c.p / G.nPA;
  c.s = 2 * (v - c.al - (lane >> 4)) + (int)(e & 1);
  c.live = c.s >= 0 && c.s < G.Ls && c.PAi * kPatch + c.al < G.NA &&
           c.PCi * kPatch + c.cl < G.NC;
  return c;
}

// Element offsets from a cell to its neighbours outside its strip: the
// c-neighbour (-c for the 16 lanes of even cl, +c for those of odd cl) sits one
// strip on, the a-neighbour across the patch face (al = 0: -a, al = 15: +a) in
// the same strip of the next patch.
__device__ inline long long pl_out_c(const PencilGeom& G, int w, bool minus) {
  // strips of consecutive patches along c are nPA patches apart
  const long long rows = (long long)G.R * 64;
  const long long far = ((long long)G.nPA * kStrips - (kStrips - 1)) * rows;
  if (minus) return -(w > 0 ? rows : far) + 64 + 32;
  return (w + 1 < kStrips ? rows : far) - 64 - 32;
}
__device__ inline long long pl_out_a(const PencilGeom& G, bool minus) {
  const long long patch = (long long)kStrips * G.R * 64;
  const long long step = (kPatch - 1) * 64 + (kPatch - 1) * 2;
  return minus ? -patch + step : patch - step;
}

// Indices of the six neighbours of a live cell (-1 where the box ends).
struct PlNbr {
  long long ms, ps, ma, pa, mc, pc;
};

__device__ inline PlNbr pl_nbr(const PencilGeom& G, const PlCell& c, long long e) {
  PlNbr n;
  n.ms = c.s > 0 ? (c.s & 1 ? e - 1 : e - 63) : -1;
  n.ps = c.s + 1 < G.Ls ? (c.s & 1 ? e + 63 : e + 1) : -1;
  if (c.al > 0) n.ma = e - 66;
  else n.ma = c.PAi > 0 ? e + pl_out_a(G, true) : -1;
  if (c.al < kPatch - 1) n.pa = e + 66;
  else n.pa = c.PAi + 1 < G.nPA ? e + pl_out_a(G, false) : -1;
  if (c.cl & 1) n.mc = e - 96;
  else n.mc = c.cl > 0 || c.PCi > 0 ? e + pl_out_c(G, c.w, true) : -1;
  if (!(c.cl & 1)) n.pc = e + 96;
  else n.pc = c.cl < kPatch - 1 || c.PCi + 1 < G.nPC ? e + pl_out_c(G, c.w, false) : -1;
  return n;
}

// s_new = z + beta s_old, q = A s_new, partial[block] = sum s_new.q.  Row order
// of the reference's sorted row for interior cells: -c, -a, -s, diagonal, +s,
// +a, +c.
//
// The previous iteration's x += alpha s_old is applied here too (alpha is
// still the previous iteration's when this kernel runs; 0 before the first).
//
// Bound by memory: 10 values per cell (z, s_old, four coefficients and x in;
// s_new, q and x out).  A block takes a chunk of steps of one patch, warp w its
// strip w, and walks them in order, a pair of cells per lane: s_new of the steps
// before, at and after the current one and the couplings of the step before
// stay in registers, and neighbours inside the strip come by shuffle, so a value
// is loaded once by its own strip.  Only the c-neighbours in the strips beside
// it (half the lanes each way, the same steps of the same block: L1) and the
// neighbours across a patch face are loaded again.  The
// former kernel, one row per block and every neighbour loaded, read each value
// of z and s_old seven times through L1 and three times through L2: 139 us an
// iteration at 256^3 in FP32, 104 here (67 at the copy rate).
constexpr int kSpmvSteps = 8;    // steps of a strip per block, at most
constexpr int kSpmvStepsMin = 2;

struct SpmvGrid {
  int steps, nchunk, blocks;
};
// Steps per block: 8 blocks per SM before a block takes more than kSpmvStepsMin
// (a chunk also reads the step before and after it, from L2), at most
// kSpmvSteps.  A solve alone and in a launch over several solves use the same
// count, so their partial sums are the same.
__host__ __device__ inline SpmvGrid pl_spmv_grid(const PencilGeom& G) {
  SpmvGrid g;
  long long n = (G.npatch * G.R + 1183) / 1184;
  n = n < kSpmvStepsMin ? kSpmvStepsMin : (n > kSpmvSteps ? kSpmvSteps : n);
  g.nchunk = (int)((G.R + n - 1) / n);
  g.steps = (int)((G.R + g.nchunk - 1) / g.nchunk);
  g.blocks = (int)(G.npatch * g.nchunk);
  return g;
}

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
  int parity;  // iterations the solve ran before, mod 2: s_old is s0 (even) or s1
};

// Block bid of nblk of one solve.
template <typename R>
__device__ __forceinline__ void pl_spmv_run(const PlSpmvArgs<R>& A, bool odd, int bid, int nblk) {
  __shared__ double sm[kRedThreads];
  double* const sc = A.sc;
  if (*(const int*)(sc + S_DONE)) return;
  constexpr unsigned full = 0xffffffffu;
  const R be = (R)sc[S_BETA];
  const R al = (R)sc[S_ALPHA];
  const PencilGeom& G = A.G;
  const R* __restrict__ const z = A.z;
  const R* __restrict__ const sold = odd ? A.s1 : A.s0;
  R* __restrict__ const snew = odd ? A.s0 : A.s1;
  R* __restrict__ const x = A.x;
  const SpmvGrid g = pl_spmv_grid(G);
  const int p = bid / g.nchunk;
  const int v0 = (bid - p * g.nchunk) * g.steps;
  const int PAi = p % G.nPA, PCi = p / G.nPA;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int NV = G.R;
  const int v1 = min(NV, v0 + g.steps);
  const int alp = lane & 15;
  const int dl = alp + (lane >> 4);
  using P2 = typename Pair<R>::T;
  const int np = (G.Ls + 1) / 2;  // pairs of a line
  const long long e0 = (((long long)p * kStrips + w) * NV) * 64 + 2 * lane;
  // c-neighbour outside the strip: lanes 0..15 the -c side, 16..31 the +c side
  const bool cm = lane < 16;
  const bool has_c = cm ? (w > 0 || PCi > 0) : (w + 1 < kStrips || PCi + 1 < G.nPC);
  const long long dc = pl_out_c(G, w, cm);
  // a-neighbour across the patch face: al = 0 the -a side, al = 15 the +a side
  const bool am = alp == 0;
  const bool has_a = (am && PAi > 0) || (alp == kPatch - 1 && PAi + 1 < G.nPA);
  const long long da = pl_out_a(G, am);
  double acc = 0;
  auto ld2 = [](const R* q, long long e) { return *reinterpret_cast<const P2*>(q + e); };
  auto st2 = [](R* q, long long e, P2 t) { *reinterpret_cast<P2*>(q + e) = t; };
  auto mix = [&](P2 a, P2 b) {  // a + beta b
    P2 t;
    t.x = a.x + be * b.x;
    t.y = a.y + be * b.y;
    return t;
  };
  if (v0 < v1) {
    P2 zero;
    zero.x = zero.y = R(0);
    // the values of one step: its own, and those of its neighbours outside
    struct Row {
      P2 ad, as, aa, ac, xv, zc, oc, cc, za, oa, ca;
    };
    auto fetch = [&](int v) {
      Row o;
      const long long e = e0 + (long long)v * 64;
      const bool live = (unsigned)(v - dl) < (unsigned)np;
      o.ad = ld2(A.AD, e);
      o.as = ld2(A.AS, e);
      o.aa = ld2(A.AA, e);
      o.ac = ld2(A.AC, e);
      o.xv = ld2(x, e);
      o.zc = o.oc = o.cc = o.za = o.oa = o.ca = zero;
      if (has_c && live) {
        o.zc = ld2(z, e + dc);
        o.oc = ld2(sold, e + dc);
        if (cm) o.cc = ld2(A.AC, e + dc);
      }
      if (has_a && live) {
        o.za = ld2(z, e + da);
        o.oa = ld2(sold, e + da);
        if (am) o.ca = ld2(A.AA, e + da);
      }
      return o;
    };
    // s_new of steps v - 1, v, v + 1; couplings of step v - 1
    P2 sm1 = zero, ps = zero, pa = zero, pc = zero;
    if (v0 > 0) {
      const long long e = e0 + (long long)(v0 - 1) * 64;
      sm1 = mix(ld2(z, e), ld2(sold, e));
      ps = ld2(A.AS, e);
      pa = ld2(A.AA, e);
      pc = ld2(A.AC, e);
    }
    long long e = e0 + (long long)v0 * 64;
    P2 so = ld2(sold, e);
    P2 s0v = mix(ld2(z, e), so);
    P2 nz = zero, ns = zero;
    if (v0 + 1 < NV) {
      nz = ld2(z, e + 64);
      ns = ld2(sold, e + 64);
    }
    for (int v = v0; v < v1; ++v, e += 64) {
      const Row cur = fetch(v);
      P2 nz2 = zero, ns2 = zero;  // two steps on: s_new of step v + 2
      if (v + 1 < v1 && v + 2 < NV) {
        nz2 = ld2(z, e + 128);
        ns2 = ld2(sold, e + 128);
      }
      const P2 sp1 = mix(nz, ns);
      const P2 sco = mix(cur.zc, cur.oc), sao = mix(cur.za, cur.oa);
      // one cell: couplings and s_new of its neighbours in the order of the row
      auto cell = [&](R o_cc, R o_sc, R o_ca, R o_sa, R m1, R ppa, R ppc, R n1, R ms_c, R ms_s,
                      R ad, R s, R ps_c, R ps_s, R aa, R ac) {
        const R m_a = __shfl_up_sync(full, m1, 1), m_pa = __shfl_up_sync(full, ppa, 1);
        const R m_c = __shfl_up_sync(full, m1, 16), m_pc = __shfl_up_sync(full, ppc, 16);
        const R p_a = __shfl_down_sync(full, n1, 1), p_c = __shfl_down_sync(full, n1, 16);
        R r = 0;
        r += (cm ? o_cc : m_pc) * (cm ? o_sc : m_c);
        r += (am ? o_ca : m_pa) * (am ? o_sa : m_a);
        r += ms_c * ms_s;
        r += ad * s;
        r += ps_c * ps_s;
        r += aa * (alp == kPatch - 1 ? o_sa : p_a);
        r += ac * (cm ? p_c : o_sc);
        return r;
      };
      P2 q2;
      q2.x = cell(cur.cc.x, sco.x, cur.ca.x, sao.x, sm1.x, pa.x, pc.x, sp1.x, ps.y, sm1.y, cur.ad.x,
                  s0v.x, cur.as.x, s0v.y, cur.aa.x, cur.ac.x);
      q2.y = cell(cur.cc.y, sco.y, cur.ca.y, sao.y, sm1.y, pa.y, pc.y, sp1.y, cur.as.x, s0v.x,
                  cur.ad.y, s0v.y, cur.as.y, sp1.x, cur.aa.y, cur.ac.y);
      P2 x2;
      x2.x = cur.xv.x + al * so.x;
      x2.y = cur.xv.y + al * so.y;
      st2(x, e, x2);
      st2(snew, e, s0v);
      st2(A.q, e, q2);
      acc += (double)s0v.x * (double)q2.x;
      acc += (double)s0v.y * (double)q2.y;
      ps = cur.as;
      pa = cur.aa;
      pc = cur.ac;
      sm1 = s0v;
      s0v = sp1;
      so = ns;
      nz = nz2;
      ns = ns2;
    }
  }
  acc = block_sum<double>(acc, sm);
  if (threadIdx.x == 0) A.part[bid] = acc;
  // the last block: alpha = rho / s.q
  if (last_block(A.done_ctr, nblk)) red_alpha_body(A.part, nblk, sc, sm);
}

template <typename R>
__global__ void __launch_bounds__(kRedThreads, sizeof(R) == 4 ? 4 : 2)
    k_pl_spmv_s(const PlSpmvArgs<R> A) {
  pl_spmv_run<R>(A, A.parity != 0, (int)blockIdx.x, (int)gridDim.x);
}

// One SpMV launch over several solves: solve s owns first[s + 1] - first[s]
// blocks; iteration it of a chunk takes s_old / s_new by the solve's iteration
// parity.
template <typename R>
__global__ void __launch_bounds__(kRedThreads, sizeof(R) == 4 ? 4 : 2)
    k_pl_spmv_batch(const PlSpmvArgs<R>* __restrict__ tab, const int* __restrict__ first,
                    int nsolve, int it) {
  const int s = batch_solve_of(first, nsolve, (int)blockIdx.x);
  const PlSpmvArgs<R> a = tab[s];
  const int b0 = __ldg(first + s);
  pl_spmv_run<R>(a, ((a.parity + it) & 1) != 0, (int)blockIdx.x - b0, __ldg(first + s + 1) - b0);
}

// status[6 s + j] = sc_s[S_RES + j] (residual, beta, tolerance, iteration,
// iteration limit, done) for each solve of a chunk
__global__ void k_pl_batch_status(double* const* __restrict__ scs, int nsolve,
                                  double* __restrict__ status) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < 6 * nsolve) status[i] = __ldcg(scs[i / 6] + S_RES + i % 6);
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
  const int nrow = (int)(G.len / kPatchLines);
  for (int row = blockIdx.x; row < nrow; row += gridDim.x) {
    const long long e = (long long)row * kPatchLines + threadIdx.x;
    const PlCell c = pl_cell(G, e);
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
  const int nrow = (int)(G.len / kPatchLines);
  for (int row = blockIdx.x; row < nrow; row += gridDim.x) {
    const long long e = (long long)row * kPatchLines + threadIdx.x;
    const PlCell c = pl_cell(G, e);
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
      const long long idx = pl_index(G, (long long)PCi * G.nPA + PAi, s, al, cl);
      v = x64 ? (R)x64[idx] : x32[idx];
    }
    p[n] = v;
  }
}

}  // namespace wcg
