// Brick form of the triangular sweeps (ILU, IC and SOR applies and the
// transposed ILU apply, src/ported.mojo:633-748, 864-952) for sweeps whose
// dependencies are the unit steps of a Cartesian grid in natural order -- the
// 5- and 7-point stencils, upwind convection-diffusion, any operator with
// that pattern.
//
// On such a grid (nx, ny, nz) a forward sweep's row r = i + nx (j + ny k)
// depends on r - 1 (i - 1), r - nx (j - 1) and r - nx ny (k - 1), each present
// exactly when that coordinate is >= 1; a backward sweep on r + 1, r + nx,
// r + nx ny (mirrored coordinates make both "coordinate minus one").  The
// dependency chain is nx + ny + nz - 2 rows long whatever the schedule, so
// what decides the speed is the cost of one link of it.  On GB300 a hand-off
// between two SMs through L2 costs ~0.5 us (store, poll and return) and a
// dependent FP64 operation 64 cycles (31 ns), during which it also holds its
// sub-partition's FP64 unit.  So the links stay in registers where they can:
//
//   * a warp takes a tile of grid lines (8 x 4 in 3-D, 32 in 2-D) and walks
//     them together, lane (tp, tq) reaching row w of its line at step
//     w + tp + tq: the value one row back is the lane's own last one, the ones
//     a line back the last ones of lanes (tp - 1, tq) and (tp, tq - 1), a
//     shuffle away.  No barrier and no memory is on that chain;
//   * the lines run along the direction whose term a row's fold takes first --
//     k forward (ascending columns k, j, i), i backward -- so the fold starts
//     from the lane's own value and the shuffles (51 cycles from one FP64
//     result to the next operation) pass behind its first operation;
//   * a CTA takes a brick of up to four such tiles, one warp (and one
//     sub-partition's FP64 unit) each.  A value on the face of a tile goes to
//     the neighbouring tile through a shared-memory ring, value-as-flag (a
//     signalling NaN marks "not yet"), indexed by the step;
//   * a value on the face of a brick goes out to global memory, and the fetch
//     warps of the neighbouring CTA poll it there, eight lanes a face line, a
//     row each, and drop each into the reader's ring the moment it is in.  A
//     brick that runs a hand-off behind its neighbour never waits on memory; on
//     128^3 the chain crosses 22 brick faces instead of 381 levels;
//   * in 3-D up to 2 x 4 bricks are a thread-block cluster: a value on a face
//     between two of them is stored straight into the reading tile's ring in the
//     other CTA's shared memory (0.9 us a face where memory takes 2, under load);
//     16 of those 22 faces are then of that kind.  A writer needs to know how far
//     its reader is: a relay warp of the reader's CTA sends that on;
//   * the faces have two copies, used in turn: a sweep reads and writes one
//     and marks the other "not yet" for the next sweep, so nothing is cleared
//     in between and the values of the rows themselves need no flags;
//   * coefficients and diagonals are stored by step, [tile][step][column]
//     [lane], so a group of kGroup steps is one contiguous piece, brought into
//     shared memory by cp.async.bulk two groups ahead; starting values come
//     by cp.async.  Loads into registers would not stay in flight over that
//     many steps: a warp has six scoreboards, and a wait on one is a wait for
//     every load that was put on it (a register ring measured 0.4 us a step);
//   * bricks (clusters of them) are handed out by a ticket in wavefront order
//     (P + Q); one depends only on those at P - 1 and Q - 1, which CTAs that are
//     already running hold, so the sweep cannot deadlock whatever the number
//     of resident CTAs.  Within a CTA a warp waits on lower steps only (for a
//     value, or for a reader a whole ring behind), and every wait has a budget.
//
// What it measures (one sweep, GB300): 122 us forward and 135 backward on 128^3
// (382 rows of chain; 163-168 with every face through memory, 370 and 466 in the
// level-ordered form), 92 and 100 on 96^3 (110 and 121), 83 and 94 on 256^2 (511 rows;
// 250 in the chunked form).  Its time is 0.24 us a row of the chain in 3-D (three
// dependent FP64 operations are 0.093, and a face's shuffle, poll and store lie
// between), 0.9 us a face inside a cluster and 2 us one through memory.
//
// Every row is the reference's fold of its terms in ascending-column order,
// with the same operations as k_ell_sweep: results are bit-identical to the
// reference's sequential sweeps and to the other forms.
#include <algorithm>
#include <atomic>
#include <climits>
#include <cstdio>
#include <cstdlib>
#include <string>
#include <type_traits>
#include <vector>

#include "gp_pc.h"

namespace gp {

constexpr int kBrickMaxLines = 128;  // forced lines of a brick
constexpr int kBrickWarps = 4;       // tiles (compute warps) of a brick
constexpr int kBrickRing = 32;       // steps a tile's ring holds (a power of two)
constexpr int kGroup = 16;           // steps staged together
constexpr int kHalf = 8;             // steps between two looks at the neighbours' progress
constexpr int kStages = 2;           // groups in shared memory
constexpr int kBrickPoll = 8;        // lanes that poll a face line, a row each (fewer for many lines)
// threads: the tiles' warps and those that fetch
constexpr int kBrickFetchMax = 7;
constexpr int kBrickMaxThreads = 32 * (kBrickWarps + kBrickFetchMax + 1);
// Doubles of a ring step: Wq p-face lines, Wp q-face lines, a column that is
// never empty and one that is never read (for lanes with no face)
__host__ __device__ constexpr int brick_pitch(bool full, bool d3) {
  return full ? (d3 ? 16 : 4) : 32;
}
__host__ __device__ constexpr int brick_ring(bool full, bool d3) {
  return kBrickRing * brick_pitch(full, d3);
}
constexpr int kBrickSmemMax = 226 * 1024;
constexpr int kBrickSpin = 1 << 22;  // polls before a wait gives up

// Shape of one sweep's layout, in the sweep's own (mirrored, if backward)
// coordinates: row (w, p, q) is f = w sw + p sp + q sq, row f of the grid or
// n - 1 - f.  Lines along w; tile (P, Q) of ntP x ntQ, lane tp + Wp tq.
struct BrickShape {
  int n, nw, np, nq;
  int sw, sp, sq;
  int Wp, Wq, LW;    // lines of a tile; LW = Wp Wq of them stored, rounded up to even
  int CP, CQ;        // tiles of a brick
  int XP, XQ;        // bricks of a cluster
  int ntP, ntQ, nbP, nbQ;
  int NS;            // steps stored a tile: nw + Wp + Wq - 2 and its phase, in whole groups
  int nwp;           // rows of a face line in memory
  int bwd, d3;
};

struct BrickArgs {
  BrickShape g;
  int nclusters;
  const int* border;      // [2 * nclusters]: (P, Q) of each cluster in hand-out order
  const double* coef;     // [tile][step][columns by lane]: brick_store
  double* faces;          // [2][fsize]: the p faces, then the q faces
  long long fsize, qface;  // doubles of one copy; where its q faces start
  int* parity;            // which copy this sweep uses
  const double* tin;      // the first sweep's values, by row
  const double* tin2;     // SOR backward: its checkpoint
  double* tout;           // first sweeps: where they go
  double* tout2;          // SOR forward: the checkpoint
  double om1;
  int write_out;
  int poll;               // fetching lanes a face line
  int nf;                 // fetch warps
  unsigned* tickets;
  DevErr* err;
};

// Modes with a stored column of diagonal factors.
__host__ __device__ constexpr bool brick_has_diag(int mode) {
  return mode == ELL_ILU_B || mode == ELL_ILUT_F || mode == ELL_ICC_F || mode == ELL_SOR_F ||
         mode == ELL_SOR_B || mode == ELL_SOR_B0;
}
__host__ __device__ constexpr bool brick_bwd(int mode) {
  return mode == ELL_ILU_B || mode == ELL_ILUT_B || mode == ELL_ICC_B || mode == ELL_SOR_B ||
         mode == ELL_SOR_B0;
}

// A row's fold is one term a direction in a fixed order -- k, j, i forward,
// i, j, k backward: the ascending columns -- for every row: a term the row
// does not have (at the grid boundary) has coefficient 0 and value `absent`,
// and c * absent = -0 for ILU / SOR (sum - c v) and IC (sum + c v) alike,
// which leaves every sum, -0 included, unchanged: the same bits as skipping
// the term.
template <int MODE>
__device__ __forceinline__ double brick_absent() {
  return (MODE == ELL_ICC_F || MODE == ELL_ICC_B) ? -0.0 : 0.0;
}

template <int MODE, bool FMA>
__device__ __forceinline__ double brick_term(double sum, double c, double v) {
  if constexpr (MODE == ELL_ICC_F || MODE == ELL_ICC_B)
    return FMA ? __fma_rn(c, v, sum) : add(sum, mul(c, v));
  else
    return FMA ? __fma_rn(-c, v, sum) : sub(sum, mul(c, v));
}

// Columns of a step: the coefficients (of the line's own direction, then of
// the two across in fold order) and the diagonal factor, in pairs of a lane's
// neighbours in memory; then, staged beside them, the starting value and (SOR's
// backward half) the forward value.
__host__ __device__ constexpr int brick_coefs(int mode, bool d3) {
  return (d3 ? 3 : 2) + (brick_has_diag(mode) ? 1 : 0);
}
__host__ __device__ constexpr int brick_cols(int mode, bool d3) {
  return brick_coefs(mode, d3) + 1 + (mode == ELL_SOR_B ? 1 : 0);
}

// What a row needs.
struct BrickRow {
  double c0, c1, c2;  // coefficients in fold order
  double sum0;        // the row's starting value
  double dv;          // diagonal factor
  double yf;          // SOR_B: the forward value's share, (1 - omega) y
};

// ---- shared-memory staging: bulk copies counted on an mbarrier, and 8-byte
// asynchronous copies by line
__device__ __forceinline__ unsigned bk_smem(const void* p) {
  return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void bk_mbar_init(unsigned long long* bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bk_smem(bar)) : "memory");
}
__device__ __forceinline__ void bk_expect(unsigned long long* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bk_smem(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void bk_bulk(void* dst, const void* src, unsigned bytes,
                                        unsigned long long* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
          "r"(bk_smem(dst)),
      "l"(src), "r"(bytes), "r"(bk_smem(bar))
      : "memory");
}
__device__ __forceinline__ bool bk_wait(unsigned long long* bar, unsigned parity) {
  for (int i = 0; i < kBrickSpin; i++) {
    unsigned done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bk_smem(bar)), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}
// 8 bytes, or zeros (reading nothing) unless `ok`.
__device__ __forceinline__ void bk_async8(unsigned dst, const double* src, bool ok) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src),
               "r"(ok ? 8 : 0)
               : "memory");
}
__device__ __forceinline__ void bk_commit() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}

__device__ __forceinline__ bool brick_failed(DevErr* err) {
  return *reinterpret_cast<volatile int*>(&err->code) != 0;
}

// Ring slots, by shared-memory address.  Not clobbering memory: their order
// among each other is kept, and nothing else reads or writes a ring.  The
// predicated forms are predicated instructions, not branches.
__device__ __forceinline__ double ring_get(unsigned a) {
  double v;
  asm volatile("ld.volatile.shared.f64 %0, [%1];" : "=d"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ void ring_put(unsigned a, double v) {
  asm volatile("st.volatile.shared.f64 [%0], %1;" ::"r"(a), "d"(v));
}
// CL: an address of cluster_addr, of this or another CTA of the cluster.
template <bool CL>
__device__ __forceinline__ void ring_put_if(bool p, unsigned a, double v) {
  if constexpr (CL)
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t"
        "@p st.relaxed.cluster.shared::cluster.f64 [%0], %1;\n\t}" ::"r"(a),
        "d"(v), "r"((unsigned)p));
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t"
        "@p st.volatile.shared.f64 [%0], %1;\n\t}" ::"r"(a),
        "d"(v), "r"((unsigned)p));
}
// Whether a slot is still empty.  The high word decides: no double with the
// flag's high word is ever computed (every one is a signalling NaN).
__device__ __forceinline__ bool empty_slot(double v) {
  return (unsigned)__double2hiint(v) == (unsigned)(kPending >> 32);
}
__device__ __forceinline__ double pending_value() {
  return __longlong_as_double((long long)kPending);
}
__device__ __forceinline__ double quiet_nan() {
  return __longlong_as_double(0x7FF8000000000000LL);
}
// A step's operands from its stage: kept where they stand in the program (a
// step before their use), past the waits that come between.
__device__ __forceinline__ double stage_get(unsigned a) {
  double v;
  asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ void stage_get2(unsigned a, double& x, double& y) {
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(x), "=d"(y) : "r"(a));
}
// A tile's next step, to the writers of its ring: after the slots it emptied.
__device__ __forceinline__ void publish(int* p, int step) {
  asm volatile("st.release.cta.shared.b32 [%0], %1;" ::"r"(bk_smem(p)), "r"(step) : "memory");
}
// A tile's progress, read by a writer of its ring: an acquire, paired with the
// release of the publishing warp (or of the relay, for a tile in another CTA of
// the cluster), so that the slots' emptying comes before the values that the
// writer stores into them next.  A plain read and the branch on it would promise
// no such order.
__device__ __forceinline__ int progress(const int* p) {
  int v;
  asm volatile("ld.acquire.cta.shared.b32 %0, [%1];" : "=r"(v) : "r"(bk_smem(p)) : "memory");
  return v;
}
__device__ __forceinline__ int progress_cluster(const int* p) {
  int v;
  asm volatile("ld.acquire.cluster.shared::cta.b32 %0, [%1];"
               : "=r"(v)
               : "r"(bk_smem(p))
               : "memory");
  return v;
}
// A face value to the other bricks.
__device__ __forceinline__ void face_put_if(bool p, double* a, double v) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t"
      "@p st.relaxed.gpu.global.f64 [%0], %1;\n\t}" ::"l"(a),
      "d"(v), "r"((unsigned)p));
}

// ---- clusters
__device__ __forceinline__ int cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return (int)r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile(
      "barrier.cluster.arrive.release;\n\t"
      "barrier.cluster.wait.acquire;" ::
          : "memory");
}
// A shared-memory address in a CTA of the cluster.
__device__ __forceinline__ unsigned cluster_addr(unsigned a, int rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
// The same shared-memory variable of another CTA of the cluster.
template <typename T>
__device__ __forceinline__ T* cluster_map(T* p, int rank) {
  unsigned long long q;
  asm volatile("mapa.u64 %0, %1, %2;" : "=l"(q) : "l"(p), "r"(rank));
  return reinterpret_cast<T*>(q);
}

// One lane of the relay warp: a tile's progress (prog) to the CTA that writes one
// of its faces (dst, in that CTA), until the tile is at `end`.  The tile's own
// warp publishes to its CTA only: a release that other SMs can see waits for the
// warp's stores on their way to the L2, a thousand cycles every kHalf steps.
__device__ void brick_relay(const int* prog, int* dst, int at, int end, bool on, DevErr* err) {
  int spins = 0;
  while (__any_sync(0xffffffffu, on)) {
    if (on) {
      const int v = progress(prog);
      if (v != at) {
        asm volatile("st.release.cluster.b32 [%0], %1;" ::"l"(dst), "r"(v) : "memory");
        at = v;
        spins = 0;
        on = v < end;
      } else if (++spins > kBrickSpin) {
        if (atomicCAS(&err->code, 0, GP_ERR_TIMEOUT) == 0) err->where = 45;
        on = false;
      }
    }
  }
}

// One lane of a fetch warp: rows i, i + poll, ... of one face line into
// the reader's ring, row i at slot i + t0.  A row goes in once the reader is
// less than a ring behind it (`prog`: its next step), and its place in the
// line's other copy is emptied for the next sweep.
template <int PITCH>
__device__ void brick_fetch(const double* line, double* next, int i, int poll, int nw, unsigned ring,
                            int t0, const int* prog, bool act, DevErr* err) {
  int spins = 0;
  if (!act) i = nw;
  while (__any_sync(0xffffffffu, i < nw)) {
    if (i < nw) {
      unsigned long long v = kPending;
      const bool room = i + t0 < progress(prog) + kBrickRing - 1;
      if (room) v = ld_relaxed_bits(line + i);
      if (++spins > kBrickSpin || ((spins & 1023) == 1023 && brick_failed(err))) {
        // never arrived (or the reader never moved): record it and hand on a
        // quiet NaN where there is room for one
        if (atomicCAS(&err->code, 0, GP_ERR_TIMEOUT) == 0) err->where = 43;
        if (!room) i = nw;
        if (room && v == kPending) v = 0x7FF8000000000000ULL;
      }
      if (v != kPending) {
        ring_put(ring + 8 * (((i + t0) & (kBrickRing - 1)) * PITCH),
                 __longlong_as_double((long long)v));
        next[i] = pending_value();
        i += poll;
        spins = 0;
      }
    }
  }
}

// Steps are counted over the whole brick: line (pb, qb) of a brick is at row w
// at step w + pb + qb, and a tile at (cp, cq) of its brick starts at the
// multiple of kHalf below step cp Wp + cq Wq, `phase` steps before its first row.
__host__ __device__ __forceinline__ int brick_phase(const BrickShape& g, int P, int Q) {
  return ((P % g.CP) * g.Wp + (Q % g.CQ) * g.Wq) % kHalf;
}

// Launched with 32 (CP CQ + NF) threads: a warp a tile, then the fetch warps.
// Dynamic shared memory: the tiles' rings, then their stages.  FULL: 32 lines
// a tile (every address within a group is then an immediate offset).  D3: a
// third direction (without it, two terms a row).
//
// A ring slot holds what was computed at the brick's step of that number, for
// the step after it; writer and reader thus use the same slot at the same
// place of a group, and no address within a group is computed.  The step's
// instructions are what is left on the chain besides its FP64 operations, so
// the loop is kept to about forty, nearly all without a branch.
template <int MODE, bool FMA, bool FULL, bool D3, bool CL>
__global__ void __launch_bounds__(kBrickMaxThreads, 1) k_brick_sweep(const int* gate, int want,
                                                                     BrickArgs a, DRef inr,
                                                                     DRef outr) {
  if (gated_off(gate, want)) return;
  constexpr bool BWD = brick_bwd(MODE);
  constexpr bool DIAG = brick_has_diag(MODE);
  constexpr int NC = brick_coefs(MODE, D3), NV = brick_cols(MODE, D3);
  constexpr unsigned full = 0xffffffffu;
  const BrickShape& g = a.g;
  // second sweeps start from the first one's values; SOR's backward half
  // without a forward one starts from the input
  const double* __restrict__ in = MODE == ELL_SOR_B            ? a.tin2
                                  : BWD && MODE != ELL_SOR_B0 ? a.tin
                                                              : inr.get();
  double* __restrict__ out = outr.get();
  extern __shared__ __align__(16) double brick_smem[];
  __shared__ unsigned long long bars[kBrickWarps][kStages];
  __shared__ int prog[kBrickWarps];  // each tile's next step
  // and of the tiles in the cluster's other CTAs that read its p and q faces
  __shared__ int rprog[2][kBrickWarps];
  __shared__ int s_brick;
  const int nw = g.nw, Wp = g.Wp, Wq = g.Wq, LW = FULL ? 32 : g.LW, NS = g.NS;
  const int nt = g.CP * g.CQ, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int PITCH = brick_pitch(FULL, D3), RING = brick_ring(FULL, D3);
  const int stage_n = kGroup * NV * LW;
  double* const stages = brick_smem + nt * RING;
  const unsigned ring0 = bk_smem(brick_smem);
  const int par = *a.parity;
  double* const f_now = a.faces + (par ? a.fsize : 0);
  double* const f_next = a.faces + (par ? 0 : a.fsize);
  const double absent = brick_absent<MODE>();
  for (int q = threadIdx.x; q < nt * RING; q += blockDim.x)
    ring_put(ring0 + 8 * q, q % PITCH == PITCH - 2 ? absent : pending_value());
  if (threadIdx.x < kBrickWarps * kStages) bk_mbar_init(&bars[0][0] + threadIdx.x);
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  const int tq = lane / Wp, tp = lane - tq * Wp;
  unsigned phases = 0;  // parity of each stage's next wait
  const int XC = CL ? g.XP * g.XQ : 1, rank = CL ? cluster_rank() : 0;
  const int xp = CL ? rank % g.XP : 0, xq = CL ? rank / g.XP : 0;
  for (;;) {
    // the last brick's reads and writes are over in the whole cluster
    if constexpr (CL) cluster_sync();
    if (threadIdx.x == 0 && rank == 0) {
      const int b = (int)atomicAdd(&a.tickets[0], 1u);
      s_brick = b;
      for (int r = 1; r < XC; r++) *cluster_map(&s_brick, r) = b;
    }
    if (threadIdx.x < nt) {
      const int cp = threadIdx.x % g.CP, cq = threadIdx.x / g.CP;
      prog[threadIdx.x] = (cp * Wp + cq * Wq) / kHalf * kHalf;
      if constexpr (CL) {
        rprog[0][threadIdx.x] = cq * Wq / kHalf * kHalf;
        rprog[1][threadIdx.x] = cp * Wp / kHalf * kHalf;
      }
    }
    if constexpr (CL)
      cluster_sync();
    else
      __syncthreads();
    const int b = s_brick;
    if (b >= a.nclusters) break;
    const int bP = a.border[2 * b] * (CL ? g.XP : 1) + xp;
    const int bQ = a.border[2 * b + 1] * (CL ? g.XQ : 1) + xq;
    if (CL && warp >= nt + a.nf) {
      // ---- relay: lane 2 w + d, tile w's progress to the writer of its p (d 0)
      // or q face, where that is in the cluster
      const int w = lane >> 1, d = lane & 1, cp = w % g.CP, cq = w / g.CP;
      const bool on = w < nt && bP * g.CP + cp < g.ntP && bQ * g.CQ + cq < g.ntQ &&
                      (d ? D3 && cq == 0 && xq > 0 : cp == 0 && xp > 0);
      const int sb = (cp * Wp + cq * Wq) / kHalf * kHalf;
      int* dst = cluster_map(&rprog[d][on ? (d ? (g.CQ - 1) * g.CP + cp : cq * g.CP + g.CP - 1) : 0],
                             on ? rank - (d ? g.XP : 1) : rank);
      brick_relay(&prog[on ? w : 0], dst, sb, sb + NS, on, a.err);
    } else if (warp >= nt) {
      // ---- fetch: the brick's p faces (CQ Wq lines), then its q faces,
      // a.poll lanes a line
      const int np = g.CQ * Wq, lines = np + (D3 ? g.CP * Wp : 0);
      const int t = threadIdx.x - 32 * nt, c = t / a.poll;
      bool act = false;
      long long line = 0;
      int w = 0, col = 0, t0 = 0;
      if (c < np) {
        const int cq = c / Wq;
        col = c - cq * Wq;
        w = cq * g.CP;
        t0 = c - 1;  // the step before row 0 of line (0, c)
        const int Q = bQ * g.CQ + cq, ql = Q * Wq + col;
        act = bP > 0 && xp == 0 && bP < g.nbP && ql < g.nq;
        line = ((long long)bP * (g.ntQ * Wq) + ql) * g.nwp;
      } else if (c < lines) {
        const int cp = (c - np) / Wp, tl = c - np - cp * Wp;
        w = cp;
        t0 = c - np - 1;
        col = Wq + tl;
        const int P = bP * g.CP + cp, pl = P * Wp + tl;
        act = bQ > 0 && xq == 0 && bQ < g.nbQ && pl < g.np;
        line = a.qface + ((long long)bQ * (g.ntP * Wp) + pl) * g.nwp;
      }
      brick_fetch<PITCH>(f_now + line, f_next + line, t % a.poll, a.poll,
                         nw, ring0 + 8 * (w * RING + col), t0, &prog[w], act, a.err);
    } else {
      // ---- compute: one tile
      const int cq = warp / g.CP, cp = warp - cq * g.CP;
      const int P = bP * g.CP + cp, Q = bQ * g.CQ + cq;
      if (P < g.ntP && Q < g.ntQ) {
        const int pl = P * Wp + tp, ql = Q * Wq + tq;
        const bool line = lane < Wp * Wq && pl < g.np && ql < g.nq;
        const int phase = (cp * Wp + cq * Wq) % kHalf;
        const int sb = cp * Wp + cq * Wq - phase;  // the tile's first step
        // the tile's step s (counted from sb) is row s - off of the lane's line
        const int off = line ? phase + tp + tq : INT_MAX / 2;  // an idle lane never starts
        const int ll = line ? lane : 0;
        // the line's row w is at row0 + rs w
        const long long rs = BWD ? -(long long)g.sw : g.sw;
        const long long f0 = line ? pl * (long long)g.sp + ql * (long long)g.sq : 0;
        const long long row0 = BWD ? g.n - 1 - f0 : f0;
        const double* const cf = a.coef + (long long)(P + g.ntP * Q) * NS * NC * LW;
        double* const stage = stages + warp * (kStages * stage_n);
        const int ngroups = NS / kGroup;
        const long long roff = row0 - rs * (line ? off : 0);  // step 0's row
        const double* src = in + roff;
        const double* src2 = MODE == ELL_SOR_B ? a.tin + roff : nullptr;
        // stage group q (steps kGroup q ..): one commit group a call, empty
        // where the sweep has no more steps
        auto fill = [&](int q, int si) {
          double* const st = stage + si * stage_n;
          if (q < ngroups) {
            if (lane == 0) {
              unsigned long long* bar = &bars[warp][si];
              constexpr unsigned cb1 = kGroup * NC * 8;
              // the stage's last readers are behind a __syncwarp
              bk_expect(bar, cb1 * LW);
              bk_bulk(st, cf + (long long)q * (kGroup * NC * LW), cb1 * LW, bar);
            }
            const int w0 = q * kGroup - off;
            const unsigned dst = bk_smem(st + kGroup * NC * LW + lane);
            if (lane < LW) {
#pragma unroll
              for (int u = 0; u < kGroup; u++) {
                const bool ok = (unsigned)(w0 + u) < (unsigned)nw;
                bk_async8(dst + u * 8 * LW, src + rs * u, ok);
                if constexpr (MODE == ELL_SOR_B)
                  bk_async8(dst + (kGroup + u) * 8 * LW, src2 + rs * u, ok);
              }
            }
            src += rs * kGroup;
            if constexpr (MODE == ELL_SOR_B) src2 += rs * kGroup;
          }
          bk_commit();
        };
        // where this tile's face values come from and go to
        const unsigned ring = ring0 + 8 * warp * RING;
        const bool fromp = line && tp == 0 && P > 0, fromq = D3 && line && tq == 0 && Q > 0;
        const bool faces = __any_sync(full, fromp || fromq);
        const bool lastp = line && tp == Wp - 1 && P + 1 < g.ntP;
        const bool lastq = D3 && line && tq == Wq - 1 && Q + 1 < g.ntQ;
        const bool ringp = cp + 1 < g.CP && P + 1 < g.ntP, ringq = cq + 1 < g.CQ && Q + 1 < g.ntQ;
        // faces that go into the ring of a tile in another CTA of the cluster
        const bool clp = CL && !ringp && P + 1 < g.ntP && xp + 1 < g.XP;
        const bool clq = CL && D3 && !ringq && Q + 1 < g.ntQ && xq + 1 < g.XQ;
        const bool rings = ringp || ringq || clp || clq;
        // this lane's columns: read from, emptied, and the neighbouring tiles'
        const unsigned colp = ring + 8 * tq, colq = ring + 8 * (Wq + tp);
        const unsigned full_col = ring + 8 * (PITCH - 2), no_col = ring + 8 * (PITCH - 1);
        const unsigned rp = fromp ? colp : full_col, rq = fromq ? colq : full_col;
        const unsigned ep = fromp ? colp : no_col, eq = fromq ? colq : no_col;
        // a neighbour in the cluster's next CTA is its tile (0, cq) or (cp, 0), and a
        // brick's step t is step t - shp (shq) there, both multiples of kHalf
        const int shp = CL && clp ? g.CP * Wp : 0, shq = CL && clq ? g.CQ * Wq : 0;
        unsigned np = lastp && ringp ? colp + 8 * RING : no_col;
        unsigned nq = lastq && ringq ? colq + 8 * g.CP * RING : no_col;
        if constexpr (CL) {
          np = cluster_addr(lastp && clp ? ring0 + 8 * (cq * g.CP * RING + tq) : np,
                            lastp && clp ? rank + 1 : rank);
          nq = cluster_addr(lastq && clq ? ring0 + 8 * (cp * RING + Wq + tp) : nq,
                            lastq && clq ? rank + g.XP : rank);
        }
        // faces that go to memory, and the lanes that write them
        const bool memp = P + 1 < g.ntP && !ringp && !clp;
        const bool memq = D3 && Q + 1 < g.ntQ && !ringq && !clq;
        const bool outp = lastp && memp, outq = lastq && memq;
        const int nwop = outp ? nw : 0, nwoq = outq ? nw : 0;
        // face lines this lane writes (row -off at the pointer)
        double* fop = f_now + ((long long)(bP + 1) * (g.ntQ * Wq) + ql) * g.nwp - (outp ? off : 0);
        double* foq = f_now + a.qface + ((long long)(bQ + 1) * (g.ntP * Wp) + pl) * g.nwp -
                      (outq ? off : 0);
        double* po = (BWD ? out : a.tout) + roff;  // step 0's row
        double* pt2 = MODE == ELL_SOR_F ? a.tout2 + roff : nullptr;
        double* pw = MODE == ELL_SOR_F && a.write_out ? out + roff : nullptr;
        for (int q = 0; q < kStages; q++) fill(q, q);
        // a face lane's value for the step at hand, `absent` where it has none
        unsigned before = 8 * ((sb - 1) & (kBrickRing - 1)) * PITCH;  // the last step's slot
        double fp = ring_get(rp + before), fq = ring_get(rq + before);
        double prev = absent;  // the lane's last value (none before its first row)
        int si = 0;
        for (int s0 = 0; s0 < NS; s0 += kGroup) {
          // the group's stage: this lane's copies (all lanes' behind the
          // __syncwarp), then the bulk copy
          asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 1) : "memory");
          if (!bk_wait(&bars[warp][si], phases >> si & 1u)) {
            if (atomicCAS(&a.err->code, 0, GP_ERR_TIMEOUT) == 0) a.err->where = 44;
          }
          phases ^= 1u << si;
          __syncwarp();
          const unsigned st = bk_smem(stage + si * stage_n);
          unsigned c0 = st + 16 * ll, v0 = st + 8 * (kGroup * NC * LW + ll);
          unsigned c1 = st + 16 * LW + (D3 && DIAG ? 16 : 8) * ll;
          auto take = [&](int u) {
            BrickRow r;
            r.sum0 = stage_get(v0 + 8 * u * LW);
            stage_get2(c0 + 8 * u * NC * LW, r.c0, r.c1);
            if constexpr (D3 && DIAG)
              stage_get2(c1 + 8 * u * NC * LW, r.c2, r.dv);
            else if constexpr (D3)
              r.c2 = stage_get(c1 + 8 * u * NC * LW);
            else if constexpr (DIAG)
              r.dv = stage_get(c1 + 8 * u * NC * LW);
            if constexpr (MODE == ELL_SOR_B) r.yf = mul(a.om1, stage_get(v0 + 8 * (kGroup + u) * LW));
            return r;
          };
          BrickRow r = take(0);
          // with_faces: some lane reads face values.  out: the last lines' values go
          // to rings (1), to the faces in memory (2), or both.  In 3-D, where a
          // tile may have one of each, all take the same code: four forms with
          // one store a direction cost 25% on 128^3, a fetch of instructions for
          // each of the SM's warps.  In 2-D the tiles of a row differ less, and
          // one store saves 6% on 256^2 (210 to 198 us a pair of sweeps).
          auto steps = [&](auto with_faces, auto out) {
            constexpr bool FACES = decltype(with_faces)::value;
            constexpr int OUT = decltype(out)::value;
            // unrolled over half a group: the code has to stay in the
            // instruction cache of the sub-partition that runs it
#pragma unroll 1
            for (int u0 = 0; u0 < kGroup; u0 += kHalf) {
              if constexpr (FACES) {
                if (u0) {  // the slots of the steps so far are free
                  __syncwarp();
                  if (lane == 0) publish(&prog[warp], sb + s0 + u0);
                }
              }
              if constexpr (OUT & 1) {
                // room in the rings of the neighbouring tiles for the next values
                if (rings) {
                  for (int spins = 0;; spins++) {
                    const int at_p = ringp ? progress(&prog[warp + 1])
                                     : clp ? progress_cluster(&rprog[0][warp]) + shp
                                           : INT_MAX / 2;
                    const int at_q = ringq ? progress(&prog[warp + g.CP])
                                     : clq ? progress_cluster(&rprog[1][warp]) + shq
                                           : INT_MAX / 2;
                    if (sb + s0 + u0 + kHalf < min(at_p, at_q) + kBrickRing) break;
                    if (spins > kBrickSpin || ((spins & 4095) == 4095 && brick_failed(a.err))) {
                      if (lane == 0 && atomicCAS(&a.err->code, 0, GP_ERR_TIMEOUT) == 0)
                        a.err->where = 42;
                      break;
                    }
                  }
                }
              }
              const unsigned slot = 8 * (((sb + s0 + u0) & (kBrickRing - 1)) * PITCH);
              const unsigned wp = np + (CL ? 8 * (((sb + s0 + u0 - shp) & (kBrickRing - 1)) * PITCH)
                                           : slot);
              const unsigned wq = nq + (CL ? 8 * (((sb + s0 + u0 - shq) & (kBrickRing - 1)) * PITCH)
                                           : slot);
#pragma unroll
              for (int h = 0; h < kHalf; h++) {
              const int u = u0 + h, w = s0 - off + u;
              const bool act = (unsigned)w < (unsigned)nw;
              double vp = __shfl_up_sync(full, prev, 1);
              double vq = absent;
              if constexpr (D3) vq = __shfl_up_sync(full, prev, Wp);
              double sum = brick_term<MODE, FMA>(r.sum0, r.c0, prev);
              // the next row's operands, behind the shuffles in the queue
              BrickRow ahead;
              if (h + 1 < kHalf || u0 == 0) ahead = take(h + 1);
              if constexpr (FACES) {
                // inactive lanes have no value to wait for, and any will do
                if (__any_sync(full, act && (empty_slot(fp) || (D3 && empty_slot(fq))))) {
                  int spins = 0;
                  do {
                    if (empty_slot(fp)) fp = ring_get(rp + before);
                    if (D3 && empty_slot(fq)) fq = ring_get(rq + before);
                    if (++spins > kBrickSpin || ((spins & 4095) == 4095 && brick_failed(a.err))) {
                      if (atomicCAS(&a.err->code, 0, GP_ERR_TIMEOUT) == 0) a.err->where = 41;
                      if (empty_slot(fp)) fp = quiet_nan();
                      if (empty_slot(fq)) fq = quiet_nan();
                    }
                  } while (__any_sync(full, act && (empty_slot(fp) || (D3 && empty_slot(fq)))));
                }
                if (tp == 0) vp = fp;
                if (D3 && tq == 0) vq = fq;
                ring_put(ep + before, pending_value());
                if constexpr (D3) ring_put(eq + before, pending_value());
                // a first look at the next step's values
                before = slot + h * (8 * PITCH);
                fp = ring_get(rp + before);
                if constexpr (D3) fq = ring_get(rq + before);
              } else {
                if (tp == 0) vp = absent;
                if (D3 && tq == 0) vq = absent;
              }
              // forward: k, j, i = own, q, p; backward: i, j, k = own, p, q
              if constexpr (!D3) {
                sum = brick_term<MODE, FMA>(sum, r.c1, vp);
              } else if constexpr (!BWD) {
                sum = brick_term<MODE, FMA>(sum, r.c1, vq);
                sum = brick_term<MODE, FMA>(sum, r.c2, vp);
              } else {
                sum = brick_term<MODE, FMA>(sum, r.c1, vp);
                sum = brick_term<MODE, FMA>(sum, r.c2, vq);
              }
              double y;
              if constexpr (MODE == ELL_ILU_B || MODE == ELL_ILUT_F || MODE == ELL_SOR_F ||
                            MODE == ELL_SOR_B0)
                y = mul(sum, r.dv);
              else if constexpr (MODE == ELL_SOR_B)
                y = add(r.yf, mul(sum, r.dv));
              else
                y = sum;
              prev = act ? y : prev;
              // the values other tiles wait on go out first
              if constexpr (OUT & 1) {
                ring_put_if<CL>(act, wp + h * (8 * PITCH), y);
                if constexpr (D3) ring_put_if<CL>(act, wq + h * (8 * PITCH), y);
              }
              if constexpr (OUT & 2) {
                face_put_if((unsigned)w < (unsigned)nwop, fop + h, y);
                if constexpr (D3) face_put_if((unsigned)w < (unsigned)nwoq, foq + h, y);
              }
              const double t = MODE == ELL_ICC_F ? mul(sum, r.dv) : y;
              if (act) po[rs * h] = t;
              if constexpr (MODE == ELL_SOR_F) {
                if (act) pt2[rs * h] = sum;
                if (act && pw) pw[rs * h] = y;
              }
              r = ahead;
              }
              c0 += 8 * kHalf * NC * LW;
              c1 += 8 * kHalf * NC * LW;
              v0 += 8 * kHalf * LW;
              fop += kHalf;
              foq += kHalf;
              po += rs * kHalf;
              if constexpr (MODE == ELL_SOR_F) {
                pt2 += rs * kHalf;
                if (pw) pw += rs * kHalf;
              }
            }
          };
          using std::integral_constant;
          if constexpr (D3) {
            steps(std::true_type{}, integral_constant<int, 3>{});
          } else if (faces) {
            if (memp)
              steps(std::true_type{}, integral_constant<int, 2>{});
            else
              steps(std::true_type{}, integral_constant<int, 1>{});
          } else if (memp) {
            steps(std::false_type{}, integral_constant<int, 2>{});
          } else if (rings) {
            steps(std::false_type{}, integral_constant<int, 1>{});
          } else {
            steps(std::false_type{}, integral_constant<int, 0>{});
          }
          __syncwarp();  // the stage is read, the ring's slots are free
          fill(s0 / kGroup + kStages, si);
          si = si + 1 == kStages ? 0 : si + 1;
          if ((D3 || faces) && lane == 0) publish(&prog[warp], sb + s0 + kGroup);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
      }
    }
    if constexpr (!CL) __syncthreads();
  }
  if (threadIdx.x == 0 && atomic_add_acq_rel(&a.tickets[1], 1u) == gridDim.x - 1) {
    a.tickets[0] = 0u;
    a.tickets[1] = 0u;
    *a.parity = par ^ 1;
  }
}

// Stored coefficients from the factor (or operator) values: one thread a
// position of [tile][step][lane], its coefficients in fold order (0 where the
// row has no such term or there is no row) and the diagonal: src[dslot[row]],
// or diag[row] for SOR.
__global__ void k_brick_refresh(BrickShape g, int nc, int npos,
                                const int* __restrict__ slot, const int* __restrict__ dslot,
                                const double* __restrict__ src, const double* __restrict__ diag,
                                double* __restrict__ coef) {
  const int nd = g.d3 ? 3 : 2;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < npos; e += gridDim.x * blockDim.x) {
    const int lane = e % g.LW, ts = e / g.LW, s = ts % g.NS, T = ts / g.NS;
    const int P = T % g.ntP, Q = T / g.ntP, tq = lane / g.Wp, tp = lane - tq * g.Wp;
    const int w = s - tp - tq - brick_phase(g, P, Q), p = P * g.Wp + tp, q = Q * g.Wq + tq;
    double v[4] = {0.0, 0.0, 0.0, 0.0};
    if (lane < g.Wp * g.Wq && w >= 0 && w < g.nw && p < g.np && q < g.nq) {
      const int f = w * g.sw + p * g.sp + q * g.sq, row = g.bwd ? g.n - 1 - f : f;
      for (int d = 0; d < nd; d++) {
        // fold order: k, j, i forward and i, j, k backward
        const int c = slot[(size_t)(g.bwd ? d : nd - 1 - d) * g.n + row];
        if (c >= 0) v[d] = src[c];
      }
      if (nc > nd) v[nd] = diag ? diag[row] : src[dslot[row]];
    }
    // columns 0 and 1 as pairs by lane, then the rest: a pair or a column
    double* const c = coef + (size_t)ts * nc * g.LW;
    c[2 * lane] = v[0];
    c[2 * lane + 1] = v[1];
    if (nc == 4) {
      c[2 * g.LW + 2 * lane] = v[2];
      c[2 * g.LW + 2 * lane + 1] = v[3];
    } else if (nc == 3) {
      c[2 * g.LW + lane] = v[2];
    }
  }
}

__global__ void k_brick_clear(long long n, double* __restrict__ faces) {
  const double p = __longlong_as_double((long long)kPending);
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n;
       q += (long long)gridDim.x * blockDim.x)
    faces[q] = p;
}

// ------------------------------------------------------------------ host
template <typename T>
static int bup(T** d, const std::vector<T>& h) {
  GP_CUDA(cudaMalloc(d, std::max<size_t>(h.size(), 1) * sizeof(T)));
  if (!h.empty()) GP_CUDA(cudaMemcpy(*d, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice));
  return GP_OK;
}

// Settings of later set-ups (gp_set_sweep_bricks; GPETSC_SWEEP_BRICKS and
// GPETSC_BRICK_LINES set the defaults).
struct BrickTuning {
  int mode = 1;      // 0 never, 1 where the model says it is faster, 2 wherever it applies
  int BJ = 0;        // lines of a brick (of one plane); 0: chosen
  int max_ctas = 0;  // cap on the persistent grid (0: none)
};
static BrickTuning& brick_tuning() {
  static BrickTuning t = [] {
    BrickTuning v;
    if (const char* e = std::getenv("GPETSC_SWEEP_BRICKS"))
      v.mode = std::max(0, std::min(2, std::atoi(e)));
    if (const char* e = std::getenv("GPETSC_BRICK_LINES"))
      v.BJ = std::max(0, std::min(kBrickMaxLines, std::atoi(e)));
    return v;
  }();
  return t;
}

void set_sweep_bricks(int mode, int lines, int max_ctas) {
  brick_tuning().mode = mode;
  brick_tuning().BJ = lines;
  brick_tuning().max_ctas = max_ctas;
}

// Grid detection: every row r (in sweep coordinates f = r forward, n-1-r
// backward; i = f % nx, j = f / nx % ny, k = f / (nx ny)) depends on exactly
// its grid neighbours r -/+ 1 (when i >= 1), nx (j >= 1) and nx ny (k >= 1),
// listed with ascending columns.  The sweep's last row has every coordinate at
// its end, so its dependencies give the grid's sizes.  On success slot[d][r]
// is the coefficient slot of row r's term in direction d (-1 where it has
// none).
static bool brick_detect(int n, bool forward, const std::vector<int>& dptr,
                         const std::vector<int>& dcol, const std::vector<int>& dsl, int* dims,
                         std::vector<int>& slot) {
  if (n < 2) return false;
  const int last = forward ? n - 1 : 0, nd = dptr[last + 1] - dptr[last];
  if (nd < 1 || nd > 3) return false;
  long long offs[3];
  for (int q = 0; q < nd; q++)
    offs[q] = std::llabs((long long)dcol[dptr[last] + q] - last);
  std::sort(offs, offs + nd);
  if (offs[0] != 1) return false;
  const long long nx = nd >= 2 ? offs[1] : n, nxny = nd >= 3 ? offs[2] : n;
  if (nx <= 1 || nxny % nx || n % nxny || nxny < nx) return false;
  const long long ny = nxny / nx;
  slot.resize((size_t)3 * n);
  std::atomic<bool> ok{true};
  host_parallel_for(n, [&](int64_t r0, int64_t r1) {
    for (int64_t r = r0; r < r1; r++) {
      const long long f = forward ? r : (long long)n - 1 - r;
      const long long c[3] = {f % nx, (f / nx) % ny, f / nxny}, o[3] = {1, nx, nxny};
      int q = dptr[r];
      // ascending columns: k, j, i forward, i, j, k backward
      for (int e = 0; e < 3; e++) {
        const int d = forward ? 2 - e : e;
        int sl = -1;
        if (c[d] >= 1) {
          if (q >= dptr[r + 1] || dcol[q] != (forward ? r - o[d] : r + o[d])) {
            ok = false;
            return;
          }
          sl = dsl[q++];
        }
        slot[(size_t)d * n + r] = sl;
      }
      if (q != dptr[r + 1]) {
        ok = false;
        return;
      }
    }
  });
  dims[0] = (int)nx;
  dims[1] = (int)ny;
  dims[2] = (int)(n / nxny);
  return ok;
}

// Modelled duration of one brick sweep (us): the chain of nx + ny + nz - 2
// rows at a step each plus a hand-off a brick face (less for one inside a
// cluster), or the bricks' steps over the SMs, whichever is longer.  The other
// forms take at least 1.25 us a dependency level in level order, or 0.4 us a
// level and the staging of a chunk (their own model, gp_sweep.cu).
constexpr double kBrickStep = 0.22, kBrickHandoff = 2.0, kBrickNear = 0.9, kBrickStart = 4.0;
static double other_model_us(int nlevels) { return std::min(1.25 * nlevels, 20.0 + 0.4 * nlevels); }
static double brick_model_us(const BrickShape& g) {
  const int ncP = (g.nbP + g.XP - 1) / g.XP, ncQ = (g.nbQ + g.XQ - 1) / g.XQ;
  const int far = ncP + ncQ - 2, near = g.nbP + g.nbQ - 2 - far;
  const double chain =
      (g.nw + g.np + g.nq - 2) * kBrickStep + far * kBrickHandoff + near * kBrickNear;
  const double rounds = std::ceil((double)g.nbP * g.nbQ / std::max(1, num_sms()));
  return kBrickStart + std::max(chain, rounds * (g.NS * kBrickStep + kBrickStart));
}

// Bricks of a cluster: 2 x 4 of those of whole 3-D tiles (whose lines across are
// multiples of kHalf, as the rings' shift between CTAs needs), eight being the
// portable limit.  ILU applies, us: 128^3 286 (2 x 2: 308, 4 x 2: 291, none: 365),
// 96^3 211 (221, 222, 235), 81^3 208 (210, 212, 223), 160^3, where the bricks take
// two rounds, 408 (410, -, 436).  In 2-D a cluster saves one or two faces of 2 us
// and its stores cost as much (256^2: 223 against 213).  The layout of the faces
// depends on it, so it is settled at set-up: by the shape, and by whether the
// device can hold such a cluster (brick_cluster_fits).
static void brick_cluster(BrickShape& g, bool clusters) {
  g.XP = g.XQ = 1;
  if (!clusters || !g.d3 || g.Wp != 8 || g.Wq != 4 || g.CP != 2 || g.CQ != 2) return;
  g.XP = std::min(2, g.nbP);
  g.XQ = std::min(4, g.nbQ);
}

static BrickShape brick_shape(const int* dims, bool bwd, int lines, bool clusters) {
  BrickShape g{};
  const int nx = dims[0], ny = dims[1], nz = dims[2];
  g.n = nx * ny * nz;
  g.bwd = bwd ? 1 : 0;
  g.d3 = nz > 1 ? 1 : 0;
  if (bwd) {  // along i, across j and k
    g.nw = nx, g.np = ny, g.nq = nz;
    g.sw = 1, g.sp = nx, g.sq = nx * ny;
  } else if (nz > 1) {  // along k, across i and j
    g.nw = nz, g.np = nx, g.nq = ny;
    g.sw = nx * ny, g.sp = 1, g.sq = nx;
  } else {  // along j, across i
    g.nw = ny, g.np = nx, g.nq = 1;
    g.sw = nx, g.sp = 1, g.sq = 0;
  }
  if (lines > 0) {
    // forced: `lines` neighbouring lines (more than a warp's in equal parts)
    const int bp = std::min({lines, nx, ny}), most = g.d3 ? 29 : 32;
    g.CP = std::min(kBrickWarps, (bp + most - 1) / most);
    g.CQ = 1;
    g.Wp = std::min(most, (bp + g.CP - 1) / g.CP);
    g.Wq = 1;
  } else {
    // 3-D: 8 x 4 lines a warp and 2 x 2 warps, the least surface of the
    // shapes that fill a warp; 2-D: 32 lines a warp and 4 warps in a row
    g.Wp = std::min(g.np, g.d3 ? 8 : 32);
    g.Wq = std::max(1, std::min(g.nq, 32 / g.Wp));
    if (g.d3) g.Wq = std::min(g.Wq, 30 - g.Wp);  // a ring step's columns
    const int tp = (g.np + g.Wp - 1) / g.Wp, tq = (g.nq + g.Wq - 1) / g.Wq;
    g.CQ = tp == 1 ? std::min(tq, kBrickWarps) : tq == 1 ? 1 : 2;
    g.CP = std::min(tp, kBrickWarps / g.CQ);
  }
  g.LW = (g.Wp * g.Wq + 1) & ~1;  // bulk copies of whole 16 bytes
  g.ntP = (g.np + g.Wp - 1) / g.Wp;
  g.ntQ = (g.nq + g.Wq - 1) / g.Wq;
  g.nbP = (g.ntP + g.CP - 1) / g.CP;
  g.nbQ = (g.ntQ + g.CQ - 1) / g.CQ;
  brick_cluster(g, clusters);
  int phase = 0;  // the largest of any tile of a brick
  for (int cp = 0; cp < g.CP; cp++)
    for (int cq = 0; cq < g.CQ; cq++)
      phase = std::max(phase, (cp * g.Wp + cq * g.Wq) % kHalf);
  g.NS = (g.nw + g.Wp + g.Wq - 2 + phase + kGroup - 1) / kGroup * kGroup;
  g.nwp = (g.nw + 3) & ~3;  // whole sectors
  return g;
}

static BrickShape shape_of(const EllSweep& e) {
  const int dims[3] = {e.gx, e.gy, e.gz};
  return brick_shape(dims, e.bwd, e.blines, e.clusters);
}

// Fetching lanes a face line (a.poll) and fetch warps: kBrickPoll lanes for every
// face line of a brick; none where one brick is the grid.
static void brick_fetchers(const BrickShape& g, int& poll, int& nf) {
  const int cols = g.CQ * g.Wq + (g.d3 ? g.CP * g.Wp : 0);
  poll = kBrickPoll;
  while (poll > 1 && cols * poll > 32 * kBrickFetchMax) poll /= 2;
  nf = g.nbP > g.XP || g.nbQ > g.XQ ? (cols * poll + 31) / 32 : 0;
}

static int brick_threads(const BrickShape& g) {
  int poll, nf;
  brick_fetchers(g, poll, nf);
  return 32 * (g.CP * g.CQ + nf + (g.XP * g.XQ > 1 ? 1 : 0));
}

// A sweep's kernel and its launch.
template <int MODE>
struct BrickLaunch {
  void (*kernel)(const int*, int, BrickArgs, DRef, DRef);
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];

  BrickLaunch(const BrickShape& g, int grid, cudaStream_t s, bool f) {
    // the other arithmetics, and tiles of other shapes, take the general addresses
    const bool full = g.LW == 32 && g.Wp + g.Wq <= (g.d3 ? 14 : 33);
    const bool cl = g.XP * g.XQ > 1;  // then the tiles are full ones (brick_cluster)
    kernel = cl       ? (f ? k_brick_sweep<MODE, true, true, true, true>
                           : k_brick_sweep<MODE, false, false, true, true>)
             : g.d3 ? (!f     ? k_brick_sweep<MODE, false, false, true, false>
                       : full ? k_brick_sweep<MODE, true, true, true, false>
                              : k_brick_sweep<MODE, true, false, true, false>)
                    : (!f     ? k_brick_sweep<MODE, false, false, false, false>
                       : full ? k_brick_sweep<MODE, true, true, false, false>
                              : k_brick_sweep<MODE, true, false, false, false>);
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(brick_threads(g));
    cfg.dynamicSmemBytes =
        (size_t)g.CP * g.CQ * 8 *
        (brick_ring(full && f, g.d3) + kStages * kGroup * brick_cols(MODE, g.d3) * g.LW);
    cfg.stream = s;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = g.XP * g.XQ;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = cl ? 1 : 0;
  }
};

template <int MODE>
static void brick_attrs() {
  for (auto k :
       {k_brick_sweep<MODE, true, true, true, true>, k_brick_sweep<MODE, false, false, true, true>,
        k_brick_sweep<MODE, true, true, true, false>, k_brick_sweep<MODE, true, false, true, false>,
        k_brick_sweep<MODE, false, false, true, false>,
        k_brick_sweep<MODE, true, true, false, false>,
        k_brick_sweep<MODE, true, false, false, false>,
        k_brick_sweep<MODE, false, false, false, false>})
    cudaFuncSetAttribute((const void*)k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         kBrickSmemMax);
}

// The modes as template arguments: M in X.
#define BRICK_MODES(X) \
  X(ELL_ILU_F) X(ELL_ILU_B) X(ELL_ILUT_F) X(ELL_ILUT_B) X(ELL_ICC_F) X(ELL_ICC_B) \
  X(ELL_SOR_F) X(ELL_SOR_B) X(ELL_SOR_B0)

// The kernels' shared-memory limit, once a device (at set-up: not capturable).
static void brick_set_attrs() {
  static std::atomic<unsigned long long> done{0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 64 && (done.load() >> dev & 1ull)) return;
#define BRICK_ATTRS(M) brick_attrs<M>();
  BRICK_MODES(BRICK_ATTRS)
#undef BRICK_ATTRS
  if (dev < 64) done |= 1ull << dev;
}

// Whether the device can hold a cluster of this sweep's bricks at all, in either
// arithmetic: eight SMs of one GPC with a CTA's shared memory each, which a
// partition or a restricted set of SMs may not have.  GPETSC_BRICK_CLUSTERS=0
// answers no.
template <int MODE>
static bool brick_cluster_fits(const BrickShape& g) {
  static const char* env = std::getenv("GPETSC_BRICK_CLUSTERS");
  if (env && std::string(env) == "0") return false;
  for (bool f : {true, false}) {
    BrickLaunch<MODE> l(g, g.XP * g.XQ, nullptr, f);
    int fit = 0;
    if (cudaOccupancyMaxActiveClusters(&fit, (const void*)l.kernel, &l.cfg) != cudaSuccess) {
      (void)cudaGetLastError();
      fit = 0;
    }
    if (fit < 1) return false;
  }
  return true;
}

static bool brick_clusters(int mode, const int* dims, int lines) {
  const BrickShape g = brick_shape(dims, brick_bwd(mode), lines, true);
  if (g.XP * g.XQ == 1) return false;
  brick_set_attrs();
#define BRICK_FITS(M) \
  case M: return brick_cluster_fits<M>(g);
  switch (mode) { BRICK_MODES(BRICK_FITS) }
#undef BRICK_FITS
  return false;
}

static int brick_layout(EllSweep& e, int mode, const int* dims, int lines, bool clusters,
                        const std::vector<int>& slot, const std::vector<int>& dslot) {
  ell_free(e);
  brick_set_attrs();
  const BrickShape g = brick_shape(dims, brick_bwd(mode), lines, clusters);
  e.clusters = clusters;
  e.brick = true;
  e.bwd = brick_bwd(mode);
  e.blines = lines;
  e.gx = dims[0];
  e.gy = dims[1];
  e.gz = dims[2];
  e.BJ = g.CP * g.Wp;
  e.BK = g.CQ * g.Wq;
  e.n = g.n;
  e.npos = g.ntP * g.ntQ * g.NS * g.LW;
  e.W = 3;
  e.bcols = brick_coefs(mode, g.d3);
  e.nbricks = g.nbP * g.nbQ;
  // hand-out order of the clusters: wavefronts P + Q, then Q
  const int ncP = (g.nbP + g.XP - 1) / g.XP, ncQ = (g.nbQ + g.XQ - 1) / g.XQ;
  std::vector<int> border;
  border.reserve(2 * (size_t)ncP * ncQ);
  for (int w = 0; w <= ncP + ncQ - 2; w++)
    for (int Q = std::max(0, w - (ncP - 1)); Q <= std::min(w, ncQ - 1); Q++) {
      border.push_back(w - Q);
      border.push_back(Q);
    }
  GP_TRY(bup(&e.border, border));
  GP_TRY(bup(&e.cslot, slot));
  if (brick_has_diag(mode) && !dslot.empty()) GP_TRY(bup(&e.dslot, dslot));
  GP_CUDA(cudaMalloc(&e.coef, (size_t)e.bcols * e.npos * sizeof(double)));
  e.qface = (long long)(g.nbP + 1) * g.ntQ * g.Wq * g.nwp;
  e.fsize = e.qface + (g.d3 ? (long long)(g.nbQ + 1) * g.ntP * g.Wp * g.nwp : 0);
  GP_CUDA(cudaMalloc(&e.faces, (size_t)(2 * e.fsize) * sizeof(double) + sizeof(int)));
  e.parity = reinterpret_cast<int*>(e.faces + 2 * e.fsize);
  GP_TRY(brick_reset(e, 0));
  GP_CUDA(cudaDeviceSynchronize());
  e.ok = true;
  return GP_OK;
}

// Both copies of the faces empty: at set-up, and after a wait ran out.
int brick_reset(EllSweep& e, cudaStream_t s) {
  if (!e.brick) return GP_OK;
  GP_CUDA(cudaMemsetAsync(e.parity, 0, sizeof(int), s));
  k_brick_clear<<<std::max(1, num_sms()), 256, 0, s>>>(2 * e.fsize, e.faces);
  GP_CHECK_LAUNCH();
  return GP_OK;
}

int brick_build(EllSweep& ef, EllSweep& eb, int mode_f, int mode_b, int n,
                const std::vector<int>& fptr, const std::vector<int>& fcol,
                const std::vector<int>& fsl, const std::vector<int>& bptr,
                const std::vector<int>& bcol, const std::vector<int>& bsl,
                const std::vector<int>& dslot, const std::vector<int>& perm, int nlevels,
                bool chosen_form, bool* built) {
  *built = false;
  const BrickTuning& tu = brick_tuning();
  if (tu.mode == 0 || (tu.mode == 1 && chosen_form) || n < 2) return GP_OK;
  for (int i = 0; i < (int)perm.size(); i++)
    if (perm[i] != i) return GP_OK;  // rows and grid in natural order only
  int df[3], db[3];
  std::vector<int> sf, sb;
  if (!brick_detect(n, true, fptr, fcol, fsl, df, sf) ||
      !brick_detect(n, false, bptr, bcol, bsl, db, sb))
    return GP_OK;
  if (df[0] != db[0] || df[1] != db[1] || df[2] != db[2]) return GP_OK;
  const int lines = std::max(0, tu.BJ);
  double est = 0.0;
  bool clusters[2];
  for (bool bwd : {false, true}) {
    clusters[bwd] = brick_clusters(bwd ? mode_b : mode_f, df, lines);
    const BrickShape g = brick_shape(df, bwd, lines, clusters[bwd]);
    // positions (steps x lanes, idle ones included) are int32, and few lanes
    // idle: a grid of very short lines keeps the other forms
    const long long pos = (long long)g.ntP * g.ntQ * g.NS * g.LW;
    const double us = brick_model_us(g);
    if (pos > INT_MAX / 4) return GP_OK;
    if (tu.mode == 1 &&
        (pos > 4LL * n + 4096 || us > other_model_us(std::max(nlevels, 1))))
      return GP_OK;
    est += us;
  }
  GP_TRY(brick_layout(ef, mode_f, df, lines, clusters[0], sf, dslot));
  GP_TRY(brick_layout(eb, mode_b, df, lines, clusters[1], sb, dslot));
  if (std::getenv("GPETSC_SWEEP_VERBOSE")) {
    const BrickShape gf = shape_of(ef), gb = shape_of(eb);
    std::fprintf(stderr,
                 "gpetsc sweep: n=%d grid %dx%dx%d bricks of %dx%d (forward) and %dx%d lines: "
                 "%d and %d, clusters of %dx%d and %dx%d, est=%.0fus\n",
                 n, df[0], df[1], df[2], ef.BJ, ef.BK, eb.BJ, eb.BK, ef.nbricks, eb.nbricks, gf.XP,
                 gf.XQ, gb.XP, gb.XQ, est);
  }
  *built = true;
  return GP_OK;
}

int brick_refresh(EllSweep& e, const double* src, const double* diag, cudaStream_t s) {
  if (!e.ok || !e.brick || e.n == 0) return GP_OK;
  const int grid = std::max(1, std::min((e.npos + 255) / 256, num_sms() * 8));
  k_brick_refresh<<<grid, 256, 0, s>>>(shape_of(e), e.bcols, e.npos, e.cslot, e.dslot, src, diag,
                                       e.coef);
  GP_CHECK_LAUNCH();
  return GP_OK;
}

int brick_sweep(int mode, const EllSweep& e, const int* gate, int want, DRef in, DRef out,
                const double* tin, const double* tin2, double* tout, double* tout2, double omega,
                int write_out, unsigned* tickets, DevErr* err, cudaStream_t s) {
  if (e.n == 0) return GP_OK;
  BrickArgs a;
  a.g = shape_of(e);
  const int xc = a.g.XP * a.g.XQ;
  a.nclusters = ((a.g.nbP + a.g.XP - 1) / a.g.XP) * ((a.g.nbQ + a.g.XQ - 1) / a.g.XQ);
  a.border = e.border;
  a.coef = e.coef;
  a.faces = e.faces;
  a.fsize = e.fsize;
  a.qface = e.qface;
  a.parity = e.parity;
  a.tin = tin;
  a.tin2 = tin2;
  a.tout = tout;
  a.tout2 = tout2;
  a.om1 = 1.0 - omega;
  a.write_out = write_out;
  a.tickets = tickets;
  a.err = err;
  brick_fetchers(a.g, a.poll, a.nf);
  int grid = std::min(a.nclusters * xc, num_sms() * 2);
  if (brick_tuning().max_ctas > 0) grid = std::min(grid, brick_tuning().max_ctas);
  grid = std::max(grid / xc, 1) * xc;
#define BRICK_LAUNCH(M)                                                                \
  case M: {                                                                            \
    const BrickLaunch<M> l(a.g, grid, s, arith_mode() == kFma);                        \
    GP_CUDA(cudaLaunchKernelEx(&l.cfg, l.kernel, gate, want, a, in, out));             \
    break;                                                                             \
  }
  switch (mode) { BRICK_MODES(BRICK_LAUNCH) }
#undef BRICK_LAUNCH
  GP_CHECK_LAUNCH();
  return GP_OK;
}

}  // namespace gp
