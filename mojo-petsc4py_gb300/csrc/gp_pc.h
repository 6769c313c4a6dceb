// Preconditioner objects: device data, host set-up analysis and applies.
#pragma once

#include <vector>

#include "gp_internal.h"

namespace gp {

enum PcType : int { PC_NONE = 0, PC_JACOBI = 2, PC_SOR = 4, PC_ILU = 5, PC_ICC = 6 };

// MatSORType bits (petscmat.h), as the reference uses them.
constexpr int kSorForward = 1 | 4;    // SOR_FORWARD_SWEEP | SOR_LOCAL_FORWARD_SWEEP
constexpr int kSorBackward = 2 | 8;   // SOR_BACKWARD_SWEEP | SOR_LOCAL_BACKWARD_SWEEP

struct PcOptions {
  int type = PC_NONE;
  int jacobi_type = 0;   // 0 diagonal, 1 rowmax, 2 rowl1, 3 rowsum
  int use_abs = 0;
  int fix_diag = 1;
  double rowl1_scale = 1.0;
  double omega = 1.0;
  double fshift = 0.0;
  int sor_flag = 12 | 16;  // LOCAL_SYMMETRIC | ZERO_INITIAL_GUESS
  int levels = 0;
  int ordering = 0;      // 0 natural, 1 rcm, 2 multicolour
};

// Processing plan of one sync-free sweep: rows in dependency-level order and
// a ticket pair for the dynamic row hand-out.
struct SweepPlan {
  int* order = nullptr;      // device, n
  int nlevels = 0;
};

// A sweep laid out in processing order for the ELL sweep kernels
// (gp_sweep.cu); `ok` is false when some row has more than kEllMaxW
// dependencies, and the CSR sweep kernels are used instead.
constexpr int kEllMaxW = 16;
enum EllMode : int {
  ELL_ILU_F, ELL_ILU_B, ELL_ICC_F, ELL_ICC_B, ELL_SOR_F, ELL_SOR_B,
  // brick form only: the two sweeps of the transposed ILU apply (U^T with the
  // diagonal, then L^T; the other forms run them as ILU_B and ILU_F) and SOR's
  // backward half without a forward one
  ELL_ILUT_F, ELL_ILUT_B, ELL_SOR_B0
};
struct EllSweep {
  int n = 0, W = 0;
  bool ok = false;
  int* cnt = nullptr;
  int* dep = nullptr;
  int* cslot = nullptr;
  int* in_idx = nullptr;
  int* out_idx = nullptr;
  int* dslot = nullptr;
  int* rowof = nullptr;
  double* coef = nullptr;
  double* dval = nullptr;
  // Tiled form (gp_sweep.cu, k_tile_sweep): positions grouped in chunks of
  // consecutive rows of the sweep's natural sequence, each chunk sorted by
  // the dependency level among its own rows and processed by one warp that
  // stages the chunk's metadata in shared memory with one bulk copy.  When
  // `tiled` is set the ELL columns above are not allocated: every index the
  // tiled kernel reads is in the blob.
  bool tiled = false;
  int nchunks = 0, C = 0, max_blob = 0, grid = 0;
  size_t smem = 0;
  unsigned char* blob = nullptr;  // per chunk: header, level offsets, columns
  long long* blob_off = nullptr;  // [nchunks + 1] byte offsets into blob
  int* cstart = nullptr;          // [nchunks + 1] first position of each chunk
  double est_us = 0.0;            // simulated duration of one tiled sweep
  int rows_per_chunk = 0;         // chunk size of the tiled layout
  // Brick form (gp_brick.cu, k_brick_sweep): the sweep's dependencies are the
  // unit steps of a grid gx x gy x gz; a CTA takes BJ x BK grid lines, a tile
  // of them a warp.  cslot is [direction][row], dslot by row, coef
  // [tile][step][bcols][lane] (npos steps x lanes, idle ones included).  The
  // two sweeps of a PC have it together.
  bool brick = false, bwd = false;
  bool clusters = false;      // bricks in thread-block clusters where the shape has them
  int gx = 0, gy = 0, gz = 0, BJ = 0, BK = 0, nbricks = 0, npos = 0, bcols = 0;
  int blines = 0;             // forced lines of a brick (0: chosen)
  int* border = nullptr;      // place (P, Q) of each cluster of bricks in hand-out order
  double* faces = nullptr;    // two copies of the bricks' face values, used in turn
  long long fsize = 0, qface = 0;
  int* parity = nullptr;      // which copy the next sweep uses (in faces' block)
};
void ell_free(EllSweep& e);
// Brick layout of a PC's two sweeps (mode_f, mode_b their EllModes) when the
// dependencies of both have the grid structure in natural order (`perm` the
// identity, or empty) and the model puts it below the other forms; *built says
// whether.  chosen_form: the caller asked for a level-ordered or chunked form,
// which only a forced brick form (mode 2) overrides.  dslot: each row's
// diagonal slot, for the modes that take it from the factor.
int brick_build(EllSweep& ef, EllSweep& eb, int mode_f, int mode_b, int n,
                const std::vector<int>& fptr, const std::vector<int>& fcol,
                const std::vector<int>& fsl, const std::vector<int>& bptr,
                const std::vector<int>& bcol, const std::vector<int>& bsl,
                const std::vector<int>& dslot, const std::vector<int>& perm, int nlevels,
                bool chosen_form, bool* built);
// Coefficients (and diagonal: from src, or diag by row) of a brick sweep from
// the current values.
int brick_refresh(EllSweep& e, const double* src, const double* diag, cudaStream_t s);
int brick_reset(EllSweep& e, cudaStream_t s);
// One brick sweep.  First sweeps read `in` and leave their values (tout) and
// SOR's checkpoint (tout2) by row, where second sweeps read them (tin, tin2).
int brick_sweep(int mode, const EllSweep& e, const int* gate, int want, DRef in, DRef out,
                const double* tin, const double* tin2, double* tout, double* tout2, double omega,
                int write_out, unsigned* tickets, DevErr* err, cudaStream_t s);
// Whether the level-ordered or a chunked form was asked for (gp_set_sweep_form).
bool sweep_form_chosen();
// Brick form of later set-ups: mode 0 never, 1 where modelled faster, 2
// wherever the structure allows; lines > 0 forces the lines of a brick;
// max_ctas > 0 caps the persistent grid.
void set_sweep_bricks(int mode, int lines, int max_ctas);
// Lay out one sweep.  forward: dependencies precede each row (ascending
// processing); otherwise they follow it.  `order` is the level order, used
// when the sweep is not tiled; nlevels its depth when known (0: counted here).
// mode: the EllMode of the kernel that will run the sweep.
int ell_build(EllSweep& e, int mode, int n, bool forward, const std::vector<int>& order,
              const std::vector<int>& dptr, const std::vector<int>& dcol,
              const std::vector<int>& dsl, const std::vector<int>& in_row,
              const std::vector<int>& out_row, const std::vector<int>& dslot_row,
              std::vector<int>* pos_of_row, int nlevels = 0);
int ell_refresh(EllSweep& e, const double* src, cudaStream_t s);
int sweep_wait_probe(int budget, int set, cudaStream_t s);
// Sweep form of later set-ups (gp_set_sweep_form).
void set_sweep_form(int tiles, int tile_rows);
// coefsrc: the array the sweep's coefficient slots index (the factor values
// for ILU/IC, the matrix values for SOR); the tiled form gathers from it.
int ell_sweep(int mode, const EllSweep& e, const int* gate, int want, DRef in, DRef out,
              double* val, const double* fval, double* aux, const double* auxin,
              const double* idiag, double omega, int use_t, int write_out, unsigned* tickets,
              DevErr* err, const double* coefsrc, cudaStream_t s);

// Host copy of a factor pattern in the reference's layout.
struct FactorPattern {
  // ILU: L rows bi[i]..bi[i+1], U rows (reversed) ending on the diagonal at
  // bdiag[i]; IC: row i = strict upper ascending then the diagonal slot
  // bdiag[i] = bi[i+1]-1.
  std::vector<int> bi, bj, bdiag;
  std::vector<int> r, ic;   // row ordering and its inverse
  int nnz = 0;              // number of factor slots
};

struct Pc {
  PcOptions opt;
  Csr* A = nullptr;  // operator the PC was set up from (not owned)
  int n = 0;
  int device = -1;
  bool ready = false;
  int epoch = 0;
  // a fresh next_uid() at every set-up (device arrays reallocated): cached
  // solve graphs compare it, never the PC's address
  unsigned long long generation = 0;

  // Jacobi
  double* diag = nullptr;
  double* diagsqrt = nullptr;

  // SOR (uses A's arrays and diagpos)
  double* idiag = nullptr;
  double* mdiag = nullptr;
  // SOR: the A->vver that the inverted diagonal and the sweeps' coefficients
  // were last computed for
  unsigned long long sor_vver = 0;

  // factor (ILU / IC), reference layout on the device
  FactorPattern pat;
  int* bi = nullptr;
  int* bj = nullptr;
  int* bdiag = nullptr;
  int* perm_r = nullptr;
  int* perm_c = nullptr;     // where row i of the factor's solution goes
  int* perm_ic = nullptr;
  double* ba = nullptr;      // factor values (what the solve reads)
  double* ba_orig = nullptr; // IC: unscaled strict rows
  int* done = nullptr;       // numeric row-done epochs
  // IC numeric: chain-ordered contributor lists (row k <- (i, slot))
  int* cptr = nullptr;
  int* crow = nullptr;
  int* cslot = nullptr;
  // IC forward sweep: transposed strict pattern, ascending source row
  int* tptr = nullptr;
  int* trow = nullptr;
  int* tslot = nullptr;
  int* amap = nullptr;       // A slot -> factor slot (or -1)
  // ILU numeric: per L slot, the (row slot, pivot U slot) updates it makes
  int* upd_ptr = nullptr;
  int* upd_dst = nullptr;
  int* upd_src = nullptr;

  SweepPlan fwd, bwd, num;
  EllSweep ef, eb;           // ELL forms of the forward and backward sweeps
  // ILU transposed apply (built on first use): sweeps over U^T (forward) and
  // L^T (backward) of the same factor
  EllSweep etf, etb;
  bool trans_ready = false;
  // sweep work: value-as-flag arrays and SOR checkpoint
  double* yf = nullptr;
  double* yb = nullptr;
  double* ys = nullptr;      // IC: scaled forward values
  double* t = nullptr;       // SOR checkpoint
  unsigned* tickets = nullptr;  // [4]: (ticket, exits) x 2
  DevErr* err = nullptr;
};

int pc_create(Pc** out);
int pc_destroy(Pc* pc);
int pc_setup(Pc* pc, Csr* A, cudaStream_t s);
// y = M^-1 x (x, y distinct device vectors).  Gate for captured loops.
int pc_apply(Pc* pc, DRef x, DRef y, cudaStream_t s, const int* gate = nullptr, int want = 0);
// y = M^-T x: the true transpose of the preconditioner (ILU: sweeps over U^T
// then L^T of the factor; none, Jacobi and IC are symmetric, so their apply;
// SOR: GP_ERR_UNSUPPORTED).  pc_transpose_prepare builds what it needs on the
// host (outside any stream capture).
int pc_transpose_prepare(Pc* pc, cudaStream_t s);
int pc_apply_transpose(Pc* pc, DRef x, DRef y, cudaStream_t s, const int* gate = nullptr,
                       int want = 0);
// IC(0)/IC(k) apply to R columns stored row-major (x, y: n * R; vf, vb, ys:
// n * R scratch), R dividing 32; no gate (not for captured solver loops of
// the single-vector drivers; the batched CG captures it).
int pc_apply_icc_cols(Pc* pc, int R, const double* x, double* y, double* vf, double* vb,
                      double* ys, cudaStream_t s);
// Jacobi symmetric half; other types fall back to pc_apply.
int pc_apply_symmetric(Pc* pc, DRef x, DRef y, cudaStream_t s, const int* gate = nullptr,
                       int want = 0);
// Read and clear the device error word (spin timeouts).  Synchronizes s.
int pc_check(Pc* pc, cudaStream_t s);

int pc_factor_numeric(Pc* pc, cudaStream_t s);
// Same operator pattern, new values: redo only the numeric phase (factor
// values, Jacobi diagonals) in the arrays of the last set-up.
int pc_update_values(Pc* pc, cudaStream_t s);
// Recompute SOR's value-derived arrays when the operator's values changed since
// (outside stream capture; a captured solve graph's owner calls it before every
// launch).
int pc_values_sync(Pc* pc, cudaStream_t s);
int pc_import_factor(Pc* pc, int type, const FactorPattern& pat, const std::vector<int>& perm_c,
                     const double* ba_host, Csr* A, cudaStream_t s);
int pc_import_jacobi(Pc* pc, int n, const double* diag, const double* diagsqrt, cudaStream_t s);
int jacobi_fill(const Csr* A, int jtype, int sym, int use_abs, int fix_diag, double scale,
                double* out, cudaStream_t s);
int sor_diagonals(Pc* pc, cudaStream_t s);

// host analysis (gp_pcsetup.cu)
int rcm_order(const std::vector<int>& rowptr, const std::vector<int>& colind, int n,
              std::vector<int>& perm);
int color_order(const std::vector<int>& rowptr, const std::vector<int>& colind, int n,
                std::vector<int>& perm, int* ncolors);
int ilu_symbolic_rows(const Csr* A, int levels, const std::vector<int>& r,
                      const std::vector<int>& ic,
                      std::vector<std::vector<std::pair<int, int>>>& rows, std::vector<int>& nL);
int icc_symbolic_rows(const Csr* A, int levels, const std::vector<int>& r,
                      const std::vector<int>& ic,
                      std::vector<std::vector<std::pair<int, int>>>& rows);
int ilu_symbolic(const Csr* A, int levels, const std::vector<int>& r,
                 const std::vector<int>& ic, FactorPattern& out);
int icc_symbolic(const Csr* A, int levels, const std::vector<int>& r,
                 const std::vector<int>& ic, FactorPattern& out);
// Levels of a DAG given as dependency lists; forward (deps < i) or backward.
void level_order(int n, const std::vector<int>& dptr, const std::vector<int>& dcol,
                 bool forward, std::vector<int>& order, int* nlevels);

}  // namespace gp
