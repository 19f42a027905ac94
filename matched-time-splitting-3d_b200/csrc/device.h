// Device-resident problem layout shared by the C ABI (capi.cu) and the
// kernels (kernels.cu).
//
// HBM layout of one problem (N = nx*ny*nz nodes, x fastest):
//   u0, u1   float64[N]   solution ping-pong (state + stage results)
//   tag      uint8[N]     bit0 outside, bit1/2/3 node is a MIB row of an
//                         x/y/z crossing block
//   ca, cb, cg  the Thomas factors of the lines that cross the interface,
//                         32 B a row, by row and line
//   u0, u1 and the FP32 fields carry kRowPad rows of slack (x-y planes)
//                         past their end: the fast form's bulk copies and
//                         the FP32 ring sweeps may read past the last row
//   lside    uint8 per line and direction: bit0 node 0, bit1 node 1, bit2
//                         node n-1 outside (the side changes only at crossings)
//   per axis: coordinates, sin 2x, cos 2x (exact-solution tables)
//   per direction: CSR offsets over grid lines -> MIB row blocks
//   per crossing: time-invariant constants of its jump data
#pragma once

#include <cstdint>

#include "../../include/mts.h"

namespace mts {

enum : uint8_t { TAG_OUT = 1, TAG_MIBX = 2, TAG_MIBY = 4, TAG_MIBZ = 8 };

// One irregular crossing (2 rows: L, L+1) or one corner pair (3 rows: L..L+2)
// on a grid line.  w[0]/w[1] are weil/weir of the (left) crossing, w[2]/w[3]
// those of the right crossing of a corner pair (Intersection_Data::wei,
// src/constant.h:119-122).  ia/ib/ic are the implicit rows after the
// Convert2Tri_irr/_cor elimination (src/temporal/douglas_adi.cc:1554-1675),
// rate[] the elimination multipliers to replay on the right-hand side.
struct MibBlock {
  int32_t line;
  int32_t L;
  int32_t kind;  // 2 or 3 rows
  int32_t c0, c1;
  int32_t sides;  // bit q: row L+q is outside
  double w[4][9];
  double ia[3], ib[3], ic[3];
  double rate[6];
};

// Time-invariant constants of one crossing's jump data for the exact
// solutions supported on the device.  For eq 8 the per-step values are
//   [u]       = R2*E - S*E
//   [beta u_d]= beta_out*((2 x_d)*E) - beta_in*(D_d*E)
//   u_dir     = pinv * (p0*[bu_x] + p1*[bu_y] + p2*[bu_z])
// with E = exp(-t), the operand order of the exact-solution code.
struct CrossConst {
  double x, y, z;
  double R2, S;
  double D[3];
  double p[3];
  double pinv;
};

struct Dev {
  int nx, ny, nz;
  int eq, method;
  int ncross;
  long long nn;
  double dt;
  double kex;   // explicit Crank-Nicolson factor coef*dt, coef = 0.5
  double cdt;   // implicit factor: dt (ADI, LOD-IE) or 0.5*dt (LOD-CN, TS)
  double hdt;   // 0.5*dt (TS source halves)
  double bi, bo, kin, c6bo;  // beta_in, beta_out, 12*beta_in-1, 6*beta_out
  double vd[3][2][3];        // [dir][side] 3-point weights beta/h^2, -(2beta)/h^2, beta/h^2
  double ia[3][2], ib[3][2], ic[3][2];  // regular implicit rows
  const double* ax[3];  // node coordinates per axis
  const double* s2[3];  // sin(2 x_i) per axis
  const double* c2[3];  // cos(2 x_i) per axis
  const uint8_t* tag;
  const uint8_t* lside[3];
  const int32_t* bstart[3];
  const MibBlock* blk[3];
  const CrossConst* cc;
  // Thomas factorisation of every line, computed once (the matrices do not
  // change between steps): bet_j = b_j - a_j*gam_j, gam_j = c_{j-1}/bet_{j-1}.
  // A line that does not cross the interface has the rows of its side (the
  // side of its row 1): taba[d][side][j] = a_j, tab[d][side][j] = (bet_j,
  // 1/bet_j), tabg[d][side][j] = gam_{j+1} (0 past the end).  The lines that
  // cross it (nfcross of them, their ids in fcross in memory order, the index
  // of a line in that list in cline[i1 + n1 i2], -1: none) have their own, by
  // row, the lines of a row side by side: ca, cb, cg[d][j nfcross + c].
  const double* taba[3][2];
  const double2* tab[3][2];
  const double* tabg[3][2];
  const int32_t* fcross[3];
  int nfcross[3];
  const int32_t* cline[3];
  // The interior lines (i1 + n1 i2) in the order of the bit-exact sweeps:
  // those that cross the interface, then the others inside, then outside.
  const int32_t* lperm[3];
  const double* ca[3];
  const double2* cb[3];
  const double* cg[3];
  int plain_div;     // a factor is out of the range of the quotients from reciprocals (kernels.cu)
  int nblk[3];
  int sweep_blocks;  // SMs
  int shape[3];      // sweep shape of the first, second and third sweep of a step
  // Mixed precision (Douglas-ADI): the step is solved for its increment
  // delta = u^{n+1} - u^n in FP32 (residual in FP64, state accumulated in
  // FP64).  Factors of the ring sweeps in FP32 (built for grids with a line
  // too long for the segmented solves): by row per side, and per node from
  // its first MIB row on for a line that crosses the interface.
  float* r32;                 // residual in, increment out [N + slack]
  float* dp32;                // [nmax + slack][sweep threads]
  const float* ptab32[3][2];  // [2*j + {0: 1/bet, 1: gam}]
  const float* fib32[3];      // per node 1/bet of crossing lines from L1
  const float* fgam32[3];
  float* rblk32[3];           // block rows' right-hand sides after Convert2Tri
  // Dense per-node coefficients of the segmented FP32 solves, built on the
  // device when the mixed form is switched on (null before, and for grids
  // whose lines are too long for them): for row j of a direction-d line,
  //   cib = 1/bet_j,  cp = -a_j/bet_j (forward multiplier, 0 on face rows),
  //   cq = -gam_{j+1} (backward multiplier, 0 on the last row).
  // They are filled only for lines that cross the interface; every other
  // interior line takes its row's values from ctab[d][side][{ib, p, q}][row]
  // by the side of its row 1.
  float* cib[3];
  float* cp[3];
  float* cq[3];
  float* ctab[3];
  int precision;              // 0 plain FP64, 1 mixed, 2 fast FP64
  // Fast FP64 form (segmented line solves, fast.cu), built when the form is
  // switched on.  Per direction: the row tables [side][1/bet, -a/bet by row
  // (32 MX each), then 2 x 5 x 32 lane-scan multipliers] of the lines
  // without crossings; per line a flag byte (bit0 the line
  // crosses the interface, bit1 the side of its row 1); the crossing lines'
  // (fcross) own rows [c][1/bet, -a/bet][32 MX]; per block the -gam_{j+1} of its rows.
  const double* ftab[3];
  const uint8_t* fline[3];
  const double* fcoef[3];
  const double* fbq[3];
  // Replayable steps (batches captured in a CUDA graph): when tsched is set,
  // kernels take the step's exp(-t) factors from tsched[3*(*tstep) + {0: t_prev,
  // 1: t_half, 2: t_next}] instead of their arguments; k_tick advances tstep.
  const double* tsched;
  int* tstep;
  int tstop;   // batched launches skip the problem once *tstep reaches it
  double* u0;  // the state (every method keeps it here)
  double* u1;  // scratch field
  const long long* mibnode;  // nodes with a MIB flag (any direction), ascending
  int nmibnode;
  const int4* mibref;        // Douglas-ADI and TS: per listed node its block in x, y, z (16 block + 4 kind + row, -1: none)
  int* status;       // reserved
};

// The ring sweeps' data (ring.cu), built before a handle's first step that takes
// one, for the directions that do (null before): by node bet_j and gam_j of the
// crossing lines from their first MIB row on; the block rows' right-hand sides
// of the sweep in flight, [3*block + q]; the partial solutions d'_j,
// [row][thread].  (Apart from Dev, which every launch carries: its 80 bytes
// cost a 33^3 step's four launches 1.9 us of host time, 9.6 against 7.7.)
struct RingData {
  const double* fbet[3];
  const double* fgam[3];
  double* rblk[3];
  double* dp;
};

// What a bit-exact line sweep does: its right-hand side (of the copied field,
// of the line's explicit stencil, of TS's z step, or the whole first
// right-hand side of Douglas-ADI) and its fields.
enum Kind { K_COPY = 0, K_STENCIL = 1, K_TS_Z = 2, K_ADI = 3 };

struct SweepIO {
  const double* stin;  // field the explicit stencil reads
  const double* add;   // field added to the explicit part (or copied)
  double* out;         // result field (may alias stin/add: a line is read
                       // completely before any of it is written)
  double e1;           // exp(-t_next): boundary data, source, jumps
  double e0;           // exp(-t_prev): TS source of the first half step
  double k;            // explicit factor: -dt (ADI), 0.5*dt (LOD-CN, TS)
  int jumps;           // MIB rows carry jump terms (LOD, TS)
  int bmode;           // boundary lines: 0 keep, 1 Outer_u(t_next), 2 + dt*f
  int last;            // LOD: epilogue adds dt*f(t_next)
};

// Line-sweep shapes: tiles (lines per tile, threads per CTA; kernels.cu), then
// rings (rows per chunk, chunks, threads per CTA; ring.cu).  All give
// bit-identical results, they differ only in speed.
constexpr int kTileShapes = 10, kRingShapes = 3;
int sweep_shape_count();
int sweep_direction(int method, int sweep);       // direction of a step's first, second, third sweep
bool sweep_shape_fits(int shape, int d, int n);   // shared memory of the shape for direction-d lines of n nodes
int sweep_shape_default(int method, int d, int n, long long lines, int sms);  // -1: no shape takes them
int tile_shape_default(int d, int n, bool adi_x);  // among the tiles; adi_x: the x sweep of Douglas-ADI
// Lets the kernels of a shape have its shared memory on the current device
// (CUDA keeps the limit per device); the others below likewise.
cudaError_t configure_shape(int shape);
// The ring sweeps (ring.cu; ring: shape - kTileShapes).
bool ring_fits(int ring, int n);
int ring_default(int method, int d, int n, double per_sm);  // lines per SM; -1: none fits
long long ring_threads(const Dev& P, int ring, int d);  // threads of the launch: columns of dp
cudaError_t configure_ring(int ring);
void build_ring_factors(const Dev& P, int d, double* fbet, double* fgam, cudaStream_t stream);
void launch_adi_rhs(const Dev& P, const double* u, double* r, double e_next, cudaStream_t stream);
void launch_ring_sweep(const Dev& P, const RingData& R, int d, int kind, const SweepIO& io, int ring, cudaStream_t stream);

// Per-step exact-solution time factors.
struct StepTimes {
  double e_prev, e_half, e_next;  // exp(-t_prev), exp(-t_half), exp(-t_next)
};

// Host-side launchers (kernels.cu).  All enqueue on `stream` and return the
// number of kernel launches made.
int launch_initialize(const Dev& P, double E, double* u, cudaStream_t stream);
// Thomas factors of the lines with MIB blocks and the MIB nodes' block
// references (once, at setup); *flags: bit 0 a zero pivot, bit 1 a factor out
// of the range of the quotients from reciprocals.
int launch_factor_lines(const Dev& P, int* flags, cudaStream_t stream);
// ev: null, or 2 events per kernel slot recorded around each launch.
// A second stream with its fork and join events (timing off), for work of a
// step that can run beside the main stream's.
struct SideStream {
  cudaStream_t stream;
  cudaEvent_t fork, join;
};
int launch_step(const Dev& P, const RingData& R, const StepTimes& T, double* u0, double* u1, cudaStream_t stream,
                cudaEvent_t* ev, const SideStream* side);
// The mixed-precision Douglas-ADI step (mixed.cu), in place on u.
int launch_step_mixed(const Dev& P, const StepTimes& T, double* u, cudaStream_t stream, cudaEvent_t* ev,
                      const SideStream* side);
cudaError_t configure_mixed_kernels();
int mixed_sweep_threads();            // threads per CTA of the FP32 sweeps
bool mixed_shape_fits(int nmax);      // their shared memory within the limit
bool mixed_segments_fit(int n);       // the segmented solves take lines of n rows (else the ring sweeps run)
// Fills Dev::cib/cp/cq (allocated by the caller) from the FP64 factors.
int build_mixed_coefs(const Dev& P, cudaStream_t stream);
// The fast FP64 Douglas-ADI step (fast.cu): u holds u^n on entry and
// u^{n+1} on return, d is scratch.  ev: null, or 6 events recorded around
// the three launches.
int launch_step_fast(const Dev& P, const StepTimes& T, double* u, double* d, cudaStream_t stream, cudaEvent_t* ev,
                     const SideStream* side);
cudaError_t configure_fast_kernels();
int fast_rows_per_lane(int n);               // MX of a direction with n rows (0: lines too long)
bool fast_fits(int nx, int ny, int nz);      // the form takes this grid
int build_fast_lines(const Dev& P, uint8_t* const fline[3], cudaStream_t stream);  // the line flags
int build_fast_tables(const Dev& P, cudaStream_t stream);  // fills ftab, fcoef, fbq (allocated by the caller)
// Batched plain steps (kernels.cu): problems of one method advance together,
// one launch per kernel of the step for all of them.  A launch's CTAs are
// listed as items (problem, the CTA's index in that problem's own grid, the
// size of that grid), so every problem sees exactly the grid its own launch
// would have; the problems' Dev records live in device memory.
struct BatchItem {
  int32_t p, cta, ncta, pad;
};
struct BatchPlan {
  int method;         // MTS_ADI .. MTS_TS, shared by all problems
  int n;              // problems
  int tile[3];        // batch_tile of each direction
  int nmax[3];        // longest line of each direction over the problems
  const Dev* Ps;      // [n] device records (tsched/tstep set)
  const BatchItem* rows;  // TS explicit half steps
  int nrows;
  const BatchItem* mib;   // MIB rows of the Douglas-ADI first right-hand side
  int nmib;
  const BatchItem* sw[3];   // line sweeps per direction
  int nsw[3];
};
// The mixed form's batched step (ADI, lines of at most 160 rows): the
// mixed kernels' bodies, one item per CTA (mixed.cu).  line[d][c]: the line
// solves of direction d for the problems of rows-per-lane class c (3, 5).
struct MixedBatchPlan {
  int n;
  const Dev* Ps;
  const BatchItem* rows;
  int nrows;
  const BatchItem* mib;
  int nmib;
  const BatchItem* blk[3];
  int nblk[3];
  const BatchItem* line[3][2];
  int nline[3][2];
};
int mixed_batch_class(const Dev& P, int d);          // -1: not batchable
unsigned mixed_line_ctas(const Dev& P, int d);      // CTAs of the line solves of direction d
int launch_step_batch_mixed(const MixedBatchPlan& plan, cudaStream_t stream);  // one step + tick
cudaError_t configure_mixed_batch_kernels();
int launch_batch_tick(const Dev* Ps, int n, cudaStream_t stream);
constexpr int kBatchClasses = 2, kBatchTiles = 2;
int batch_tile(int d, int n);              // tiles of the batched sweeps for direction-d lines of up to n nodes; -1: none
int batch_class(const Dev& P);             // a class is launched together; -1: the problem steps by itself
unsigned ts_explicit_grid(const Dev& P);
cudaError_t configure_batch(int tile);
int launch_step_batch(const BatchPlan& plan, cudaStream_t stream);  // one step + tick
unsigned mib_grid(const Dev& P);
unsigned block_grid(const Dev& P, int d);
unsigned batch_sweep_grid(const Dev& P, int tile, int d);

// Shared by both step forms (kernels.cu).
void launch_tick(const Dev& P, cudaStream_t stream);  // ++(*P.tstep)
unsigned pointwise_rows_grid(const Dev& P);
constexpr int kProfileSlots = 8;
constexpr int kRowPad = 16;  // rows of slack after each staged field (>= chunk rows)
// The fictitious points' relative errors (Refresh_Fp): two per crossing
// into err, for the records cr sorted by (direction, line, position) whose
// indices in the handle's list are ci; role[i] 0 single, 1 left of a corner
// pair, 2 its right (diag.cu).
int launch_fp_errors(const Dev& P, const mts_crossing* cr, const int32_t* ci, const int8_t* role, int n, double E,
                     double* err, cudaStream_t stream);
// The jumps' relative errors (Refresh_Jump's jump.err): one per record of
// the same sorted list into err (diag.cu).
int launch_jump_errors(const Dev& P, const mts_crossing* cr, const int32_t* ci, int n, double E, double* err,
                       cudaStream_t stream);

int launch_norms(const Dev& P, double E, const double* u, double* partial, int nblocks,
                 double* out3, cudaStream_t stream);
int norms_blocks(const Dev& P);

// Error norms through a statically sized module array instead of handle
// buffers (mts_norms_noalloc).  The array holds the ticket counter, the
// result triple and the partials of at most kNoAllocMaxBlocks blocks, i.e.
// grids of at most kNoAllocMaxBlocks * 2048 nodes (norms_blocks).
constexpr int kNoAllocMaxBlocks = 2048;
constexpr int kNoAllocScratchDoubles = 64 + 3 * kNoAllocMaxBlocks;  // 48.5 KiB
cudaError_t noalloc_scratch_address(double** p);  // call with the device current
int launch_norms_noalloc(const Dev& P, double E, const double* u, double* scratch, int nb, cudaStream_t stream);

}  // namespace mts
