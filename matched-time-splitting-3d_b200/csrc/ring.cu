// The bit-exact line sweeps of grids with many long lines: one line per
// thread over a ring of staged rows.
//
// A sweep runs as one persistent CTA per SM; each thread solves one grid line
// at a time, lines of a warp being consecutive in the fast index.  Per line:
//   * forward: the inputs of the line (and its per-node factors from its
//     first MIB row on) are staged into a shared-memory ring with cp.async,
//     chunks ahead of use; each row's right-hand side is built from the ring
//     (3-point stencil, source terms), the MIB row blocks' right-hand sides
//     come from the block pre-pass (Convert2Tri row operations replayed on
//     them), and the elimination recurrence runs over the chunk;
//   * the partial solutions d'_j go to per-thread scratch laid out
//     [row][thread] (coalesced in every direction, reused line after line);
//   * backward: the scratch is staged back through the same ring and the
//     solution is written once.
// The inside/outside side of a node, which selects the stencil weights and
// the source, changes along a line only at its recorded crossings, so it is
// tracked from the line's block list instead of being read per node.
//
// An SM has as many lines on the chain as the CTA has threads, whatever their
// length, where the line tiles (kernels.cu) have as many as its shared memory
// holds.  Which of the two a sweep takes, with both measured:
// sweep_shape_default (kernels.cu).
//
// Compiled with -fmad=false like kernels.cu: the same operations in the same
// order, so the two give the same bits.
#include <cuda_runtime.h>

#include <cmath>

#include "device.h"

#include "device_common.cuh"

namespace mts {
namespace {

// ---------------------------------------------------------------------------
// Douglas-ADI first right-hand side (douglas_adi.cc:89-359):
//   uhs = ((dt*D_yy u + dt*D_zz u) + u) + dt*src
// at the regular rows, Outer_u(t_next) on the faces: a pass of its own before
// the x ring sweep (an x tile forms it itself).
template <int G>
__global__ void __launch_bounds__(TPB, 8) k_adi_rhs(const __grid_constant__ Dev P, const double* __restrict__ un,
                                                 double* __restrict__ R, double E) {
  E = step_e(P, E, 2);
  const int lane = threadIdx.x & 31;
  const int nx = P.nx, nrows = P.ny * P.nz;
  const long long sy = nx, sz = (long long)nx * P.ny;
  const double dt = P.dt;
  // a node's side selects one of two specialised bodies (uniform over a warp
  // away from the interface), whose stencil weights are fixed kernel
  // parameters (constant-bank operands) instead of weights indexed per node
  for (int row = blockIdx.x * (TPB / 32) + (threadIdx.x >> 5); row < nrows; row += gridDim.x * (TPB / 32)) {
    const int iy = row % P.ny, iz = row / P.ny;
    const long long m0 = (long long)nx * row;
    const RowExact q = row_exact(P, iy, iz);
    double* const Rr = R + m0;
    if (iy == 0 || iz == 0 || iy == P.ny - 1 || iz == P.nz - 1) {
      for (int ix = lane; ix < nx; ix += 32) Rr[ix] = row_outer(P, q, ix, E);
      continue;
    }
    // the row's two face nodes, then its interior in groups of G x 32
    if (lane < 2) {
      const int ix = lane ? nx - 1 : 0;
      Rr[ix] = row_outer(P, q, ix, E);
    }
    const double* const uc_r = un + m0;
    const double* const uym_r = uc_r - sy;
    const double* const uyp_r = uc_r + sy;
    const double* const uzm_r = uc_r - sz;
    const double* const uzp_r = uc_r + sz;
    const uint8_t* const tg_r = P.tag + m0;
    for (int ix0 = 1; ix0 < nx - 1; ix0 += 32 * G) {
      double uc[G], uym[G], uyp[G], uzm[G], uzp[G];
      int tg[G];
#pragma unroll
      for (int g = 0; g < G; g++) {
        const int ix = ix0 + 32 * g + lane;
        if (ix < nx - 1) {
          tg[g] = tg_r[ix];
          uc[g] = uc_r[ix];
          uym[g] = uym_r[ix];
          uyp[g] = uyp_r[ix];
          uzm[g] = uzm_r[ix];
          uzp[g] = uzp_r[ix];
        }
      }
#pragma unroll
      for (int g = 0; g < G; g++) {
        const int ix = ix0 + 32 * g + lane;
        if (ix >= nx - 1) break;
        if (tg[g] & (TAG_MIBX | TAG_MIBY | TAG_MIBZ)) continue;  // a MIB row: k_adi_mib writes it
        auto node = [&](auto S) {
          constexpr int sd = decltype(S)::value;
          double sum = 0.0;
          sum += uym[g] * P.vd[1][sd][0];
          sum += uc[g] * P.vd[1][sd][1];
          sum += uyp[g] * P.vd[1][sd][2];
          const double ydt = dt * sum;
          sum = 0.0;
          sum += uzm[g] * P.vd[2][sd][0];
          sum += uc[g] * P.vd[2][sd][1];
          sum += uzp[g] * P.vd[2][sd][2];
          const double zdt = dt * sum;
          const double src = row_source(P, q, ix, E, sd);
          double r = ydt + zdt;
          r += uc[g];
          r += dt * src;
          return r;
        };
        Rr[ix] = (tg[g] & TAG_OUT) ? node(IntC<1>{}) : node(IntC<0>{});
      }
    }
  }
}

// ---------------------------------------------------------------------------
// The sweep.  Shape: CH rows per staged chunk, NS chunks in the ring (both
// powers of two), NT threads per CTA (one CTA per SM).
//
// Shared memory per thread column: three staged fields of NS*CH rows
// (forward: stencil field, added field, bet from the first MIB row on;
// backward: d'_j, gam_{j+1}).  Whole chunks are staged without per-row bound
// checks: every field the sweep reads (the solution fields, the per-node
// factors, the d' scratch) carries kRowPad rows of slack past its last row,
// so the rows of a line's last chunk beyond n are readable (and never used).
// The forward pass handles a chunk of regular rows (no MIB row, no line end)
// with a fully unrolled loop at compile-time shared-memory offsets whose
// stencil window slides in registers; chunks that hold a MIB block or a line
// end take the row-by-row path.  The backward pass does the same for chunks
// without the line end (and without the LOD epilogue).

struct BlockHead {
  int L, kind, sides;
  double a0, a1, a2;  // sub-diagonal of the block's rows after Convert2Tri
  double r0, r1, r2;  // their right-hand sides this sweep (block pre-pass)
};

__device__ __forceinline__ void load_head(const MibBlock* blk, const double* rblk, int k, int end,
                                          BlockHead& h) {
  if (k < end) {
    const MibBlock& b = blk[k];
    h.L = b.L;
    h.kind = b.kind;
    h.sides = b.sides;
    h.a0 = b.ia[0];
    h.a1 = b.ia[1];
    h.a2 = b.ia[2];
    h.r0 = rblk[3 * k];
    h.r1 = rblk[3 * k + 1];
    h.r2 = rblk[3 * k + 2];
  } else {
    h.L = 0x7fffffff;
    h.kind = 0;
    h.sides = 0;
  }
}

// Block pre-pass of a sweep: one thread per MIB block of direction D computes
// the right-hand sides of the block's rows and stores them for the sweep.
template <int D, int KIND>
__global__ void __launch_bounds__(TPB) k_block_rhs(const __grid_constant__ Dev P, const SweepIO io, double* rblk) {
  const int k = blockIdx.x * TPB + threadIdx.x;
  if (k >= P.nblk[D]) return;
  const int n2 = D == 2 ? P.ny : P.nz;
  const int line = P.blk[D][k].line;
  Line L;
  decode_line<D>(P, (long long)(line % n2) * (D == 0 ? P.ny : P.nx) + line / n2, L);
  double r[3];
  block_rhs<D, KIND>(P, io, step_e(P, io.e0, 0), step_e(P, io.e1, 2), k, L.base, L.i1, L.i2, r);
  for (int q = 0; q < 3; q++) rblk[3 * k + q] = r[q];
}

// Exact-solution parts along a line: the fixed axes are read once per line,
// the sweep axis from shared memory.  S = (sin2x cos2y) sin2z and
// R2 = (x*x + y*y) + z*z keep the operand order of the exact-solution code,
// so S*E and R2*E are the inner and outer solutions bit for bit.
struct LineExact {
  double x, y, z, s2x, c2y, s2z;
};

template <int D>
__device__ __forceinline__ void line_exact(const Dev& P, const Line& L, LineExact& f) {
  int ix, iy, iz;
  node_of<D>(L, 0, ix, iy, iz);
  f.x = P.ax[0][ix];
  f.y = P.ax[1][iy];
  f.z = P.ax[2][iz];
  f.s2x = P.s2[0][ix];
  f.c2y = P.c2[1][iy];
  f.s2z = P.s2[2][iz];
}

// sX: [coordinate | sin 2x | cos 2x] of the sweep axis, nd rows each.
template <int D>
__device__ __forceinline__ void row_parts(const LineExact& f, const double* sX, int nd, int j, double& S,
                                          double& R2) {
  if (D == 0) {
    const double x = sX[j];
    S = (sX[nd + j] * f.c2y) * f.s2z;
    R2 = (x * x + f.y * f.y) + f.z * f.z;
  } else if (D == 1) {
    const double y = sX[j];
    S = (f.s2x * sX[2 * nd + j]) * f.s2z;
    R2 = (f.x * f.x + y * y) + f.z * f.z;
  } else {
    const double z = sX[j];
    S = (f.s2x * f.c2y) * sX[nd + j];
    R2 = (f.x * f.x + f.y * f.y) + z * z;
  }
}
__device__ __forceinline__ double outer_from(const Dev& P, double R2, double E) {
  return P.eq == 0 ? 100.0 : R2 * E;
}
__device__ __forceinline__ double source_from(const Dev& P, double S, double R2, double E, int out) {
  if (P.eq == 0) return 0.0;
  if (out) return -(R2 * E) - P.c6bo * E;
  return P.kin * (S * E);
}

// Shared memory of a shape: the staging ring, the two prefix factor tables
// of the sweep direction (2 sides x 2 values x n rows) and its exact-solution
// tables (3 x n).
template <int CH, int NS, int NT, int D = 0>
constexpr size_t ring_smem(int n) {
  // D = 0 pads each ring row by 4 doubles (the x sweeps' cooperative staging);
  // the default D = 0 is the largest, used for the fit check
  return sizeof(double) * ((size_t)3 * NS * CH * (D == 0 ? NT + 4 : NT) + (size_t)7 * n);
}


template <int D, int KIND, int CH, int NS, int NT>
__global__ void __launch_bounds__(NT, 1) k_sweep(const __grid_constant__ Dev P, const __grid_constant__ RingData R,
                                                 const SweepIO io) {
  static_assert((CH & (CH - 1)) == 0 && (NS & (NS - 1)) == 0 && NS >= 4 && CH >= 4, "shape");
  static_assert(CH <= kRowPad, "chunk rows past a line end must stay within the fields' slack");
  constexpr int RING = NS * CH;    // rows in a field's ring
  // x lines (kCoop, below) are staged by the warp together, with 4 doubles of
  // padding per ring row so that a copy instruction's lanes, which write
  // CH rows of 32/CH columns, fall on distinct banks in pairs
  constexpr int RS = D == 0 ? NT + 4 : NT;  // doubles per ring row
  constexpr int SLOT = CH * RS;    // doubles per chunk slot
  extern __shared__ double sm[];
  const int tid = threadIdx.x;
  double* const sA = sm + tid;             // [NS][CH][NT]
  double* const sB = sA + NS * SLOT;       // [NS][CH][NT]
  double* const sC = sB + NS * SLOT;       // [NS][CH][NT]
#define SA(j) sA[((j) & (RING - 1)) * RS]
#define SB(j) sB[((j) & (RING - 1)) * RS]
#define SC(j) sC[((j) & (RING - 1)) * RS]
  const long long T = (long long)gridDim.x * NT;
  const long long gt = (long long)blockIdx.x * NT + tid;
  double* const dp = R.dp + gt;
  const long long nl = nlines<D>(P);
  const MibBlock* __restrict__ blk = P.blk[D];
  const double* __restrict__ fbet = R.fbet[D];
  const double* __restrict__ fgam = R.fgam[D];
  const double* __restrict__ rblk = R.rblk[D];
  const double E1 = step_e(P, io.e1, 2);
  const double E0 = step_e(P, io.e0, 0);
  const double kx = io.k;
  // per-direction constants by side (0 inside, 1 outside), in registers
  const double v0i = P.vd[D][0][0], v0o = P.vd[D][1][0];
  const double v1i = P.vd[D][0][1], v1o = P.vd[D][1][1];
  const double v2i = P.vd[D][0][2], v2o = P.vd[D][1][2];
  const double cai = P.ia[D][0], cao = P.ia[D][1];
  // prefix factor tables [side][row][bet, gam] and exact-solution tables of
  // the sweep axis [coordinate | sin 2x | cos 2x] into shared memory (they sit
  // on the recurrence chain; the staging stream would evict them from L1)
  const int nd = D == 0 ? P.nx : D == 1 ? P.ny : P.nz;
  double* const sP = sm + 3 * NS * SLOT;
  double* const sX = sP + 4 * nd;
  for (int i = tid; i < 2 * nd; i += NT) {
    const int side = i >= nd, j = side ? i - nd : i;
    sP[2 * i] = P.tab[D][side][j].x;
    sP[2 * i + 1] = j ? P.tabg[D][side][j - 1] : 0.0;
  }
  for (int i = tid; i < nd; i += NT) {
    sX[i] = P.ax[D][i];
    sX[nd + i] = P.s2[D][i];
    sX[2 * nd + i] = P.c2[D][i];
  }
  __syncthreads();

  // x lines are contiguous in memory and 2 KB apart, so a thread staging its
  // own line would touch 32 segments per warp instruction.  There the warp
  // stages and stores its 32 lines together (kCoop): lane e of copy q moves
  // row e % CH of line e / CH, so runs of CH lanes read one line's
  // consecutive rows, into that line's column of the ring.  The warp then
  // walks its lines' chunks in step, including lanes whose line is a face
  // line or past the end, which only help with the copies.
  constexpr bool kCoop = D == 0;
  const int lane = tid & 31;
  double* const sAw = sm + (tid - lane);  // the warp's first column of ring A
  const long long nxl = P.nx;

  for (long long t0 = gt - (kCoop ? lane : 0); t0 < nl; t0 += T) {
    const long long t = kCoop ? t0 + lane : t0;
    const bool act = t < nl;
    Line L;
    decode_line<D>(P, act ? t : nl - 1, L);
    const int n = L.n;
    const long long s = L.s;
    LineExact fx;
    line_exact<D>(P, L, fx);
    if (L.boundary && act) {
      if (io.bmode) {
        for (int j = 0; j < n; j++) {
          long long m = L.base + (long long)j * s;
          double S, R2;
          row_parts<D>(fx, sX, nd, j, S, R2);
          double v = outer_from(P, R2, E1);
          if (io.bmode == 2) v = v + P.dt * source_from(P, S, R2, E1, P.tag[m] & TAG_OUT);
          io.out[m] = v;
        }
      }
    }
    const bool solve = act && !L.boundary;
    if (!kCoop && !solve) continue;
    unsigned solvers = 0;
    if (kCoop) {
      __syncwarp();
      solvers = __ballot_sync(0xffffffffu, solve);
      if (!solvers) continue;
    }
    const int nch = (n + CH - 1) / CH;
    const int ls = P.lside[D][L.lid];
    const int bfirst = P.bstart[D][L.lid];
    const int bend = P.bstart[D][L.lid + 1];
    const int L1 = bfirst < bend ? blk[bfirst].L : n;  // first MIB row
    const double* pt = sP + ((ls >> 1) & 1) * 2 * nd;
    const bool two = KIND != K_COPY && io.add != io.stin;
    // row j of a field: g[j*s]; rows up to nch*CH-1 are readable (the fields
    // carry one chunk of slack past their end)
    const double* gA = (KIND == K_COPY ? io.add : io.stin) + L.base;
    const double* gB = io.add + L.base;
    const double* gC = fbet + L.base;
    // kCoop: the first MIB row of the line each of this lane's copies serves
    int L1q[CH];
    long long gq[CH];  // start of the line each copy serves, or -1 past the end
    if (kCoop) {
#pragma unroll
      for (int q = 0; q < CH; q++) {
        const int l = (q * 32 + lane) / CH;
        L1q[q] = __shfl_sync(0xffffffffu, L1, l);
        gq[q] = t0 + l < nl ? (t0 + l) * nxl + (q * 32 + lane) % CH : -1;
      }
    }
    auto stage = [&](int c) {
      if (kCoop) {
        if (c < nch) {
          const double* fA = KIND == K_COPY ? io.add : io.stin;
          double* aw = sAw + (c & (NS - 1)) * SLOT;
          double* bw = aw + NS * SLOT;
          double* cw = bw + NS * SLOT;
#pragma unroll
          for (int q = 0; q < CH; q++) {
            const int e = q * 32 + lane, l = e / CH, r = e % CH;
            if (gq[q] >= 0) {
              const long long g = gq[q] + (long long)c * CH;
              cp_async8(aw + r * RS + l, fA + g);
              if (two) cp_async8(bw + r * RS + l, io.add + g);
              if ((c + 1) * CH > L1q[q] && L1q[q] < n) cp_async8(cw + r * RS + l, fbet + g);
            }
          }
        }
        cp_async_commit();
        return;
      }
      if (c < nch) {
        const long long off = (long long)c * CH * s;
        double* a = sA + (c & (NS - 1)) * SLOT;
#pragma unroll
        for (int r = 0; r < CH; r++) cp_async8(a + r * RS, gA + off + r * s);
        if (two) {
          double* b = sB + (c & (NS - 1)) * SLOT;
#pragma unroll
          for (int r = 0; r < CH; r++) cp_async8(b + r * RS, gB + off + r * s);
        }
        if ((c + 1) * CH > L1 && L1 < n) {  // per-node factors exist only for lines with blocks
          double* cc = sC + (c & (NS - 1)) * SLOT;
#pragma unroll
          for (int r = 0; r < CH; r++) cp_async8(cc + r * RS, gC + off + r * s);
        }
      }
      cp_async_commit();
    };
    auto outer_at = [&](int j) -> double {
      double S, R2;
      row_parts<D>(fx, sX, nd, j, S, R2);
      return outer_from(P, R2, E1);
    };
    // right-hand side of a regular row from its stencil values
    auto rhs = [&](int j, double xm, double x0, double xp, double addv, double w0, double w1, double w2,
                   int side) -> double {
      if (KIND == K_COPY) return x0;
      double sum = 0.0;
      sum += xm * w0;
      sum += x0 * w1;
      sum += xp * w2;
      double r = kx * sum + addv;
      if (KIND == K_TS_Z) {
        double S, R2;
        row_parts<D>(fx, sX, nd, j, S, R2);
        r = r + P.hdt * source_from(P, S, R2, E0, side);
        r = r + P.hdt * source_from(P, S, R2, E1, side);
      }
      return r;
    };

    // ---- forward substitution with the precomputed factors (TDMA,
    // douglas_adi.cc:1794-1800): d'_j = (r_j - a_j d'_{j-1}) / bet_j
    for (int c = 0; c < NS - 2; c++) stage(c);
    int mb = bfirst;
    BlockHead hb, hb2;  // the next block and the one after (prefetched)
    load_head(blk, rblk, mb, bend, hb);
    load_head(blk, rblk, mb + 1, bend, hb2);
    int mside = (ls >> 1) & 1;
    double dprev = 0.0;
    int j = 1;
    for (int c = 0; c < nch; c++) {
      if (kCoop) __syncwarp();  // every lane is done with the slot restaged next
      stage(c + NS - 2);
      cp_async_wait<NS - 3>();  // chunks c-1, c, c+1 resident
      if (kCoop) {
        __syncwarp();  // and the other lanes' copies into this lane's column visible
        if (!solve) continue;
      }
      if (c == 0) {
        dprev = outer_at(0) / pt[0];
        dp[0] = dprev;
      }
      const int c0 = c * CH;
      const int cend = min(c0 + CH, n - 1);
      if (j >= cend) continue;
      if (j == c0 && cend == c0 + CH && hb.L >= cend && (cend <= L1 || c0 >= L1)) {
        // a chunk of regular rows, same side, factors from one source
        const double w0 = mside ? v0o : v0i, w1 = mside ? v1o : v1i, w2 = mside ? v2o : v2i;
        const double ac = mside ? cao : cai;
        const double* a = sA + (c & (NS - 1)) * SLOT;
        const double* ap = sA + ((c - 1) & (NS - 1)) * SLOT;
        const double* an = sA + ((c + 1) & (NS - 1)) * SLOT;
        const double* b = sB + (c & (NS - 1)) * SLOT;
        double* q = dp + (long long)c0 * T;
        auto run = [&](auto tag) {
          // tag: bet from the staged per-node factors, else from the prefix table
          constexpr bool kField = decltype(tag)::value;
          const double* bt = kField ? sC + (c & (NS - 1)) * SLOT : pt + 2 * c0;
          double xm = ap[(CH - 1) * RS];
          double x0 = a[0];
#pragma unroll
          for (int rr = 0; rr < CH; rr++) {
            const double xp = rr == CH - 1 ? an[0] : a[(rr + 1) * RS];
            const double r = rhs(c0 + rr, xm, x0, xp, two ? b[rr * RS] : x0, w0, w1, w2, mside);
            const double bet = kField ? bt[rr * RS] : bt[2 * rr];
            const double d = (r - ac * dprev) / bet;
            q[rr * T] = d;
            dprev = d;
            xm = x0;
            x0 = xp;
          }
        };
        if (c0 >= L1)
          run(BoolC<true>{});
        else
          run(BoolC<false>{});
        j = cend;
      } else {
        while (j < cend) {
          const double bet = j >= L1 ? SC(j) : pt[2 * j];
          if (j == hb.L) {
            // a MIB block: its rows' right-hand sides come mixed from the
            // block pre-pass (k_block_rhs); substitute them
            double d = (hb.r0 - hb.a0 * dprev) / bet;
            dp[(long long)j * T] = d;
            dprev = d;
            d = (hb.r1 - hb.a1 * dprev) / SC(j + 1);
            dp[(long long)(j + 1) * T] = d;
            dprev = d;
            if (hb.kind == 3) {
              d = (hb.r2 - hb.a2 * dprev) / SC(j + 2);
              dp[(long long)(j + 2) * T] = d;
              dprev = d;
            }
            mside = (hb.sides >> (hb.kind - 1)) & 1;
            j += hb.kind;
            mb++;
            hb = hb2;
            load_head(blk, rblk, mb + 1, bend, hb2);
          } else {
            const double r = rhs(j, SA(j - 1), SA(j), SA(j + 1), two ? SB(j) : SA(j), mside ? v0o : v0i,
                                 mside ? v1o : v1i, mside ? v2o : v2i, mside);
            const double d = (r - (mside ? cao : cai) * dprev) / bet;
            dp[(long long)j * T] = d;
            dprev = d;
            j++;
          }
        }
      }
    }
    if (solve) {
      // last row: the Dirichlet identity row (a = 0)
      const double r = outer_at(n - 1);
      const double a = 0.0;
      const double bet = n - 1 >= L1 ? SC(n - 1) : pt[2 * (n - 1)];
      dp[(long long)(n - 1) * T] = (r - a * dprev) / bet;
    }
    cp_async_wait<0>();

    // ---- back substitution u_j = d'_j - gam_{j+1} u_{j+1} (douglas_adi.cc:
    // 1805-1806), staged back through the ring: field A = d'_j, field B =
    // gam_{j+1} where it comes from the per-node factors.  The fence orders
    // this thread's d' stores before the asynchronous copies that read them.
    __threadfence_block();
    const double* gG = fgam + L.base;
    auto bstage = [&](int c) {
      if (c >= 0) {
        double* a = sA + (c & (NS - 1)) * SLOT;
        const double* g = dp + (long long)c * CH * T;
#pragma unroll
        for (int r = 0; r < CH; r++) cp_async8(a + r * RS, g + r * T);
        if ((c + 1) * CH >= L1 && L1 < n) {
          double* b = sB + (c & (NS - 1)) * SLOT;
          const long long off = ((long long)c * CH + 1) * s;
#pragma unroll
          for (int r = 0; r < CH; r++) cp_async8(b + r * RS, gG + off + r * s);
        }
      }
      cp_async_commit();
    };
    // side tracking downwards (only the LOD epilogue needs it): below a block
    // the side is that of the block's first row, above the last block that of
    // its last row.
    int db = bend - 1;
    int dbL = db >= bfirst ? blk[db].L : -1, dbK = db >= bfirst ? blk[db].kind : 0;
    int dbS = db >= bfirst ? blk[db].sides : 0;
    int dside = db >= bfirst ? (dbS >> (dbK - 1)) & 1 : (ls >> 1) & 1;
    double unext = 0.0;
    for (int c = nch - 1; c > nch - NS; c--) bstage(c);
    for (int c = nch - 1; c >= 0; c--) {
      if (kCoop) __syncwarp();  // the previous chunk's stores have read its slot
      bstage(c - NS + 1);
      cp_async_wait<NS - 1>();
      const int c0 = c * CH;
      // kCoop: results go to this lane's column of the slot, then the warp
      // stores its lines' rows together
      double* const aslot = sA + (c & (NS - 1)) * SLOT;
      if (!solve) {
      } else if (!io.last && c0 + CH <= n - 1 && (c0 + CH < L1 || c0 + 1 >= L1)) {
        // every row has a successor; gam_{j+1} from one source
        double* a = aslot;
        double* o = io.out + L.base + (long long)c0 * s;
        auto run = [&](auto tag) {
          // tag: gam_{j+1} from the staged per-node factors, else from the
          // prefix table (pt + 2*c0 + 3 is gam of row c0 + 1)
          constexpr bool kField = decltype(tag)::value;
          const double* gb = kField ? sB + (c & (NS - 1)) * SLOT : pt + 2 * c0 + 3;
#pragma unroll
          for (int rr = CH - 1; rr >= 0; rr--) {
            const double gm = kField ? gb[rr * RS] : gb[2 * rr];
            double u = a[rr * RS];
            u -= gm * unext;
            unext = u;
            if (kCoop)
              a[rr * RS] = u;
            else
              o[rr * s] = u;
          }
        };
        if (c0 + 1 >= L1)
          run(BoolC<true>{});
        else
          run(BoolC<false>{});
      } else {
        for (int rr = CH - 1; rr >= 0; rr--) {
          const int jj = c0 + rr;
          if (jj >= n) continue;
          double u = SA(jj);
          if (jj != n - 1) u -= (jj + 1 >= L1 ? SB(jj) : pt[2 * (jj + 1) + 1]) * unext;
          unext = u;
          double v = u;
          if (io.last) {
            int side;
            if (jj == 0) {
              side = ls & 1;
            } else if (jj == n - 1) {
              side = (ls >> 2) & 1;
            } else if (jj >= dbL && jj < dbL + dbK) {
              side = (dbS >> (jj - dbL)) & 1;
              if (jj == dbL) {
                dside = dbS & 1;
                db--;
                if (db >= bfirst) {
                  dbL = blk[db].L;
                  dbK = blk[db].kind;
                  dbS = blk[db].sides;
                } else {
                  dbL = -1;
                  dbK = 0;
                }
              }
            } else {
              side = dside;
            }
            double S, R2;
            row_parts<D>(fx, sX, nd, jj, S, R2);
            v = u + P.dt * source_from(P, S, R2, E1, side);
          }
          if (kCoop)
            SA(jj) = v;
          else
            io.out[L.base + (long long)jj * s] = v;
        }
      }
      if (kCoop) {
        __syncwarp();
        const double* aw = sAw + (c & (NS - 1)) * SLOT;
#pragma unroll
        for (int q = 0; q < CH; q++) {
          const int e = q * 32 + lane, l = e / CH, r = e % CH;
          if (((solvers >> l) & 1u) && c0 + r < n) io.out[gq[q] + c0] = aw[r * RS + l];
        }
      }
    }
    cp_async_wait<0>();
  }
#undef SA
#undef SB
#undef SC
}
// The crossing lines' factors by node, from the first MIB row on (bet_j and
// gam_j at row j's node): one thread per listed line and row.
template <int D>
__global__ void __launch_bounds__(TPB) k_ring_factors(const __grid_constant__ Dev P, double* fbet, double* fgam) {
  const int n = D == 0 ? P.nx : D == 1 ? P.ny : P.nz;
  const int nc = P.nfcross[D];
  const long long t = (long long)blockIdx.x * TPB + threadIdx.x;
  if (t >= (long long)nc * n) return;
  const int c = (int)(t % nc), j = (int)(t / nc);
  const int lid = P.fcross[D][c];
  if (j < P.blk[D][P.bstart[D][lid]].L) return;
  const int n2 = D == 2 ? P.ny : P.nz;
  Line L;
  decode_line<D>(P, (long long)(lid % n2) * (D == 0 ? P.ny : P.nx) + lid / n2, L);
  const long long m = L.base + (long long)j * L.s;
  fbet[m] = P.cb[D][t].x;
  fgam[m] = P.cg[D][t - nc];
}

// Sweep shapes (rows per chunk, ring chunks, threads per CTA): ids from 0 here.
#define MTS_RINGS(X) X(0, 4, 4, 384) X(1, 4, 4, 448) X(2, 4, 4, 128)

template <int D, int KIND>
void sweep(const Dev& P, const RingData& R, const SweepIO& io, int ring, cudaStream_t st) {
  const int nd = D == 0 ? P.nx : D == 1 ? P.ny : P.nz;
  if (P.nblk[D] > 0) k_block_rhs<D, KIND><<<(P.nblk[D] + TPB - 1) / TPB, TPB, 0, st>>>(P, io, R.rblk[D]);
  switch (ring) {
#define MTS_CASE(id, ch, ns, nt)                                                                               \
  case id:                                                                                                     \
    k_sweep<D, KIND, ch, ns, nt><<<sweep_grid(P, nlines<D>(P), nt), nt, ring_smem<ch, ns, nt, D>(nd), st>>>(P, R, io); \
    break;
    MTS_RINGS(MTS_CASE)
#undef MTS_CASE
  }
}

template <int CH, int NS, int NT>
cudaError_t allow_rings() {
  return allow_smem(kMaxSweepSmem,
                    {(const void*)k_sweep<0, K_COPY, CH, NS, NT>, (const void*)k_sweep<1, K_COPY, CH, NS, NT>,
                     (const void*)k_sweep<2, K_COPY, CH, NS, NT>, (const void*)k_sweep<0, K_STENCIL, CH, NS, NT>,
                     (const void*)k_sweep<1, K_STENCIL, CH, NS, NT>, (const void*)k_sweep<2, K_STENCIL, CH, NS, NT>,
                     (const void*)k_sweep<2, K_TS_Z, CH, NS, NT>});
}

}  // namespace

bool ring_fits(int ring, int n) {
  switch (ring) {
#define MTS_FITS(id, ch, ns, nt) \
  case id:                       \
    return ring_smem<ch, ns, nt>(n) <= (size_t)kMaxSweepSmem;
    MTS_RINGS(MTS_FITS)
#undef MTS_FITS
    default:
      return false;
  }
}

// 384 threads a CTA; 448 where that saves a round of lines (353^3 y, ADI: 402
// against 453 us; from 400 rows on their larger d' scratch costs more, 513^3 y
// 1593 against 1158, but for the z sweep of LOD, which waits row by row,
// 65 x 900 x 900: 984 against 1561); 128 where the lines would not fill the
// SMs otherwise (1000 x 257 x 129 x, ADI: 661 against 790
// with 87 CTAs of 384).
int ring_default(int method, int d, int n, double per_sm) {
  const bool lod_z = d == 2 && (method == MTS_LOD_IE || method == MTS_LOD_CN);
  int k = 0;
  if (per_sm < (d == 0 ? 240 : 120))
    k = 2;
  else if ((n <= 400 || lod_z) && std::ceil(per_sm / 448) < std::ceil(per_sm / 384))
    k = 1;
  for (int c : {k, 0, 2})
    if (ring_fits(c, n)) return c;
  return -1;
}

long long ring_threads(const Dev& P, int ring, int d) {
  const int nt = ring == 0 ? 384 : ring == 1 ? 448 : 128;
  return (long long)nt * sweep_grid(P, d == 0 ? nlines<0>(P) : d == 1 ? nlines<1>(P) : nlines<2>(P), nt);
}

cudaError_t configure_ring(int ring) {
  switch (ring) {
#define MTS_ALLOW(id, ch, ns, nt) \
  case id:                        \
    return allow_rings<ch, ns, nt>();
    MTS_RINGS(MTS_ALLOW)
#undef MTS_ALLOW
    default:
      return cudaErrorInvalidValue;
  }
}

void build_ring_factors(const Dev& P, int d, double* fbet, double* fgam, cudaStream_t st) {
  const int n = d == 0 ? P.nx : d == 1 ? P.ny : P.nz;
  const unsigned nb = (unsigned)(((long long)P.nfcross[d] * n + TPB - 1) / TPB);
  if (nb == 0) return;
  if (d == 0)
    k_ring_factors<0><<<nb, TPB, 0, st>>>(P, fbet, fgam);
  else if (d == 1)
    k_ring_factors<1><<<nb, TPB, 0, st>>>(P, fbet, fgam);
  else
    k_ring_factors<2><<<nb, TPB, 0, st>>>(P, fbet, fgam);
}

void launch_adi_rhs(const Dev& P, const double* u, double* r, double e_next, cudaStream_t st) {
  k_adi_rhs<2><<<pointwise_rows_grid(P), TPB, 0, st>>>(P, u, r, e_next);
}

void launch_ring_sweep(const Dev& P, const RingData& R, int d, int kind, const SweepIO& io, int ring, cudaStream_t st) {
  if (d == 0) {
    if (kind == K_COPY)
      sweep<0, K_COPY>(P, R, io, ring, st);
    else
      sweep<0, K_STENCIL>(P, R, io, ring, st);
  } else if (d == 1) {
    if (kind == K_COPY)
      sweep<1, K_COPY>(P, R, io, ring, st);
    else
      sweep<1, K_STENCIL>(P, R, io, ring, st);
  } else {
    if (kind == K_COPY)
      sweep<2, K_COPY>(P, R, io, ring, st);
    else if (kind == K_TS_Z)
      sweep<2, K_TS_Z>(P, R, io, ring, st);
    else
      sweep<2, K_STENCIL>(P, R, io, ring, st);
  }
}

}  // namespace mts
