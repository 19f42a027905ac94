// Time-stepping kernels for sm_100a.
//
// Implicit line sweeps (the Thomas solves, douglas_adi.cc:1784-1807 and the
// LOD/TS copies): a CTA holds a tile of lines in shared memory, builds their
// right-hand sides (stencils, sources, MIB rows with their jumps) with all
// threads, solves them with one warp, a lane per line, and writes them back
// (k_line).  The Thomas factors (bet, gam) are computed once at setup.
//
// The TS explicit half steps are plain grid-stride kernels.
//
// The file is compiled with -fmad=false: every product and sum is rounded on
// its own, in the operand order of the reference statement it restates, which
// makes the plain FP64 path bit-identical to the reference CPU build.
#include <cuda_runtime.h>

#include <algorithm>

#include "device.h"

#include "device_common.cuh"

namespace mts {
namespace {

// ---------------------------------------------------------------------------
// Pointwise passes

// Pointwise kernels run one warp per grid row (iy, iz), lanes over ix.
#define FOR_EACH_NODE(P)                                                                          \
  for (int row_ = blockIdx.x * (TPB / 32) + (threadIdx.x >> 5); row_ < (P).ny * (P).nz;          \
       row_ += gridDim.x * (TPB / 32))                                                            \
    for (int ix = threadIdx.x & 31, iy = row_ % (P).ny, iz = row_ / (P).ny; ix < (P).nx; ix += 32) \
      if (long long m = ix + (long long)(P).nx * row_; true)

// The MIB rows of the Douglas-ADI first right-hand side (douglas_adi.cc:
// 89-359): uhs = ((dt*D_yy u + dt*D_zz u) + u) + dt*src with src = f + the x,
// y, z jump terms, into R at those nodes; the x sweep takes them from there.
// A pass of its own because a node waits on three loads in a row (its block,
// the block's weights and crossings, the field): all nodes of the grid wait
// at once here, a tile's would wait in turn.
__device__ __forceinline__ void k_adi_mib_body(const Dev& P, unsigned cta_, unsigned ncta_,
                                               const double* __restrict__ un, double* __restrict__ R, double E) {
  const double dt = P.dt;
  mib_nodes(P, un, step_e(P, E, 2), cta_ * (TPB / 32) + (threadIdx.x >> 5), ncta_ * (TPB / 32),
            [&](long long m, int, int, int, double, double sy, double sz, double src) {
              double r = sy * dt + sz * dt;
              r += un[m];
              r += dt * src;
              R[m] = r;
            });
}

__global__ void __launch_bounds__(TPB) k_adi_mib(const __grid_constant__ Dev P, const double* __restrict__ un,
                                                 double* __restrict__ R, double E) {
  k_adi_mib_body(P, blockIdx.x, gridDim.x, un, R, E);
}

// TS explicit half step along D = x or y (TS::D_xx_r / D_yy_r, the LOD
// Crank-Nicolson operators, trapezoidal.cc:319-895), then Set_bc at t_half.
// At a MIB row of a D block, with its jump terms.  The block comes from ref
// (Dev::mibref) and not from a search of the line's list, whose loads a thread
// waits on one by one (113 x 97 x 141, 48 steps: 5.28 -> 4.95 ms).
template <int D>
__device__ __forceinline__ double ts_explicit_mib(const Dev& P, const double* in, double E1, long long m, int ref,
                                                  int side) {
  const long long s = D == 0 ? 1 : (long long)P.nx;
  const MibBlock& b = P.blk[D][ref >> 4];
  const int kind = (ref >> 2) & 3, row = ref & 3;
  const double* const p = in + m - (row + b.L) * s;  // row 0 of the line
  const double2 Jl = jump_at(P, b.c0, E1), Jr = kind == 3 ? jump_at(P, b.c1, E1) : Jl;
  const double sum = mib_sum(b, row, [&](int j) { return p[j * s]; }, P.vd[D][side], true, Jl, Jr);
  return P.kex * sum + in[m];
}

// CTAs of the pass that take the MIB rows, a thread per listed node, after
// the ones that walk the grid's rows.
__host__ __device__ __forceinline__ unsigned mib_ctas(const Dev& P) { return (unsigned)((P.nmibnode + TPB - 1) / TPB); }

template <int D>
__device__ __forceinline__ void k_ts_explicit_body(const Dev& P, unsigned cta_, unsigned ncta_,
                                                   const double* __restrict__ in, double* __restrict__ out,
                                                   double eh, double e1) {
  const long long s = D == 0 ? 1 : (long long)P.nx;
  const int flag = D == 0 ? TAG_MIBX : TAG_MIBY;
  const unsigned nrow = ncta_ - mib_ctas(P);
  if (cta_ >= nrow) {
    const int k = (int)(cta_ - nrow) * TPB + threadIdx.x;
    if (k >= P.nmibnode) return;
    const long long m = P.mibnode[k];
    const int ref = reinterpret_cast<const int*>(P.mibref)[4 * (long long)k + D];
    if (ref >= 0) out[m] = ts_explicit_mib<D>(P, in, step_e(P, e1, 2), m, ref, P.tag[m] & TAG_OUT);
    return;
  }
  eh = step_e(P, eh, 1);
  const int lane = threadIdx.x & 31;
  const int nrows = P.ny * P.nz;
  const double kex = P.kex;
  const double w0i = P.vd[D][0][0], w1i = P.vd[D][0][1], w2i = P.vd[D][0][2];
  const double w0o = P.vd[D][1][0], w1o = P.vd[D][1][1], w2o = P.vd[D][1][2];
  for (int row = cta_ * (TPB / 32) + (threadIdx.x >> 5); row < nrows; row += nrow * (TPB / 32)) {
    const int iy = row % P.ny, iz = row / P.ny;
    const long long m0 = (long long)P.nx * row;
    const RowExact q = row_exact(P, iy, iz);
    if (iy == 0 || iz == 0 || iy == P.ny - 1 || iz == P.nz - 1) {
      for (int ix = lane; ix < P.nx; ix += 32) out[m0 + ix] = row_outer(P, q, ix, eh);
      continue;
    }
    for (int ix0 = 0; ix0 < P.nx; ix0 += 32 * ROW_G) {
      double um[ROW_G], uc[ROW_G], up[ROW_G];
      int tg[ROW_G];
#pragma unroll
      for (int g = 0; g < ROW_G; g++) {
        const int ix = ix0 + 32 * g + lane;
        if (ix < P.nx) {
          const long long m = m0 + ix;
          tg[g] = P.tag[m];
          uc[g] = in[m];
          um[g] = in[m - s];
          up[g] = in[m + s];
        }
      }
#pragma unroll
      for (int g = 0; g < ROW_G; g++) {
        const int ix = ix0 + 32 * g + lane;
        if (ix >= P.nx) break;
        const long long m = m0 + ix;
        double v;
        if (ix == 0 || ix == P.nx - 1) {
          v = row_outer(P, q, ix, eh);
        } else if (!(tg[g] & flag)) {
          const int side = tg[g] & TAG_OUT;
          double sum = 0.0;
          sum += um[g] * (side ? w0o : w0i);
          sum += uc[g] * (side ? w1o : w1i);
          sum += up[g] * (side ? w2o : w2i);
          v = kex * sum + uc[g];
        } else {
          continue;  // a MIB row of a D block: the CTAs past the rows write it
        }
        out[m] = v;
      }
    }
  }
}

template <int D>
__global__ void __launch_bounds__(TPB) k_ts_explicit(const __grid_constant__ Dev P, const double* __restrict__ in,
                                                     double* __restrict__ out, double eh, double e1) {
  k_ts_explicit_body<D>(P, blockIdx.x, gridDim.x, in, out, eh, e1);
}

// ---------------------------------------------------------------------------
// The line solves of one direction.  A CTA takes a tile of NL lines, keeps it
// in shared memory from the right-hand side to the solution, and leaves:
//   load    all threads build the right-hand sides of the tile's regular rows
//           (the line's stencil, or for the Douglas-ADI x solve the whole
//           first right-hand side, douglas_adi.cc:89-359) with every load
//           coalesced and several rows in flight per thread;
//   blocks  a thread per MIB block builds its rows' right-hand sides (the
//           explicit MIB stencil of douglas_adi.cc:112-210 / lod.cc:337-496,
//           the jump terms of D_xx_l lod.cc:960-1097, the Convert2Tri row
//           operations) from the line's own values;
//   solve   one warp runs the Thomas recurrences, a lane per line, forward
//           and back, in place in shared memory, the rows' factors copied in
//           ahead of use;
//   store   all threads write the tile back, coalesced.
// Interior lines are taken in the order of Dev::lperm: the lines that cross
// the interface, whose tiles take longest, then the others by side, each in
// memory order.  Tiles are full whatever the grid's extents.  CTAs past the
// tiles write the face lines.
//
// What bounds it: the recurrence is one dependent chain a row, so a tile
// costs its line's length whatever its width (one warp, B200: 88 clocks a row
// forward and back, 130 with the lines' own factors), and an SM solves as many
// lines at once as its shared memory holds (32 lines of 257 rows take 72 KB
// for x, three tiles, and 76 KB for y and z, two); the other tiles' loads and
// stores overlap the chains.  Up to 4 tiles an SM (129^3) a sweep is one
// tile's latency; with many more the loads are the longer part, held to about
// 3.9 TB/s by the small L1 that the tiles leave (a plain tile copy: 5.9 TB/s
// with 1 KB of shared memory per CTA, 3.9 with 36 KB or more).  Against one
// line per thread over a ring of staged rows with the partial solutions in a
// global scratch (ring.cu, which takes the sweeps of many long lines), us per
// step: 65^3 Douglas-ADI 138 -> 55, 129^3 LOD-CN 256 -> 81, 193^3 LOD-CN 655 ->
// 241, 225^3 Douglas-ADI 513 -> 463.

// Lines per tile and threads per CTA of each shape (mts_set_sweep_shape).
#define MTS_SHAPES(X)                                                                           \
  X(0, 32, 256) X(1, 32, 128) X(2, 32, 192) X(3, 16, 256) X(4, 8, 96) X(5, 16, 96) X(6, 8, 128) \
  X(7, 16, 128) X(8, 4, 128) X(9, 4, 96)

// Doubles per row of a tile: an x tile is written along its lines, so its
// rows are padded to an odd stride.
template <int D, int NL>
__host__ __device__ constexpr int tile_row() { return D == 0 ? NL + 1 : NL; }
// Rows of a chunk of the lines' own factors while a tile is solved: 8, or 4
// for x lines, where the smaller buffers let an SM hold three 257-row tiles
// (us with 4 / 8: 257^3 Douglas-ADI x 227 / 240, LOD-IE x 176 / 184, 400 x 129
// x 129 LOD-IE x 83 / 91; LOD-CN x, whose tiles hold more registers, 225^3 121
// / 111).  For y and z 8 rows are better at 129 (25 / 27, LOD-IE y), 193 (87 /
// 92, Douglas-ADI y) and from 257 rows on (LOD-IE z 224 / 210), and 4 where
// they make room for one more tile, at 161 (48 / 59, Douglas-ADI y) and 225
// rows (120 / 153).
template <int D>
__host__ __device__ constexpr int own_rows() { return D == 0 ? 4 : 8; }
// Bytes for the factors: those of a side ((bet, 1/bet), gam by row), or two
// chunks of the lines' own ((bet, 1/bet), a).
template <int D, int NL>
__host__ __device__ constexpr int factor_bytes(int n) {
  const int side = (24 * n + 15) / 16 * 16, own = 2 * 24 * NL * own_rows<D>();
  return side > own ? side : own;
}
template <int D, int NL>
constexpr size_t tile_smem(int n) {
  return factor_bytes<D, NL>(n) + sizeof(double) * (size_t)n * tile_row<D, NL>();
}

// Interior lines of direction D.
template <int D>
__host__ __device__ __forceinline__ long long interior_lines(const Dev& P) {
  return (long long)((D == 0 ? P.ny : P.nx) - 2) * ((D == 2 ? P.ny : P.nz) - 2);
}

template <int D>
__device__ __forceinline__ long long line_base(const Dev& P, int i1, int i2) {
  if (D == 0) return (long long)P.nx * (i1 + (long long)P.ny * i2);
  if (D == 1) return i1 + (long long)P.nx * P.ny * i2;
  return i1 + (long long)P.nx * i2;
}

// Face lines of direction D, all their nodes: Outer_u(t_next), with dt f
// added after the last sweep of a LOD step.
template <int D>
__device__ __forceinline__ void face_lines(const Dev& P, unsigned cta, unsigned ncta, const SweepIO& io, double E1) {
  if (!io.bmode) return;
  const int n = D == 0 ? P.nx : D == 1 ? P.ny : P.nz;
  const int n1 = D == 0 ? P.ny : P.nx, n2 = D == 2 ? P.ny : P.nz;
  const long long s = D == 0 ? 1 : D == 1 ? (long long)P.nx : (long long)P.nx * P.ny;
  const int nf = 2 * n1 + 2 * (n2 - 2);
  const long long total = (long long)nf * n;
  for (long long e = (long long)cta * blockDim.x + threadIdx.x; e < total; e += (long long)ncta * blockDim.x) {
    int f, j;  // neighbouring threads: neighbouring nodes in memory
    if (D == 0) {
      f = (int)(e / n);
      j = (int)(e % n);
    } else {
      j = (int)(e / nf);
      f = (int)(e % nf);
    }
    int i1, i2;
    if (f < 2 * n1) {
      i1 = f % n1;
      i2 = f < n1 ? 0 : n2 - 1;
    } else {
      i2 = 1 + (f - 2 * n1) % (n2 - 2);
      i1 = f - 2 * n1 < n2 - 2 ? 0 : n1 - 1;
    }
    const long long m = line_base<D>(P, i1, i2) + j * s;
    const int ix = D == 0 ? j : i1;
    const int iy = D == 0 ? i1 : D == 1 ? j : i2;
    const int iz = D == 2 ? j : i2;
    double v = outer_u(P, E1, ix, iy, iz);
    if (io.bmode == 2) v = v + P.dt * source(P, E1, P.tag[m] & TAG_OUT, ix, iy, iz);
    io.out[m] = v;
  }
}

// The Convert2Tri row operations of x block k on the first right-hand side's
// rows in shared memory (Douglas-ADI).
template <int RS>
__device__ __forceinline__ void block_ops(const Dev& P, int k, double* row0) {
  const MibBlock& b = P.blk[0][k];
  double* const r0 = row0 + b.L * RS;
  double r[3] = {r0[0], r0[RS], b.kind == 3 ? r0[2 * RS] : 0.0};
  implicit_rows(P, b, r, nullptr, nullptr, nullptr, false, make_double2(0.0, 0.0), make_double2(0.0, 0.0));
  for (int q = 0; q < b.kind; q++) r0[q * RS] = r[q];
}

__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gsrc) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gsrc) : "memory");
}

// Quotients from the reciprocal.  With y = 1/b rounded to nearest, the
// quotient of n by b is formed as
//   t = n (y (1 - b y)),  q0 = n y + t,  q = q0 + (n - b q0) y
// with fused multiply-adds.  1 - b y is exact, so q0 is n (1/b) to a relative
// 2^-104 before its own rounding, one of the two doubles around n/b, and then
// q is the correctly rounded quotient (Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", 1990: from y correctly
// rounded and q0 within one unit, one correction by the exact remainder).
// That holds while nothing over- or underflows on the way: |b| in [2^-100,
// 2^100] (checked where the factors are made, Dev::plain_div) and |q| in
// [2^-800, 2^800].  A tile with a quotient outside that (zeros, infinities
// and NaN among them) is built and solved again with the divide: a field that
// is zero throughout, boundary data and source included, costs 129^3
// Douglas-ADI 298 against 97 us a step, 257^3 1282 against 623 (rings alone:
// 386 and 932).  Between boundary values of order one zeros do not last a row.
// (Letting +0 by a positive factor pass takes the numerator's bits too: 102
// against 97 us at 129^3 on ordinary fields.)
// One warp alone (B200): 52 clocks a row of the recurrence against 125 with
// the divide, whose own reciprocal and tests are on the chain.
constexpr unsigned kQLo = (1023u - 800u) << 21, kQRange = 1600u << 21;
__device__ __forceinline__ bool quotient_out(double q) {
  return ((unsigned)__double2hiint(q) << 1) - kQLo >= kQRange;
}

// G rows of the forward recurrence d_j = (r_j - a_j d_{j-1}) / bet_j (TDMA,
// douglas_adi.cc:1794-1800): r in, d out, d_{j-1} of the first row in d.
// f: (bet, 1/bet) by row.
template <int G, bool PLAIN>
__device__ __forceinline__ void forward_rows(double (&r)[G], const double (&a)[G], const double2 (&f)[G], double& d) {
#pragma unroll
  for (int k = 0; k < G; k++) {
    const double nn = r[k] - a[k] * d;
    const double b = f[k].x, y = f[k].y;
    if (PLAIN) {
      d = nn / b;
    } else {
      const double yl = y * __fma_rn(-b, y, 1.0);
      const double q0 = __fma_rn(nn, y, nn * yl);
      d = __fma_rn(__fma_rn(-b, q0, nn), y, q0);
    }
    r[k] = d;
  }
}

// The recurrences of a line whose rows are its side's, with the row factors
// of that side in shared memory ((bet, 1/bet) and gam_{j+1} by row); row0:
// row 0 of the line, right-hand sides in, solution out.  Returns whether a
// quotient is out of range.
template <int RS, bool PLAIN>
__device__ __forceinline__ bool solve_side(const double2* bet, const double* gam, double ac, double* row0, int n) {
  constexpr int G = 4;
  const int last = n - 1;
  double d = 0.0;
  auto single = [&](int j, double aj) {
    const double a[1] = {aj};
    const double2 f[1] = {bet[j]};
    double r[1] = {row0[j * RS]};
    forward_rows<1, PLAIN>(r, a, f, d);
    row0[j * RS] = d;
  };
  single(0, 0.0);  // (the end rows are identities)
  double a[G], r[G], rn[G];
  double2 f[G], fn[G];
#pragma unroll
  for (int k = 0; k < G; k++) a[k] = ac;
  int j = 1;
  auto ahead = [&](int at) {
#pragma unroll
    for (int k = 0; k < G; k++) {
      rn[k] = row0[(at + k) * RS];
      fn[k] = bet[at + k];
    }
  };
  if (j + G <= last) ahead(j);
  for (; j + G <= last; j += G) {
#pragma unroll
    for (int k = 0; k < G; k++) {
      r[k] = rn[k];
      f[k] = fn[k];
    }
    // the next rows, off the chain (for the last group any will do)
    ahead(j + 2 * G <= last ? j + G : j);
    forward_rows<G, PLAIN>(r, a, f, d);
#pragma unroll
    for (int k = 0; k < G; k++) row0[(j + k) * RS] = r[k];
  }
  for (; j < n; j++) single(j, j == last ? 0.0 : ac);

  // back: u_j = d_j - gam_{j+1} u_{j+1} (douglas_adi.cc:1805-1806)
  double u = d, g[G], gn[G];
  bool out = quotient_out(d);
  j = n - 2;
  auto behind = [&](int at) {
#pragma unroll
    for (int k = 0; k < G; k++) {
      rn[k] = row0[(at - k) * RS];
      gn[k] = gam[at - k];
    }
  };
  if (j - G + 1 >= 0) behind(j);
  for (; j - G + 1 >= 0; j -= G) {
#pragma unroll
    for (int k = 0; k < G; k++) {
      r[k] = rn[k];
      g[k] = gn[k];
    }
    behind(j - 2 * G + 1 >= 0 ? j - G : j);
#pragma unroll
    for (int k = 0; k < G; k++) {
      out |= quotient_out(r[k]);
      r[k] -= g[k] * u;
      u = r[k];
      row0[(j - k) * RS] = u;
    }
  }
  for (; j >= 0; j--) {
    double v = row0[j * RS];
    out |= quotient_out(v);
    v -= gam[j] * u;
    u = v;
    row0[j * RS] = u;
  }
  return out;
}

// Named barriers of two warps: one arrives and goes on, the other waits.
__device__ __forceinline__ void pair_sync(int id) { asm volatile("bar.sync %0, 64;\n" ::"r"(id) : "memory"); }
__device__ __forceinline__ void pair_arrive(int id) { asm volatile("bar.arrive %0, 64;\n" ::"r"(id) : "memory"); }

// The same for a tile with lines of their own factors, called by the whole
// CTA: of row j of this lane's line a_j at fa[j st], (bet_j, 1/bet_j) at
// fb[j st], gam_{j+1} at g[j st].  Up to seven other warps bring the factors
// in, OWN_C rows a chunk in turn: each holds its next chunk in registers and
// puts it down in one of two buffers (buf) once warp ws, which solves, is
// done with the chunk two before.  Barrier 1 + p: a chunk of producer p is
// down; 8 + p: its buffer is free.  (Two producers at least: a producer's
// next chunk waits for a chunk that the solving warp takes no earlier than
// its last one, so neither barrier is arrived at twice in a round.)
template <int NL, int RS, int NW, int C, bool PLAIN>
__device__ __forceinline__ bool solve_own(const double* __restrict__ fa, const double2* __restrict__ fb,
                                          const double* __restrict__ g, long long st, double* buf, double* row0, int n,
                                          int ws) {
  constexpr int NP = NW - 1 < 7 ? NW - 1 : 7;  // producers
  static_assert(NP >= 2, "two producers");
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const bool on = lane < NL;
  const int last = n - 1;
  double2* const bb = reinterpret_cast<double2*>(buf) + lane;  // [2][C][NL]
  double* const ba = buf + 4 * C * NL + lane;                  // [2][C][NL]
  const int chunks = (n + C - 1) / C;
  if (w != ws) {
    const int p = (w - ws - 1 + NW) % NW;
    double a[C];
    double2 f[C];
    if (p < NP) {
      auto fetch = [&](int k) {
        if (on && k < chunks) {
#pragma unroll
          for (int e = 0; e < C; e++) {
            const long long o = (long long)min(k * C + e, last) * st;
            a[e] = fa[o];
            f[e] = fb[o];
          }
        }
      };
      fetch(p);
      for (int k = p; k < chunks; k += NP) {
        if (k >= 2) pair_sync(8 + p);
        if (on) {
#pragma unroll
          for (int e = 0; e < C; e++) {
            ba[((k & 1) * C + e) * NL] = a[e];
            bb[((k & 1) * C + e) * NL] = f[e];
          }
        }
        __syncwarp();
        pair_arrive(1 + p);
        fetch(k + NP);
      }
    }
    __syncthreads();
    if (p < NP) {
      const double* const gl = g + (long long)last * st;
      auto fetch = [&](int k) {
        if (on && k < chunks) {
#pragma unroll
          for (int e = 0; e < C; e++) a[e] = gl[-(long long)min(k * C + e, last) * st];
        }
      };
      fetch(p);
      for (int k = p; k < chunks; k += NP) {
        if (k >= 2) pair_sync(8 + p);
        if (on) {
#pragma unroll
          for (int e = 0; e < C; e++) ba[((k & 1) * C + e) * NL] = a[e];
        }
        __syncwarp();
        pair_arrive(1 + p);
        fetch(k + NP);
      }
    }
    return false;
  }
  // the solving warp: forward
  bool out = false;
  double d = 0.0;
  for (int k = 0, q = 0, q2 = 2 % NP; k < chunks; k++) {
    pair_sync(1 + q);
    if (on) {
      double a[C], r[C];
      double2 f[C];
#pragma unroll
      for (int e = 0; e < C; e++) {
        a[e] = ba[((k & 1) * C + e) * NL];
        f[e] = bb[((k & 1) * C + e) * NL];
        r[e] = row0[min(k * C + e, last) * RS];
      }
      // (rows past the end repeat the last one's inputs; not stored)
      forward_rows<C, PLAIN>(r, a, f, d);
#pragma unroll
      for (int e = 0; e < C; e++)
        if (k * C + e < n) row0[(k * C + e) * RS] = r[e];
    }
    __syncwarp();
    if (k + 2 < chunks) pair_arrive(8 + q2);
    q = q + 1 < NP ? q + 1 : 0;
    q2 = q2 + 1 < NP ? q2 + 1 : 0;
  }
  __syncthreads();
  // back, rows counted from the last (gam_n = 0)
  double* const rl = row0 + last * RS;
  double u = 0.0;
  for (int k = 0, q = 0, q2 = 2 % NP; k < chunks; k++) {
    pair_sync(1 + q);
    if (on) {
      double a[C], r[C];
#pragma unroll
      for (int e = 0; e < C; e++) {
        a[e] = ba[((k & 1) * C + e) * NL];
        r[e] = rl[-min(k * C + e, last) * RS];
      }
#pragma unroll
      for (int e = 0; e < C; e++) {
        if (k * C + e < n) {
          out |= quotient_out(r[e]);
          r[e] -= a[e] * u;
          u = r[e];
          rl[-(k * C + e) * RS] = u;
        }
      }
    }
    __syncwarp();
    if (k + 2 < chunks) pair_arrive(8 + q2);
    q = q + 1 < NP ? q + 1 : 0;
    q2 = q2 + 1 < NP ? q2 + 1 : 0;
  }
  return out;
}

// What the phases of a tile share.
template <int NL>
struct TileState {
  int i1[NL], i2[NL];  // the tile's lines
  int next_task;       // of the load phase
  int side;            // the side whose factors all its lines have, -1: not so
  int again;           // a quotient was out of range
};

// The MIB rows' right-hand sides (the warps from BW on).
template <int D, int KIND, int NL, int NT>
__device__ __forceinline__ void tile_blocks(const Dev& P, const SweepIO& io, const TileState<NL>& T, double* sm,
                                         int nlive) {
  constexpr int RS = tile_row<D, NL>(), NW = NT / 32, BW = NW / 2;
  const int tid = threadIdx.x, w = tid >> 5;
  const double E1 = step_e(P, io.e1, 2);
  if (KIND != K_ADI && P.nblk[D] > 0) {
    const int e = tid - 32 * BW, c = e % NL;
    if (c < nlive) {
      const int i1 = T.i1[c], i2 = T.i2[c];
      const int lid = i1 * (D == 2 ? P.ny : P.nz) + i2;
      const int bend = P.bstart[D][lid + 1];
      const long long base = line_base<D>(P, i1, i2);
      const double E0 = KIND == K_TS_Z ? step_e(P, io.e0, 0) : 0.0;
      for (int k = P.bstart[D][lid] + e / NL; k < bend; k += (NT - 32 * BW) / NL) {
        double r[3];
        block_rhs<D, KIND>(P, io, E0, E1, k, base, i1, i2, r);
        const MibBlock& b = P.blk[D][k];
        for (int q = 0; q < b.kind; q++) sm[(b.L + q) * RS + c] = r[q];
      }
    }
  }
}

// The regular rows' right-hand sides: warps take tasks (a few rows of the
// tile each) until none is left; all loads of a task are issued before any is
// used.
constexpr int TASK_ROWS = 6;
template <int D, int KIND, int NL, int NT>
__device__ __forceinline__ void tile_rows(const Dev& P, const SweepIO& io, TileState<NL>& T, double* sm, int nlive) {
  constexpr int RS = tile_row<D, NL>();
  const int lane = threadIdx.x & 31;
  constexpr int SUB = 32 / NL;
  const int n = D == 0 ? P.nx : D == 1 ? P.ny : P.nz;
  const double E1 = step_e(P, io.e1, 2);
  const double kx = io.k;
  auto task = [&]() {
    int t = 0;
    if (lane == 0) t = atomicAdd(&T.next_task, 1);
    return __shfl_sync(0xffffffffu, t, 0);
  };
  if (D != 0) {
    // lanes: lines (32 / NL runs of rows at a time), U rows a lane; the last
    // run is moved back to end with the line (the rows it shares with the one
    // before get the same values twice)
    const long long s = D == 1 ? (long long)P.nx : (long long)P.nx * P.ny;
    const int c = lane % NL, sub = lane / NL;
    const int i1 = T.i1[c], i2 = T.i2[c];
    const long long base = line_base<D>(P, i1, i2);
    const bool two = KIND != K_COPY && io.add != io.stin;
    const double E0 = KIND == K_TS_Z ? step_e(P, io.e0, 0) : 0.0;
    constexpr int flag = D == 1 ? TAG_MIBY : TAG_MIBZ;
    auto run = [&](auto UU) {
      constexpr int U = decltype(UU)::value;
      for (int t = task(); t * (U * SUB) < n; t = task()) {
        const int j0 = min((t * SUB + sub) * U, n - U);
        const long long g0 = base + (long long)j0 * s;
        double u[U + 2], av[U];
        int tt[U];
        {
          const uint8_t* tg = P.tag + g0;
          const double* gb = io.add + g0;
#pragma unroll
          for (int k = 0; k < U; k++, tg += s) tt[k] = *tg;
          if (KIND == K_COPY || two) {
#pragma unroll
            for (int k = 0; k < U; k++, gb += s) av[k] = __ldcg(gb);
          }
        }
        if (KIND != K_COPY) {
          // (the neighbours past the line's ends are not used)
          const double* ga = io.stin + g0;
          u[0] = j0 > 0 ? __ldcg(ga - s) : 0.0;
#pragma unroll
          for (int k = 1; k <= U; k++, ga += s) u[k] = __ldcg(ga);
          u[U + 1] = j0 + U < n ? __ldcg(ga) : 0.0;
        }
#pragma unroll
        for (int k = 0; k < U; k++) {
          const int j = j0 + k;
          double r;
          if (KIND == K_COPY) {
            r = av[k];
          } else {
            auto val = [&](auto S) {
              constexpr int sd = decltype(S)::value;
              double sum = 0.0;
              sum += u[k] * P.vd[D][sd][0];
              sum += u[k + 1] * P.vd[D][sd][1];
              sum += u[k + 2] * P.vd[D][sd][2];
              double v = kx * sum + (two ? av[k] : u[k + 1]);
              if (KIND == K_TS_Z) {
                v = v + P.hdt * source(P, E0, sd, i1, i2, j);
                v = v + P.hdt * source(P, E1, sd, i1, i2, j);
              }
              return v;
            };
            r = (tt[k] & TAG_OUT) ? val(IntC<1>{}) : val(IntC<0>{});
          }
          if (j == 0 || j == n - 1) r = outer_u(P, E1, i1, D == 1 ? j : i2, D == 1 ? i2 : j);
          if (!(tt[k] & flag) && c < nlive) sm[j * RS + c] = r;
        }
      }
    };
    if (n >= TASK_ROWS)
      run(IntC<TASK_ROWS>{});
    else
      run(IntC<1>{});
    return;
  }
  // lanes: 32 columns of U lines; the interior columns, then the two ends
  constexpr int U = 4, GROUPS = (NL + U - 1) / U;
  const int chunks = (n - 2 + 31) / 32;
  for (int t = task(); t <= chunks * GROUPS; t = task()) {
    if (t == chunks * GROUPS) {
      for (int e = lane; e < 2 * nlive; e += 32) {
        const int ix = (e & 1) ? n - 1 : 0;
        sm[ix * RS + (e >> 1)] = outer_u(P, E1, ix, T.i1[e >> 1], T.i2[e >> 1]);
      }
      continue;
    }
    const int c0 = t / chunks * U;
    if (c0 >= nlive) continue;
    const int ixl = 1 + t % chunks * 32 + lane;
    const int ix = min(ixl, n - 2);
    const bool in = ixl < n - 1;
    if (KIND != K_ADI) {
      double um[U], uc[U], up[U], av[U];
      int tt[U];
#pragma unroll
      for (int k = 0; k < U; k++) {
        const int c = min(c0 + k, nlive - 1);
        const long long m = line_base<0>(P, T.i1[c], T.i2[c]) + ix;
        tt[k] = P.tag[m];
        if (KIND == K_COPY) {
          av[k] = io.add[m];
        } else {
          uc[k] = io.stin[m];
          um[k] = io.stin[m - 1];
          up[k] = io.stin[m + 1];
          av[k] = io.add[m];
        }
      }
#pragma unroll
      for (int k = 0; k < U; k++) {
        double r;
        if (KIND == K_COPY) {
          r = av[k];
        } else {
          const bool out = tt[k] & TAG_OUT;
          double sum = 0.0;
          sum += um[k] * (out ? P.vd[0][1][0] : P.vd[0][0][0]);
          sum += uc[k] * (out ? P.vd[0][1][1] : P.vd[0][0][1]);
          sum += up[k] * (out ? P.vd[0][1][2] : P.vd[0][0][2]);
          r = kx * sum + av[k];
        }
        if (in && c0 + k < nlive && !(tt[k] & TAG_MIBX)) sm[ix * RS + c0 + k] = r;
      }
    } else {
      // Douglas-ADI: the first right-hand side ((dt D_yy u + dt D_zz u) + u)
      // + dt src (douglas_adi.cc:89-359); the lines' y neighbours are one
      // another where they lie in one plane
      const double* const un = io.stin;
      const long long sy = P.nx, sz = (long long)P.nx * P.ny;
      const double dt = P.dt;
      double um[U], uc[U], up[U], zm[U], zp[U];
      int tt[U], yy[U], zz[U];
      const double xv = P.ax[0][ix], s2x = P.s2[0][ix];
      const double x2 = xv * xv;
#pragma unroll
      for (int k = 0; k < U; k++) {
        const int c = min(c0 + k, nlive - 1);
        yy[k] = T.i1[c];
        zz[k] = T.i2[c];
      }
      bool plane = c0 + U <= nlive;  // four neighbours
#pragma unroll
      for (int k = 1; k < U; k++) plane = plane && yy[k] == yy[0] + k && zz[k] == zz[0];
      if (plane) {
        const long long m0 = line_base<0>(P, yy[0], zz[0]) + ix;
        double u[U + 2];
#pragma unroll
        for (int k = 0; k < U + 2; k++) u[k] = un[m0 + (k - 1) * sy];
#pragma unroll
        for (int k = 0; k < U; k++) {
          zm[k] = __ldcg(un + m0 + k * sy - sz);
          zp[k] = __ldcg(un + m0 + k * sy + sz);
          tt[k] = P.tag[m0 + k * sy];
        }
#pragma unroll
        for (int k = 0; k < U; k++) {
          um[k] = u[k];
          uc[k] = u[k + 1];
          up[k] = u[k + 2];
        }
      } else {
#pragma unroll
        for (int k = 0; k < U; k++) {
          const long long m = line_base<0>(P, yy[k], zz[k]) + ix;
          um[k] = un[m - sy];
          uc[k] = un[m];
          up[k] = un[m + sy];
          zm[k] = un[m - sz];
          zp[k] = un[m + sz];
          tt[k] = P.tag[m];
        }
      }
#pragma unroll
      for (int k = 0; k < U; k++) {
        if (!in || c0 + k >= nlive) continue;
        if (tt[k] & (TAG_MIBX | TAG_MIBY | TAG_MIBZ)) {
          sm[ix * RS + c0 + k] = io.out[line_base<0>(P, yy[k], zz[k]) + ix];  // a MIB row: from k_adi_mib
          continue;
        }
        const RowExact q = row_exact(P, yy[k], zz[k]);
        auto val = [&](auto S) {
          constexpr int sd = decltype(S)::value;
          double sum = 0.0;
          sum += um[k] * P.vd[1][sd][0];
          sum += uc[k] * P.vd[1][sd][1];
          sum += up[k] * P.vd[1][sd][2];
          const double ydt = dt * sum;
          sum = 0.0;
          sum += zm[k] * P.vd[2][sd][0];
          sum += uc[k] * P.vd[2][sd][1];
          sum += zp[k] * P.vd[2][sd][2];
          const double zdt = dt * sum;
          double src = 0.0;
          if (P.eq != 0) {
            if (sd)
              src = -(((x2 + q.y2) + q.z2) * E1) - P.c6bo * E1;
            else
              src = P.kin * (((s2x * q.c2y) * q.s2z) * E1);
          }
          double v = ydt + zdt;
          v += uc[k];
          v += dt * src;
          return v;
        };
        sm[ix * RS + c0 + k] = (tt[k] & TAG_OUT) ? val(IntC<1>{}) : val(IntC<0>{});
      }
    }
  }
}

// A tile from its fields to its solution in shared memory.
template <int D, int KIND, int NL, int NT, bool PLAIN>
__device__ __forceinline__ void tile_solution(const Dev& P, const SweepIO& io, TileState<NL>& T, double* sm_,
                                              int nlive) {
  constexpr int RS = tile_row<D, NL>();
  constexpr int NW = NT / 32;
  constexpr int BW = NW / 2;  // the warps from this one on take the blocks first
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int n = D == 0 ? P.nx : D == 1 ? P.ny : P.nz;
  const int n1 = D == 0 ? P.ny : P.nx, n2 = D == 2 ? P.ny : P.nz;
  double* const sm = sm_ + factor_bytes<D, NL>(n) / 8;  // [n][RS]
  const int ws = (blockIdx.x / P.sweep_blocks) % NW;  // the solving warp: another sub-core CTA by CTA
  // ---- which factors the solve needs (the first warp): one side's, copied
  // into shared memory here, or the lines' own
  if (w == 0) {
    const int i1 = T.i1[lane % NL], i2 = T.i2[lane % NL];
    const int c = P.cline[D] ? P.cline[D][i1 + n1 * i2] : -1;
    const int side = (P.lside[D][i1 * n2 + i2] >> 1) & 1;
    const int side0 = __shfl_sync(0xffffffffu, side, 0);
    const bool same = __all_sync(0xffffffffu, c < 0 && side == side0);
    if (lane == 0) T.side = same ? side : -1;
    if (same) {
      for (int j = lane; j < n; j += 32) {
        cp_async16(sm_ + 2 * j, P.tab[D][side] + j);
        cp_async8(sm_ + 2 * n + j, P.tabg[D][side] + j);
      }
    }
  }
  // ---- load
  if (w >= BW) tile_blocks<D, KIND, NL, NT>(P, io, T, sm, nlive);
  tile_rows<D, KIND, NL, NT>(P, io, T, sm, nlive);
  if (w == 0) {
    cp_async_commit();
    cp_async_wait<0>();
  }
  __syncthreads();
  const int side = T.side;
  if (KIND == K_ADI && side < 0) {
    // the x blocks' row operations on their right-hand sides
    const int c = tid % NL;
    if (c < nlive) {
      const int lid = T.i1[c] * n2 + T.i2[c];
      const int bend = P.bstart[0][lid + 1];
      for (int k = P.bstart[0][lid] + tid / NL; k < bend; k += NT / NL) block_ops<RS>(P, k, sm + c);
    }
    __syncthreads();
  }
  // ---- solve: one warp
  if (side >= 0) {
    if (w == ws && lane < nlive) {
      if (solve_side<RS, PLAIN>(reinterpret_cast<const double2*>(sm_), sm_ + 2 * n, side ? P.ia[D][1] : P.ia[D][0],
                                sm + lane, n))
        T.again = 1;
    }
  } else {
    // (lanes past the tile's lines run the last line's factors on columns
    // that are not stored)
    const int cl = min(lane, nlive - 1);
    const int i1 = T.i1[cl], i2 = T.i2[cl];
    const int c = P.cline[D] ? P.cline[D][i1 + n1 * i2] : -1;
    const int ls = (P.lside[D][i1 * n2 + i2] >> 1) & 1;
    if (solve_own<NL, RS, NW, own_rows<D>(), PLAIN>(c >= 0 ? P.ca[D] + c : P.taba[D][ls], c >= 0 ? P.cb[D] + c : P.tab[D][ls],
                                     c >= 0 ? P.cg[D] + c : P.tabg[D][ls], c >= 0 ? P.nfcross[D] : 1, sm_,
                                     sm + min(lane, NL - 1), n, ws) &&
        lane < nlive)
      T.again = 1;
  }
  __syncthreads();
}

// The same with the divide, out of line (rare).
template <int D, int KIND, int NL, int NT>
__device__ __noinline__ void tile_solution_plain(const Dev& P, const SweepIO& io, TileState<NL>& T, double* sm_,
                                                 int nlive) {
  tile_solution<D, KIND, NL, NT, true>(P, io, T, sm_, nlive);
}

template <int D, int KIND, int NL, int NT>
__device__ __forceinline__ void k_line_body(const Dev& P, unsigned cta_, unsigned ncta_, const SweepIO& io) {
  static_assert(NT % 32 == 0 && NT >= 96 && NL <= 32 && 32 % NL == 0, "shape");
  static_assert(D == 0 || KIND != K_ADI, "the first right-hand side belongs to the x solve");
  constexpr int RS = tile_row<D, NL>();
  constexpr int NW = NT / 32;
  const int tid = threadIdx.x;
  const int n = D == 0 ? P.nx : D == 1 ? P.ny : P.nz;
  const int nint = (int)interior_lines<D>(P);
  const int ntile = (nint + NL - 1) / NL;
  if ((int)cta_ >= ntile) {
    face_lines<D>(P, cta_ - ntile, ncta_ - ntile, io, step_e(P, io.e1, 2));
    return;
  }
  extern __shared__ __align__(16) double sm_[];
  __shared__ TileState<NL> T;
  const int t0 = (int)cta_ * NL;
  const int nlive = min(NL, nint - t0);
  if (tid < NL) {
    const int n1 = D == 0 ? P.ny : P.nx;
    const int v = P.lperm[D][min(t0 + tid, nint - 1)];
    const int q = v / n1;
    T.i1[tid] = v - q * n1;
    T.i2[tid] = q;
  }
  if (tid == 0) {
    T.next_task = 0;
    T.again = P.plain_div;
  }
  __syncthreads();
  if (!P.plain_div) tile_solution<D, KIND, NL, NT, false>(P, io, T, sm_, nlive);
  if (T.again) {
    __syncthreads();
    if (tid == 0) T.next_task = 0;
    __syncthreads();
    tile_solution_plain<D, KIND, NL, NT>(P, io, T, sm_, nlive);
  }

  // ---- store
  const double* const sm = sm_ + factor_bytes<D, NL>(n) / 8;
  if (D != 0) {
    constexpr int SUB = NT / NL;
    const long long s = D == 1 ? (long long)P.nx : (long long)P.nx * P.ny;
    const int c = tid % NL;
    if (c < nlive) {
      const int i1 = T.i1[c], i2 = T.i2[c];
      const long long base = line_base<D>(P, i1, i2);
      double* const o = io.out + base;
      if (io.last) {
        const uint8_t* const tg = P.tag + base;
        const double E1 = step_e(P, io.e1, 2);
#pragma unroll 4
        for (int j = tid / NL; j < n; j += SUB)
          o[j * s] = sm[j * RS + c] +
                     P.dt * source(P, E1, tg[j * s] & TAG_OUT, i1, D == 1 ? j : i2, D == 1 ? i2 : j);
      } else {
#pragma unroll 8
        for (int j = tid / NL; j < n; j += SUB) o[j * s] = sm[j * RS + c];
      }
    }
  } else {
    for (int c = tid >> 5; c < nlive; c += NW) {
      double* const o = io.out + line_base<0>(P, T.i1[c], T.i2[c]);
#pragma unroll 8
      for (int ix = tid & 31; ix < n; ix += 32) o[ix] = sm[ix * RS + c];
    }
  }
}

// CTAs of a direction's line solves: its tiles, and for the face lines one
// per 4096 nodes.
template <int D>
unsigned line_grid(const Dev& P, int nl, bool faces) {
  const long long tiles = (interior_lines<D>(P) + nl - 1) / nl;
  const long long n1 = D == 0 ? P.ny : P.nx, n2 = D == 2 ? P.ny : P.nz, n = D == 0 ? P.nx : D == 1 ? P.ny : P.nz;
  const long long fn = (2 * n1 + 2 * (n2 - 2)) * n;
  return (unsigned)(tiles + (faces ? (fn + 4095) / 4096 : 0));
}

// CTAs per SM that the registers should allow: four of 256 threads, three for
// the first right-hand side, which holds more.  It pays where the shared memory
// allows as many, and costs spills where it does not (us with this rule / with
// one CTA less: LOD-CN x, y, z 129^3 27, 27, 33 / 31, 31, 40, 161^3 43, 47, 58
// / 46, 46, 58, 241^3 151, 155, 201 / 133, 148, 199; Douglas-ADI x 129^3 39 /
// 37, 193^3 87 / 111, 257^3 227 / 235, 353^3 690 / 645; 16-line tiles, LOD-IE z
// 289^3 298 / 350).
template <int KIND, int NT>
constexpr int line_min_ctas() { return NT == 256 ? (KIND == K_ADI ? 3 : 4) : NT == 192 ? 4 : NT == 128 ? 5 : 6; }

template <int D, int KIND, int NL, int NT>
__global__ void __launch_bounds__(NT, line_min_ctas<KIND, NT>()) k_line(const __grid_constant__ Dev P,
                                                                       const __grid_constant__ SweepIO io) {
  k_line_body<D, KIND, NL, NT>(P, blockIdx.x, gridDim.x, io);
}

// Thomas factors of the lines that cross the interface (the factor half of
// TDMA, douglas_adi.cc:1790-1798: gam_j = c_{j-1}/bet, bet = b_j - a_j*gam_j,
// the same IEEE operations as the host's side tables), once at setup, one
// thread per listed line.  A line's rows are the identity on its faces, the
// regular three-point rows of the node's side elsewhere, and the Convert2Tri
// rows of its blocks; a_j, (bet_j, 1/bet_j) and gam_{j+1} are stored by row,
// the lines of a row side by side, and for the FP32 ring sweeps (where fib32 is there)
// 1/bet and gam per node from the first MIB row on.  A zero pivot sets bit 0
// of *flags, a factor out of the range of the quotients from reciprocals bit
// 1.
template <int D>
__global__ void __launch_bounds__(TPB) k_factor_lines(const __grid_constant__ Dev P, int* flags) {
  const int l = blockIdx.x * TPB + threadIdx.x;
  const int nc = P.nfcross[D];
  if (l >= nc) return;
  const int lid = P.fcross[D][l];
  const int n2 = D == 2 ? P.ny : P.nz;
  Line L;
  decode_line<D>(P, (long long)(lid % n2) * (D == 0 ? P.ny : P.nx) + lid / n2, L);
  const int bfirst = P.bstart[D][lid], bend = P.bstart[D][lid + 1];
  const MibBlock* const blk = P.blk[D];
  const int n = L.n;
  const int L1 = blk[bfirst].L;
  // (the factors are read-only to the step kernels; setup fills them here)
  double* const fa = const_cast<double*>(P.ca[D]) + l;
  double2* const fb = const_cast<double2*>(P.cb[D]) + l;
  double* const g = const_cast<double*>(P.cg[D]) + l;
  fa[0] = 0.0;
  fb[0] = make_double2(1.0, 1.0);
  int b = bfirst;
  double bet = 1.0;   // row 0: b = 1
  double cprev = 0.0; // c of the previous row
  for (int j = 1; j < n; j++) {
    double aj, bj, cj;
    if (j == n - 1) {
      aj = 0.0;
      bj = 1.0;
      cj = 0.0;
    } else if (b < bend && j >= blk[b].L) {
      const int q = j - blk[b].L;
      aj = blk[b].ia[q];
      bj = blk[b].ib[q];
      cj = blk[b].ic[q];
      if (q == blk[b].kind - 1) b++;
    } else {
      const int side = (P.tag[L.base + (long long)j * L.s] & TAG_OUT) ? 1 : 0;
      aj = P.ia[D][side];
      bj = P.ib[D][side];
      cj = P.ic[D][side];
    }
    const double gm = cprev / bet;
    bet = bj - aj * gm;
    if (bet == 0.0) {
      atomicOr(flags, 1);
      return;
    }
    fa[(long long)j * nc] = aj;
    fb[(long long)j * nc] = make_double2(bet, 1.0 / bet);
    if (!(fabs(bet) >= 0x1p-100 && fabs(bet) <= 0x1p100)) atomicOr(flags, 2);
    g[(long long)(j - 1) * nc] = gm;
    if (j >= L1 && P.fib32[D]) {
      const long long m = L.base + (long long)j * L.s;
      const_cast<float*>(P.fib32[D])[m] = (float)(1.0 / bet);
      const_cast<float*>(P.fgam32[D])[m] = (float)gm;
    }
    cprev = cj;
  }
  g[(long long)(n - 1) * nc] = 0.0;
}

// Per MIB node its block in x, y, z, once at setup: 16 block + 4 kind + row,
// -1: none.
__global__ void __launch_bounds__(TPB) k_mibref(const __grid_constant__ Dev P) {
  const int k = blockIdx.x * TPB + threadIdx.x;
  if (k >= P.nmibnode) return;
  const long long m = P.mibnode[k];
  const int tg = P.tag[m];
  int ix, iy, iz;
  node_xyz(P, m, ix, iy, iz);
  int4 r = make_int4(-1, -1, -1, 0);
  int row = 0;
  if (tg & TAG_MIBX) {
    const MibBlock* b = find_block<0>(P, iy * P.nz + iz, ix, row);
    if (b) r.x = (int)(b - P.blk[0]) * 16 + b->kind * 4 + row;
  }
  if (tg & TAG_MIBY) {
    const MibBlock* b = find_block<1>(P, ix * P.nz + iz, iy, row);
    if (b) r.y = (int)(b - P.blk[1]) * 16 + b->kind * 4 + row;
  }
  if (tg & TAG_MIBZ) {
    const MibBlock* b = find_block<2>(P, ix * P.ny + iy, iz, row);
    if (b) r.z = (int)(b - P.blk[2]) * 16 + b->kind * 4 + row;
  }
  const_cast<int4*>(P.mibref)[k] = r;
}

__global__ void __launch_bounds__(TPB) k_init(const Dev P, double E, double* u) {
  FOR_EACH_NODE(P) { u[m] = (P.tag[m] & TAG_OUT) ? outer_u(P, E, ix, iy, iz) : inner_u(P, E, ix, iy, iz); }
}

// Error norms: block partials of (max |e|, first argmax key, sum e^2), the key
// being the position in the reference's [ix][iy][iz] loop order.
constexpr int NB_TPB = 256;

__device__ __forceinline__ void better(double& v, long long& k, double v2, long long k2) {
  if (v2 > v || (v2 == v && k2 < k)) {
    v = v2;
    k = k2;
  }
}

__global__ void __launch_bounds__(NB_TPB) k_norms_partial(const Dev P, double E, const double* u, double* part) {
  __shared__ double smax[NB_TPB], ssum[NB_TPB];
  __shared__ long long skey[NB_TPB];
  double vmax = 0.0, vsum = 0.0;
  long long vkey = 0x7fffffffffffffffLL;
  for (long long m = (long long)blockIdx.x * NB_TPB + threadIdx.x; m < P.nn; m += (long long)gridDim.x * NB_TPB) {
    int ix, iy, iz;
    node_xyz(P, m, ix, iy, iz);
    double ex = (P.tag[m] & TAG_OUT) ? outer_u(P, E, ix, iy, iz) : inner_u(P, E, ix, iy, iz);
    double e = fabs(u[m] - ex);
    long long key = ((long long)ix * P.ny + iy) * P.nz + iz;
    better(vmax, vkey, e, key);
    vsum += e * e;
  }
  smax[threadIdx.x] = vmax;
  skey[threadIdx.x] = vkey;
  ssum[threadIdx.x] = vsum;
  __syncthreads();
  for (int w = NB_TPB / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) {
      better(smax[threadIdx.x], skey[threadIdx.x], smax[threadIdx.x + w], skey[threadIdx.x + w]);
      ssum[threadIdx.x] += ssum[threadIdx.x + w];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    part[3 * blockIdx.x + 0] = smax[0];
    part[3 * blockIdx.x + 1] = (double)skey[0];
    part[3 * blockIdx.x + 2] = ssum[0];
  }
}

__global__ void __launch_bounds__(NB_TPB) k_norms_final(const Dev P, const double* part, int nb, double* out3) {
  __shared__ double smax[NB_TPB], ssum[NB_TPB];
  __shared__ long long skey[NB_TPB];
  double vmax = 0.0, vsum = 0.0;
  long long vkey = 0x7fffffffffffffffLL;
  for (int i = threadIdx.x; i < nb; i += NB_TPB) {
    better(vmax, vkey, part[3 * i], (long long)part[3 * i + 1]);
    vsum += part[3 * i + 2];
  }
  smax[threadIdx.x] = vmax;
  skey[threadIdx.x] = vkey;
  ssum[threadIdx.x] = vsum;
  __syncthreads();
  for (int w = NB_TPB / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) {
      better(smax[threadIdx.x], skey[threadIdx.x], smax[threadIdx.x + w], skey[threadIdx.x + w]);
      ssum[threadIdx.x] += ssum[threadIdx.x + w];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    out3[0] = smax[0];
    out3[1] = smax[0] > 0.0 ? (double)skey[0] : 0.0;
    out3[2] = sqrt(ssum[0] / (1.0 * P.nx * P.ny * P.nz));
  }
}

unsigned pointwise_blocks(const Dev& P) {
  long long rows = (long long)P.ny * P.nz;
  long long b = (rows + TPB / 32 - 1) / (TPB / 32);
  long long cap = (long long)P.sweep_blocks * 32;
  return (unsigned)(b < cap ? b : cap);
}

// Whether the sweep of direction d of a step writes the face lines: the
// Douglas-ADI y solve and the TS y and x solves keep them.
bool sweep_faces(int method, int d) { return method == 0 ? d != 1 : method == 3 ? d == 2 : true; }

template <int D, int KIND, int NL, int NT>
void sweep_shape(const Dev& P, const SweepIO& io, cudaStream_t st) {
  const int nd = D == 0 ? P.nx : D == 1 ? P.ny : P.nz;
  k_line<D, KIND, NL, NT>
      <<<line_grid<D>(P, NL, sweep_faces(P.method, D)), NT, tile_smem<D, NL>(nd), st>>>(P, io);
}

// One sweep in the shape selected for it (Dev::shape).
template <int D, int KIND>
void sweep(const Dev& P, const RingData& R, const SweepIO& io, int shape, cudaStream_t st) {
  switch (shape) {
#define MTS_CASE(id, nl, nt)                    \
  case id:                                      \
    sweep_shape<D, KIND, nl, nt>(P, io, st);    \
    break;
    MTS_SHAPES(MTS_CASE)
#undef MTS_CASE
    default:
      // a ring, where its data could be built
      if (KIND != K_ADI && R.rblk[D])
        launch_ring_sweep(P, R, D, KIND, io, shape - kTileShapes, st);
      else
        sweep<D, KIND>(P, R, io, tile_shape_default(D, D == 0 ? P.nx : D == 1 ? P.ny : P.nz, KIND == K_ADI), st);
  }
}

template <int NL, int NT>
cudaError_t allow_tiles() {
  return allow_smem(kMaxTileSmem, {(const void*)k_line<0, K_COPY, NL, NT>, (const void*)k_line<1, K_COPY, NL, NT>,
                                   (const void*)k_line<2, K_COPY, NL, NT>, (const void*)k_line<0, K_STENCIL, NL, NT>,
                                   (const void*)k_line<1, K_STENCIL, NL, NT>, (const void*)k_line<2, K_STENCIL, NL, NT>,
                                   (const void*)k_line<0, K_ADI, NL, NT>, (const void*)k_line<2, K_TS_Z, NL, NT>});
}

}  // namespace

int sweep_shape_count() { return kTileShapes + kRingShapes; }

// TS runs its implicit sweeps z, y, x, the others x, y, z.
int sweep_direction(int method, int sweep) { return method == 3 ? 2 - sweep : sweep; }

bool sweep_shape_fits(int shape, int d, int n) {
  switch (shape) {
#define MTS_FITS(id, nl, nt) \
  case id:                   \
    return n <= kMaxLineRows && (d == 0 ? tile_smem<0, nl>(n) : tile_smem<1, nl>(n)) <= (size_t)kMaxTileSmem;
    MTS_SHAPES(MTS_FITS)
#undef MTS_FITS
    default:
      return n <= kMaxLineRows && ring_fits(shape - kTileShapes, n);
  }
}

// Lines that an SM solves at once with tiles of a shape (0: too long for it).
template <int NL, int NT>
int lines_at_once(int d, int n, bool adi_x) {
  const size_t bytes = d == 0 ? tile_smem<0, NL>(n) : tile_smem<1, NL>(n);
  if (n > kMaxLineRows || bytes > (size_t)kMaxTileSmem) return 0;
  const int regs = adi_x ? line_min_ctas<K_ADI, NT>() : line_min_ctas<K_COPY, NT>();
  return NL * (int)std::min<size_t>(regs, (228 * 1024) / (bytes + 1024 + sizeof(TileState<NL>)));
}

// The tile with the most lines on an SM at once, the narrower of two with as
// many (more tiles overlap their loads).  32 lines up to 258 (x) and 243 rows
// (y, z), then 16 lines, then 32 again where two 32-line tiles beat three
// 16-line ones, and so on.  B200, us per sweep with 32 / 16 lines: LOD-CN x,
// 241 rows 148 / 160, 289 rows 300 / 264, 385 rows 698 / 730, 449 rows 1928 /
// 1157; Douglas-ADI y, 193 rows 84 / 92, 257 rows 226 / 197, 513 rows 2842 /
// 2185.
int tile_shape_default(int d, int n, bool adi_x) {
  const int id[4] = {0, 3, 6, 8};
  const int lines[4] = {lines_at_once<32, 256>(d, n, adi_x), lines_at_once<16, 256>(d, n, adi_x),
                        lines_at_once<8, 128>(d, n, adi_x), lines_at_once<4, 128>(d, n, adi_x)};
  int k = 0;
  for (int i = 1; i < 4; i++)
    if (lines[i] >= lines[k]) k = i;
  return lines[k] > 0 ? id[k] : -1;
}

// Tiles or a ring (ring.cu).  A ring has as many lines on the chain as its CTA
// has threads, whatever their length, but waits for global memory on every
// step of it and fills an SM with few lines poorly: it pays where an SM has
// much to do (w: nodes per SM) in long lines, or very many short ones.  The
// lines lie where the two measured equal (B200, 70 grids of 17 to 1600 rows an
// axis); us per sweep, tiles / ring:
//   x, LOD-IE                 353^3 465 / 508, 385^3 727 / 620, 449^3 1139 / 955
//   x, Douglas-ADI, with its first right-hand side (a pass of its own before a
//   ring)                     321^3 500 / 553, 385 x 298 x 384 689 / 744, 449^3 1468 / 1414
//   y, z                      ADI y 225^3 142 / 136, 257^3 197 / 190, 385^3 738 / 515;
//                             LOD-IE y (copied) 249^3 142 / 155, 273^3 201 / 190
//   z of LOD (adds the source on the way out, row by row in a ring)
//                             LOD-CN 345 x 254 x 352 468 / 548, 353^3 652 / 593, 385^3 878
//                             / 815, 220 x 260 x 640 770 / 642
//   33 x 700 x 700 x, TS      209 / 169; 500 x 33 x 500 y, ADI 115 / 98
int sweep_shape_default(int method, int d, int n, long long lines, int sms) {
  const double per_sm = (double)lines / sms, w = per_sm * n;
  bool ring;
  if (d == 0)
    ring = (n >= (method == MTS_ADI ? 420 : 360) && w >= 110e3) ||
           (method != MTS_ADI && n <= 50 && per_sm >= 1500);
  else if (d == 2 && (method == MTS_LOD_IE || method == MTS_LOD_CN))
    ring = (n >= 340 && w >= 280e3) || (n >= 600 && w >= 210e3) || (n <= 50 && per_sm >= 1500);
  else if (method == MTS_LOD_IE || (method == MTS_TS && d == 1))
    ring = (n >= 150 && w >= 110e3) || (n <= 82 && per_sm >= 1000);
  else
    ring = (n >= 150 && w >= 100e3) || per_sm >= 1000;
  const int k = ring ? ring_default(method, d, n, per_sm) : -1;
  return k >= 0 && n <= kMaxLineRows ? kTileShapes + k : tile_shape_default(d, n, method == MTS_ADI && d == 0);
}

cudaError_t configure_shape(int shape) {
  switch (shape) {
#define MTS_ALLOW(id, nl, nt) \
  case id:                    \
    return allow_tiles<nl, nt>();
    MTS_SHAPES(MTS_ALLOW)
#undef MTS_ALLOW
    default:
      return configure_ring(shape - kTileShapes);
  }
}

__global__ void k_tick(int* step) { ++*step; }

void launch_tick(const Dev& P, cudaStream_t st) { k_tick<<<1, 1, 0, st>>>(P.tstep); }

unsigned pointwise_rows_grid(const Dev& P) { return pointwise_blocks(P); }

int launch_factor_lines(const Dev& P, int* flags, cudaStream_t st) {
  int launches = 0;
  if (P.mibref && P.nmibnode > 0) {
    k_mibref<<<(P.nmibnode + TPB - 1) / TPB, TPB, 0, st>>>(P);
    launches++;
  }
  if (P.nfcross[0] > 0) {
    k_factor_lines<0><<<(P.nfcross[0] + TPB - 1) / TPB, TPB, 0, st>>>(P, flags);
    launches++;
  }
  if (P.nfcross[1] > 0) {
    k_factor_lines<1><<<(P.nfcross[1] + TPB - 1) / TPB, TPB, 0, st>>>(P, flags);
    launches++;
  }
  if (P.nfcross[2] > 0) {
    k_factor_lines<2><<<(P.nfcross[2] + TPB - 1) / TPB, TPB, 0, st>>>(P, flags);
    launches++;
  }
  return launches;
}

int launch_initialize(const Dev& P, double E, double* u, cudaStream_t st) {
  k_init<<<pointwise_blocks(P), TPB, 0, st>>>(P, E, u);
  return 1;
}

int norms_blocks(const Dev& P) {
  long long nb = (P.nn + NB_TPB * 8 - 1) / (NB_TPB * 8);
  if (nb > 4096) nb = 4096;
  if (nb < 1) nb = 1;
  return (int)nb;
}

int launch_norms(const Dev& P, double E, const double* u, double* partial, int nb, double* out3, cudaStream_t st) {
  k_norms_partial<<<nb, NB_TPB, 0, st>>>(P, E, u, partial);
  k_norms_final<<<1, NB_TPB, 0, st>>>(P, partial, nb, out3);
  return 2;
}

// One time step.  u0 holds u^n on entry and u^{n+1} on return; u1 is scratch.
int launch_step(const Dev& P, const RingData& R, const StepTimes& T, double* u0, double* u1, cudaStream_t st,
                cudaEvent_t* ev, const SideStream* side) {
  int launches = 0;
  int slot = 0;
  auto mark = [&](int k) {
    if (ev) cudaEventRecord(ev[2 * slot + k], st);
    if (k == 1) slot++;
  };
  // (slot 0, once the jump pass: the kernels evaluate the jumps they use)
  mark(0);
  mark(1);
  SweepIO io{};
  io.e1 = T.e_next;
  io.e0 = T.e_prev;
  if (P.method == 0) {
    // Douglas-ADI.  The x sweep forms uhs of its lines from u0 and solves it
    // into u1 (u*); the y sweep builds uhss = -dt D_yy u^n + u* and solves in
    // place (u**); the z sweep builds uh1 = -dt D_zz u^n + u** and writes
    // u^{n+1} over u^n in u0 (a z line reads only its own nodes of u^n).  The
    // faces get Outer_u(t_next) in u1 and in u0.  The state stays in u0, u1
    // is scratch.  Before an x ring sweep uhs is formed in u1 by passes of its
    // own, the MIB rows on the side stream beside the others (they write
    // disjoint nodes and read only u0).
    const bool ring_x = P.shape[0] >= kTileShapes && R.rblk[0];
    const bool fork = ring_x && side && side->stream && P.nmibnode > 0;
    cudaStream_t sst = fork ? side->stream : st;
    mark(0);
    if (fork) {
      cudaEventRecord(side->fork, st);
      cudaStreamWaitEvent(sst, side->fork, 0);
    }
    if (P.nmibnode > 0) {
      k_adi_mib<<<mib_nodes_grid(P), TPB, 0, sst>>>(P, u0, u1, T.e_next);
      launches++;
    }
    if (ring_x) {
      launch_adi_rhs(P, u0, u1, T.e_next, st);
      launches++;
    }
    if (fork) {
      cudaEventRecord(side->join, sst);
      cudaStreamWaitEvent(st, side->join, 0);
    }
    mark(1);
    io.stin = u0;
    io.add = u0;
    io.out = u1;
    io.jumps = 0;
    io.bmode = 1;
    mark(0);
    if (ring_x) {
      io.stin = u1;
      io.add = u1;
      io.bmode = 0;
      sweep<0, K_COPY>(P, R, io, P.shape[0], st);
      io.stin = u0;
    } else {
      sweep<0, K_ADI>(P, R, io, P.shape[0], st);
    }
    mark(1);
    io.add = u1;
    io.bmode = 0;
    io.k = -P.dt;
    mark(0);
    sweep<1, K_STENCIL>(P, R, io, P.shape[1], st);
    mark(1);
    io.out = u0;
    io.bmode = 1;
    mark(0);
    sweep<2, K_STENCIL>(P, R, io, P.shape[2], st);
    mark(1);
    launches += 3;
  } else if (P.method == 1 || P.method == 2) {
    // LOD, in place on u0.
    io.jumps = 1;
    io.k = P.kex;
    io.stin = u0;
    io.add = u0;
    io.out = u0;
    io.bmode = 1;
    mark(0);
    if (P.method == 2)
      sweep<0, K_STENCIL>(P, R, io, P.shape[0], st);
    else
      sweep<0, K_COPY>(P, R, io, P.shape[0], st);
    mark(1);
    mark(0);
    if (P.method == 2)
      sweep<1, K_STENCIL>(P, R, io, P.shape[1], st);
    else
      sweep<1, K_COPY>(P, R, io, P.shape[1], st);
    mark(1);
    io.last = 1;
    io.bmode = 2;
    mark(0);
    if (P.method == 2)
      sweep<2, K_STENCIL>(P, R, io, P.shape[2], st);
    else
      sweep<2, K_COPY>(P, R, io, P.shape[2], st);
    mark(1);
    launches += 3;
  } else {
    // TS: explicit x (u0 -> u1) and y (u1 -> u0) half steps, fused explicit
    // z + sources + implicit z in place on u0, then implicit y and x in place.
    const unsigned rows = pointwise_blocks(P) + mib_ctas(P);
    mark(0);
    k_ts_explicit<0><<<rows, TPB, 0, st>>>(P, u0, u1, T.e_half, T.e_next);
    mark(1);
    mark(0);
    k_ts_explicit<1><<<rows, TPB, 0, st>>>(P, u1, u0, T.e_half, T.e_next);
    mark(1);
    io.jumps = 1;
    io.k = P.kex;
    io.stin = u0;
    io.add = u0;
    io.out = u0;
    io.bmode = 1;
    mark(0);
    sweep<2, K_TS_Z>(P, R, io, P.shape[0], st);
    mark(1);
    io.bmode = 0;
    mark(0);
    sweep<1, K_COPY>(P, R, io, P.shape[1], st);
    mark(1);
    mark(0);
    sweep<0, K_COPY>(P, R, io, P.shape[2], st);
    mark(1);
    launches += 5;
  }
  return launches;
}

// ---------------------------------------------------------------------------
// Error norms with no allocation (mts_norms_noalloc).  A caller that cannot
// allocate device memory still needs somewhere for the per-block partials of
// the reduction, so they live in one statically sized module array instead
// of a buffer owned by a handle.  Layout, in doubles:
//   [0]        ticket counter (read as unsigned): MUST be zero when the
//              kernel starts; the host clears it before each launch and the
//              last block leaves it at zero
//   [32..34]   the result triple (max |e|, argmax key, L2)
//   [64 ..)    3 doubles of partials per block, kNoAllocMaxBlocks blocks
// Every call on a device uses the same array, so calls that overlap in time
// on one device (two handles, two streams, two host threads) race.

static __device__ __align__(256) double g_noalloc_scratch[kNoAllocScratchDoubles];

cudaError_t noalloc_scratch_address(double** p) { return cudaGetSymbolAddress((void**)p, g_noalloc_scratch); }

namespace {

// One launch: each block reduces its share exactly as k_norms_partial does;
// the block that takes the last ticket then combines the partials exactly as
// k_norms_final does, so the triple is bit-identical to launch_norms' with
// the same block count.
__global__ void __launch_bounds__(NB_TPB) k_norms_noalloc(const Dev P, double E, const double* u, double* scratch) {
  __shared__ double smax[NB_TPB], ssum[NB_TPB];
  __shared__ long long skey[NB_TPB];
  __shared__ int last;
  unsigned* const ticket = reinterpret_cast<unsigned*>(scratch);
  double* const res = scratch + 32;
  double* const part = scratch + 64;
  double vmax = 0.0, vsum = 0.0;
  long long vkey = 0x7fffffffffffffffLL;
  for (long long m = (long long)blockIdx.x * NB_TPB + threadIdx.x; m < P.nn; m += (long long)gridDim.x * NB_TPB) {
    int ix, iy, iz;
    node_xyz(P, m, ix, iy, iz);
    double ex = (P.tag[m] & TAG_OUT) ? outer_u(P, E, ix, iy, iz) : inner_u(P, E, ix, iy, iz);
    double e = fabs(u[m] - ex);
    long long key = ((long long)ix * P.ny + iy) * P.nz + iz;
    better(vmax, vkey, e, key);
    vsum += e * e;
  }
  smax[threadIdx.x] = vmax;
  skey[threadIdx.x] = vkey;
  ssum[threadIdx.x] = vsum;
  __syncthreads();
  for (int w = NB_TPB / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) {
      better(smax[threadIdx.x], skey[threadIdx.x], smax[threadIdx.x + w], skey[threadIdx.x + w]);
      ssum[threadIdx.x] += ssum[threadIdx.x + w];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    part[3 * blockIdx.x + 0] = smax[0];
    part[3 * blockIdx.x + 1] = (double)skey[0];
    part[3 * blockIdx.x + 2] = ssum[0];
    __threadfence();  // the partial is visible device-wide before the ticket
    last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  const int nb = gridDim.x;
  vmax = 0.0;
  vsum = 0.0;
  vkey = 0x7fffffffffffffffLL;
  for (int i = threadIdx.x; i < nb; i += NB_TPB) {
    // other blocks wrote these: read through L2, past this SM's L1
    better(vmax, vkey, __ldcg(part + 3 * i), (long long)__ldcg(part + 3 * i + 1));
    vsum += __ldcg(part + 3 * i + 2);
  }
  smax[threadIdx.x] = vmax;
  skey[threadIdx.x] = vkey;
  ssum[threadIdx.x] = vsum;
  __syncthreads();
  for (int w = NB_TPB / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) {
      better(smax[threadIdx.x], skey[threadIdx.x], smax[threadIdx.x + w], skey[threadIdx.x + w]);
      ssum[threadIdx.x] += ssum[threadIdx.x + w];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    res[0] = smax[0];
    res[1] = smax[0] > 0.0 ? (double)skey[0] : 0.0;
    res[2] = sqrt(ssum[0] / (1.0 * P.nx * P.ny * P.nz));
    *ticket = 0u;
  }
}

}  // namespace

int launch_norms_noalloc(const Dev& P, double E, const double* u, double* scratch, int nb, cudaStream_t st) {
  k_norms_noalloc<<<nb, NB_TPB, 0, st>>>(P, E, u, scratch);
  return 1;
}

// ---------------------------------------------------------------------------
// Batched plain steps: the kernels above, launched once for many problems.

namespace {

struct Roles {
  int stin, add, out;  // fields: 0 = u0, 1 = u1
  int ksel;            // explicit factor: 0 none, 1 -dt (ADI), 2 0.5*dt (LOD-CN, TS)
  int jumps, bmode, last;
};

__device__ __forceinline__ SweepIO make_io(const Dev& P, const Roles& r) {
  SweepIO io{};
  io.stin = r.stin ? P.u1 : P.u0;
  io.add = r.add ? P.u1 : P.u0;
  io.out = r.out ? P.u1 : P.u0;
  io.k = r.ksel == 1 ? -P.dt : r.ksel == 2 ? P.kex : 0.0;
  io.jumps = r.jumps;
  io.bmode = r.bmode;
  io.last = r.last;
  io.e0 = io.e1 = 0.0;  // from the step table
  return io;
}

__global__ void __launch_bounds__(TPB) kb_adi_mib(const Dev* __restrict__ Ps, const BatchItem* __restrict__ items) {
  BATCH_PROLOGUE
  k_adi_mib_body(P, w.cta, w.ncta, P.u0, P.u1, 0.0);
}

template <int D>
__global__ void __launch_bounds__(TPB) kb_ts_explicit(const Dev* __restrict__ Ps,
                                                      const BatchItem* __restrict__ items, int in) {
  BATCH_PROLOGUE
  k_ts_explicit_body<D>(P, w.cta, w.ncta, in ? P.u1 : P.u0, in ? P.u0 : P.u1, 0.0, 0.0);
}

template <int D, int KIND, int BNL, int BNT>
__global__ void __launch_bounds__(BNT, line_min_ctas<KIND, BNT>()) kb_line(const Dev* __restrict__ Ps,
                                                                           const BatchItem* __restrict__ items,
                                                                           Roles r) {
  BATCH_PROLOGUE
  __shared__ SweepIO io;
  if (threadIdx.x == 0) io = make_io(P, r);
  __syncthreads();
  k_line_body<D, KIND, BNL, BNT>(P, w.cta, w.ncta, io);
}

__global__ void kb_tick(const Dev* __restrict__ Ps, int n) {
  const int i = blockIdx.x * TPB + threadIdx.x;
  if (i < n && *Ps[i].tstep < Ps[i].tstop) ++*Ps[i].tstep;
}

// Lines per tile and threads per CTA of the batched sweeps (batch_tile).
#define MTS_BATCH_TILES(X) X(0, 32, 128) X(1, 16, 256)

template <int D, int KIND>
void bsweep(const BatchPlan& b, const Roles& r, cudaStream_t st, int& launches) {
  if (b.nsw[D] == 0) return;
  switch (b.tile[D]) {
#define MTS_CASE(id, nl, nt)                                                                            \
  case id:                                                                                              \
    kb_line<D, KIND, nl, nt><<<b.nsw[D], nt, tile_smem<D, nl>(b.nmax[D]), st>>>(b.Ps, b.sw[D], r);      \
    break;
    MTS_BATCH_TILES(MTS_CASE)
#undef MTS_CASE
  }
  launches++;
}

template <int NL, int NT>
cudaError_t allow_batch_tiles() {
  return allow_smem(kMaxBatchTileSmem,
                    {(const void*)kb_line<0, K_COPY, NL, NT>, (const void*)kb_line<1, K_COPY, NL, NT>,
                     (const void*)kb_line<2, K_COPY, NL, NT>, (const void*)kb_line<0, K_STENCIL, NL, NT>,
                     (const void*)kb_line<1, K_STENCIL, NL, NT>, (const void*)kb_line<2, K_STENCIL, NL, NT>,
                     (const void*)kb_line<0, K_ADI, NL, NT>, (const void*)kb_line<2, K_TS_Z, NL, NT>});
}

}  // namespace

int batch_tile(int d, int n) {
  auto fits = [&](size_t x, size_t yz, int limit) { return (d == 0 ? x : yz) <= (size_t)limit; };
  if (fits(tile_smem<0, 32>(n), tile_smem<1, 32>(n), kBatchTileSmem)) return 0;
  return fits(tile_smem<0, 16>(n), tile_smem<1, 16>(n), kMaxBatchTileSmem) ? 1 : -1;
}

// Problems whose lines all fit three 32-line tiles to an SM (232 rows) always
// batch.  Of the others a solo step costs 14 to 19 us of launches, and the
// batched tiles take about as long for 200 thousand nodes (100 thousand for
// TS with long y or z lines, whose z sweep spills; 260 thousand for ADI and TS
// with long x lines alone): the smaller ones batch, in launches of their own.
// B200, us per step of 64 problems, solo / batched: 17 x 17 x 300 ADI 1018 /
// 598, 300 x 17 x 17 TS 1227 / 609, 9 x 1500 x 9 LOD-CN 1646 / 1220, 780 x 17 x
// 17 ADI 1753 / 1502; 33 x 33 x 240 TS 1306 / 1771, 25 x 25 x 500 ADI 1353 /
// 1511, 780 x 17 x 17 LOD-CN 1291 / 1423.
int batch_class(const Dev& P) {
  const int t[3] = {batch_tile(0, P.nx), batch_tile(1, P.ny), batch_tile(2, P.nz)};
  if (std::min(t[0], std::min(t[1], t[2])) < 0) return -1;
  if (std::max(t[0], std::max(t[1], t[2])) == 0) return 0;
  const bool yz = t[1] > 0 || t[2] > 0, lod = P.method == MTS_LOD_IE || P.method == MTS_LOD_CN;
  const long long most = yz && P.method == MTS_TS ? 100000 : yz || lod ? 200000 : 260000;
  return P.nn <= most ? 1 : -1;
}

int launch_batch_tick(const Dev* Ps, int n, cudaStream_t st) {
  kb_tick<<<(n + TPB - 1) / TPB, TPB, 0, st>>>(Ps, n);
  return 1;
}

unsigned mib_grid(const Dev& P) { return mib_nodes_grid(P); }
unsigned block_grid(const Dev& P, int d) { return (unsigned)((P.nblk[d] + TPB - 1) / TPB); }
unsigned ts_explicit_grid(const Dev& P) { return pointwise_blocks(P) + mib_ctas(P); }
unsigned batch_sweep_grid(const Dev& P, int tile, int d) {
  const int nl = tile == 0 ? 32 : 16;
  const bool faces = sweep_faces(P.method, d);
  return d == 0 ? line_grid<0>(P, nl, faces) : d == 1 ? line_grid<1>(P, nl, faces) : line_grid<2>(P, nl, faces);
}

cudaError_t configure_batch(int tile) { return tile == 0 ? allow_batch_tiles<32, 128>() : allow_batch_tiles<16, 256>(); }

// One step of every problem of the plan, the launch sequence of launch_step.
int launch_step_batch(const BatchPlan& b, cudaStream_t st) {
  int launches = 0;
  if (b.method == 0) {
    if (b.nmib > 0) {
      kb_adi_mib<<<b.nmib, TPB, 0, st>>>(b.Ps, b.mib);
      launches++;
    }
    bsweep<0, K_ADI>(b, Roles{0, 0, 1, 0, 0, 1, 0}, st, launches);
    bsweep<1, K_STENCIL>(b, Roles{0, 1, 1, 1, 0, 0, 0}, st, launches);
    bsweep<2, K_STENCIL>(b, Roles{0, 1, 0, 1, 0, 1, 0}, st, launches);
  } else if (b.method == 1 || b.method == 2) {
    if (b.method == 2) {
      bsweep<0, K_STENCIL>(b, Roles{0, 0, 0, 2, 1, 1, 0}, st, launches);
      bsweep<1, K_STENCIL>(b, Roles{0, 0, 0, 2, 1, 1, 0}, st, launches);
      bsweep<2, K_STENCIL>(b, Roles{0, 0, 0, 2, 1, 2, 1}, st, launches);
    } else {
      bsweep<0, K_COPY>(b, Roles{0, 0, 0, 2, 1, 1, 0}, st, launches);
      bsweep<1, K_COPY>(b, Roles{0, 0, 0, 2, 1, 1, 0}, st, launches);
      bsweep<2, K_COPY>(b, Roles{0, 0, 0, 2, 1, 2, 1}, st, launches);
    }
  } else {
    kb_ts_explicit<0><<<b.nrows, TPB, 0, st>>>(b.Ps, b.rows, 0);
    kb_ts_explicit<1><<<b.nrows, TPB, 0, st>>>(b.Ps, b.rows, 1);
    launches += 2;
    bsweep<2, K_TS_Z>(b, Roles{0, 0, 0, 2, 1, 1, 0}, st, launches);
    bsweep<1, K_COPY>(b, Roles{0, 0, 0, 2, 1, 0, 0}, st, launches);
    bsweep<0, K_COPY>(b, Roles{0, 0, 0, 2, 1, 0, 0}, st, launches);
  }
  kb_tick<<<(b.n + TPB - 1) / TPB, TPB, 0, st>>>(b.Ps, b.n);
  return launches + 1;
}

}  // namespace mts
