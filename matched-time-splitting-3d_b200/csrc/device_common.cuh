// Device helpers shared by the plain FP64 kernels (kernels.cu) and the mixed
// precision kernels (mixed.cu): the exact solutions, line geometry, cp.async
// staging, the MIB row sums and the Convert2Tri row operations.
#pragma once

#include <cuda_runtime.h>

#include <initializer_list>

#include "device.h"

namespace mts {
namespace {

constexpr int TPB = 128;                // pointwise kernels and small kernels
constexpr int kMaxSweepSmem = 232448;  // 227 KB: the sm_100 per-CTA limit
constexpr int kMaxTileSmem = kMaxSweepSmem - 1024;  // the line tiles keep a few words of static shared memory too
// The longest line the bit-exact form takes: what its smallest ring holds (3 x
// 16 rows of 132 doubles and 7 doubles a row of the line in 227 KB; 4-line
// tiles hold 3616).
constexpr int kMaxLineRows = 3245;
// The batched line tiles, with their problem's record beside them in static
// shared memory: three to an SM, and at all.
constexpr int kBatchTileSmem = 70 * 1024;
constexpr int kMaxBatchTileSmem = kMaxSweepSmem - 3 * 1024;

// ---------------------------------------------------------------------------
// Exact solutions (eq 0: src/equation/eq_0.cc; eq 8: see oracle/ref_harness.cc
// Eq8 for the operand order).

__device__ __forceinline__ double outer_u(const Dev& P, double E, int ix, int iy, int iz) {
  if (P.eq == 0) return 100.0;
  double x = P.ax[0][ix], y = P.ax[1][iy], z = P.ax[2][iz];
  return ((x * x + y * y) + z * z) * E;
}
__device__ __forceinline__ double inner_u(const Dev& P, double E, int ix, int iy, int iz) {
  if (P.eq == 0) return 80.0;
  return ((P.s2[0][ix] * P.c2[1][iy]) * P.s2[2][iz]) * E;
}
__device__ __forceinline__ double source(const Dev& P, double E, int out, int ix, int iy, int iz) {
  if (P.eq == 0) return 0.0;
  if (out) return -outer_u(P, E, ix, iy, iz) - P.c6bo * E;
  return P.kin * inner_u(P, E, ix, iy, iz);
}

// Lets each kernel have `bytes` of dynamic shared memory on the current device.
inline cudaError_t allow_smem(int bytes, std::initializer_list<const void*> kernels) {
  for (const void* k : kernels) {
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// CTAs of a persistent line sweep: one per SM at most, no more than nl lines
// of nt threads need.
inline unsigned sweep_grid(const Dev& P, long long nl, int nt) {
  const long long b = (nl + nt - 1) / nt;
  return (unsigned)(b < P.sweep_blocks ? (b > 0 ? b : 1) : P.sweep_blocks);
}

// The step's time factor k (0: exp(-t_prev), 1: exp(-t_half), 2: exp(-t_next)):
// the launch argument, or the step table of a replayed graph.
__device__ __forceinline__ double step_e(const Dev& P, double given, int k) {
  return P.tsched ? P.tsched[3 * (*P.tstep) + k] : given;
}

// The exact jumps at crossing q for time factor E: [u] (Equation::Jump_u) and
// [beta u_x], [beta u_y], [beta u_z] (the Eq's Jump_betau_x/y/z), with the
// operations of src/equation/eq_0.cc and of the measured problem in their
// order.
__device__ __forceinline__ void exact_jumps(const Dev& P, const CrossConst& q, double E, double& ju, double jb[3]) {
  if (P.eq == 0) {
    ju = 100.0 - 80.0;
    for (int d = 0; d < 3; d++) jb[d] = P.bi * 0.0 - P.bo * 0.0;
  } else {
    ju = q.R2 * E - q.S * E;
    const double xyz[3] = {q.x, q.y, q.z};
    for (int d = 0; d < 3; d++) jb[d] = P.bo * ((2.0 * xyz[d]) * E) - P.bi * (q.D[d] * E);
  }
}

// Jump data of crossing c (Refresh_Jump, intersection.cc:2294-2490): [u] and
// u_dir at the step's exp(-t).
__device__ __forceinline__ double2 jump_at(const Dev& P, int c, double E) {
  const CrossConst& q = P.cc[c];
  double ju, jb[3];
  exact_jumps(P, q, E, ju, jb);
  const double bxi = q.p[0] * jb[0] + q.p[1] * jb[1] + q.p[2] * jb[2];
  return make_double2(ju, q.pinv * bxi);
}

// ---------------------------------------------------------------------------
// Line geometry.  Direction D lines are indexed (i1, i2) as in the reference
// (src/constant.h:83-89): x -> (iy, iz), y -> (ix, iz), z -> (ix, iy); the
// line number runs over i1 fastest.

struct Line {
  long long base, s;
  int n, lid, i1, i2;
  bool boundary;
};

template <int D>
__host__ __device__ __forceinline__ long long nlines(const Dev& P) {
  int n1 = D == 0 ? P.ny : P.nx;
  int n2 = D == 2 ? P.ny : P.nz;
  return (long long)n1 * n2;
}

template <int D>
__device__ __forceinline__ void decode_line(const Dev& P, long long t, Line& L) {
  int n1 = D == 0 ? P.ny : P.nx;
  int n2 = D == 2 ? P.ny : P.nz;
  // a direction has n1*n2 < 2^31 lines: 32-bit division
  L.i1 = (int)t % n1;
  L.i2 = (int)t / n1;
  L.lid = L.i1 * n2 + L.i2;
  if (D == 0) {
    L.base = (long long)P.nx * (L.i1 + (long long)P.ny * L.i2);
    L.s = 1;
    L.n = P.nx;
  } else if (D == 1) {
    L.base = L.i1 + (long long)P.nx * P.ny * L.i2;
    L.s = P.nx;
    L.n = P.ny;
  } else {
    L.base = L.i1 + (long long)P.nx * L.i2;
    L.s = (long long)P.nx * P.ny;
    L.n = P.nz;
  }
  L.boundary = L.i1 == 0 || L.i1 == n1 - 1 || L.i2 == 0 || L.i2 == n2 - 1;
}

template <int D>
__device__ __forceinline__ void node_of(const Line& L, int j, int& ix, int& iy, int& iz) {
  if (D == 0) {
    ix = j;
    iy = L.i1;
    iz = L.i2;
  } else if (D == 1) {
    ix = L.i1;
    iy = j;
    iz = L.i2;
  } else {
    ix = L.i1;
    iy = L.i2;
    iz = j;
  }
}

__device__ __forceinline__ void node_xyz(const Dev& P, long long m, int& ix, int& iy, int& iz) {
  ix = (int)(m % P.nx);
  long long q = m / P.nx;
  iy = (int)(q % P.ny);
  iz = (int)(q / P.ny);
}

// ---------------------------------------------------------------------------
// cp.async (8-byte, L1-allocating) staging

__device__ __forceinline__ void cp_async8(double* smem_dst, const double* gsrc) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// ---------------------------------------------------------------------------
// MIB rows

__device__ __forceinline__ double corner_jumps(const double* w, double2 l, double2 r) {
  return l.x * w[5] + l.y * w[6] + r.x * w[7] + r.y * w[8];
}

// Explicit 3-point sum of row r of block b with fictitious points, before the
// dt factor: the MIB branches of douglas_adi.cc:112-210 (jumps = 0) and
// lod.cc:337-496 (jumps = 1).  U(j) returns the field at row j of the line.
// Jl, Jr: the jump data of the block's crossings (read when jumps).
template <class UF>
__device__ double mib_sum(const MibBlock& b, int r, UF U, const double* vd, bool jumps, double2 Jl, double2 Jr) {
  const int L = b.L;
  double sum = 0.0;
  if (b.kind == 2) {
    if (r == 0) {
      sum += vd[0] * U(L - 1);
      sum += vd[1] * U(L);
      for (int i = 0; i < 4; i++) sum += vd[2] * U(L - 1 + i) * b.w[1][i];
      if (jumps) sum += vd[2] * (Jl.x * b.w[1][4] + Jl.y * b.w[1][5]);
    } else {
      sum += vd[1] * U(L + 1);
      sum += vd[2] * U(L + 2);
      for (int i = 0; i < 4; i++) sum += vd[0] * U(L - 1 + i) * b.w[0][i];
      if (jumps) sum += vd[0] * (Jl.x * b.w[0][4] + Jl.y * b.w[0][5]);
    }
  } else {
    if (r == 0) {
      sum += vd[0] * U(L - 1);
      sum += vd[1] * U(L);
      for (int i = 0; i < 5; i++) sum += vd[2] * U(L - 1 + i) * b.w[1][i];
      if (jumps) sum += vd[2] * corner_jumps(b.w[1], Jl, Jr);
    } else if (r == 1) {
      for (int i = 0; i < 5; i++) sum += vd[0] * U(L - 1 + i) * b.w[0][i];
      if (jumps) sum += vd[0] * corner_jumps(b.w[0], Jl, Jr);
      sum += vd[1] * U(L + 1);
      for (int i = 0; i < 5; i++) sum += vd[2] * U(L - 1 + i) * b.w[3][i];
      if (jumps) sum += vd[2] * corner_jumps(b.w[3], Jl, Jr);
    } else {
      sum += vd[1] * U(L + 2);
      sum += vd[2] * U(L + 3);
      for (int i = 0; i < 5; i++) sum += vd[0] * U(L - 1 + i) * b.w[2][i];
      if (jumps) sum += vd[0] * corner_jumps(b.w[2], Jl, Jr);
    }
  }
  return sum;
}

// LOD/TS: jump terms on the right-hand side of the implicit MIB rows
// (D_xx_l, lod.cc:960-1097), then the Convert2Tri row operations.
__device__ __forceinline__ void implicit_rows(const Dev& P, const MibBlock& b, double* r,
                                              const double* vd0, const double* vd1, const double* vd2,
                                              bool jumps, double2 Jl, double2 Jr) {
  const double cdt = P.cdt;
  if (jumps) {
    if (b.kind == 2) {
      r[0] = r[0] + cdt * vd0[2] * (Jl.x * b.w[1][4] + Jl.y * b.w[1][5]);
      r[1] = r[1] + cdt * vd1[0] * (Jl.x * b.w[0][4] + Jl.y * b.w[0][5]);
    } else {
      r[0] = r[0] + cdt * vd0[2] * corner_jumps(b.w[1], Jl, Jr);
      r[1] = r[1] + cdt * vd1[0] * corner_jumps(b.w[0], Jl, Jr);
      r[1] += cdt * vd1[2] * corner_jumps(b.w[3], Jl, Jr);
      r[2] = r[2] + cdt * vd2[0] * corner_jumps(b.w[2], Jl, Jr);
    }
  }
  if (b.kind == 2) {
    r[1] -= b.rate[0] * r[0];
    r[0] -= b.rate[1] * r[1];
  } else {
    r[1] -= b.rate[0] * r[0];
    r[2] -= b.rate[1] * r[0];
    r[0] -= b.rate[2] * r[2];
    r[1] -= b.rate[3] * r[2];
    r[2] -= b.rate[4] * r[1];
    r[0] -= b.rate[5] * r[1];
  }
}

template <int DD>
__device__ __forceinline__ const MibBlock* find_block(const Dev& P, int lid, int j, int& row) {
  int be = P.bstart[DD][lid + 1];
  for (int k = P.bstart[DD][lid]; k < be; k++) {
    const MibBlock* b = &P.blk[DD][k];
    if (j >= b->L && j < b->L + b->kind) {
      row = j - b->L;
      return b;
    }
  }
  row = 0;
  return nullptr;
}

// Right-hand sides of block k's rows (K_COPY, K_STENCIL, K_TS_Z) from the
// fields, jump terms and Convert2Tri row operations included (the explicit MIB
// stencil of douglas_adi.cc:112-210 / lod.cc:337-496, the jump terms of D_xx_l
// lod.cc:960-1097).
template <int D, int KIND>
__device__ __forceinline__ void block_rhs(const Dev& P, const SweepIO& io, double E0, double E1, int k, long long base,
                                          int i1, int i2, double (&r)[3]) {
  const long long s = D == 0 ? 1 : D == 1 ? (long long)P.nx : (long long)P.nx * P.ny;
  const MibBlock& b = P.blk[D][k];
  double2 Jl = make_double2(0.0, 0.0), Jr = Jl;
  if (io.jumps) {
    Jl = jump_at(P, b.c0, E1);
    if (b.kind == 3) Jr = jump_at(P, b.c1, E1);
  }
  const double* const stin = KIND == K_COPY ? io.add : io.stin;
  auto U = [&](int j) { return stin[base + (long long)j * s]; };
  r[0] = r[1] = r[2] = 0.0;
  for (int q = 0; q < b.kind; q++) {
    const int jj = b.L + q;
    const int side = (b.sides >> q) & 1;
    const double av = io.add[base + (long long)jj * s];
    if (KIND == K_COPY) {
      r[q] = av;
    } else {
      const double sum = mib_sum(b, q, U, P.vd[D][side], io.jumps, Jl, Jr);
      double v = io.k * sum + av;
      if (KIND == K_TS_Z) {
        v = v + P.hdt * source(P, E0, side, i1, i2, jj);
        v = v + P.hdt * source(P, E1, side, i1, i2, jj);
      }
      r[q] = v;
    }
  }
  implicit_rows(P, b, r, P.vd[D][b.sides & 1], P.vd[D][(b.sides >> 1) & 1], P.vd[D][(b.sides >> 2) & 1], io.jumps,
                Jl, Jr);
}

// The Douglas-ADI data of a MIB node in one direction: the explicit sum of
// D_dd u there (the MIB sum of douglas_adi.cc:112-210 where the node is a row
// of a d block, else the three-point sum), and the jump terms that Src_2nd
// adds (douglas_adi.cc:1156-1427; nt of them, in their order).  ref: the
// node's block of that direction (Dev::mibref), -1: none.  Every load's
// address comes from ref alone, so they are in flight together.
struct MibDir {
  double sum, t0, t1;
  int nt;
};
__device__ __forceinline__ MibDir mib_direction(const Dev& P, const double* __restrict__ un, double E, long long m,
                                                int ref, int d, int side) {
  const long long s = d == 0 ? 1 : d == 1 ? (long long)P.nx : (long long)P.nx * P.ny;
  const double vd0 = P.vd[d][side][0], vd1 = P.vd[d][side][1], vd2 = P.vd[d][side][2];
  MibDir r;
  r.sum = 0.0;
  r.t0 = r.t1 = 0.0;
  r.nt = 0;
  if (ref < 0) {
    r.sum += un[m - s] * vd0;
    r.sum += un[m] * vd1;
    r.sum += un[m + s] * vd2;
    return r;
  }
  const MibBlock& b = (d == 0 ? P.blk[0] : d == 1 ? P.blk[1] : P.blk[2])[ref >> 4];
  const int kind = (ref >> 2) & 3, row = ref & 3;
  const double* const p = un + m - (row + 1) * s;  // row L-1
  double u[5], w[9];
  for (int i = 0; i < 4; i++) u[i] = p[i * s];
  u[4] = kind == 3 ? p[4 * s] : 0.0;
  // the fictitious value's weights: right of the first row, left of the others
  const double* const wp = b.w[row == 0 ? 1 : row == 1 ? 0 : 2];
  for (int i = 0; i < 9; i++) w[i] = wp[i];
  const double2 Jl = jump_at(P, b.c0, E);
  const double2 Jr = kind == 3 ? jump_at(P, b.c1, E) : Jl;
  const double vf = row == 0 ? vd2 : vd0;
  if (kind == 3 && row == 1) {
    for (int i = 0; i < 5; i++) r.sum += vf * u[i] * w[i];
    r.sum += vd1 * u[2];
    const double* const wq = b.w[3];
    for (int i = 0; i < 5; i++) r.sum += vd2 * u[i] * wq[i];
    r.t0 = vf * (Jl.x * w[5] + Jl.y * w[6] + Jr.x * w[7] + Jr.y * w[8]);
    r.t1 = vd2 * (Jl.x * wq[5] + Jl.y * wq[6] + Jr.x * wq[7] + Jr.y * wq[8]);
    r.nt = 2;
    return r;
  }
  r.sum += row == 0 ? vd0 * u[0] : vd1 * (kind == 2 ? u[2] : u[3]);
  r.sum += row == 0 ? vd1 * u[1] : vd2 * (kind == 2 ? u[3] : u[4]);
  for (int i = 0; i < 4; i++) r.sum += vf * u[i] * w[i];
  if (kind == 3) r.sum += vf * u[4] * w[4];
  r.t0 = kind == 2 ? vf * (Jl.x * w[4] + Jl.y * w[5]) : vf * (Jl.x * w[5] + Jl.y * w[6] + Jr.x * w[7] + Jr.y * w[8]);
  r.nt = 1;
  return r;
}

// The listed MIB nodes, shared out over nw warps (this one is w): three lanes
// a node, one per direction.  done(m, ix, iy, iz, sx, sy,
// sz, src) gets a node's three sums and its source with the jump terms.
template <class F>
__device__ __forceinline__ void mib_nodes(const Dev& P, const double* __restrict__ un, double E, int w, int nw,
                                          F done) {
  constexpr unsigned ALL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int d = lane % 3, g = lane / 3;
  for (int kb = 10 * w; kb < P.nmibnode; kb += 10 * nw) {
    const int k = kb + g;
    const bool act = g < 10 && k < P.nmibnode;
    MibDir r{0.0, 0.0, 0.0, 0};
    long long m = 0;
    int side = 0;
    if (act) {
      m = P.mibnode[k];
      const int ref = reinterpret_cast<const int*>(P.mibref)[4 * (long long)k + d];
      side = P.tag[m] & TAG_OUT;
      r = mib_direction(P, un, E, m, ref, d, side);
    }
    MibDir q[2];
    for (int e = 0; e < 2; e++) {
      q[e].sum = __shfl_down_sync(ALL, r.sum, e + 1);
      q[e].t0 = __shfl_down_sync(ALL, r.t0, e + 1);
      q[e].t1 = __shfl_down_sync(ALL, r.t1, e + 1);
      q[e].nt = __shfl_down_sync(ALL, r.nt, e + 1);
    }
    if (act && d == 0) {
      int ix, iy, iz;
      node_xyz(P, m, ix, iy, iz);
      double src = source(P, E, side, ix, iy, iz);
      if (r.nt > 0) src = src + r.t0;
      if (r.nt > 1) src = src + r.t1;
      for (int e = 0; e < 2; e++) {
        if (q[e].nt > 0) src = src + q[e].t0;
        if (q[e].nt > 1) src = src + q[e].t1;
      }
      done(m, ix, iy, iz, r.sum, q[0].sum, q[1].sum, src);
    }
  }
}

inline unsigned mib_nodes_grid(const Dev& P) { return (unsigned)((P.nmibnode + 10 * (TPB / 32) - 1) / (10 * (TPB / 32))); }

// Rows of the pointwise passes: a warp takes one x-row (iy, iz) at a time and
// covers it in groups of G x 32 nodes (ROW_G, or 2 for the five-load ADI
// RHS).  All loads of a group are issued before any of them is used, so each
// warp keeps G rows' worth of DRAM reads in flight; the exact-solution parts
// fixed along the row are computed once.
constexpr int ROW_G = 4;

struct RowExact {
  double y2, z2;   // y*y, z*z
  double c2y, s2z; // cos 2y, sin 2z
};
__device__ __forceinline__ RowExact row_exact(const Dev& P, int iy, int iz) {
  const double y = P.ax[1][iy], z = P.ax[2][iz];
  return {y * y, z * z, P.c2[1][iy], P.s2[2][iz]};
}
// outer_u and source in the operand order of outer_u / inner_u / source
__device__ __forceinline__ double row_outer(const Dev& P, const RowExact& q, int ix, double E) {
  if (P.eq == 0) return 100.0;
  const double x = P.ax[0][ix];
  return ((x * x + q.y2) + q.z2) * E;
}
__device__ __forceinline__ double row_source(const Dev& P, const RowExact& q, int ix, double E, int out) {
  if (P.eq == 0) return 0.0;
  if (out) return -row_outer(P, q, ix, E) - P.c6bo * E;
  return P.kin * (((P.s2[0][ix] * q.c2y) * q.s2z) * E);
}

template <bool B>
struct BoolC {
  static constexpr bool value = B;
};
template <int I>
struct IntC {
  static constexpr int value = I;
};

// The CTA's item and its problem's record, copied into shared memory.
#define BATCH_PROLOGUE                                                                \
  __shared__ __align__(16) long long sdev_[(sizeof(Dev) + 7) / 8];                    \
  const BatchItem w = items[blockIdx.x];                                              \
  {                                                                                   \
    const long long* src_ = reinterpret_cast<const long long*>(Ps + w.p);             \
    for (int i_ = threadIdx.x; i_ < (int)((sizeof(Dev) + 7) / 8); i_ += blockDim.x) \
      sdev_[i_] = src_[i_];                                                           \
  }                                                                                   \
  __syncthreads();                                                                    \
  const Dev& P = *reinterpret_cast<const Dev*>(sdev_);                                \
  if (*P.tstep >= P.tstop) return; /* this problem's steps of the batch are done */


}  // namespace
}  // namespace mts
