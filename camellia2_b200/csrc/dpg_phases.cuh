// dpg_phases.cuh — the phases of the per-cell assembly and their device helpers, shared by the
// kernels that walk cells with one CTA (assembly, work queue, reverse mode, energy error, DLS)
// and by the large-bucket kernel.  Each kernel family is a translation unit of its own.
#pragma once
#include "../../include/dpg_b200.h"
#include "dpg_internal.h"
#include "dpg_plan.h"

#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cstring>
#include <mutex>
#include <type_traits>
#include <vector>

// The CTA's dynamic shared memory; every shared pointer below is derived from it
// so the compiler keeps shared-space (LDS/STS) addressing inside the phase functions.
extern __shared__ __align__(128) double dpg_smem[];

namespace {

// Warps per CTA and CTAs per SM of this translation unit: 16 and one, or (DPG_CTA_WARPS defined) the
// small buckets' 8 and two.
#ifndef DPG_CTA_WARPS
#define DPG_CTA_WARPS DPG_NWARPS
#endif
constexpr int NW = DPG_CTA_WARPS;
constexpr int NT = NW * 32;
constexpr int CTAS_PER_SM = DPG_NWARPS / NW;
constexpr int MAX_MBT = NW == DPG_NWARPS ? DPG_MAX_MBT : NW;  // trial tiles: one column tile per warp
constexpr int MAX_KB = (MAX_MBT * MAX_MBT / 4 + NW - 1) / NW;  // 16x8 blocks of K_ext per warp (even MAX_MBT)
constexpr int MBAR_SPIN_LIMIT = 1 << 22;
constexpr int ERR_TIMEOUT_FLAG = 0x7fff0000;
constexpr int GEO = 24;  // doubles per point geometry record: J(9) Ji(9) det w*|J| n(3) 1/det

__device__ __forceinline__ void dmma(double2& c, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(c.x), "+d"(c.y)
               : "d"(a), "d"(b));
}

// D(16x8) += A(16x16) B(16x8), FP64.  Fragments: a[2i] = A[g][t+4i], a[2i+1] = A[g+8][t+4i],
// b[i] = B[t+4i][g]; c = {C[g][2t], C[g][2t+1], C[g+8][2t], C[g+8][2t+1]}.
__device__ __forceinline__ void dmma16(double* c, const double* a, const double* b) {
  asm("mma.sync.aligned.m16n8k16.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7,%8,%9,%10,%11}, "
      "{%12,%13,%14,%15}, {%0,%1,%2,%3};"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(a[4]), "d"(a[5]), "d"(a[6]), "d"(a[7]), "d"(b[0]),
        "d"(b[1]), "d"(b[2]), "d"(b[3]));
}

// D(16x8) += A(16x4) B(4x8): a0 = A[g][t], a1 = A[g+8][t]; b = B[t][g].
__device__ __forceinline__ void dmma16x4(double* c, double a0, double a1, double b) {
  asm("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a0), "d"(a1), "d"(b));
}

// D(16x8) += A(16x8) B(8x8), operands as dmma16x8's.
__device__ __forceinline__ void dmma16k8(double* c, double a0, double a1, double a2, double a3, double b0, double b1) {
  asm("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a0), "d"(a1), "d"(a2), "d"(a3), "d"(b0), "d"(b1));
}

// D(16x8) += A(16x8) * B(8x8): a0 = A[g][t], a1 = A[g+8][t], a2 = A[g][t+4], a3 = A[g+8][t+4];
// b0 = B[t][g], b1 = B[t+4][g]; c_lo holds rows g, c_hi rows g+8 (columns 2t, 2t+1 each).
__device__ __forceinline__ void dmma16x8(double2& c_lo, double2& c_hi, double a0, double a1, double a2, double a3,
                                         double b0, double b1) {
  asm("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+d"(c_lo.x), "+d"(c_lo.y), "+d"(c_hi.x), "+d"(c_hi.y)
      : "d"(a0), "d"(a1), "d"(a2), "d"(a3), "d"(b0), "d"(b1));
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* b, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* b, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(b)), "r"(bytes) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(b)) : "memory");
}

// Global -> shared bulk copy completing on an mbarrier (16-byte aligned, bytes % 16 == 0).
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* b) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(b))
               : "memory");
}

// Bounded wait on an mbarrier phase; false if the limit was reached.
__device__ __forceinline__ bool mbar_wait(uint64_t* b, uint32_t parity, int limit = MBAR_SPIN_LIMIT) {
  for (int it = 0; it < limit; it++) {
    uint32_t done;
    asm volatile(
        "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
        : "=r"(done)
        : "r"(smem_u32(b)), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

// AK layout index of element (r, c) of an 8x8 tile
__device__ __forceinline__ int ak(int r, int c) { return ((c >> 2) * 8 + r) * 4 + (c & 3); }

// Offset of the C-fragment pair (g, 2t..2t+1) in AK layout
__device__ __forceinline__ int ak_cfrag(int g, int t) { return ((t >> 1) * 8 + g) * 4 + (t & 1) * 2; }

// Convert a C-fragment (rows g, cols 2t, 2t+1) into the two B-fragments of the
// same 8x8 matrix used as the k x n operand: B_h[t][g] = X[4h + t][g].
__device__ __forceinline__ void cfrag_to_bfrag(const double2 c, int lane, double& b0, double& b1) {
  const int g = lane >> 2, t = lane & 3;
  const int src0 = t * 4 + (g >> 1);
  const int src1 = 16 + t * 4 + (g >> 1);
  double x0 = __shfl_sync(0xffffffffu, c.x, src0);
  double y0 = __shfl_sync(0xffffffffu, c.y, src0);
  double x1 = __shfl_sync(0xffffffffu, c.x, src1);
  double y1 = __shfl_sync(0xffffffffu, c.y, src1);
  b0 = (g & 1) ? y0 : x0;
  b1 = (g & 1) ? y1 : x1;
}

// Geometry record of one point: Jacobian, inverse, determinant, weighted
// measure (w*detJ, or w*|side Jacobian| when tang != nullptr) and, on a side,
// the outward unit normal.  All vertex-shape derivatives are loaded up front.
__device__ __forceinline__ void point_geometry(int d, int nv, const double* __restrict__ X,
                                               const double* __restrict__ dN, double w,
                                               const double* __restrict__ tang, double* gq) {
  double dn[24];
#pragma unroll
  for (int i = 0; i < 24; i++) dn[i] = (i < nv * d) ? __ldg(dN + i) : 0.0;
  double tg[6];
  if (tang) {
#pragma unroll
    for (int i = 0; i < 6; i++) tg[i] = __ldg(tang + i);
  }
  double J[9];
#pragma unroll
  for (int i = 0; i < 9; i++) J[i] = 0.0;
  if (d == 3) {
#pragma unroll
    for (int a = 0; a < 8; a++) {
      if (a < nv) {
#pragma unroll
        for (int i = 0; i < 3; i++) {
          double xa = X[a * 3 + i];
#pragma unroll
          for (int j = 0; j < 3; j++) J[i * 3 + j] += xa * dn[a * 3 + j];
        }
      }
    }
  } else {
#pragma unroll
    for (int a = 0; a < 4; a++) {
      if (a < nv) {
#pragma unroll
        for (int i = 0; i < 2; i++) {
          double xa = X[a * 2 + i];
#pragma unroll
          for (int j = 0; j < 2; j++) J[i * 3 + j] += xa * dn[a * 2 + j];
        }
      }
    }
  }
  double Ji[9], det;
  if (d == 2) {
    det = J[0] * J[4] - J[1] * J[3];
    double id = 1.0 / det;
    Ji[0] = J[4] * id; Ji[1] = -J[1] * id; Ji[2] = 0;
    Ji[3] = -J[3] * id; Ji[4] = J[0] * id; Ji[5] = 0;
    Ji[6] = 0; Ji[7] = 0; Ji[8] = 1;
  } else {
    double c00 = J[4] * J[8] - J[5] * J[7];
    double c01 = J[5] * J[6] - J[3] * J[8];
    double c02 = J[3] * J[7] - J[4] * J[6];
    det = J[0] * c00 + J[1] * c01 + J[2] * c02;
    double id = 1.0 / det;
    Ji[0] = c00 * id;
    Ji[3] = c01 * id;
    Ji[6] = c02 * id;
    Ji[1] = (J[2] * J[7] - J[1] * J[8]) * id;
    Ji[4] = (J[0] * J[8] - J[2] * J[6]) * id;
    Ji[7] = (J[1] * J[6] - J[0] * J[7]) * id;
    Ji[2] = (J[1] * J[5] - J[2] * J[4]) * id;
    Ji[5] = (J[2] * J[3] - J[0] * J[5]) * id;
    Ji[8] = (J[0] * J[4] - J[1] * J[3]) * id;
  }
#pragma unroll
  for (int i = 0; i < 9; i++) { gq[i] = J[i]; gq[9 + i] = Ji[i]; }
  gq[18] = det;
  gq[23] = 1.0 / det;
  gq[20] = gq[21] = gq[22] = 0.0;
  if (!tang) {
    gq[19] = w * det;
    return;
  }
  double T0[3] = {0, 0, 0}, T1[3] = {0, 0, 0};
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) {
      T0[i] += J[i * 3 + j] * tg[j];
      T1[i] += J[i * 3 + j] * tg[3 + j];
    }
  double meas;
  if (d == 2) {
    meas = sqrt(T0[0] * T0[0] + T0[1] * T0[1]);
    gq[20] = T0[1] / meas;
    gq[21] = -T0[0] / meas;
  } else {
    double c0 = T0[1] * T1[2] - T0[2] * T1[1];
    double c1 = T0[2] * T1[0] - T0[0] * T1[2];
    double c2 = T0[0] * T1[1] - T0[1] * T1[0];
    meas = sqrt(c0 * c0 + c1 * c1 + c2 * c2);
    gq[20] = c0 / meas; gq[21] = c1 / meas; gq[22] = c2 / meas;
  }
  gq[19] = w * meas;
}

// Row `m` of the slot transform T of a test var at a point: physical value of
// the operator in physical slot m = sum_k T[m][k] * reference slot k.
//   HGRAD slots (value, d/dx_0..): T[0][0] = 1, T[1+c][1+j] = Ji[j][c]
//   HDIV  slots (v_0.., div):      T[c][j] = J[c][j]/det, T[d][d] = 1/det
__device__ __forceinline__ void trow_slot(int space, int d, int m, const double* gq, double* r) {
  r[0] = r[1] = r[2] = r[3] = 0.0;
  if (space == DPG_SPACE_HGRAD) {
    if (m == 0) r[0] = 1.0;
    else if (m <= d) {
      int c = m - 1;
      for (int j = 0; j < d; j++) r[1 + j] = gq[9 + j * 3 + c];
    }
  } else {
    const double id = gq[23];
    if (m < d) {
      for (int j = 0; j < d; j++) r[j] = gq[m * 3 + j] * id;
    } else if (m == d) {
      r[d] = id;
    }
  }
}

// Row of T for a physical operator (incl. tau . n on a side; normal at gq[20..22]).
__device__ __forceinline__ void trow_op(int space, int d, int op, const double* gq, double* r) {
  if (space == DPG_SPACE_HGRAD) {
    trow_slot(space, d, op == DPG_OP_VALUE ? 0 : 1 + (op - DPG_OP_DX), gq, r);
    return;
  }
  if (op == DPG_OP_DOT_NORMAL) {
    const double id = gq[23];
    r[0] = r[1] = r[2] = r[3] = 0.0;
    for (int c = 0; c < d; c++)
      for (int j = 0; j < d; j++) r[j] += gq[20 + c] * gq[c * 3 + j] * id;
    return;
  }
  trow_slot(space, d, op == DPG_OP_DIV ? d : op - DPG_OP_X, gq, r);
}

// Element (r, c) of the symmetric matrix stored as lower AK tiles at base.
__device__ __forceinline__ double sym_get(const double* base, int r, int c) {
  if (r < c) { int x = r; r = c; c = x; }
  int I = r >> 3, J = c >> 3;
  return base[(I * (I + 1) / 2 + J) * 64 + ak(r & 7, c & 7)];
}

// Shared-memory views of the persistent region (derived from dpg_smem).
#define DPG_SMEM_VIEWS(P)                                                              \
  double* const sm = dpg_smem;                                                         \
  int* const flag_s = reinterpret_cast<int*>(sm + (P).sm_nodes + 24);                  \
  uint64_t* const mbar_s = reinterpret_cast<uint64_t*>(sm + (P).sm_nodes + DPG_SM_BARS); \
  const int* const tri_s = reinterpret_cast<const int*>(sm + (P).sm_nodes + 32);       \
  const double* const nodes_s = sm + (P).sm_nodes;                                     \
  const double* const coef_s = sm + (P).sm_coef;                                       \
  (void)flag_s; (void)mbar_s; (void)tri_s; (void)nodes_s; (void)coef_s;

// Factor the diagonal tile k (one warp) and invert the factor.  Every lane loads the lower
// triangle and runs the whole factorisation in its own registers, so the pivot chain is eight
// reciprocal square roots (70 cycles each), each followed by one multiply and one FMA (8), with no
// shuffle on it; lane c forms column c of the inverse tile L_kk^-1 row by row beside it.  Only
// the inverse (AK layout, linv[64 k]) is written: the panel and the solves multiply by it,
// and nothing reads L_kk.  First failing pivot (1-based) -> *flag (sign sgn).
__device__ __forceinline__ void factor_diag(const double* __restrict__ T, int k, int* flag, int sgn, double* linv) {
  const int lane = threadIdx.x & 31;
  const double* Tkk = T + (k * (k + 1) / 2 + k) * 64;
  double a[36];  // a[r (r + 1) / 2 + c], c <= r
#pragma unroll
  for (int r = 0; r < 8; r++)
#pragma unroll
    for (int c = 0; c <= r; c++) a[r * (r + 1) / 2 + c] = Tkk[ak(r, c)];
  const int c0 = lane & 7;
  double x[8];
  bool failed = false;
  int fail_j = 0;
#pragma unroll
  for (int j = 0; j < 8; j++) {
    const double piv = a[j * (j + 1) / 2 + j];
    if (!(piv > 0.0) && !failed) { failed = true; fail_j = j; }
    const double inv = rsqrt(piv);
#pragma unroll
    for (int r = j + 1; r < 8; r++) a[r * (r + 1) / 2 + j] *= inv;
#pragma unroll
    for (int c = j + 1; c < 8; c++)
#pragma unroll
      for (int r = c; r < 8; r++) a[r * (r + 1) / 2 + c] -= a[r * (r + 1) / 2 + j] * a[c * (c + 1) / 2 + j];
    // row j of the inverse's column c0
    double v = (j == c0) ? 1.0 : 0.0;
#pragma unroll
    for (int m = 0; m < j; m++) v -= a[j * (j + 1) / 2 + m] * x[m];
    x[j] = (j < c0) ? 0.0 : v * inv;
  }
  if (lane == 0 && failed && *flag == 0) *flag = sgn * (k * 8 + fail_j + 1);
  if (lane < 8) {
#pragma unroll
    for (int r = 0; r < 8; r++) linv[k * 64 + ak(r, c0)] = x[r];
  }
  __syncwarp();
}

// The blocked Cholesky of 8x8 tiles (AK layout, lower tiles row by row) is left-looking: after
// step k's panel L_ik = A_ik L_kk^-T, column k+1 receives all its updates
// A_i,k+1 -= sum_{j <= k} L_ij L_k+1,j^T at once, each tile in one warp's registers.  A
// right-looking update reads and writes every trailing tile in every step (7.4 K cycles for
// the first step of 22 tiles, a dozen warps each waiting on load, two products and store per
// tile); here a tile is loaded and stored once, its products run in two chains joined at the
// end, and the work of a step stays below the time of the diagonal tile next door.  That chain of
// diagonal tiles is what bounds the factorisation: warp 0 does nothing else, with its sub-partition
// to itself (warps 4, 8, 12 only keep the barriers), and it needs from the others only the sum over
// j < k of tile (k+1, k+1), formed a step ahead.
constexpr int CHOL_NW = NW - NW / 4;  // warps that update: those of the other sub-partitions

__device__ __forceinline__ int chol_rank(int warp) { return warp - (warp >> 2) - 1; }

// Warp 0: panel tile (k+1, k), then update and factorisation of tile (k+1, k+1).
__device__ __forceinline__ void chol_chain(double* T, int nb, int nsteps, int* flag, int sgn, double* linv) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  factor_diag(T, 0, flag, sgn, linv);
  asm volatile("bar.sync 0, %0;" ::"n"(NT) : "memory");
#pragma unroll 1
  for (int k = 0; k < nsteps; k++) {
    const int i = k + 1;
    double* Lik = T + (i * (i + 1) / 2 + k) * 64;
    double2 c2 = make_double2(0.0, 0.0);
    if (i < nsteps) c2 = *reinterpret_cast<const double2*>(Lik + 64 + ak_cfrag(g, t));
    if (i < nb) {
      const double* Li = linv + k * 64;
      const double a0 = Lik[lane], a1 = Lik[32 + lane];
      double2 c = make_double2(0.0, 0.0);
      dmma(c, a0, Li[lane]);
      dmma(c, a1, Li[32 + lane]);
      __syncwarp();
      *reinterpret_cast<double2*>(Lik + ak_cfrag(g, t)) = c;
    }
    asm volatile("bar.arrive 1, %0;" ::"n"(NT) : "memory");  // it needs no other warp's panel tile
    __syncwarp();
    if (i < nsteps) {
      double* Tii = Lik + 64;
      dmma(c2, -Lik[lane], Lik[lane]);
      dmma(c2, -Lik[32 + lane], Lik[32 + lane]);
      *reinterpret_cast<double2*>(Tii + ak_cfrag(g, t)) = c2;
      __syncwarp();
      factor_diag(T, i, flag, sgn, linv);
    }
    asm volatile("bar.sync 0, %0;" ::"n"(NT) : "memory");
  }
}

// Panel tiles L_ik = A_ik L_kk^-T of step k, i > k + 1 (warps of rank r).
__device__ __forceinline__ void chol_panel(double* T, const double* Li, int nb, int k, int r, int lane) {
  const int g = lane >> 2, t = lane & 3;
#pragma unroll 1
  for (int i = k + 2 + r; i < nb; i += CHOL_NW) {
    double* Tik = T + (i * (i + 1) / 2 + k) * 64;
    const double a0 = Tik[lane], a1 = Tik[32 + lane];
    double2 c = make_double2(0.0, 0.0);
    dmma(c, a0, Li[lane]);
    dmma(c, a1, Li[32 + lane]);
    __syncwarp();
    *reinterpret_cast<double2*>(Tik + ak_cfrag(g, t)) = c;
  }
}

// A_ij -= sum_{m < n} L_im L_jm^T of one tile.
__device__ __forceinline__ void chol_tile(double* T, int i, int j, int n, int lane) {
  const int g = lane >> 2, t = lane & 3;
  const double* pa = T + (i * (i + 1) / 2) * 64 + lane;
  const double* pb = T + (j * (j + 1) / 2) * 64 + lane;
  double* C = T + (i * (i + 1) / 2 + j) * 64 + ak_cfrag(g, t);
  // two chains of products (m8n8k4: 26 cycles to its result, 16 on the pipe)
  double2 c = *reinterpret_cast<const double2*>(C), c1 = make_double2(0.0, 0.0);
#pragma unroll 2
  for (int m = 0; m < n; m++) {
    const double a0 = -pa[m * 64], a1 = -pa[m * 64 + 32];
    const double b0 = pb[m * 64], b1 = pb[m * 64 + 32];
    dmma(c, a0, b0);
    dmma(c1, a1, b1);
  }
  c.x += c1.x;
  c.y += c1.y;
  *reinterpret_cast<double2*>(C) = c;
}

// After the panel of step k: column k+1 below its diagonal tile, and tile (k+2, k+2) up to
// column k (warps of rank r).
__device__ __forceinline__ void chol_column(double* T, int nb, int nsteps, int k, int r, int lane) {
  if (k + 1 >= nsteps) return;
#pragma unroll 1
  for (int e = r; e < nb - 1 - k; e += CHOL_NW) {
    if (e > 0) chol_tile(T, k + 1 + e, k + 1, k + 1, lane);
    else if (k + 2 < nsteps) chol_tile(T, k + 2, k + 2, k + 1, lane);
  }
}

// Factors the leading nsteps tiles of a tile-lower matrix with nb tiles in shared memory; the
// trailing block is left with its Schur complement.  linv (nsteps x 64) receives the
// inverses of the diagonal tiles.
__device__ __noinline__ void tile_cholesky(int T_off, int nb, int nsteps, int flag_idx, int sgn, int tri_off,
                                           int linv_off) {
  double* const T = dpg_smem + T_off;
  int* const flag = reinterpret_cast<int*>(dpg_smem) + flag_idx;
  const int* const tri = reinterpret_cast<const int*>(dpg_smem + tri_off);
  double* const linv = dpg_smem + linv_off;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (nsteps <= 0) return;
  if (warp == 0) {
    chol_chain(T, nb, nsteps, flag, sgn, linv);
  } else {
    const int r = chol_rank(warp);
    asm volatile("bar.sync 0, %0;" ::"n"(NT) : "memory");
#pragma unroll 1
    for (int k = 0; k < nsteps; k++) {
      if (warp & 3) chol_panel(T, linv + k * 64, nb, k, r, lane);
      asm volatile("bar.sync 1, %0;" ::"n"(NT) : "memory");
      if (warp & 3) chol_column(T, nb, nsteps, k, r, lane);
      asm volatile("bar.sync 0, %0;" ::"n"(NT) : "memory");
    }
  }
  // the trailing block
  const int m = nb - nsteps, ntr = m * (m + 1) / 2;
#pragma unroll 1
  for (int u = warp; u < ntr; u += NW) chol_tile(T, nsteps + (tri[u] & 255), nsteps + (tri[u] >> 8), nsteps, lane);
  __syncthreads();
}

// ---------------------------------------------------------------------------
// Phase 1: B and F -> per-CTA scratch (or the B/F outputs in parts mode)
// ---------------------------------------------------------------------------
// Term rows of chunk c of segment sgi (or of the next segment's first chunk): row[lq][term][m] = w|J| (or the
// side measure) x coef x slot x (n) x (parity) x T_op[m], one thread per point and term, counted from the
// last thread; buf: which of the two row buffers.
__device__ __forceinline__ void b_term_rows(const DpgPlanDev& P, const DpgLaunch& L, const int8_t* par_c,
                                            const double* geo, int sgi, int c, int buf) {
  DPG_SMEM_VIEWS(P);
  if (c >= P.seg[sgi].nchunk) {
    c = 0;
    sgi++;
    while (sgi < P.nseg && P.seg[sgi].nterm == 0) sgi++;
    if (sgi >= P.nseg) return;
  }
  const DpgSeg& S = P.seg[sgi];
  const int q0 = c * S.chunk, n = min(S.chunk, S.npts - q0) * S.nterm;
  double* const rows = sm + P.b_row + buf * P.max_chunk * P.max_nterm * 4;
  for (int task = NT - 1 - (int)threadIdx.x; task < n; task += NT) {
    const int lq = task / S.nterm, lt = task - lq * S.nterm, q = q0 + lq;
    const double* gq = geo + (S.geo0 + q) * GEO;
    const DpgBTerm& Tm = P.bterm[S.term0 + lt];
    double v = gq[19] * Tm.coef;
    if (Tm.slot >= 0) v *= coef_s[Tm.slot * P.Ptot + S.pbase + q];
    if (Tm.normal_comp >= 0) v *= gq[20 + Tm.normal_comp];
    if (Tm.kind == DPG_VAR_FLUX) v *= (double)par_c[S.side];
    double tr[4];
    trow_op(P.test[Tm.test_var].space, P.d, Tm.test_op, gq, tr);
    double* dst = rows + task * 4;
    dst[0] = tr[0] * v; dst[1] = tr[1] * v; dst[2] = tr[2] * v; dst[3] = tr[3] * v;
  }
}

template <int BTW>
__device__ __noinline__ void phase_b(const DpgPlanDev& P, const DpgLaunch& L, int cell) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int d = P.d, nv = P.nv;
  DPG_SMEM_VIEWS(P);
  double* geo = sm + P.b_geo;
  double* U = sm + P.b_u;
  const int8_t* par_c = L.parity + (size_t)cell * P.ns;
  double2* scr = reinterpret_cast<double2*>(L.scratch + (size_t)blockIdx.x * P.scratch_per_cta);
  // prologue: first chunk's records in flight while the geometry is computed
  int first_seg = 0;
  while (first_seg < P.nseg && P.seg[first_seg].nterm == 0) first_seg++;
  if (tid == 0 && first_seg < P.nseg) {
    const DpgSeg& S = P.seg[first_seg];
    const uint32_t bytes = (uint32_t)(((min(S.chunk, S.npts) + 3) & ~3) * S.rec_len * sizeof(double));
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    mbar_expect_tx(&mbar_s[DPG_BAR_B], bytes);
    bulk_g2s(sm + P.b_rec0, S.rec, bytes, &mbar_s[DPG_BAR_B]);
  }
  // [B | F] tiles accumulate in this CTA's scratch slot, C-fragment layout per tile
  for (int i = tid; i < P.MBT * P.NBT * 32; i += NT) scr[i] = make_double2(0.0, 0.0);
  for (int q = tid; q < P.nbpts; q += NT)
    point_geometry(d, nv, nodes_s, P.dNB + (size_t)q * nv * d, P.wB[q], q >= P.QB ? P.tangB + (size_t)q * 6 : nullptr,
                   geo + q * GEO);
  // separable side terms, while the first volume chunk is in flight: per-point factors,
  // then one thread per entry (scratch element); entries are unique, and an element
  // that a bilinear block also writes is read-modified-written (the blocks add to it
  // after the chunk loop's barriers)
  __syncthreads();  // geometry complete, scratch zeroed
  if (first_seg < P.nseg) b_term_rows(P, L, par_c, geo, first_seg, 0, 0);
  if (P.nse > 0) {
    double* fac = sm + P.b_fac;  // [nse][QS]
    for (int task = tid; task < P.nse * P.QS; task += NT) {
      const int se = task / P.QS, q = task - se * P.QS;
      const DpgSideTerm& E = P.se[se];
      const double* gq = geo + (P.QB + E.side * P.QS + q) * GEO;
      double v = E.coef;
      if (E.use_meas) v *= gq[19];
      if (E.slot >= 0) v *= coef_s[E.slot * P.Ptot + E.pbase + q];
      if (E.normal_comp >= 0) v *= gq[20 + E.normal_comp];
      if (E.flux) v *= (double)par_c[E.side];
      fac[task] = v;
    }
    __syncthreads();
    double* scd = reinterpret_cast<double*>(scr);
    for (int e = tid; e < P.nsent; e += NT) {
      const int4 en = __ldg(P.sent + e);
      double acc = 0.0;
      if (en.z == 1) {
        const double* f = fac + (en.w & 0xffff) * P.QS;
        const double* w = P.scon_w + en.y;
        for (int q = 0; q < P.QS; q++) acc += __ldg(w + (size_t)q * P.ncon) * f[q];
      } else {
        for (int c = en.y; c < en.y + en.z; c++) {
          const double* f = fac + __ldg(P.scon_se + c) * P.QS;
          for (int q = 0; q < P.QS; q++) acc += __ldg(P.scon_w + (size_t)q * P.ncon + c) * f[q];
        }
      }
      if (en.w >> 16) scd[en.x] = acc;
      else scd[en.x] += acc;
    }
  }
  int gc = 0;  // global chunk counter (buffer parity)
  for (int sgi = first_seg; sgi < P.nseg; sgi++) {
    const DpgSeg& S = P.seg[sgi];
    if (S.nterm == 0) continue;
    // this warp's active 16x8 blocks of the segment: operand offsets and accumulators
    const int bbase = S.ntile / NW, bextra = S.ntile % NW;
    const int my0 = S.tile0 + warp * bbase + min(warp, bextra);
    const int nmine = bbase + (warp < bextra ? 1 : 0);
    uint32_t pk[BTW];
    double acc[BTW][4];
#pragma unroll
    for (int u = 0; u < BTW; u++) {
      acc[u][0] = acc[u][1] = acc[u][2] = acc[u][3] = 0.0;
      uint32_t v = 0;
      if (u < nmine) {
        const int4 td = P.btiles[my0 + u];
        const DpgBBlock& Bk = S.blk[td.z];
        const DpgTestVar& V = P.test[Bk.var];
        v = (uint32_t)(V.foff + t * V.ldA + (td.x - V.ntile0) * 8 + g) | ((uint32_t)(Bk.off + t * DPG_ULD + g) << 16);
      }
      pk[u] = v;
    }
    for (int c = 0; c < S.nchunk; c++, gc++) {
      const int buf = gc & 1;
      double* rec = sm + (buf ? P.b_rec1 : P.b_rec0);
      __syncthreads();  // the other buffer and U are free; geometry is complete
      if (tid == 0) {
        // prefetch the next chunk (this segment or the next one with terms)
        int ns = sgi, nc = c + 1;
        if (nc >= S.nchunk) {
          ns = sgi + 1;
          nc = 0;
          while (ns < P.nseg && P.seg[ns].nterm == 0) ns++;
        }
        if (ns < P.nseg) {
          const DpgSeg& S2 = P.seg[ns];
          // the records of the chunk's points, rounded up to a whole k-step (the table is padded)
          const uint32_t bytes =
              (uint32_t)(((min(S2.chunk, S2.npts - nc * S2.chunk) + 3) & ~3) * S2.rec_len * sizeof(double));
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          mbar_expect_tx(&mbar_s[DPG_BAR_B + (buf ^ 1)], bytes);
          bulk_g2s(sm + (buf ? P.b_rec0 : P.b_rec1), S2.rec + (size_t)nc * S2.chunk * S2.rec_len, bytes,
                   &mbar_s[DPG_BAR_B + (buf ^ 1)]);
        }
        const int par = flag_s[3];  // bit i: parity of the next wait on buffer i
        if (!mbar_wait(&mbar_s[DPG_BAR_B + buf], (par >> buf) & 1)) flag_s[2] = 1;
        flag_s[3] = par ^ (1 << buf);
      }
      const int nq = min(S.chunk, S.npts - c * S.chunk);
      __syncthreads();
      // U blocks: U[lq][blk][m][col] = sum over the (block, column)'s terms of row[lq][term][m] x trial value;
      // beside them the last threads form the next chunk's term rows
      b_term_rows(P, L, par_c, geo, sgi, c + 1, (gc + 1) & 1);
      {
        const double* const rows = sm + P.b_row + (gc & 1) * P.max_chunk * P.max_nterm * 4;
        const int per = S.nblk * 8, nterm = S.nterm, rl = S.rec_len, us = S.ustride;
        const int *const ustart = S.ustart, *const ucon = S.ucon;
        for (int task = tid; task < S.chunk * per; task += NT) {
          const int lq = task / per, rem = task - lq * per;
          double u0 = 0.0, u1 = 0.0, u2 = 0.0, u3 = 0.0;
          if (lq < nq) {
            const double* rq = rec + lq * rl;
            const int i1 = __ldg(ustart + rem + 1);
            for (int i = __ldg(ustart + rem); i < i1; i++) {
              const int v = __ldg(ucon + i);
              const double psi = rq[v & 0xffff];
              const double2* R = reinterpret_cast<const double2*>(rows + (lq * nterm + (v >> 16)) * 4);
              const double2 r01 = R[0], r23 = R[1];
              u0 += r01.x * psi; u1 += r01.y * psi; u2 += r23.x * psi; u3 += r23.y * psi;
            }
          }
          double* uq = U + lq * us + (rem >> 3) * 4 * DPG_ULD + (rem & 7);
          uq[0] = u0; uq[DPG_ULD] = u1; uq[2 * DPG_ULD] = u2; uq[3 * DPG_ULD] = u3;
        }
      }
      __syncthreads();
      // DMMA over this warp's active blocks of the segment: m16n8k16, one k-step = 4 points x 4 slots
#pragma unroll 1
      for (int s4 = 0; s4 < nq; s4 += 4) {
        const double* ra = rec + s4 * S.rec_len;
        const double* ub = U + s4 * S.ustride;
        uint32_t prevA = 0xffffffffu;
        double av[8];
#pragma unroll
        for (int u = 0; u < BTW; u++) {
          if (u < nmine) {
            const uint32_t ao = pk[u] & 0xffffu, bo = pk[u] >> 16;
            if (ao != prevA) {
#pragma unroll
              for (int i = 0; i < 4; i++) {
                av[2 * i] = ra[i * S.rec_len + ao];
                av[2 * i + 1] = ra[i * S.rec_len + ao + 8];
              }
              prevA = ao;
            }
            double bv[4];
#pragma unroll
            for (int i = 0; i < 4; i++) bv[i] = ub[i * S.ustride + bo];
            dmma16(acc[u], av, bv);
          }
        }
      }
    }
    // segment contributions into the scratch tiles (each block has one owner per segment)
#pragma unroll
    for (int u = 0; u < BTW; u++) {
      if (u < nmine) {
        const int4 td = P.btiles[my0 + u];
        const int s0 = (td.y * P.NBT + td.x) * 32 + lane;
        double2 v0 = scr[s0];
        v0.x += acc[u][0]; v0.y += acc[u][1];
        scr[s0] = v0;
        if (!td.w) {  // the block has a second row tile
          double2 v1 = scr[s0 + 32];
          v1.x += acc[u][2]; v1.y += acc[u][3];
          scr[s0 + 32] = v1;
        }
      }
    }
  }
  if (!L.parts) return;
  __syncthreads();
  double* Bc = L.B ? L.B + (size_t)cell * P.M * P.N : nullptr;
  double* Fc = L.F ? L.F + (size_t)cell * P.N : nullptr;
  for (int tile = warp; tile < P.MBT * P.NBT; tile += NW) {
    const int J = tile / P.NBT, I = tile - J * P.NBT;
    const double2 v = scr[tile * 32 + lane];
    const int ur = P.dev2user_test[I * 8 + g];
    if (ur < 0) continue;
#pragma unroll
    for (int e = 0; e < 2; e++) {
      const int col = J * 8 + 2 * t + e;
      const double x = e ? v.y : v.x;
      const int uc = P.dev2user_trial[col];
      if (Bc && uc >= 0) Bc[(size_t)uc * P.N + ur] = x;
      if (Fc && col == P.fcol) Fc[ur] = x;
    }
  }
}

// One k-step of the Gram products over a warp's blocks.  The row var's slots f_a go through the
// point's coupling D first (A' = f_a D, formed when the row pair or the column var changes), so the
// column var's slots are the B operand as staged.  blk[u]: offset of block u's column slots | slot
// stride << 16 | 1 << 31 where A' changes; tdesc: the block table (lane-independent).
// 3D, two points: A' is an m16n8k8 of the two points' slots with the block diagonal of
// their couplings; its columns 2t, 2t + 1 = (point t >> 1, slots 2 (t & 1), + 1) leave the lane that holds
// them as A operand of the products, which take k = t and k = t + 4 from those columns.
template <int GTM>
__device__ __forceinline__ void gram_step3d(const double* __restrict__ f, const double* __restrict__ Dm, int fs, int dstride,
                                            const int4* tdesc, const uint32_t (&blk)[GTM], int ntw,
                                            double (&acc)[GTM][4]) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  double av[4];
#pragma unroll
  for (int u = 0; u < GTM; u++) {
    if (u < ntw) {
      const uint32_t v = blk[u];
      if (v >> 31) {
        const int4 T = tdesc[u];
        const double* fa = f + (T.z & 0xffff) + t * (T.y & 0xffff) + g;
        const double d = Dm[(g >> 2) * dstride + (T.z >> 16) * 16 + t * 4 + (g & 3)];
        av[0] = av[1] = av[2] = av[3] = 0.0;
        dmma16k8(av, fa[0], fa[8], fa[fs], fa[fs + 8], g < 4 ? d : 0.0, g < 4 ? 0.0 : d);
      }
      const int ldb = (v >> 16) & 0x7fff;
      const double* b = f + (t >> 1) * fs + 2 * (t & 1) * ldb + g + (v & 0xffffu);
      dmma16k8(acc[u], av[0], av[2], av[1], av[3], b[0], b[ldb]);
    }
  }
}

// 2D, four points with three slots each (lane t: point t), three m16n8k4: a fourth slot would be
// zeros, a quarter of the tensor work.  A' by FMAs (lane t has its point's slots and coupling).
template <int GTM>
__device__ __forceinline__ void gram_step2d(const double* __restrict__ f, const double* __restrict__ Dm, int fs, int dstride,
                                            const int4* tdesc, const uint32_t (&blk)[GTM], int ntw,
                                            double (&acc)[GTM][4]) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  double av[6];
#pragma unroll
  for (int u = 0; u < GTM; u++) {
    if (u < ntw) {
      const uint32_t v = blk[u];
      if (v >> 31) {
        const int4 T = tdesc[u];
        const int ld = T.y & 0xffff;
        const double* fa = f + (T.z & 0xffff) + t * fs + g;
        const double* D = Dm + (T.z >> 16) * 16 + t * dstride;
#pragma unroll
        for (int k = 0; k < 3; k++) {
          const double lo = fa[k * ld], hi = fa[k * ld + 8];
          const double2 d01 = *reinterpret_cast<const double2*>(D + k * 4);
          const double dk[3] = {d01.x, d01.y, D[k * 4 + 2]};
#pragma unroll
          for (int l = 0; l < 3; l++) {
            av[2 * l] = k == 0 ? lo * dk[l] : fma(lo, dk[l], av[2 * l]);
            av[2 * l + 1] = k == 0 ? hi * dk[l] : fma(hi, dk[l], av[2 * l + 1]);
          }
        }
      }
      const int ldb = (v >> 16) & 0x7fff;
      const double* b = f + t * fs + g + (v & 0xffffu);
      const double b0 = b[0], b1 = b[ldb], b2 = b[2 * ldb];
      dmma16x4(acc[u], av[0], av[1], b0);
      dmma16x4(acc[u], av[2], av[3], b1);
      dmma16x4(acc[u], av[4], av[5], b2);
    }
  }
}

// What the chunk loop needs of the plan, in shared memory (cta_setup): read again once a chunk
// (volatile), because kept in registers it would push accumulators to local memory.  GP_PAR: bit i
// is the parity of the next first use of ring stage i.
enum { GP_CHG, GP_QG, GP_RING, GP_STAGE, GP_STAGES, GP_FLUSH, GP_D, GP_NGB, GP_TILES, GP_FS, GP_DS, GP_GT, GP_PAR, GP_N };

// The Gram chunk loop.  The chunks travel through a ring of stages: warps arrive on a stage's empty
// mbarrier and warp 0 refills it while the next chunk is worked on, so no block barrier is left in
// the loop and the warps drift apart by up to a ring.  Every GP_FLUSH chunks (except after the last)
// each thread adds the accumulators of its flushed blocks (P.gflushmask) into its own running sums
// in the scratch slot ([block][lane][4]; plain L2 loads and stores, one writer per element, so the
// order of additions is fixed) and restarts them from zero.
__device__ __forceinline__ uint32_t gram_flush_bits(const DpgPlanDev& P, int tau0) {
  return __funnelshift_r(P.gflushmask[tau0 >> 5], P.gflushmask[(tau0 >> 5) + 1], tau0 & 31);
}

template <int GTM, int DIM>
__device__ __forceinline__ void gram_body(const DpgPlanDev& P, const DpgLaunch& L, int sm_nodes) {
  const volatile int* const gp = reinterpret_cast<const volatile int*>(dpg_smem + sm_nodes + DPG_SM_GRAM);
  double acc[GTM][4];
#pragma unroll
  for (int u = 0; u < GTM; u++) acc[u][0] = acc[u][1] = acc[u][2] = acc[u][3] = 0.0;
  // owned 16x8 blocks, balanced: warps 0 .. extra-1 take one block more, so the four SM
  // sub-partitions (warps w, w+4, w+8, w+12) carry equal tensor work
  int ntw, tau0;
  {
    const int ngb = gp[GP_NGB], warp = threadIdx.x >> 5;
    ntw = ngb / NW + (warp < ngb % NW ? 1 : 0);
    tau0 = warp * (ngb / NW) + min(warp, ngb % NW);
  }
  const int4* const tdesc = reinterpret_cast<const int4*>(dpg_smem + gp[GP_TILES]) + tau0;
  const int fs = gp[GP_FS], dstride = gp[GP_DS];
  uint32_t blk[GTM];
  {
    int lastA = -1;
#pragma unroll
    for (int u = 0; u < GTM; u++) {
      blk[u] = 0;
      if (u < ntw) {
        const int4 T = tdesc[u];
        blk[u] = (uint32_t)T.w | ((uint32_t)(T.y >> 16) << 16) | (T.z != lastA ? 0x80000000u : 0u);
        lastA = T.z;
      }
    }
  }
#pragma unroll 1
  for (int c = 0; c * gp[GP_CHG] < gp[GP_QG]; c++) {
    const double* f;
    const double* Dm;
    int nq;  // points of the chunk, in whole k-steps of four
    {
      const int chg = gp[GP_CHG], stages = gp[GP_STAGES], use = c >> (stages >> 1), st = c & (stages - 1);  // 1, 2 or 4 stages
      uint64_t* const full = reinterpret_cast<uint64_t*>(dpg_smem + sm_nodes + DPG_SM_BARS);
      if (c > 0 && threadIdx.x == 0 && (c - 1 + stages) * chg < gp[GP_QG]) {
        // refill the stage of chunk c - 1 with chunk c - 1 + stages
        const int pu = (c - 1) >> (stages >> 1), ps = (c - 1) & (stages - 1);
        const uint32_t par = (uint32_t)gp[GP_PAR] >> (DPG_GSTAGES + ps);
        if (!mbar_wait(&full[DPG_BAR_EMPTY + ps], (par ^ pu) & 1u)) reinterpret_cast<int*>(dpg_smem + sm_nodes + 24)[2] = 1;
        const uint32_t bytes = (uint32_t)(chg * fs * sizeof(double));
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        mbar_expect_tx(&full[ps], bytes);
        bulk_g2s(dpg_smem + gp[GP_RING] + ps * gp[GP_STAGE], P.frefG + (size_t)(c - 1 + stages) * chg * fs, bytes, &full[ps]);
      }
      __syncwarp();
      if (!mbar_wait(&full[st], (((uint32_t)gp[GP_PAR] >> st) ^ use) & 1u)) reinterpret_cast<int*>(dpg_smem + sm_nodes + 24)[2] = 1;
      f = dpg_smem + gp[GP_RING] + st * gp[GP_STAGE];
      Dm = dpg_smem + gp[GP_D] + c * chg * dstride;
      nq = (min(chg, gp[GP_QG] - c * chg) + 3) & ~3;
    }
    constexpr int STEP = DIM == 3 ? 2 : 4;
#pragma unroll 1
    for (; nq > 0; nq -= STEP, f += STEP * fs, Dm += STEP * dstride) {
      if (DIM == 3) gram_step3d<GTM>(f, Dm, fs, dstride, tdesc, blk, ntw, acc);
      else gram_step2d<GTM>(f, Dm, fs, dstride, tdesc, blk, ntw, acc);
    }
    const int chg = gp[GP_CHG], stages = gp[GP_STAGES], gflush = gp[GP_FLUSH];
    if ((c + stages) * chg < gp[GP_QG]) {  // the stage will be refilled
      __syncwarp();
      if ((threadIdx.x & 31) == 0)
        mbar_arrive(reinterpret_cast<uint64_t*>(dpg_smem + sm_nodes + DPG_SM_BARS) + DPG_BAR_EMPTY + (c & (stages - 1)));
    }
    if ((c + 1) % gflush == 0 && (c + 1) * chg < gp[GP_QG]) {
      const bool first = (c + 1) == gflush;
      const uint32_t fb = gram_flush_bits(P, tau0);
      double* const gsum = L.scratch + (size_t)blockIdx.x * P.scratch_per_cta + P.gsum_off + tau0 * 128 + (threadIdx.x & 31) * 4;
#pragma unroll
      for (int u = 0; u < GTM; u++) {
        if (u < ntw && ((fb >> u) & 1u)) {
          double2* sp = reinterpret_cast<double2*>(gsum + u * 128);
          double2 lo = make_double2(acc[u][0], acc[u][1]), hi = make_double2(acc[u][2], acc[u][3]);
          if (!first) {
            const double2 a = __ldcg(sp), b = __ldcg(sp + 1);
            lo.x = a.x + lo.x; lo.y = a.y + lo.y; hi.x = b.x + hi.x; hi.y = b.y + hi.y;
          }
          __stcg(sp, lo);
          __stcg(sp + 1, hi);
          acc[u][0] = acc[u][1] = acc[u][2] = acc[u][3] = 0.0;
        }
      }
    }
  }
  __syncthreads();  // every warp is done with the ring, which the tiles overlap
  if (threadIdx.x == 0) {
    const int chg = gp[GP_CHG], stages = gp[GP_STAGES], nch = (gp[GP_QG] + chg - 1) / chg;
    int par = gp[GP_PAR];
    for (int i = 0; i < stages; i++) {
      const int uses = (nch - i + stages - 1) / stages;  // a stage is emptied once less than it is filled
      par ^= ((uses & 1) << i) | (((uses - 1) & 1) << (DPG_GSTAGES + i));
    }
    reinterpret_cast<int*>(dpg_smem + sm_nodes + DPG_SM_GRAM)[GP_PAR] = par;
  }
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  double* const GT = dpg_smem + gp[GP_GT];
  const bool join = gp[GP_FLUSH] * gp[GP_CHG] < gp[GP_QG];  // the last group joins the running sums
  const uint32_t fb = gram_flush_bits(P, tau0);
  const double* const gsum = L.scratch + (size_t)blockIdx.x * P.scratch_per_cta + P.gsum_off + tau0 * 128 + lane * 4;
#pragma unroll
  for (int u = 0; u < GTM; u++) {
    if (u < ntw) {
      double2 lo = make_double2(acc[u][0], acc[u][1]), hi = make_double2(acc[u][2], acc[u][3]);
      if (join && ((fb >> u) & 1u)) {
        const double2* sp = reinterpret_cast<const double2*>(gsum + u * 128);
        const double2 a = __ldcg(sp), b = __ldcg(sp + 1);
        lo.x = a.x + lo.x; lo.y = a.y + lo.y; hi.x = b.x + hi.x; hi.y = b.y + hi.y;
      }
      const int T = tdesc[u].x;
      const int I = T & 0xffff, J = (T >> 16) & 0xff;
      if (J <= I) *reinterpret_cast<double2*>(GT + (I * (I + 1) / 2 + J) * 64 + ak_cfrag(g, t)) = lo;
      if (!(T >> 24)) *reinterpret_cast<double2*>(GT + ((I + 1) * (I + 2) / 2 + J) * 64 + ak_cfrag(g, t)) = hi;
    }
  }
}

// ---------------------------------------------------------------------------
// Phase 2: Gram matrix -> lower tiles in shared memory
// ---------------------------------------------------------------------------
template <int GTM>
__device__ __forceinline__ void phase_gram(const DpgPlanDev& P, const DpgLaunch& L, int cell) {
  const int tid = threadIdx.x;
  const int d = P.d, nv = P.nv;
  DPG_SMEM_VIEWS(P);
  double* geo = sm + P.g_geo;
  double* Dm = sm + P.g_D;  // [q][pair][16], points 2 doubles apart in bank position
  double* GT = sm + P.sm_gt;
  const uint32_t chunk_bytes = (uint32_t)(P.chg * P.featstride * sizeof(double));
  if (tid == 0) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    mbar_expect_tx(&mbar_s[0], chunk_bytes);
    bulk_g2s(sm + P.g_fref, P.frefG, chunk_bytes, &mbar_s[0]);
  }
  const int qg4 = (P.QG + 3) & ~3;
  for (int q = tid; q < qg4; q += NT)
    point_geometry(d, nv, nodes_s, P.dNG + (size_t)q * nv * d, P.wG[q], nullptr, geo + q * GEO);
  __syncthreads();
  // beta_r,a[k] = sum over row-r entries on var a of coef * slot * T_a[slot_e][k]
  double* beta = sm + P.g_beta;  // [q][row][4 * ntest]
  const int F = 4 * P.ntest;
  for (int task = tid; task < qg4 * P.niprows * P.ntest; task += NT) {
    const int q = task / (P.niprows * P.ntest);
    const int rem = task - q * P.niprows * P.ntest;
    const int r = rem / P.ntest, a = rem - r * P.ntest;
    const double* gq = geo + q * GEO;
    double b0 = 0.0, b1 = 0.0, b2 = 0.0, b3 = 0.0;
    for (int e = P.rowstart[r]; e < P.rowstart[r + 1]; e++) {
      const DpgIPEnt& E = P.ipent[e];
      if ((E.gslot >> 2) != a) continue;
      double v = E.coef;
      if (E.slot >= 0) v *= (q < P.QG) ? coef_s[E.slot * P.Ptot + q] : 0.0;
      double tr[4];
      trow_slot(P.test[a].space, d, E.gslot & 3, gq, tr);
      b0 += v * tr[0]; b1 += v * tr[1]; b2 += v * tr[2]; b3 += v * tr[3];
    }
    double* dst = beta + (q * P.niprows + r) * F + 4 * a;
    dst[0] = b0; dst[1] = b1; dst[2] = b2; dst[3] = b3;
  }
  __syncthreads();
  // coupling D_ab[k][l] = wdet * sum_r beta_r,a[k] beta_r,b[l]
  for (int task = tid; task < qg4 * P.npairs * 16; task += NT) {
    const int q = task / (P.npairs * 16);
    const int rem = task - q * P.npairs * 16;
    const int p = rem >> 4, k = (rem >> 2) & 3, l = rem & 3;
    const double* bq = beta + q * P.niprows * F;
    const int ia = 4 * P.pair_a[p] + k, ib = 4 * P.pair_b[p] + l;
    double sacc = 0.0;
    for (int r = 0; r < P.niprows; r++) sacc += bq[r * F + ia] * bq[r * F + ib];
    Dm[q * (P.npairs * 16 + 2) + rem] = sacc * geo[q * GEO + 19];
  }
  __syncthreads();
  if (tid == 0) {  // the stages that beta overlapped
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    for (int c = 1; c < P.gstages && c * P.chg < P.QG; c++) {
      mbar_expect_tx(&mbar_s[c], chunk_bytes);
      bulk_g2s(sm + P.g_fref + c * P.gstage, P.frefG + (size_t)c * P.chg * P.featstride, chunk_bytes, &mbar_s[c]);
    }
  }
  if (d == 3) gram_body<GTM, 3>(P, L, P.sm_nodes);
  else gram_body<GTM, 2>(P, L, P.sm_nodes);
  // tiles of uncoupled var pairs are zero
  for (int e = tid; e < P.ngz * 64; e += NT) GT[P.gzero[e >> 6] * 64 + (e & 63)] = 0.0;
  __syncthreads();
  // padded rows decouple: unit diagonal
  for (int r = tid; r < P.Np; r += NT)
    if (P.dev2user_test[r] < 0) GT[((r >> 3) * ((r >> 3) + 1) / 2 + (r >> 3)) * 64 + ak(r & 7, r & 7)] = 1.0;
  __syncthreads();
  if (L.parts && L.G) {
    double* Gc = L.G + (size_t)cell * P.N * P.N;
    for (int e = tid; e < P.Np * P.Np; e += NT) {
      int r = e / P.Np, c2 = e - r * P.Np;
      int ur = P.dev2user_test[r], uc = P.dev2user_test[c2];
      if (ur >= 0 && uc >= 0) Gc[(size_t)ur * P.N + uc] = sym_get(GT, r, c2);
    }
  }
}

// ---------------------------------------------------------------------------
// Phase 3: equilibrated Cholesky of G and inverses of its diagonal tiles
// ---------------------------------------------------------------------------
__device__ __forceinline__ void phase_factor(const DpgPlanDev& P) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  DPG_SMEM_VIEWS(P);
  double* GT = sm + P.sm_gt;
  double* scale = sm + P.sm_scale;
  for (int r = tid; r < P.Np; r += NT) {
    int I = r >> 3;
    double dg = GT[(I * (I + 1) / 2 + I) * 64 + ak(r & 7, r & 7)];
    scale[r] = (dg > 0.0) ? rsqrt(dg) : 1.0;
  }
  __syncthreads();
  for (int u = warp; u < P.ngt; u += NW) {
    int ij = tri_s[u];
    int I = ij & 255, J = ij >> 8;
    double2* p = reinterpret_cast<double2*>(GT + u * 64 + ak_cfrag(g, t));
    double si = scale[I * 8 + g];
    double2 v = *p;
    v.x *= si * scale[J * 8 + 2 * t];
    v.y *= si * scale[J * 8 + 2 * t + 1];
    *p = v;
  }
  __syncthreads();
  tile_cholesky(P.sm_gt, P.NBT, P.NBT, 2 * (P.sm_nodes + 24), 1, P.sm_nodes + 32, P.sm_linv);
}

// ---------------------------------------------------------------------------
// Phase 4: W = L^-1 [B | F] per column tile in registers, W^T tiles to shared memory
// ---------------------------------------------------------------------------

// Column tile J of S [B | F] (S: the equilibration scales), C-fragments per row tile.
template <int NBTM>
__device__ __forceinline__ void solve_load(const DpgPlanDev& P, const DpgLaunch& L, int cell, int J, const double* scale,
                                           double2 (&y)[NBTM]) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  if (L.solve_only) {
    const double* Bc = L.Bin + (size_t)cell * P.M * P.N;
    const double* Fc = L.Fin + (size_t)cell * P.N;
#pragma unroll
    for (int I = 0; I < NBTM; I++) {
      y[I] = make_double2(0.0, 0.0);
      const int row = I * 8 + g;
      if (I < P.NBT && row < P.N) {
        double v[2];
#pragma unroll
        for (int e = 0; e < 2; e++) {
          const int col = J * 8 + 2 * t + e;
          v[e] = col < P.M ? Bc[(size_t)col * P.N + row] : (col == P.fcol ? Fc[row] : 0.0);
        }
        y[I] = make_double2(v[0], v[1]);
      }
    }
  } else {
    const double2* scr = reinterpret_cast<const double2*>(L.scratch + (size_t)blockIdx.x * P.scratch_per_cta) +
                         (size_t)J * P.NBT * 32 + lane;
#pragma unroll
    for (int I = 0; I < NBTM; I++) y[I] = I < P.NBT ? scr[I * 32] : make_double2(0.0, 0.0);
  }
#pragma unroll
  for (int I = 0; I < NBTM; I++)
    if (I < P.NBT) {
      const double si = scale[I * 8 + g];
      y[I].x *= si;
      y[I].y *= si;
    }
}

// x_k = L_kk^-1 y_k, returned as a C-fragment and as negated B-fragments.
__device__ __forceinline__ double2 solve_diag(const double* Li, const double2 yk, int lane, double& x0, double& x1) {
  double y0, y1;
  cfrag_to_bfrag(yk, lane, y0, y1);
  double2 x = make_double2(0.0, 0.0);
  dmma(x, Li[lane], y0);
  dmma(x, Li[32 + lane], y1);
  cfrag_to_bfrag(x, lane, x0, x1);
  x0 = -x0;
  x1 = -x1;
  return x;
}

// y_i -= L_ik x_k for i > k: tiles (2j, 2j + 1) together, one m16n8k8 on the stacked tiles
// [L_ik; L_i+1,k].  The pairs are the same in every step: an m16n8k8 accumulates into eight
// consecutive registers, so pairs that shift with k would move every tile each step.
// k is a compile-time value in the unrolled callers.
template <int NBTM>
__device__ __forceinline__ void solve_update(const double* __restrict__ GT, int NBT, int k, int lane, double2 (&y)[NBTM],
                                             double x0, double x1) {
  if (!(k & 1) && k + 1 < NBTM && k + 1 < NBT) {
    const double* Lik = GT + ((k + 1) * (k + 2) / 2 + k) * 64;
    dmma(y[k + 1], Lik[lane], x0);
    dmma(y[k + 1], Lik[32 + lane], x1);
  }
#pragma unroll
  for (int r = 0; r < NBTM; r += 2) {
    if (r <= k) continue;
    const double* Lik = GT + (r * (r + 1) / 2 + k) * 64;
    const double* Ln = GT + ((r + 1) * (r + 2) / 2 + k) * 64;
    if (r + 1 < NBTM && r + 1 < NBT) {  // (an odd NBTM has no pair at its end)
      dmma16x8(y[r], y[r + 1], Lik[lane], Ln[lane], Lik[32 + lane], Ln[32 + lane], x0, x1);
    } else if (r < NBT) {
      dmma(y[r], Lik[lane], x0);
      dmma(y[r], Lik[32 + lane], x1);
    }
  }
}

// W^T tiles (trial J, test I) in AK layout, over L's tiles.
template <int NBTM>
__device__ __forceinline__ void solve_store(double* WT, int NBT, int J, const double2 (&y)[NBTM]) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  double* tile = WT + J * NBT * 64 + ((g >> 2) * 8 + 2 * t) * 4 + (g & 3);
#pragma unroll
  for (int I = 0; I < NBTM; I++) {
    if (I < NBT) {
      tile[I * 64] = y[I].x;
      tile[I * 64 + 4] = y[I].y;
    }
  }
}

// W = Ls^-1 S [B | F] = L^-1 [B | F], one warp per column tile; then W^T over L's tiles.
template <int NBTM>
__device__ __forceinline__ void phase_trsm(const DpgPlanDev& P, const DpgLaunch& L, int cell) {
  const int lane = threadIdx.x & 31, J = threadIdx.x >> 5;
  const double* const GT = dpg_smem + P.sm_gt;
  const double* const LINV = dpg_smem + P.sm_linv;
  const int NBT = P.NBT;
  if (J < P.MBT) {
    double2 y[NBTM];
    solve_load<NBTM>(P, L, cell, J, dpg_smem + P.sm_scale, y);
#pragma unroll
    for (int k = 0; k < NBTM; k++) {
      if (k >= NBT) break;
      double x0, x1;
      y[k] = solve_diag(LINV + k * 64, y[k], lane, x0, x1);
      solve_update<NBTM>(GT, NBT, k, lane, y, x0, x1);
    }
    asm volatile("bar.sync 0, %0;" ::"n"(NT) : "memory");
    solve_store<NBTM>(dpg_smem + P.sm_w, NBT, J, y);
  } else {
    asm volatile("bar.sync 0, %0;" ::"n"(NT) : "memory");
  }
  __syncthreads();
}

// ---------------------------------------------------------------------------
// Phase 5/6: K_ext = W^T W, outputs, condensation
// ---------------------------------------------------------------------------
// K_ext's lower tiles as 16x8 blocks of the row pairs (r, r + 1), r = 2p + o (o = MBT & 1), by the
// columns J <= r, and what is left of the diagonal, the 8x8 tiles of every second row: no product is
// done twice or for padding.  A warp's blocks k0 .. k0 + N - 1 (row by row) and, with SINGLE, the diagonal
// tile of row I1, then their stores over W^T behind the block barrier.  Bound by the tensor pipe (18.5 K
// cycles for 14 trial and 22 test tiles).  N and SINGLE are template arguments: with up to nine guarded
// 8x8 tiles per warp every load waited behind a branch (31 K cycles).  48^3 hexes 144.9 -> 142.1 ms,
// quads of k = 4 14.27 -> 14.15 ms; two steps of R per pass: 14.45 ms for the latter.
template <int N, bool SINGLE>
__device__ __forceinline__ void syrk_blocks(const double* __restrict__ WT, double* KT, int NBT, int o, int k0, int I1,
                                            int lane) {
  double acc[N + 1][4];
  double2 acc1 = make_double2(0.0, 0.0);
  int ai[N + 1], bj[N + 1];
  uint32_t newrow = 1;  // bit u: block u is the first of its row pair
  int p = 0;
#pragma unroll
  for (int u = 0; u < N; u++) {
    while ((p + 1) * (p + 1 + o) <= k0 + u) p++;
    ai[u] = (2 * p + o) * NBT * 64 + lane;
    if (k0 + u == p * (p + o)) newrow |= 1u << u;
    bj[u] = (k0 + u - p * (p + o)) * NBT * 64 + lane;
#pragma unroll
    for (int e = 0; e < 4; e++) acc[u][e] = 0.0;
  }
  const int row = NBT * 64;
#pragma unroll 1
  for (int R = 0; R < NBT; R++, WT += 64) {
    double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
#pragma unroll
    for (int u = 0; u < N; u++) {
      if (newrow >> u & 1) {
        a0 = WT[ai[u]];
        a1 = WT[ai[u] + row];
        a2 = WT[ai[u] + 32];
        a3 = WT[ai[u] + row + 32];
      }
      dmma16k8(acc[u], a0, a1, a2, a3, WT[bj[u]], WT[bj[u] + 32]);
    }
    if (SINGLE) {
      const double w0 = WT[I1 * row + lane], w1 = WT[I1 * row + lane + 32];
      dmma(acc1, w0, w0);
      dmma(acc1, w1, w1);
    }
  }
  asm volatile("bar.sync 0, %0;" ::"n"(NT) : "memory");
  const int c = ak_cfrag(lane >> 2, lane & 3);
  p = 0;
#pragma unroll
  for (int u = 0; u < N; u++) {
    while ((p + 1) * (p + 1 + o) <= k0 + u) p++;
    const int I = 2 * p + o, J = k0 + u - p * (p + o);
    *reinterpret_cast<double2*>(KT + (I * (I + 1) / 2 + J) * 64 + c) = make_double2(acc[u][0], acc[u][1]);
    *reinterpret_cast<double2*>(KT + ((I + 1) * (I + 2) / 2 + J) * 64 + c) = make_double2(acc[u][2], acc[u][3]);
  }
  if (SINGLE) *reinterpret_cast<double2*>(KT + (I1 * (I1 + 3) / 2) * 64 + c) = acc1;
}

// The instance for n blocks (at most N).
template <int N, bool SINGLE>
__device__ __forceinline__ void syrk_pick(int n, const double* WT, double* KT, int NBT, int o, int k0, int I1, int lane) {
  if (n == N) syrk_blocks<N, SINGLE>(WT, KT, NBT, o, k0, I1, lane);
  else if constexpr (N > 0) syrk_pick<N - 1, SINGLE>(n, WT, KT, NBT, o, k0, I1, lane);
}

__device__ __forceinline__ void syrk(int w_off, int k_off, int NBT, int MBT) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double* const WT = dpg_smem + w_off;
  double* const KT = dpg_smem + k_off;
  // the first warps take the blocks that do not divide evenly, the last ones the diagonal tiles
  const int o = MBT & 1, np = MBT >> 1, nk = np * (np + o);
  const int kbase = nk / NW, kextra = nk % NW;
  const int k0 = warp * kbase + min(warp, kextra), I1 = 2 * (NW - 1 - warp) + 1 - o;
  const int n = kbase + (warp < kextra ? 1 : 0);
  if (I1 < MBT) syrk_pick<MAX_KB, true>(n, WT, KT, NBT, o, k0, I1, lane);
  else syrk_pick<MAX_KB, false>(n, WT, KT, NBT, o, k0, I1, lane);
}

__device__ __forceinline__ void phase_syrk_out(const DpgPlanDev& P, const DpgLaunch& L, int cell) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  DPG_SMEM_VIEWS(P);
  double* KT = sm + P.sm_k;
  syrk(P.sm_w, P.sm_k, P.NBT, P.MBT);
  __syncthreads();
  // K and l out (user numbering; fields first: dev = i for i < nf, nfp + (i - nf) otherwise);
  // streaming stores, so the outputs do not evict the CTA's scratch slot from L2
  if (L.K) {
    double* Kc = L.K + (size_t)cell * P.M * P.M;
    for (int i = warp; i < P.M; i += NW) {
      const int di = i < P.nf ? i : P.nfp + (i - P.nf);
      for (int j = lane; j < P.M; j += 32) {
        const int dj = j < P.nf ? j : P.nfp + (j - P.nf);
        __stcs(&Kc[(size_t)i * P.M + j], sym_get(KT, di, dj));
      }
    }
    double* lc = L.l + (size_t)cell * P.M;
    for (int i = tid; i < P.M; i += NT) {
      int di = i < P.nf ? i : P.nfp + (i - P.nf);
      __stcs(&lc[i], sym_get(KT, P.fcol, di));
    }
  }
  if (L.S && P.nt > 0) {
    if (P.nfb > 0) {
      __syncthreads();
      for (int r = P.nf + tid; r < P.nfp; r += NT) {
        int I = r >> 3;
        KT[(I * (I + 1) / 2 + I) * 64 + ak(r & 7, r & 7)] = 1.0;
      }
      __syncthreads();
      tile_cholesky(P.sm_k, P.MBT, P.nfb, 2 * (P.sm_nodes + 24) + 1, -1, P.sm_nodes + 32, P.sm_linv);
    }
    double* Sc = L.S + (size_t)cell * P.nt * P.nt;
    for (int i = warp; i < P.nt; i += NW)
      for (int j = lane; j < P.nt; j += 32) __stcs(&Sc[(size_t)i * P.nt + j], sym_get(KT, P.nfp + i, P.nfp + j));
    double* sc = L.s + (size_t)cell * P.nt;
    for (int i = tid; i < P.nt; i += NT) __stcs(&sc[i], sym_get(KT, P.fcol, P.nfp + i));
  }
}

// Element (r, c) of a C-fragment tiled N x (M+1) matrix in a scratch slot
// (tile (I, J) at ((J * NBT + I) * 32 + lane) double2, lane = r * 4 + c / 2).
__device__ __forceinline__ size_t cfrag_index(int NBT, int r, int c) {
  return ((size_t)((c >> 3) * NBT + (r >> 3)) * 32 + (r & 7) * 4 + ((c & 7) >> 1)) * 2 + (c & 1);
}

__device__ __forceinline__ void mbar_inval(uint64_t* b) {
  asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(smem_u32(b)) : "memory");
}

// Per-CTA tables of one plan: triangular tile index, G block list, mbarriers.
__device__ __forceinline__ void cta_setup(const DpgPlanDev& P) {
  const int tid = threadIdx.x;
  double* const sm = dpg_smem;
  int* tri_s = reinterpret_cast<int*>(sm + P.sm_nodes + 32);
  DpgGTile* tiles_s = reinterpret_cast<DpgGTile*>(sm + P.sm_tiles);
  uint64_t* mbar_s = reinterpret_cast<uint64_t*>(sm + P.sm_nodes + DPG_SM_BARS);
  const int ntri = DPG_MAX_NBT * (DPG_MAX_NBT + 1) / 2;
  for (int u = tid; u < ntri; u += NT) {
    int I = (int)((sqrt(8.0 * u + 1.0) - 1.0) * 0.5);
    while ((I + 1) * (I + 2) / 2 <= u) I++;
    while (I * (I + 1) / 2 > u) I--;
    tri_s[u] = I | ((u - I * (I + 1) / 2) << 8);
  }
  for (int u = tid; u < P.ngb && P.gtiles; u += NT) tiles_s[u] = P.gtiles[u];
  if (tid == 0) {
    for (int i = 0; i < DPG_NBARS; i++) mbar_init(&mbar_s[i], i < DPG_BAR_EMPTY ? 1 : NW);
    int* const gp = reinterpret_cast<int*>(sm + P.sm_nodes + DPG_SM_GRAM);
    reinterpret_cast<int*>(sm + P.sm_nodes + 24)[3] = 0;
    gp[GP_CHG] = P.chg; gp[GP_QG] = P.QG; gp[GP_RING] = P.g_fref; gp[GP_STAGE] = P.gstage; gp[GP_STAGES] = P.gstages;
    gp[GP_FLUSH] = P.gflush; gp[GP_D] = P.g_D; gp[GP_NGB] = P.ngb; gp[GP_TILES] = P.sm_tiles; gp[GP_FS] = P.featstride;
    gp[GP_DS] = P.npairs * 16 + 2; gp[GP_GT] = P.sm_gt; gp[GP_PAR] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
}

typedef DpgKernelFn KernelFn;

}  // namespace
