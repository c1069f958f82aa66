// dpg_big.cuh — large buckets (N > 192 or M > 120 after padding), included by dpg_big.cu.
//
// One persistent CTA (16 warps) per SM walks the cells, or, with few cells, a cluster of CTAs takes each.
// A cell's matrices do not fit in shared memory, so each CTA or cluster owns a workspace in global memory
// (L2-resident for the smaller buckets) holding the lower triangle of
//
//     Z = [[ S G S , S E ],        E = [B^T | F]  (N x (M + 1), device trial order),
//          [ E^T S ,  0  ]]        S = diag(G_ii^-1/2)  (DPOEQU scaling, BF.cpp:944-960)
//
// rows/columns: device test rows, then device trial columns (fields, traces, F).
//   1. Per-point factors: w|J| and the IP rows' Piola-mapped coefficients at the Gram points,
//      the terms' (w|J| or side measure) x coefficient x normal x parity x Piola row at the
//      B points (LinearTerm::integrate, LinearTerm.cpp:427-627; BasisEvaluation.cpp:182-390).
//   2. Formation by 64 x 64 tiles on the FP64 tensor cores (mma.m16n8k16.f64): a G tile sums
//      w|J| L_r(v_i) L_r(v_j) over the points and the IP rows r touching both tiles'
//      test vars (IP::computeInnerProductMatrix, IP.cpp:215-292); an E tile sums trial value x
//      test-operator value over the points of every segment and term touching the tile
//      (TBF::stiffnessMatrix, BF.cpp:575-656), the load's row is summed apart (RHS.cpp:68-82).  The diagonal G tiles come
//      first and give the scales S.
//   3. Np steps of a blocked right-looking Cholesky: the 64 x 64 diagonal block is factored in
//      shared memory as 8 x 8 tiles (the single-CTA kernel's tile Cholesky) and inverted by block
//      forward substitution, the rows below it become L panels (the rows of
//      W^T = (L^-1 E)^T, BF.cpp:987-988) and the trailing update subtracts L_I L_J^T
//      (DSYRK, BF.cpp:993-1005).  The trailing block is then -E^T G^-1 E = -[[K, l], [l^T, .]].
//   4. K, l are written out, the trailing block is negated, and nfp more steps over the field
//      columns leave [S s] = the Schur complement (CondensedDofInterpreter.cpp:1138-1192).
// A CTA waits on the CTAs of its own cluster (cluster barriers: they are resident together) and on its own
// asynchronous copies (cp.async groups), on nothing else.

constexpr int ZT = 64;  // tile edge
constexpr int ZL = 68;  // shared row stride, == 4 (mod 16) doubles: conflict-free DMMA fragments
// ZK (template parameter below): k-chunk of a formation tile, 16 or 32 points (one or two
// m16n8k16 steps per chunk); the plan's big_zk, chosen by dpg_plan_autotune
constexpr int BIG_NOFAIL = 0x7fffffff;
static_assert(DPG_MAX_IPROWS <= 32 && DPG_MAX_BF <= 120, "relevance lists of a formation tile");

// A cell's CTAs: one, or the CTAs of a cluster (few cells: the idle SMs share each cell's tiles).
// They share the cell's workspace; big_sync orders its writes before the other CTAs' reads.
struct BigTeam {
  int rank, size;
};
__device__ __forceinline__ BigTeam big_team() {
  BigTeam t;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(t.rank));
  asm("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(t.size));
  return t;
}
template <bool TEAM>
__device__ __forceinline__ void big_sync() {
  if (TEAM) {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  } else {
    __syncthreads();
  }
}

// A relevant entry of an E tile (one segment and term), in shared memory.
struct BigEntry {
  const double* rec;     // the segment's point records
  int rec_len, tv;       // doubles per record; trial value of device column j at tv + j
  int col0, col1;        // device trial columns
  int var, foff, ld;     // test var, its slots in a record
  int vt;                // first row of per-point factors
  int k0, k1;            // its k range
};

struct BigSm {
  double* D;   // [64][ZL] diagonal block, factored in place
  double* Xi;  // [64][ZL] inverse of its factor
  double* LI;  // [64][ZL] L panel rows of the current row block
  double* LJ;  // [64][ZL] panel rows of the column block / staging of the raw panel
  double* LJ1; // [64][ZL] second panel buffer (double buffering of the column blocks)
  double* fa;  // [2][2][ZK][ZL] formation operands (rows, columns) x two chunks (aliases D..LJ1)
  double* sc;  // [Np] equilibration scales
  int* col;    // [Np] test row record: var << 16 | local dof, or -1 (padding row)
  int* ints;   // [0] first failing G column, [1] first failing field column, [64..] relevance lists
  double* nodes;
};

__device__ __forceinline__ BigSm big_views(const DpgPlanDev& P) {
  double* const sm = dpg_smem;
  BigSm S;
  S.D = sm;
  S.Xi = sm + ZT * ZL;
  S.LI = sm + 2 * ZT * ZL;
  S.LJ = sm + 3 * ZT * ZL;
  S.LJ1 = sm + 4 * ZT * ZL;
  S.fa = sm;
  S.sc = sm + P.bs_sc;
  S.col = reinterpret_cast<int*>(sm + P.bs_col);
  S.ints = reinterpret_cast<int*>(sm + P.bs_int);
  S.nodes = sm + P.bs_nodes;
  return S;
}

// acc (a 16 x 16 warp tile: rows wr.., columns wc..) += A B over one ZK chunk, operands stored
// k-major: A[r][k] = fa[k][r], B[k][c] = fb[k][c].  The k16 steps alternate between acc and
// acc2, so four independent DMMA chains are in flight.
template <int ZK>
__device__ __forceinline__ void big_mma_kmajor(const double* fa, const double* fb, int wr, int wc, int g, int t,
                                               double (&acc)[2][4], double (&acc2)[2][4]) {
#pragma unroll
  for (int s16 = 0; s16 < ZK / 16; s16++) {
    const double* fa_s = fa + s16 * 16 * ZL;
    const double* fb_s = fb + s16 * 16 * ZL;
    double a[8];
#pragma unroll
    for (int i = 0; i < 4; i++) {
      a[2 * i] = fa_s[(t + 4 * i) * ZL + wr + g];
      a[2 * i + 1] = fa_s[(t + 4 * i) * ZL + wr + g + 8];
    }
#pragma unroll
    for (int nb = 0; nb < 2; nb++) {
      double b[4];
#pragma unroll
      for (int i = 0; i < 4; i++) b[i] = fb_s[(t + 4 * i) * ZL + wc + nb * 8 + g];
      dmma16((s16 & 1) ? acc2[nb] : acc[nb], a, b);
    }
  }
}

// acc += A B^T over k in [0, kn) (kn a multiple of 16, at most 64), both stored row-major [row][k].  Odd
// k-steps go to a second set of accumulators, so four independent DMMA chains are in flight (the caller joins
// them: big_join).  f0 and f1 run after the first and the second k-step: copies and loads of a tile issued
// there cost nothing, between two tiles the tensor pipe waits for them.
template <class F0, class F1>
__device__ __forceinline__ void big_mma_rows(const double* A, const double* B, int kn, int wr, int wc, int g, int t,
                                             double (&acc)[2][4], double (&acc2)[2][4], F0 f0, F1 f1) {
#pragma unroll
  for (int s16 = 0; s16 < ZT / 16; s16++) {
    const int kk = 16 * s16;
    if (kk < kn) {
      double a[8];
#pragma unroll
      for (int i = 0; i < 4; i++) {
        a[2 * i] = A[(wr + g) * ZL + kk + t + 4 * i];
        a[2 * i + 1] = A[(wr + g + 8) * ZL + kk + t + 4 * i];
      }
#pragma unroll
      for (int nb = 0; nb < 2; nb++) {
        double b[4];
#pragma unroll
        for (int i = 0; i < 4; i++) b[i] = B[(wc + nb * 8 + g) * ZL + kk + t + 4 * i];
        dmma16((s16 & 1) ? acc2[nb] : acc[nb], a, b);
      }
    }
    if (s16 == 0) f0();
    if (s16 == 1) f1();
  }
}

__device__ __forceinline__ void big_zero(double (&a)[2][4], double (&b)[2][4]) {
#pragma unroll
  for (int nb = 0; nb < 2; nb++)
#pragma unroll
    for (int e = 0; e < 4; e++) a[nb][e] = b[nb][e] = 0.0;
}

__device__ __forceinline__ void big_join(double (&a)[2][4], const double (&b)[2][4]) {
#pragma unroll
  for (int nb = 0; nb < 2; nb++)
#pragma unroll
    for (int e = 0; e < 4; e++) a[nb][e] += b[nb][e];
}

// Test vars whose (padded) rows meet [r0, r0 + 64).
__device__ __forceinline__ int big_var_mask(const DpgPlanDev& P, int r0) {
  int m = 0;
  for (int a = 0; a < P.ntest; a++) {
    const int lo = P.test[a].dev_off, hi = lo + P.test[a].ntiles * 8;
    if (lo < r0 + ZT && hi > r0) m |= 1 << a;
  }
  return m;
}

// Per-point factors of one cell (workspace): wq[q] = w|J| at the Gram points;
// bh[q][r][a][k] = sum over IP entries of row r on var a of coef x slot x T_a[slot_e][k];
// vt[row][k] = (w|J| or side measure) x coef x slot x (n_c) x (parity) x T_op[k] per term and point.
__device__ void big_prep(const DpgPlanDev& P, const DpgLaunch& L, int cell, const BigSm& S, double* wq, double* bh,
                         double* vt, const BigTeam team) {
  const int tid = team.rank * NT + threadIdx.x, nth = team.size * NT;
  const int d = P.d, nv = P.nv;
  const double* co = L.coeff ? L.coeff + (size_t)cell * P.nslots * P.Ptot : nullptr;
  for (int task = tid; task < P.QG * P.niprows; task += nth) {
    const int q = task / P.niprows, r = task - q * P.niprows;
    double gq[GEO];
    point_geometry(d, nv, S.nodes, P.dNG + (size_t)q * nv * d, P.wG[q], nullptr, gq);
    if (r == 0) wq[q] = gq[19];
    for (int a = 0; a < P.ntest; a++) {
      double b0 = 0.0, b1 = 0.0, b2 = 0.0, b3 = 0.0;
      for (int e = P.rowstart[r]; e < P.rowstart[r + 1]; e++) {
        const DpgIPEnt& E = P.ipent[e];
        if ((E.gslot >> 2) != a) continue;
        double v = E.coef;
        if (E.slot >= 0) v *= (q < P.QG && co) ? co[E.slot * P.Ptot + q] : 0.0;
        double tr[4];
        trow_slot(P.test[a].space, d, E.gslot & 3, gq, tr);
        b0 += v * tr[0]; b1 += v * tr[1]; b2 += v * tr[2]; b3 += v * tr[3];
      }
      double* dst = bh + ((size_t)(q * P.niprows + r) * P.ntest + a) * 4;
      dst[0] = b0; dst[1] = b1; dst[2] = b2; dst[3] = b3;
    }
  }
  const int nvt = P.nbe > 0 ? P.be[P.nbe - 1].z + P.be[P.nbe - 1].w : 0;
  const int8_t* par = L.parity + (size_t)cell * P.ns;
  for (int task = tid; task < nvt; task += nth) {
    int e = 0;
    while (task >= P.be[e].z + P.be[e].w) e++;
    const int4 be = P.be[e];
    const int q = task - be.z;
    const DpgSeg& Sg = P.seg[be.x];
    const DpgBTerm& Tm = P.bterm[Sg.term0 + be.y];
    const int pt = Sg.geo0 + q;
    double gq[GEO];
    point_geometry(d, nv, S.nodes, P.dNB + (size_t)pt * nv * d, P.wB[pt], Sg.side >= 0 ? P.tangB + (size_t)pt * 6 : nullptr,
                   gq);
    double v = gq[19] * Tm.coef;
    if (Tm.slot >= 0) v *= co ? co[Tm.slot * P.Ptot + Sg.pbase + q] : 0.0;
    if (Tm.normal_comp >= 0) v *= gq[20 + Tm.normal_comp];
    if (Tm.kind == DPG_VAR_FLUX) v *= (double)par[Sg.side];
    double tr[4];
    trow_op(P.test[Tm.test_var].space, d, Tm.test_op, gq, tr);
    double* dst = vt + (size_t)task * 4;
    dst[0] = v * tr[0]; dst[1] = v * tr[1]; dst[2] = v * tr[2]; dst[3] = v * tr[3];
  }
}

// One formation tile.  kind 0: G rows r0.., columns c0.. (test rows); kind 1: E^T rows
// (device trial columns) r0.., columns c0.. (test rows), without the F row (big_load_row).
template <int ZK>
__device__ void big_form_tile(const DpgPlanDev& P, int* fail, double* sc_out, int kind, int r0, int c0, bool diag, double* Z,
                              const BigSm& S, const double* wq, const double* bh, const double* vt) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int wr = (warp >> 2) * 16, wc = (warp & 3) * 16;
  int* rel = S.ints + 64;    // relevant IP rows (kind 0) or E entries (kind 1)
  int* relk = S.ints + 192;  // kind 1: first k of each relevant entry, then the total
  BigEntry* const ent = reinterpret_cast<BigEntry*>(S.ints + 512);  // kind 1: the relevant entries
  __syncthreads();           // lists and operand buffers free
  if (warp == 0) {  // ordered lists by ballots (one thread walking a hundred entries took 10 K cycles)
    const unsigned below = (1u << lane) - 1u;
    int n = 0, k = 0;
    const int mc = big_var_mask(P, c0);
    if (kind == 0) {
      const int mr = big_var_mask(P, r0);
      const bool in = lane < P.niprows && (P.ipmask[lane] & mr) && (P.ipmask[lane] & mc);
      const unsigned m = __ballot_sync(0xffffffffu, in);
      if (in) rel[__popc(m & below)] = lane;
      n = __popc(m);
      k = n * P.QG;
    } else {
      for (int e0 = 0; e0 < P.nbe; e0 += 32) {
        const int e = e0 + lane;
        bool in = e < P.nbe;
        int w = 0;
        if (in) {
          const int4 be = P.be[e];
          const DpgBTerm& Tm = P.bterm[P.seg[be.x].term0 + be.y];
          in = Tm.kind >= 0 && ((mc >> Tm.test_var) & 1) && Tm.col0 < r0 + ZT && Tm.col0 + Tm.ncol > r0;
          if (in) w = be.w;
        }
        const unsigned m = __ballot_sync(0xffffffffu, in);
        int sum = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int x = __shfl_up_sync(0xffffffffu, sum, o);
          if (lane >= o) sum += x;
        }
        if (in) {
          const int at = n + __popc(m & below);
          rel[at] = e;
          relk[at] = k + sum - w;
        }
        n += __popc(m);
        k += __shfl_sync(0xffffffffu, sum, 31);
      }
    }
    if (lane == 0) {
      relk[120] = n;
      relk[121] = k;
    }
  }
  __syncthreads();
  const int nrel = relk[120], nk = relk[121];
  if (kind == 1) {
    if (tid < nrel) {
      const int4 be = P.be[rel[tid]];
      const DpgSeg& Sg = P.seg[be.x];
      const DpgBTerm& Tm = P.bterm[Sg.term0 + be.y];
      BigEntry E;
      E.rec = Sg.rec;
      E.rec_len = Sg.rec_len;
      E.tv = Sg.tvoff[be.y] - Tm.col0;
      E.col0 = Tm.col0;
      E.col1 = Tm.col0 + Tm.ncol;
      E.var = Tm.test_var;
      E.foff = P.test[Tm.test_var].foff;
      E.ld = P.test[Tm.test_var].ldA;
      E.vt = be.z;
      E.k0 = relk[tid];
      E.k1 = relk[tid] + be.w;
      ent[tid] = E;
    }
    __syncthreads();
  }
  double acc[2][4], acc2[2][4];
#pragma unroll
  for (int nb = 0; nb < 2; nb++)
#pragma unroll
    for (int e = 0; e < 4; e++) acc[nb][e] = acc2[nb][e] = 0.0;
  // operands of k-chunk k0 (2 sides x ZK x 64 values) into buffer pair buf; chunk c + 1 is
  // formed while the MMAs of chunk c run on the other pair, one barrier per chunk.  A thread's
  // column is the same for every value it forms (NT is a multiple of 64), so its column records
  // are read once per tile; all of a thread's values are computed before any is stored, so
  // their loads overlap instead of waiting behind the shared-memory stores.
  constexpr int NU = 2 * ZK * ZT / NT;
  const int cc = tid & (ZT - 1);
  int crec[2];
#pragma unroll
  for (int side = 0; side < 2; side++) {
    const int i = (side ? c0 : r0) + cc;
    crec[side] = (kind == 1 && side == 0) ? -1 : (i < P.Np ? S.col[i] : -1);
  }
  int fo[2], fl[2];  // the column's slots inside a Gram point's
#pragma unroll
  for (int side = 0; side < 2; side++) {
    const DpgTestVar& V = P.test[crec[side] >= 0 ? crec[side] >> 16 : 0];
    fo[side] = V.foff + (crec[side] & 0xffff);
    fl[side] = V.ldA;
  }
  // A thread forms KPT consecutive k of each side.  G tiles number k point-major (k = q nrel +
  // row), so a thread's run mostly stays on one point and reads its column's four reference slot
  // values once for all the IP rows.  k only grows, by ZK per chunk: point and row (kind 0) or entry
  // (kind 1) of the run's first k come from cursors, without divisions.
  constexpr int KPT = ZK / (NT / ZT);
  const int kl0 = (tid >> 6) * KPT;
  int cq = 0, cr = 0, dq = 0, dr = 0, ecur = 0;
  if (kind == 0 && nrel > 0) {
    cq = kl0 / nrel;
    cr = kl0 - cq * nrel;
    dq = ZK / nrel;
    dr = ZK - dq * nrel;
  }
  // part 0: the column side of a G tile, or the first half of an E tile's k; part 1: the rest
  double vals[NU];
  auto operands = [&](int k0, int buf, auto part_c) {
    constexpr int part = decltype(part_c)::value;
    double* const fa = S.fa + buf * 2 * ZK * ZL;
    const int kk0 = k0 + kl0;
    if (kind == 0) {
      constexpr int side = 1 - part;
      if (side == 0 && diag) {  // the same columns: times the weight
        int q = cq, r = cr;
#pragma unroll
        for (int u = 0; u < KPT; u++) {
          vals[u] = kk0 + u < nk ? vals[KPT + u] * wq[q] : 0.0;
          if (++r >= nrel) { r = 0; q++; }
        }
      } else {
        int q = cq, r = cr, lastq = -1;
        double fv[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int u = 0; u < KPT; u++) {
          double val = 0.0;
          if (kk0 + u < nk && crec[side] >= 0) {
            if (q != lastq) {
              const double* f = P.frefG + (size_t)q * P.featstride + fo[side];
              fv[0] = __ldg(f); fv[1] = __ldg(f + fl[side]); fv[2] = __ldg(f + 2 * fl[side]); fv[3] = __ldg(f + 3 * fl[side]);
              lastq = q;
            }
            const double* b = bh + ((size_t)(q * P.niprows + rel[r]) * P.ntest + (crec[side] >> 16)) * 4;
            const double2 b01 = *reinterpret_cast<const double2*>(b), b23 = *reinterpret_cast<const double2*>(b + 2);
            val = b01.x * fv[0] + b01.y * fv[1] + b23.x * fv[2] + b23.y * fv[3];
            if (side == 0) val *= wq[q];
          }
          vals[side * KPT + u] = val;
          if (++r >= nrel) { r = 0; q++; }
        }
      }
      if (part == 1) {
        cq += dq;
        cr += dr;
        if (cr >= nrel) { cr -= nrel; cq++; }
      }
#pragma unroll
      for (int u = 0; u < KPT; u++) fa[side * ZK * ZL + (kl0 + u) * ZL + cc] = vals[side * KPT + u];
    } else {
      const int j = r0 + cc, rec = crec[1];
#pragma unroll
      for (int u = part * KPT / 2; u < (part + 1) * KPT / 2; u++) {
        double v0 = 0.0, v1 = 0.0;
        if (kk0 + u < nk) {
          while (kk0 + u >= ent[ecur].k1) ecur++;
          const BigEntry& E = ent[ecur];
          const int q = kk0 + u - E.k0;
          const double* rq = E.rec + (size_t)q * E.rec_len;
          if (j >= E.col0 && j < E.col1) v0 = __ldg(rq + E.tv + j);
          if (rec >= 0 && (rec >> 16) == E.var) {
            const int ld = E.ld;
            const double* f = rq + E.foff + (rec & 0xffff);
            const double* v4 = vt + (size_t)(E.vt + q) * 4;
            const double2 v01 = *reinterpret_cast<const double2*>(v4), v23 = *reinterpret_cast<const double2*>(v4 + 2);
            v1 = v01.x * __ldg(f) + v01.y * __ldg(f + ld) + v23.x * __ldg(f + 2 * ld) + v23.y * __ldg(f + 3 * ld);
          }
        }
        vals[u] = v0;
        vals[KPT + u] = v1;
      }
#pragma unroll
      for (int u = part * KPT / 2; u < (part + 1) * KPT / 2; u++) {
        fa[(kl0 + u) * ZL + cc] = vals[u];
        fa[(ZK + kl0 + u) * ZL + cc] = vals[KPT + u];
      }
    }
  };
  constexpr std::integral_constant<int, 0> part0{};
  constexpr std::integral_constant<int, 1> part1{};
  if (nk > 0) {
    operands(0, 0, part0);
    operands(0, 0, part1);
  }
  __syncthreads();
  for (int k0 = 0, c = 0; k0 < nk; k0 += ZK, c++) {
    // chunk c + 1's operands are formed between and after the products of chunk c, which run meanwhile
    const double* fa = S.fa + (c & 1) * 2 * ZK * ZL;
    const bool more = k0 + ZK < nk;
    big_mma_kmajor<16>(fa, fa + ZK * ZL, wr, wc, g, t, acc, acc2);
    if (more) operands(k0 + ZK, (c + 1) & 1, part0);
    if (ZK == 32) big_mma_kmajor<16>(fa + 16 * ZL, fa + (ZK + 16) * ZL, wr, wc, g, t, acc2, acc);
    if (more) operands(k0 + ZK, (c + 1) & 1, part1);
    __syncthreads();
  }
#pragma unroll
  for (int nb = 0; nb < 2; nb++)
#pragma unroll
    for (int e = 0; e < 4; e++) acc[nb][e] += acc2[nb][e];
  const int ld = P.ldz;
  if (kind == 0) {
    if (diag) {
      // the diagonal of G gives the scales of these rows
#pragma unroll
      for (int nb = 0; nb < 2; nb++)
#pragma unroll
        for (int e = 0; e < 4; e++) {
          const int row = wr + g + (e >> 1) * 8, cl = wc + nb * 8 + 2 * t + (e & 1);
          const int i = r0 + row;
          if (row == cl && i < P.Np) {
            double s = 1.0;
            if (S.col[i] >= 0) {
              const double gii = acc[nb][e];
              if (gii > 0.0) s = 1.0 / sqrt(gii);
              else atomicMin(fail, i);
            }
            S.sc[i] = s;
            if (sc_out) sc_out[i] = s;
          }
        }
      __syncthreads();
    }
#pragma unroll
    for (int nb = 0; nb < 2; nb++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int i = r0 + wr + g + h * 8, j = c0 + wc + nb * 8 + 2 * t;
        if (i < P.Np && j < P.Np) {
          const double si = S.sc[i];
          double2 v = make_double2(acc[nb][2 * h] * si * S.sc[j], acc[nb][2 * h + 1] * si * S.sc[j + 1]);
          if (diag && S.col[i] < 0) {
            if (i == j) v.x = 1.0;
            if (i == j + 1) v.y = 1.0;
          }
          *reinterpret_cast<double2*>(Z + (size_t)i * ld + j) = v;
        }
      }
  } else {
#pragma unroll
    for (int nb = 0; nb < 2; nb++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int j = r0 + wr + g + h * 8, i = c0 + wc + nb * 8 + 2 * t;
        if (j < P.Mp && i < P.Np && j != P.fcol)
          *reinterpret_cast<double2*>(Z + (size_t)(P.Np + j) * ld + i) =
              make_double2(acc[nb][2 * h] * S.sc[i], acc[nb][2 * h + 1] * S.sc[i + 1]);
      }
  }
}

// The F row of E^T in blocks of 64 test rows; eight threads per row take every eighth point, their sums are joined in
// order.  The products of a tile meet every entry with every row, zeros included: a load that is not finite must
// not share them with B, nor a side of zero length with F.  Bound by the latency of its loads (records in L2): 148
// Poisson quads of k = 5 425 us with F in the tiles, 435 with one thread per row, 429 so; 37 Stokes quads of
// p = 6 1.778 -> 1.761 ms.  (Not inlined: the 32 values in flight would spill in the cell's body.)
__device__ __noinline__ void big_load_row(const DpgPlanDev& P, double* row, const int* col, const double* sc, const double* vt,
                                          double* red, int first, int step) {
  const double* const rec = P.seg[0].rec;
  const int rl = P.seg[0].rec_len, part = threadIdx.x >> 6, lr = threadIdx.x & 63;
  for (int b = first, k = 0; b * ZT < P.Np; b += step, k ^= NT) {
    const int i = b * ZT + lr, c = i < P.Np ? col[i] : -1;
    double f = 0.0;
    for (int e = 0; e < P.nle; e++) {
      const int4 E = P.le[e];
      if (c < 0 || E.w >> 24 != c >> 16) continue;
      const double* const r = rec + E.x + (c & 0xffff);
      const double* const v = vt + (size_t)(E.w & 0xffffff) * 4;
#pragma unroll 1
      for (int q0 = part; q0 < E.z; q0 += 64) {  // all loads of eight points in flight: no branch between them
        double x[8][4];
#pragma unroll
        for (int u = 0; u < 8; u++)
#pragma unroll
          for (int m = 0; m < 4; m++) x[u][m] = __ldg(r + (size_t)min(q0 + 8 * u, E.z - 1) * rl + m * E.y);
#pragma unroll
        for (int u = 0; u < 8; u++) {
          const int q = min(q0 + 8 * u, E.z - 1);
          const double2 a = *reinterpret_cast<const double2*>(v + q * 4), d = *reinterpret_cast<const double2*>(v + q * 4 + 2);
          const double g = a.x * x[u][0] + a.y * x[u][1] + d.x * x[u][2] + d.y * x[u][3];
          f += q0 + 8 * u < E.z ? g : 0.0;
        }
      }
    }
    red[k + threadIdx.x] = f;  // two buffers, one barrier per block
    __syncthreads();
    if (part == 0 && i < P.Np) {
#pragma unroll
      for (int p = 1; p < NT / ZT; p++) f += red[k + p * ZT + lr];
      row[i] = f * sc[i];
    }
  }
}

// The diagonal block Z[k0 .. k0+w) (w <= 64, padded to 64 with a unit diagonal): factored as
// 8 x 8 tiles in AK layout (in D) by the single-CTA kernel's blocked Cholesky (tile_cholesky:
// look-ahead, diagonal tiles factored in registers), then X = L_kk^-1 by block forward
// substitution, one warp per 8-column block (X_cc = L_cc^-1, X_ic = -L_ii^-1 sum_k L_ik X_kc),
// into Xi (row-major, zero above the diagonal).  The first column whose pivot is not positive
// goes to *fail (atomicMin).
__device__ __forceinline__ void big_diag_block(const double* Z, int ld, int k0, int w, const BigSm& S, int* fail) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  constexpr int NBD = ZT / 8;                 // 8 tiles
  constexpr int NTD = NBD * (NBD + 1) / 2;    // 36 lower tiles
  double* const T = S.D;
  double* const linv = S.LI;                  // [8][64] inverse diagonal tiles
  int* const tri = reinterpret_cast<int*>(S.LI + NBD * 64);
  int* const flag = tri + 64;
  __syncthreads();
  for (int e = tid; e < NTD * 64; e += NT) {
    const int tau = e >> 6, idx = e & 63;
    int I = 0;
    while ((I + 1) * (I + 2) / 2 <= tau) I++;
    const int J = tau - I * (I + 1) / 2;
    const int r = 8 * I + ((idx >> 2) & 7), c = 8 * J + (idx >> 5) * 4 + (idx & 3);
    double v = (r == c) ? 1.0 : 0.0;
    if (r < w && c <= r) v = Z[(size_t)(k0 + r) * ld + k0 + c];
    T[e] = v;
    if (idx == 0) tri[tau] = I | (J << 8);
  }
  if (tid == 0) *flag = 0;
  __syncthreads();
  tile_cholesky((int)(T - dpg_smem), NBD, NBD, (int)(flag - reinterpret_cast<int*>(dpg_smem)), 1,
                (int)(reinterpret_cast<double*>(tri) - dpg_smem), (int)(linv - dpg_smem));
  if (tid == 0 && *flag > 0) atomicMin(fail, k0 + *flag - 1);
  if (warp < NBD) {
    const int cb = warp;
    double2 acc[NBD];
#pragma unroll
    for (int i = 0; i < NBD; i++)
      acc[i] = (i == cb) ? make_double2(g == 2 * t ? 1.0 : 0.0, g == 2 * t + 1 ? 1.0 : 0.0) : make_double2(0.0, 0.0);
#pragma unroll
    for (int k = 0; k < NBD; k++) {
      if (k >= cb) {
        double y0, y1;
        cfrag_to_bfrag(acc[k], lane, y0, y1);
        const double* Li = linv + k * 64;
        double2 x = make_double2(0.0, 0.0);
        dmma(x, Li[lane], y0);
        dmma(x, Li[32 + lane], y1);
        acc[k] = x;
        double x0, x1;
        cfrag_to_bfrag(x, lane, x0, x1);
        x0 = -x0;
        x1 = -x1;
#pragma unroll
        for (int i = k + 1; i < NBD; i += 2) {
          const double* Lik = T + (i * (i + 1) / 2 + k) * 64;
          if (i + 1 < NBD) {
            const double* Li1k = T + ((i + 1) * (i + 2) / 2 + k) * 64;
            dmma16x8(acc[i], acc[i + 1], Lik[lane], Li1k[lane], Lik[32 + lane], Li1k[32 + lane], x0, x1);
          } else {
            dmma(acc[i], Lik[lane], x0);
            dmma(acc[i], Lik[32 + lane], x1);
          }
        }
      }
    }
#pragma unroll
    for (int i = 0; i < NBD; i++)
      *reinterpret_cast<double2*>(S.Xi + (8 * i + g) * ZL + 8 * cb + 2 * t) = acc[i];
  }
  __syncthreads();
}

// Rows r0 .. r0 + 63 of panel columns k0 .. k0 + w - 1 of Z into a [64][ZL] block by asynchronous copies, zeros
// beyond the matrix and the panel (k0, w and the row stride are even: 16-byte pieces; ld is a multiple of 8).
__device__ __forceinline__ void big_copy_block(double* dst, const double* Z, int ld, int Zn, int r0, int k0, int w) {
#pragma unroll
  for (int u = 0; u < ZT * ZT / 2 / NT; u++) {
    const int e = threadIdx.x + u * NT, r = e >> 5, c = 2 * (e & 31);
    const bool in = r0 + r < Zn && c < w;
    const double* src = in ? Z + (size_t)(r0 + r) * ld + k0 + c : Z;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst + r * ZL + c)), "l"(src), "r"(in ? 16 : 0)
                 : "memory");
  }
}

// Steps kb .. ke-1 of a right-looking Cholesky of the lower triangle of Z (order Zn).  The
// first column whose pivot is not positive goes to *fail (atomicMin); the cell's outputs are
// then undefined (info reports the column).
__device__ void big_cholesky(const DpgPlanDev& P, double* Z, int kb, int ke, const BigSm& S, int* fail) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int wr = (warp >> 2) * 16, wc = (warp & 3) * 16;
  const int ld = P.ldz, Zn = P.Zn;
  for (int k0 = kb; k0 < ke; k0 += ZT) {
    const int w = min(ZT, ke - k0);
    const int wk = (w + 15) & ~15;
    big_diag_block(Z, ld, k0, w, S, fail);
    // rows below the block: panel L_I = Z_I,k L_kk^-T (stored back), then Z_IJ -= L_I L_J^T.  The
    // next raw panel (in D, free after the diagonal block) and the next column block's panel are
    // copied asynchronously while the products of a tile run; one barrier per tile.
    const int rbeg = k0 + w;
    const int nrb = (Zn - rbeg + ZT - 1) / ZT;
    if (nrb > 0) big_copy_block(S.D, Z, ld, Zn, rbeg, k0, w);
    for (int bi = 0; bi < nrb; bi++) {
      const int ri0 = rbeg + bi * ZT, nri = min(ZT, Zn - ri0);
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncthreads();
      double acc[2][4], acc2[2][4];
      big_zero(acc, acc2);
      big_mma_rows(S.D, S.Xi, wk, wr, wc, g, t, acc, acc2, [] {}, [] {});
      big_join(acc, acc2);
#pragma unroll
      for (int nb = 0; nb < 2; nb++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int r = wr + g + h * 8, c = wc + nb * 8 + 2 * t;
          const double2 v = make_double2(acc[nb][2 * h], acc[nb][2 * h + 1]);
          *reinterpret_cast<double2*>(S.LI + r * ZL + c) = v;
          if (r < nri && c < w) *reinterpret_cast<double2*>(Z + (size_t)(ri0 + r) * ld + k0 + c) = v;
        }
      __syncthreads();
      if (bi + 1 < nrb) big_copy_block(S.D, Z, ld, Zn, ri0 + ZT, k0, w);
      for (int bj = 0; bj <= bi; bj++) {
        const int rj0 = rbeg + bj * ZT, nrj = min(ZT, Zn - rj0);
        const double* Lj = bj == bi ? S.LI : ((bj & 1) ? S.LJ : S.LJ1);
        double2 zo[2][2];
        big_zero(acc, acc2);
        // column blocks bj < bi come from the stored panels; the first one of the next row block last
        auto next_block = [&]() {
          if (bj + 1 < bi) big_copy_block(((bj + 1) & 1) ? S.LJ : S.LJ1, Z, ld, Zn, rj0 + ZT, k0, w);
          else if (bj == bi && bi + 1 < nrb) big_copy_block(S.LJ1, Z, ld, Zn, rbeg, k0, w);
        };
        auto old_values = [&]() {
#pragma unroll
          for (int nb = 0; nb < 2; nb++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
              const int r = wr + g + h * 8, c = wc + nb * 8 + 2 * t;
              zo[nb][h] = (r < nri && c < nrj) ? *reinterpret_cast<const double2*>(Z + (size_t)(ri0 + r) * ld + rj0 + c)
                                               : make_double2(0.0, 0.0);
            }
        };
        // on the diagonal tile, warp tiles wholly above the diagonal are not needed
        const bool upper = bj == bi && wc >= wr + 16;
        big_mma_rows(S.LI, Lj, upper ? 0 : wk, wr, wc, g, t, acc, acc2, next_block, old_values);
        // the barrier before the sums are touched: their products drain while the warps meet
        if (bj < bi) {
          asm volatile("cp.async.wait_all;" ::: "memory");
          __syncthreads();
        }
        big_join(acc, acc2);
#pragma unroll
        for (int nb = 0; nb < 2; nb++)
#pragma unroll
          for (int h = 0; h < 2; h++) {
            const int r = wr + g + h * 8, c = wc + nb * 8 + 2 * t;
            if (!upper && r < nri && c < nrj)
              *reinterpret_cast<double2*>(Z + (size_t)(ri0 + r) * ld + rj0 + c) =
                  make_double2(zo[nb][h].x - acc[nb][2 * h], zo[nb][h].y - acc[nb][2 * h + 1]);
          }
      }
    }
  }
  __syncthreads();
}

// The same steps by the CTAs of a cluster: every CTA factors the diagonal block for itself, the row
// blocks' panels and then the trailing tiles are dealt out (a contiguous run of the row-major tile list
// per CTA, so a row's panel is loaded once), with a cluster barrier after each.  Same products
// in the same order as big_cholesky.
__device__ void big_cholesky_team(const DpgPlanDev& P, double* Z, int kb, int ke, const BigSm& S, int* fail,
                                  const BigTeam team) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int wr = (warp >> 2) * 16, wc = (warp & 3) * 16;
  const int ld = P.ldz, Zn = P.Zn;
  auto load_block = [&](double* dst, int r0, int k0, int w) {
    const int nr = min(ZT, Zn - r0);
    double pre[ZT * ZT / NT];
#pragma unroll
    for (int u = 0; u < ZT * ZT / NT; u++) {
      const int e = tid + u * NT, r = e >> 6, c = e & (ZT - 1);
      pre[u] = (r < nr && c < w) ? Z[(size_t)(r0 + r) * ld + k0 + c] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < ZT * ZT / NT; u++) {
      const int e = tid + u * NT;
      dst[(e >> 6) * ZL + (e & (ZT - 1))] = pre[u];
    }
  };
  for (int k0 = kb; k0 < ke; k0 += ZT) {
    const int w = min(ZT, ke - k0);
    const int wk = (w + 15) & ~15;
    big_diag_block(Z, ld, k0, w, S, fail);
    const int rbeg = k0 + w;
    const int nrb = (Zn - rbeg + ZT - 1) / ZT;
    for (int bi = team.rank; bi < nrb; bi += team.size) {
      const int ri0 = rbeg + bi * ZT, nri = min(ZT, Zn - ri0);
      __syncthreads();
      load_block(S.LJ, ri0, k0, w);
      __syncthreads();
      double acc[2][4], acc2[2][4];
      big_zero(acc, acc2);
      big_mma_rows(S.LJ, S.Xi, wk, wr, wc, g, t, acc, acc2, [] {}, [] {});
      big_join(acc, acc2);
#pragma unroll
      for (int nb = 0; nb < 2; nb++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int r = wr + g + h * 8, c = wc + nb * 8 + 2 * t;
          if (r < nri && c < w)
            *reinterpret_cast<double2*>(Z + (size_t)(ri0 + r) * ld + k0 + c) =
                make_double2(acc[nb][2 * h], acc[nb][2 * h + 1]);
        }
    }
    big_sync<true>();
    const int ntile = nrb * (nrb + 1) / 2;
    const int t0 = (int)((long long)ntile * team.rank / team.size), t1 = (int)((long long)ntile * (team.rank + 1) / team.size);
    int bi = 0;
    while ((bi + 1) * (bi + 2) / 2 <= t0) bi++;
    int bj = t0 - bi * (bi + 1) / 2, have = -1;
    for (int tt = t0; tt < t1; tt++) {
      const int ri0 = rbeg + bi * ZT, nri = min(ZT, Zn - ri0);
      const int rj0 = rbeg + bj * ZT, nrj = min(ZT, Zn - rj0);
      __syncthreads();  // the buffers are free
      if (bi != have) load_block(S.LI, ri0, k0, w);
      have = bi;
      if (bj != bi) load_block(S.LJ, rj0, k0, w);
      double2 zo[2][2];
#pragma unroll
      for (int nb = 0; nb < 2; nb++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int r = wr + g + h * 8, c = wc + nb * 8 + 2 * t;
          zo[nb][h] = (r < nri && c < nrj) ? *reinterpret_cast<const double2*>(Z + (size_t)(ri0 + r) * ld + rj0 + c)
                                           : make_double2(0.0, 0.0);
        }
      __syncthreads();
      double acc[2][4], acc2[2][4];
      big_zero(acc, acc2);
      const bool upper = bj == bi && wc >= wr + 16;
      if (!upper) big_mma_rows(S.LI, bj == bi ? S.LI : S.LJ, wk, wr, wc, g, t, acc, acc2, [] {}, [] {});
      big_join(acc, acc2);
#pragma unroll
      for (int nb = 0; nb < 2; nb++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int r = wr + g + h * 8, c = wc + nb * 8 + 2 * t;
          if (!upper && r < nri && c < nrj)
            *reinterpret_cast<double2*>(Z + (size_t)(ri0 + r) * ld + rj0 + c) =
                make_double2(zo[nb][h].x - acc[nb][2 * h], zo[nb][h].y - acc[nb][2 * h + 1]);
        }
      if (++bj > bi) { bi++; bj = 0; }
    }
    big_sync<true>();
  }
}

// Per-CTA table of a large plan: the test var and local dof of every device test row.
__device__ __forceinline__ void big_cta_setup(const DpgPlanDev& P, const BigSm& S) {
  for (int i = threadIdx.x; i < P.Np; i += NT) {
    int rec = -1;
    for (int a = 0; a < P.ntest; a++) {
      const int il = i - P.test[a].dev_off;
      if (il >= 0 && il < P.test[a].card) rec = (a << 16) | il;
    }
    S.col[i] = rec;
  }
}

// One cell of a large plan; Z is the workspace of its CTA or cluster (bz_per_cta doubles).
template <int ZK, bool TEAM>
__device__ __forceinline__ void big_cell_body(const DpgPlanDev& P, const DpgLaunch& L, int cell, const BigSm& S, double* const Z, const BigTeam team) {
  const int tid = threadIdx.x, gtid = team.rank * NT + tid, nth = team.size * NT;
  int* const fail = TEAM ? reinterpret_cast<int*>(Z + P.bz_sc + P.Np) : S.ints;  // first failing G column, field column
  double* const sc_out = TEAM ? Z + P.bz_sc : nullptr;
  double* const wq = Z + P.bz_wq;
  double* const bh = Z + P.bz_bh;
  double* const vt = Z + P.bz_vt;
  const int Np = P.Np, Mp = P.Mp, M = P.M, ld = P.ldz;
  {
    __syncthreads();
    if (gtid == 0) { fail[0] = BIG_NOFAIL; fail[1] = BIG_NOFAIL; }
    if (tid < P.nv * P.d) S.nodes[tid] = L.nodes[(size_t)cell * P.nv * P.d + tid];
    __syncthreads();
    big_prep(P, L, cell, S, wq, bh, vt, team);
    for (size_t e = gtid; e < (size_t)Mp * Mp; e += nth) {
      const int r = (int)(e / Mp), c = (int)(e - (size_t)r * Mp);
      if (c <= r) Z[(size_t)(Np + r) * ld + Np + c] = 0.0;
    }
    big_sync<TEAM>();
    const int nbg = (Np + ZT - 1) / ZT, nbm = (Mp + ZT - 1) / ZT;
    for (int I = team.rank; I < nbg; I += team.size)
      big_form_tile<ZK>(P, fail, sc_out, 0, I * ZT, I * ZT, true, Z, S, wq, bh, vt);
    if (TEAM) {
      big_sync<TEAM>();
      for (int i = tid; i < Np; i += NT) S.sc[i] = sc_out[i];
      __syncthreads();
    }
    int deal = 0;  // the other tiles, dealt round robin
    for (int I = 1; I < nbg; I++)
      for (int J = 0; J < I; J++)
        if (!TEAM || deal++ % team.size == team.rank)
          big_form_tile<ZK>(P, fail, nullptr, 0, I * ZT, J * ZT, false, Z, S, wq, bh, vt);
    for (int J = 0; J < nbm; J++)
      for (int I = 0; I < nbg; I++)
        if (!TEAM || deal++ % team.size == team.rank)
          big_form_tile<ZK>(P, fail, nullptr, 1, J * ZT, I * ZT, false, Z, S, wq, bh, vt);
    big_load_row(P, Z + (size_t)(Np + P.fcol) * ld, S.col, S.sc, vt, S.fa, team.rank, team.size);
    if (TEAM) big_sync<TEAM>();
    if (L.parts) {
      // G (N, N), B (M, N) and F (N) in user numbering: Z unscaled (dpg_assemble_parts)
      __syncthreads();
      const int N = P.N;
      if (L.G)
        for (int e = gtid; e < N * N; e += nth) {
          const int ur = e / N, uc = e - ur * N;
          const int dr = __ldg(P.u2d_test + ur), dc = __ldg(P.u2d_test + uc);
          L.G[(size_t)cell * N * N + e] = Z[(size_t)max(dr, dc) * ld + min(dr, dc)] / (S.sc[dr] * S.sc[dc]);
        }
      if (L.B)
        for (int e = gtid; e < M * N; e += nth) {
          const int ut = e / N, us = e - ut * N;
          const int ds = __ldg(P.u2d_test + us);
          L.B[(size_t)cell * M * N + e] = Z[(size_t)(Np + __ldg(P.u2d_trial + ut)) * ld + ds] / S.sc[ds];
        }
      if (L.F)
        for (int us = gtid; us < N; us += nth) {
          const int ds = __ldg(P.u2d_test + us);
          L.F[(size_t)cell * N + us] = Z[(size_t)(Np + P.fcol) * ld + ds] / S.sc[ds];
        }
      big_sync<TEAM>();
      return;
    }
    if (TEAM) big_cholesky_team(P, Z, 0, Np, S, &fail[0], team);
    else big_cholesky(P, Z, 0, Np, S, &fail[0]);
    if (L.energy) {
      // energy error (dpg_energy_error): the rows below the test block now hold W = L^-1 E, so
      // e^2 = || L^-1 F - L^-1 B^T x ||^2 is a sum over the test rows, with no cancellation
      const double* x = L.xsol + (size_t)cell * M;
      double part = 0.0;
      for (int k = tid; k < Np; k += NT) {
        double r = Z[(size_t)(Np + P.fcol) * ld + k];
        for (int ut = 0; ut < M; ut++) r -= Z[(size_t)(Np + __ldg(P.u2d_trial + ut)) * ld + k] * x[ut];
        part += r * r;
      }
      for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
      double* red = S.LI;  // free after the factorisation
      if ((tid & 31) == 0) red[tid >> 5] = part;
      __syncthreads();
      if (gtid == 0) {
        double e2 = 0.0;
        for (int w = 0; w < NT / 32; w++) e2 += red[w];
        // a failed factorisation of the test block leaves no energy to report
        L.energy[cell] = fail[0] == BIG_NOFAIL ? sqrt(e2) : __longlong_as_double(0x7ff8000000000000ll);
      }
    } else if (L.B) {
      // DLS local matrices (dpg_assemble_dls): the rows below the test block hold
      // W^T = (L^-1 E)^T, so W = L^-1 B^T and y = L^-1 F are read out in user numbering
      const int N = P.N;
      double* Wc = L.B + (size_t)cell * M * N;
      for (size_t e = gtid; e < (size_t)M * N; e += nth) {
        const int ut = (int)(e / N), us = (int)(e - (size_t)ut * N);
        Wc[e] = Z[(size_t)(Np + __ldg(P.u2d_trial + ut)) * ld + __ldg(P.u2d_test + us)];
      }
      if (L.F)
        for (int us = gtid; us < N; us += nth) L.F[(size_t)cell * N + us] = Z[(size_t)(Np + P.fcol) * ld + __ldg(P.u2d_test + us)];
    } else {
    // trailing block = -[K_ext]: K, l out, then negate (padded field columns get a unit pivot)
    const double* T = Z + (size_t)Np * ld + Np;
    if (L.K)
      for (size_t e = gtid; e < (size_t)M * M; e += nth) {
        const int ur = (int)(e / M), uc = (int)(e - (size_t)ur * M);
        const int dr = __ldg(P.u2d_trial + ur), dc = __ldg(P.u2d_trial + uc);
        L.K[(size_t)cell * M * M + e] = -T[(size_t)max(dr, dc) * ld + min(dr, dc)];
      }
    if (L.l)
      for (int u = gtid; u < M; u += nth) L.l[(size_t)cell * M + u] = -T[(size_t)P.fcol * ld + __ldg(P.u2d_trial + u)];
    if (L.S || L.s) {
      big_sync<TEAM>();
      for (size_t e = gtid; e < (size_t)Mp * Mp; e += nth) {
        const int r = (int)(e / Mp), c = (int)(e - (size_t)r * Mp);
        if (c <= r) {
          double* p = Z + (size_t)(Np + r) * ld + Np + c;
          *p = (r == c && r < P.nfp && __ldg(P.dev2user_trial + r) < 0) ? 1.0 : -*p;
        }
      }
      big_sync<TEAM>();
      if (TEAM) big_cholesky_team(P, Z, Np, Np + P.nfp, S, &fail[1], team);
      else big_cholesky(P, Z, Np, Np + P.nfp, S, &fail[1]);
      const int nt = P.nt, nf = P.nf;
      if (L.S)
        for (size_t e = gtid; e < (size_t)nt * nt; e += nth) {
          const int ur = (int)(e / nt), uc = (int)(e - (size_t)ur * nt);
          const int dr = __ldg(P.u2d_trial + nf + ur), dc = __ldg(P.u2d_trial + nf + uc);
          L.S[(size_t)cell * nt * nt + e] = T[(size_t)max(dr, dc) * ld + min(dr, dc)];
        }
      if (L.s)
        for (int u = gtid; u < nt; u += nth) L.s[(size_t)cell * nt + u] = T[(size_t)P.fcol * ld + __ldg(P.u2d_trial + nf + u)];
    }
    }
    big_sync<TEAM>();  // the cell's workspace is free for the next one
    if (gtid == 0 && L.info) {
      int v = 0;
      if (fail[0] != BIG_NOFAIL) {
        const int u = P.dev2user_test[fail[0]];
        v = (u >= 0 ? u : fail[0]) + 1;
      } else if (fail[1] != BIG_NOFAIL) {
        const int u = P.dev2user_trial[fail[1] - Np];
        v = -((u >= 0 ? u : fail[1] - Np) + 1);
      }
      L.info[cell] = v;
    }
  }
}

template <int ZK, bool TEAM>
__global__ void __launch_bounds__(NT, 1) dpg_big_kernel(const __grid_constant__ DpgPlanDev P,
                                                        const __grid_constant__ DpgLaunch L) {
  const BigSm S = big_views(P);
  big_cta_setup(P, S);
  BigTeam team{0, 1};
  if (TEAM) team = big_team();
  const int first = TEAM ? blockIdx.x / team.size : blockIdx.x, step = TEAM ? gridDim.x / team.size : gridDim.x;
  double* const Z = L.scratch + (size_t)first * P.bz_per_cta;
  for (int cell = first; cell < L.C; cell += step) big_cell_body<ZK, TEAM>(P, L, cell, S, Z, team);
}
