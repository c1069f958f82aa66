// dpg_kernel.cu — fused FP64 per-cell DPG assembly for sm_100a.
//
// Persistent CTAs (16 warps, one per SM; small buckets: 8 warps, two per SM) walk the
// cells.  Per cell:
//   1. B and F (TBF::stiffnessMatrix, BF.cpp:575-656; RHS.cpp:68-82).  Volume: the
//      per-point records (reference slots of the test bases plus each term's trial
//      values) arrive by bulk (TMA) copy, double buffered; each point's and term's row
//      (weight x coefficient x Piola row) is formed a chunk ahead, U = row x trial
//      value per active (test var, column tile) block and column, and each warp accumulates its 16x8 blocks with mma.m16n8k16.f64 over k-steps of 4
//      points x 4 slots.  Boundary terms with a cell-independent side transform
//      (HGRAD value; HDIV normal trace by the Piola identity) are separable: compact
//      per-entry sums over the test rows nonzero on the side.  The tiles wait in a
//      per-CTA scratch slot (L2-resident).
//   2. Gram matrix G (IP::computeInnerProductMatrix, IP.cpp:215-292): the same slot
//      form; per point and coupled test-var pair a 4x4 coupling D = T_a^T C T_b (C:
//      graph-norm coefficients, T: Piola maps), folded into the row operand, and
//      each warp accumulates its 16x8 blocks of the lower triangle from the staged
//      slots (m16n8k8, 2D: m16n8k4).
//   3. Equilibrated Cholesky of G (BF.cpp:944-982: DPOEQU scaling, DPOTRF('L'),
//      the solves take the scaled factor), blocked left-looking on 8x8 tiles in shared
//      memory, the chain of diagonal tiles on a warp of its own.
//   4. W = L^-1 [B | F] in registers (BF.cpp:987-988, 1013-1014): each warp runs a
//      blocked forward substitution on its own column tile; diagonal blocks use
//      precomputed inverses, row pairs update with mma.m16n8k8.f64.
//   5. K_ext = W^T W (DSYRK, BF.cpp:993-1005) including l = W^T y (BF.cpp:1016).
//   6. Static condensation (CondensedDofInterpreter.cpp:1138-1192): the first
//      field-tile steps of a blocked Cholesky of K_ext leave the Schur complement
//      [S s; s^T .] in the trailing block.
// Numerical failures are reported per cell in info (DPOTRF INFO semantics).  The
// reverse mode, the energy error and the multi-bucket launch reuse these phases.
#include "dpg_phases.cuh"

#include <climits>

namespace {

#include "dpg_cell.cuh"

}  // namespace

namespace dpg {
namespace {
constexpr int kMaxDevices = 64;
std::mutex g_dev_mu;
int g_dev_sms[kMaxDevices] = {0};
cudaMemPool_t g_dev_pool[kMaxDevices] = {nullptr};
bool g_dev_pool_tried[kMaxDevices] = {false};
}  // namespace

int num_sms() {
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= kMaxDevices) return 148;
  std::lock_guard<std::mutex> g(g_dev_mu);
  if (g_dev_sms[dev] == 0) {
    int n = 0;
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    g_dev_sms[dev] = n > 0 ? n : 1;
    cudaGetLastError();
  }
  return g_dev_sms[dev];
}

cudaError_t ws_alloc(void** p, size_t bytes, cudaStream_t s) {
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &cap) != cudaSuccess) {
    cudaGetLastError();
    cap = cudaStreamCaptureStatusNone;
  }
  int dev = 0;
  cudaGetDevice(&dev);
  cudaMemPool_t pool = nullptr;
  if (cap == cudaStreamCaptureStatusNone && dev >= 0 && dev < kMaxDevices) {
    std::lock_guard<std::mutex> g(g_dev_mu);
    if (!g_dev_pool_tried[dev]) {
      g_dev_pool_tried[dev] = true;
      cudaMemPoolProps props;
      std::memset(&props, 0, sizeof(props));
      props.allocType = cudaMemAllocationTypePinned;
      props.location.type = cudaMemLocationTypeDevice;
      props.location.id = dev;
      cudaMemPool_t created = nullptr;
      if (cudaMemPoolCreate(&created, &props) == cudaSuccess) {
        uint64_t thr = UINT64_MAX;
        cudaMemPoolSetAttribute(created, cudaMemPoolAttrReleaseThreshold, &thr);
        g_dev_pool[dev] = created;
      }
      cudaGetLastError();
    }
    pool = g_dev_pool[dev];
  }
  if (pool) return cudaMallocFromPoolAsync(p, bytes, pool, s);
  return cudaMallocAsync(p, bytes, s);
}
}  // namespace dpg

// The small buckets run two CTAs per SM when there are cells for them.
static DpgKernelChoice choose_kernel(const DpgPlanDev* plan, int C) {
  DpgKernelChoice c = dpg_small_kernel(plan, DPG_KIND_ASSEMBLE, C);
  if (!c.k) c = DpgKernelChoice{pick_kernel(plan), NT, 1};
  return c;
}

int dpg_configure_kernels(const DpgPlanDev* plan) {
  if (plan->big) return dpg_configure_big(plan);
  // Several plans may share a kernel instance: the opt-in limit is the device's
  // maximum, so configuring one plan never lowers another's.
  int dev = 0, optin = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  size_t bytes = (size_t)plan->sm_total * sizeof(double);
  if (optin > 0 && bytes > (size_t)optin) return dpg::fail(DPG_ERR_UNSUPPORTED, "bucket needs more shared memory than one CTA has");
  if (optin > 0) bytes = (size_t)optin;
  for (int C : {1, INT_MAX}) {  // few cells, many cells (a small bucket's other kernel)
    if (C > 1 && !plan->small) break;
    const DpgKernelChoice kc = choose_kernel(plan, C);
    KernelFn k = kc.k;
    if (!k) return dpg::fail(DPG_ERR_UNSUPPORTED, "no kernel instance for this bucket size");
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess && kc.per_sm > 1)
      e = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return dpg::fail(DPG_ERR_CUDA, std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e));
  }
  return plan->adj_ok ? dpg_configure_adjoint(plan, (int)bytes) : DPG_OK;
}

int dpg_launch_assemble(const DpgPlanDev* plan, const DpgPlanDev* d_plan, const DpgLaunch* Lin, cudaStream_t stream) {
  (void)d_plan;
  if (Lin->C <= 0) return DPG_OK;
  if (plan->big) return dpg_launch_big(plan, Lin, stream);
  const DpgKernelChoice kc = choose_kernel(plan, Lin->C);
  KernelFn k = kc.k;
  if (!k) return dpg::fail(DPG_ERR_UNSUPPORTED, "no kernel instance for this bucket size");
  const int grid = std::min(Lin->C, dpg::num_sms() * kc.per_sm);
  DpgLaunch L = *Lin;
  void* scratch = nullptr;
  const bool need_scratch = !L.solve_only && plan->scratch_per_cta > 0 && !L.scratch;
  if (need_scratch) {
    cudaError_t ea = dpg::ws_alloc(&scratch, (size_t)grid * plan->scratch_per_cta * sizeof(double), stream);
    if (ea != cudaSuccess) {
      cudaGetLastError();
      return dpg::fail(DPG_ERR_OUT_OF_MEMORY, std::string("scratch allocation: ") + cudaGetErrorString(ea));
    }
    L.scratch = (double*)scratch;
  }
  size_t bytes = (size_t)plan->sm_total * sizeof(double);
  k<<<grid, kc.threads, bytes, stream>>>(*plan, L);
  cudaError_t e = cudaGetLastError();
  if (scratch) cudaFreeAsync(scratch, stream);
  if (e != cudaSuccess) return dpg::fail(DPG_ERR_CUDA, std::string("kernel launch: ") + cudaGetErrorString(e));
  return DPG_OK;
}

// Field recovery after the global solve (CondensedDofInterpreter::
// interpretGlobalCoefficients, CondensedDofInterpreter.cpp:1229-1346): per cell,
// K_ff u_f = l_f - K_ft t for the field dofs u_f given the cell's trace dofs t, with
// the local K, l of the assembly (user numbering: fields first).  One CTA per cell:
// K_ff is equilibrated (s_i = K_ii^-1/2) and Cholesky-factored in shared memory; the
// local coefficients [u_f | t] are written out.  info: 0, or the first non-positive
// pivot (1-based).
namespace {
__global__ void __launch_bounds__(256) recover_fields_kernel(int C, int M, int nf, const double* __restrict__ K,
                                                             const double* __restrict__ l,
                                                             const double* __restrict__ t_in, double* __restrict__ u,
                                                             int32_t* __restrict__ info) {
  extern __shared__ double rs[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  const int nt = M - nf;
  double* A = rs;                 // nf x nf, row-major (lower triangle used)
  double* sc = A + nf * nf;       // scaling
  double* b = sc + nf;            // right-hand side, then the solution
  __shared__ int fail;
  for (int cell = blockIdx.x; cell < C; cell += gridDim.x) {
    const double* Kc = K + (size_t)cell * M * M;
    const double* lc = l + (size_t)cell * M;
    const double* tc = t_in + (size_t)cell * nt;
    if (tid == 0) fail = 0;
    for (int i = tid; i < nf; i += blockDim.x) {
      const double d = Kc[(size_t)i * M + i];
      sc[i] = d > 0.0 ? rsqrt(d) : 1.0;
    }
    __syncthreads();
    for (int e = tid; e < nf * nf; e += blockDim.x) {
      const int i = e / nf, j = e - i * nf;
      A[e] = sc[i] * Kc[(size_t)i * M + j] * sc[j];
    }
    // b = S (l_f - K_ft t): one warp per row
    for (int i = warp; i < nf; i += nw) {
      double acc = 0.0;
      for (int j = lane; j < nt; j += 32) acc += Kc[(size_t)i * M + nf + j] * tc[j];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if (lane == 0) b[i] = sc[i] * (lc[i] - acc);
    }
    __syncthreads();
    // right-looking Cholesky, column by column
    for (int k = 0; k < nf; k++) {
      const double piv = A[k * nf + k];
      if (!(piv > 0.0)) {
        if (tid == 0 && fail == 0) fail = k + 1;
      }
      const double inv = rsqrt(piv);
      __syncthreads();
      for (int i = k + tid; i < nf; i += blockDim.x) A[i * nf + k] = (i == k) ? piv * inv : A[i * nf + k] * inv;
      __syncthreads();
      const int m = nf - 1 - k;
      for (int e = tid; e < m * m; e += blockDim.x) {
        const int i = k + 1 + e / m, j = k + 1 + e % m;
        if (j <= i) A[i * nf + j] -= A[i * nf + k] * A[j * nf + k];
      }
      __syncthreads();
    }
    // L z = b, L^T y = z (warp 0; lanes split the dot products)
    if (warp == 0) {
      for (int i = 0; i < nf; i++) {
        double acc = 0.0;
        for (int j = lane; j < i; j += 32) acc += A[i * nf + j] * b[j];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) b[i] = (b[i] - acc) / A[i * nf + i];
        __syncwarp();
      }
      for (int i = nf - 1; i >= 0; i--) {
        double acc = 0.0;
        for (int j = i + 1 + lane; j < nf; j += 32) acc += A[j * nf + i] * b[j];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) b[i] = (b[i] - acc) / A[i * nf + i];
        __syncwarp();
      }
    }
    __syncthreads();
    double* uc = u + (size_t)cell * M;
    for (int i = tid; i < M; i += blockDim.x) uc[i] = i < nf ? sc[i] * b[i] : tc[i - nf];
    if (tid == 0 && info) info[cell] = fail;
    __syncthreads();
  }
}

// nf <= 32: one warp per cell, no block barrier.  The lower 8x8 tiles of K_ff go to shared memory by
// 8-byte asynchronous copies, K_ft t is formed meanwhile from coalesced reads of the K_ft rows, each
// lane holding partial sums of all rows, which one butterfly reduce-scatter (31 shuffles) turns into
// lane i's row sum.  K_ff is then equilibrated and factored as tiles like G (factor_diag, panels and
// updates by m8n8k4), four diagonal tiles of ~1 K cycles: a row per lane in registers takes 32 steps of
// pivot, reciprocal square root, broadcast and update (200-300 cycles each), and the kernel is bound by
// that chain.  The two solves multiply by the inverse diagonal tiles.  Same info as the block kernel.
// 64,000 hex cells (nf 32, M 110; HBM floor 0.29 ms): 0.96 ms with rows in registers and shuffles, 0.68 ms now;
// 20 warps per SM at 96 registers spill: 0.71 ms
constexpr int RF_TILES = 10;  // lower tiles of a 32 x 32 matrix
constexpr int RF_SM = RF_TILES * 64 + 4 * 64 + 3 * 32 + 2;  // tiles, inverses, scales, two vectors, flag (then t)

__global__ void __launch_bounds__(32) recover_fields_warp_kernel(int C, int M, int nf, const double* __restrict__ K,
                                                                 const double* __restrict__ l,
                                                                 const double* __restrict__ t_in,
                                                                 double* __restrict__ u, int32_t* __restrict__ info) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x, i = lane, g = lane >> 2, t = lane & 3;
  double* const T = dpg_smem;
  double* const linv = T + RF_TILES * 64;
  double* const scl = linv + 4 * 64;
  double* const vb = scl + 32;
  double* const vz = vb + 32;
  int* const flag = reinterpret_cast<int*>(vz + 32);
  double* const ts = vz + 34;
  const int nt = M - nf, nb = (nf + 7) >> 3;
  for (int cell = blockIdx.x; cell < C; cell += gridDim.x) {
    const double* Kc = K + (size_t)cell * M * M;
    const double* tc = t_in + (size_t)cell * nt;
    if (lane == 0) *flag = 0;
    for (int r = 0; r < nb * 8; r++) {
      const int I = r >> 3;
      if ((lane >> 3) <= I) {
        double* dst = T + (I * (I + 1) / 2 + (lane >> 3)) * 64 + ak(r & 7, lane & 7);
        if (r < nf && lane < nf)
          asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(Kc + (size_t)r * M + lane)
                       : "memory");
        else *dst = r == lane ? 1.0 : 0.0;
      }
    }
    for (int j = lane; j < nt; j += 32)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(ts + j)), "l"(tc + j) : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
    // partial sums of K_ft(i,:) t over this lane's columns, all rows
    double p[32];
#pragma unroll
    for (int r = 0; r < 32; r++) p[r] = 0.0;
    for (int c0 = 0; c0 < nt; c0 += 32) {
      const int c = c0 + lane;
      const double tv = c < nt ? tc[c] : 0.0;
#pragma unroll
      for (int r = 0; r < 32; r++)
        if (r < nf && c < nt) p[r] += Kc[(size_t)r * M + nf + c] * tv;
    }
    // reduce-scatter: after the step with offset o a lane keeps the rows whose bit o
    // matches its own; at the end lane i holds row i's sum in p[0]
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
      const bool hi = (lane & o) != 0;
#pragma unroll
      for (int r = 0; r < o; r++) {
        const double send = hi ? p[r] : p[r + o];
        const double keep = hi ? p[r + o] : p[r];
        p[r] = keep + __shfl_xor_sync(FULL, send, o);
      }
    }
    const double li = i < nf ? l[(size_t)cell * M + i] : 0.0;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
    // equilibrate (rows and columns nf .. are padded with the identity)
    double sc = 1.0;
    if (i < nf) {
      const double d = T[((i >> 3) * ((i >> 3) + 1) / 2 + (i >> 3)) * 64 + ak(i & 7, i & 7)];
      if (d > 0.0) sc = rsqrt(d);
    }
    scl[i] = sc;
    vb[i] = i < nf ? (li - p[0]) * sc : 0.0;
    __syncwarp();
    for (int I = 0, tau = 0; I < nb; I++)
      for (int J = 0; J <= I; J++, tau++) {
        double2* q = reinterpret_cast<double2*>(T + tau * 64 + ak_cfrag(g, t));
        double2 v = *q;
        const double si = scl[I * 8 + g];
        v.x *= si * scl[J * 8 + 2 * t];
        v.y *= si * scl[J * 8 + 2 * t + 1];
        *q = v;
      }
    __syncwarp();
    for (int k = 0; k < nb; k++) {
      factor_diag(T, k, flag, 1, linv);
      const double* Li = linv + k * 64;
      for (int I = k + 1; I < nb; I++) {  // panel
        double* Tik = T + (I * (I + 1) / 2 + k) * 64;
        const double a0 = Tik[lane], a1 = Tik[32 + lane];
        double2 c = make_double2(0.0, 0.0);
        dmma(c, a0, Li[lane]);
        dmma(c, a1, Li[32 + lane]);
        __syncwarp();
        *reinterpret_cast<double2*>(Tik + ak_cfrag(g, t)) = c;
      }
      __syncwarp();
      for (int I = k + 1; I < nb; I++)  // trailing update
        for (int J = k + 1; J <= I; J++) {
          const double* Lik = T + (I * (I + 1) / 2 + k) * 64;
          const double* Ljk = T + (J * (J + 1) / 2 + k) * 64;
          double2* q = reinterpret_cast<double2*>(T + (I * (I + 1) / 2 + J) * 64 + ak_cfrag(g, t));
          double2 c = *q;
          dmma(c, -Lik[lane], Ljk[lane]);
          dmma(c, -Lik[32 + lane], Ljk[32 + lane]);
          *q = c;
        }
      // z_k = L_kk^-1 b_k (four lanes per row), then b_I -= L_Ik z_k, a lane per row
      double z = Li[ak(g, t)] * vb[k * 8 + t] + Li[ak(g, t + 4)] * vb[k * 8 + t + 4];
      z += __shfl_xor_sync(FULL, z, 1);
      z += __shfl_xor_sync(FULL, z, 2);
      if (t == 0) vz[k * 8 + g] = z;
      __syncwarp();
      if ((i >> 3) > k && (i >> 3) < nb) {
        const double* Lik = T + ((i >> 3) * ((i >> 3) + 1) / 2 + k) * 64;
        double b = vb[i];
#pragma unroll
        for (int m = 0; m < 8; m++) b -= Lik[ak(i & 7, m)] * vz[k * 8 + m];
        vb[i] = b;
      }
      __syncwarp();
    }
    // y_k = L_kk^-T z_k, then z_J -= L_kJ^T y_k for J < k
    for (int k = nb - 1; k >= 0; k--) {
      const double* Li = linv + k * 64;
      double y = Li[ak(t, g)] * vz[k * 8 + t] + Li[ak(t + 4, g)] * vz[k * 8 + t + 4];
      y += __shfl_xor_sync(FULL, y, 1);
      y += __shfl_xor_sync(FULL, y, 2);
      if (t == 0) vb[k * 8 + g] = y;
      __syncwarp();
      if ((i >> 3) < k) {
        const double* Lk = T + (k * (k + 1) / 2 + (i >> 3)) * 64;
        double z = vz[i];
#pragma unroll
        for (int m = 0; m < 8; m++) z -= Lk[ak(m, i & 7)] * vb[k * 8 + m];
        vz[i] = z;
      }
      __syncwarp();
    }
    double* uc = u + (size_t)cell * M;
    if (i < nf) uc[i] = sc * vb[i];
    for (int j = lane; j < nt; j += 32) uc[nf + j] = ts[j];
    if (lane == 0 && info) info[cell] = *flag;
    __syncwarp();
  }
}
}  // namespace

int dpg_launch_recover_fields(int C, int M, int nf, const double* K, const double* l, const double* t, double* u,
                              int32_t* info, cudaStream_t stream) {
  if (C <= 0) return DPG_OK;
  const size_t per_warp = ((size_t)RF_SM + M) * sizeof(double);
  if (nf <= 32 && per_warp <= 100 * 1024) {
    // one-warp blocks: as many resident per SM as the staging tiles allow
    static int wconfigured = 0;
    if (!wconfigured) {
      cudaFuncSetAttribute(recover_fields_warp_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024);
      wconfigured = 1;
    }
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, recover_fields_warp_kernel, 32, per_warp);
    const int sms = dpg::num_sms();
    const int grid = (int)std::min<long long>(C, (long long)sms * std::max(1, per_sm));
    recover_fields_warp_kernel<<<grid, 32, per_warp, stream>>>(C, M, nf, K, l, t, u, info);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return dpg::fail(DPG_ERR_CUDA, std::string("kernel launch: ") + cudaGetErrorString(e));
    return DPG_OK;
  }
  const size_t bytes = ((size_t)nf * nf + 2 * (size_t)nf) * sizeof(double);
  if (bytes > 200 * 1024) return dpg::fail(DPG_ERR_UNSUPPORTED, "too many field dofs for the recovery kernel");
  static int configured = 0;
  if (!configured) {
    cudaFuncSetAttribute(recover_fields_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    configured = 1;
  }
  const int grid = std::min(C, (dpg::num_sms()) * 4);
  recover_fields_kernel<<<grid, 256, bytes, stream>>>(C, M, nf, K, l, t, u, info);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return dpg::fail(DPG_ERR_CUDA, std::string("kernel launch: ") + cudaGetErrorString(e));
  return DPG_OK;
}

// Bounded-wait probe: one thread waits, with the kernels' own wait routine, on an
// mbarrier whose transaction never arrives (a flag nothing sets), and reports the
// status the assembly kernels turn into info = 0x7fff0000.  Lets a test check that a
// stalled staging copy ends the wait with an error instead of hanging the GPU.
namespace {
__global__ void wait_probe_kernel(int limit, int* status) {
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    mbar_expect_tx(&bar, 16);  // no copy will deliver these bytes
    status[0] = mbar_wait(&bar, 0, limit) ? 0 : ERR_TIMEOUT_FLAG;
  }
}
}  // namespace

extern "C" int dpg_debug_wait_probe(int limit, int* status_dev, void* stream) {
  if (limit <= 0 || !status_dev) return dpg::fail(DPG_ERR_INVALID_ARGUMENT, "bad probe arguments");
  wait_probe_kernel<<<1, 32, 0, (cudaStream_t)stream>>>(limit, status_dev);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return dpg::fail(DPG_ERR_CUDA, std::string("kernel launch: ") + cudaGetErrorString(e));
  return DPG_OK;
}

// ---------------------------------------------------------------------------
// Allocation-free launch: the per-CTA scratch comes from a fixed device array
// instead of a stream-ordered allocation.  32 MiB (4 Mi doubles): the 3D hex k=2
// bucket needs 286 KiB per CTA (B tiles 154 KiB, Gram running sums 132 KiB), so
// 114 CTAs fit; smaller buckets run one CTA per SM, or two of 8 warps.
// ---------------------------------------------------------------------------
#define DPG_NOALLOC_SCRATCH_DOUBLES ((size_t)4 << 20)

static __device__ __align__(256) double g_noalloc_scratch[DPG_NOALLOC_SCRATCH_DOUBLES];

namespace {
std::mutex g_noalloc_mu;
double* g_noalloc_ptr[64] = {nullptr};           // device address of the array, per device ordinal
unsigned long long g_noalloc_ctx[64] = {0};      // id of the context that address belongs to

// Id of the current CUDA context (0 if the driver cannot tell).  A device reset
// followed by a new context changes it, and the array's address must then be looked
// up again.  The driver functions are reached through the runtime's entry-point query,
// so the library needs no link against the driver library.
unsigned long long current_context_id() {
  typedef int (*CtxGetCurrent)(void**);
  typedef int (*CtxGetId)(void*, unsigned long long*);
  static CtxGetCurrent get_current = nullptr;
  static CtxGetId get_id = nullptr;
  static bool looked_up = false;
  if (!looked_up) {  // called with g_noalloc_mu held
    looked_up = true;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuCtxGetCurrent", (void**)&get_current, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      get_current = nullptr;
    if (cudaGetDriverEntryPoint("cuCtxGetId", (void**)&get_id, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      get_id = nullptr;
    cudaGetLastError();
  }
  void* ctx = nullptr;
  unsigned long long id = 0;
  if (get_current && get_id && get_current(&ctx) == 0 && ctx && get_id(ctx, &id) == 0) return id;
  return 0;
}
}  // namespace

int dpg_launch_assemble_noalloc(const DpgPlanDev* plan, const DpgLaunch* Lin, cudaStream_t stream) {
  if (Lin->C <= 0) return DPG_OK;
  if (plan->big) return dpg::fail(DPG_ERR_UNSUPPORTED, "dpg_assemble_noalloc: large-bucket plans need dpg_assemble");
  const DpgKernelChoice kc = choose_kernel(plan, Lin->C);
  KernelFn k = kc.k;
  if (!k) return dpg::fail(DPG_ERR_UNSUPPORTED, "no kernel instance for this bucket size");
  if (plan->scratch_per_cta > DPG_NOALLOC_SCRATCH_DOUBLES)
    return dpg::fail(DPG_ERR_UNSUPPORTED,
                     "dpg_assemble_noalloc: the bucket needs more per-CTA scratch than the fixed 32 MiB array holds");
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
    cudaGetLastError();
    return dpg::fail(DPG_ERR_CUDA, "dpg_assemble_noalloc: no current CUDA device");
  }
  double* base = nullptr;
  {
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    const unsigned long long ctx = current_context_id();
    if (!g_noalloc_ptr[dev] || (ctx != 0 && ctx != g_noalloc_ctx[dev])) {
      void* p = nullptr;
      cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
      if (e != cudaSuccess || !p) {
        cudaGetLastError();
        return dpg::fail(DPG_ERR_CUDA, std::string("dpg_assemble_noalloc: cudaGetSymbolAddress: ") +
                                           cudaGetErrorString(e));
      }
      g_noalloc_ptr[dev] = (double*)p;
      g_noalloc_ctx[dev] = current_context_id();  // the lookup made the context current if none was
    }
    base = g_noalloc_ptr[dev];
  }
  const size_t fit = plan->scratch_per_cta > 0 ? DPG_NOALLOC_SCRATCH_DOUBLES / plan->scratch_per_cta : (size_t)Lin->C;
  int grid = std::min(Lin->C, dpg::num_sms() * kc.per_sm);
  grid = (int)std::min<size_t>((size_t)grid, fit);
  DpgLaunch L = *Lin;
  L.scratch = base;
  size_t bytes = (size_t)plan->sm_total * sizeof(double);
  k<<<grid, kc.threads, bytes, stream>>>(*plan, L);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return dpg::fail(DPG_ERR_CUDA, std::string("kernel launch: ") + cudaGetErrorString(e));
  return DPG_OK;
}
