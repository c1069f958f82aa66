// dpg_big.cu — the large-bucket kernel's instances, workspace and launch.
#include "dpg_phases.cuh"

namespace {
#include "dpg_big.cuh"
}  // namespace

int dpg_configure_big(const DpgPlanDev* plan) {
  int dev = 0, optin = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  size_t bytes = (size_t)plan->bs_total * sizeof(double);
  if (optin > 0 && bytes > (size_t)optin) return dpg::fail(DPG_ERR_UNSUPPORTED, "bucket needs more shared memory than one CTA has");
  // every large plan shares the kernel: opt in to the device maximum so that configuring one
  // plan never lowers the limit another plan needs
  if (optin > 0) bytes = (size_t)optin;
  for (KernelFn k : {dpg_big_kernel<16, false>, dpg_big_kernel<32, false>, dpg_big_kernel<16, true>, dpg_big_kernel<32, true>}) {
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return dpg::fail(DPG_ERR_CUDA, std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e));
  }
  return DPG_OK;
}

static void cluster_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr, int grid, int size, size_t smem,
                           cudaStream_t stream) {
  std::memset(&cfg, 0, sizeof(cfg));
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = size;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(NT);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
}

// CTAs per cell of a call of C cells, and the clusters that run at once.  With at most half as many cells as SMs the
// others would idle, so a cluster shares each cell: the size with the least waves x (serial tenth + rest / size),
// at most half the cell's 64-row blocks (a step's panels and trailing tiles are what is dealt out).  ms of a
// call, one CTA per cell -> the size chosen; in brackets the fastest of all sizes where it is another:
//   Stokes quads p = 6      10 cells 3.95 -> 0.85 (8)  37: 4.02 -> 1.79 (3)  60: 4.05 -> 2.46 (2)  74: 4.08 -> 2.49 (2)
//   Stokes quads p = 4      37: 1.36 -> 0.67 (3)  60: 1.37 -> 0.85 (2)  74: 1.37 -> 0.85 (2)
//   Stokes triangles p = 4  10: 0.50 -> 0.28 (3) [0.23 (8)]  37: 0.51 -> 0.28 (3)  74: 0.51 -> 0.38 (2)
//   3D Poisson hexes k = 3  10: 2.43 -> 0.75 (5) [0.56 (8)]  37: 2.49 -> 1.08 (3)  74: 2.50 -> 1.48 (2)
// Beyond half the SMs clusters lose where one wave of CTAs holds the cells (quads p = 6, best cluster: 100 cells 4.14
// -> 4.72, 148: 4.27 -> 4.95: a cluster reloads a step's panels in every CTA and waits at two barriers per step), and
// would win where the last wave is nearly empty (75: 4.08 -> 3.54, 200: 8.32 -> 7.36); those keep one CTA.
static int team_size(const DpgPlanDev* plan, int C, KernelFn k, int* clusters) {
  const int sms = dpg::num_sms();
  *clusters = std::min(C, sms);
  int best = 1;
  double cost = 1.0;
  if (2 * C > sms) return best;
  for (int size = 2; size <= 8 && size <= (plan->Zn + 127) / 128; size++) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[1];
    cluster_config(cfg, attr, size, size, (size_t)plan->bs_total * sizeof(double), nullptr);
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, k, &cfg) != cudaSuccess || n < 1) {
      cudaGetLastError();
      break;
    }
    const double c = ((C + n - 1) / n) * (0.1 + 0.9 / size);
    if (c < cost) {
      cost = c;
      best = size;
      *clusters = std::min(C, n);
    }
  }
  return best;
}

static KernelFn team_kernel(const DpgPlanDev* plan) {
  return plan->big_zk == 16 ? dpg_big_kernel<16, true> : dpg_big_kernel<32, true>;
}

int dpg_big_team(const DpgPlanDev* plan, int C) {
  int clusters = 0;
  return team_size(plan, C, team_kernel(plan), &clusters);
}

// Large buckets: one CTA per SM, or a cluster per cell, each with its own workspace (Z and the per-point
// factors).
int dpg_launch_big(const DpgPlanDev* plan, const DpgLaunch* Lin, cudaStream_t stream) {
  if (Lin->solve_only)
    return dpg::fail(DPG_ERR_UNSUPPORTED, "large-bucket plans support the assembly entry points only");
  KernelFn kt = team_kernel(plan);
  int grid = 0;  // workspaces: CTAs or clusters
  const int team = team_size(plan, Lin->C, kt, &grid);
  DpgLaunch L = *Lin;
  void* ws = nullptr;
  if (!L.scratch) {  // a caller-provided workspace holds dpg_big_workspace_bytes(plan, C)
    cudaError_t ea = dpg::ws_alloc(&ws, (size_t)grid * plan->bz_per_cta * sizeof(double), stream);
    if (ea != cudaSuccess) {
      cudaGetLastError();
      return dpg::fail(DPG_ERR_OUT_OF_MEMORY, std::string("workspace allocation: ") + cudaGetErrorString(ea));
    }
    L.scratch = (double*)ws;
  }
  const size_t smem = (size_t)plan->bs_total * sizeof(double);
  cudaError_t e;
  if (team > 1) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[1];
    cluster_config(cfg, attr, grid * team, team, smem, stream);
    e = cudaLaunchKernelEx(&cfg, kt, *plan, (const DpgLaunch)L);
  } else {
    KernelFn k = plan->big_zk == 16 ? dpg_big_kernel<16, false> : dpg_big_kernel<32, false>;
    k<<<grid, NT, smem, stream>>>(*plan, L);
    e = cudaGetLastError();
  }
  if (ws) cudaFreeAsync(ws, stream);
  if (e != cudaSuccess) return dpg::fail(DPG_ERR_CUDA, std::string("kernel launch: ") + cudaGetErrorString(e));
  return DPG_OK;
}

size_t dpg_big_workspace_bytes(const DpgPlanDev* plan, int C) {
  const int grid = std::min(std::max(C, 1), dpg::num_sms());
  return (size_t)grid * plan->bz_per_cta * sizeof(double);
}
