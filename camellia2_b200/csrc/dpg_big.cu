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
  for (KernelFn k : {dpg_big_kernel<16>, dpg_big_kernel<32>}) {
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return dpg::fail(DPG_ERR_CUDA, std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e));
  }
  return DPG_OK;
}

// Large buckets: one CTA per SM, each with its own workspace (Z and the per-point factors).
int dpg_launch_big(const DpgPlanDev* plan, const DpgLaunch* Lin, cudaStream_t stream) {
  if (Lin->solve_only)
    return dpg::fail(DPG_ERR_UNSUPPORTED, "large-bucket plans support the assembly entry points only");
  const int grid = std::min(Lin->C, dpg::num_sms());
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
  KernelFn k = plan->big_zk == 16 ? dpg_big_kernel<16> : dpg_big_kernel<32>;
  k<<<grid, NT, (size_t)plan->bs_total * sizeof(double), stream>>>(*plan, L);
  cudaError_t e = cudaGetLastError();
  if (ws) cudaFreeAsync(ws, stream);
  if (e != cudaSuccess) return dpg::fail(DPG_ERR_CUDA, std::string("kernel launch: ") + cudaGetErrorString(e));
  return DPG_OK;
}

size_t dpg_big_workspace_bytes(const DpgPlanDev* plan, int C) {
  const int grid = std::min(std::max(C, 1), dpg::num_sms());
  return (size_t)grid * plan->bz_per_cta * sizeof(double);
}
