// dpg_energy.cu — the energy error's and the DLS matrices' kernel instances and launch.
#include "dpg_phases.cuh"

namespace {
#include "dpg_energy.cuh"
}  // namespace

int dpg_launch_energy(const DpgPlanDev* plan, const DpgLaunch* Lin, cudaStream_t stream) {
  if (Lin->C <= 0) return DPG_OK;
  if (plan->big) return dpg_launch_big(plan, Lin, stream);  // energy error or DLS output
  DpgKernelChoice kc = dpg_small_kernel(plan, Lin->xsol ? DPG_KIND_ENERGY : DPG_KIND_DLS, Lin->C);
  if (!kc.k) kc = DpgKernelChoice{Lin->xsol ? pick_energy_kernel(plan) : pick_dls_kernel(plan), NT, 1};
  KernelFn k = kc.k;
  if (!k) return dpg::fail(DPG_ERR_UNSUPPORTED, "no kernel instance for this bucket size");
  int dev = 0, optin = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       optin > 0 ? optin : (int)(plan->sm_total * sizeof(double)));
  if (e == cudaSuccess && kc.per_sm > 1)
    e = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
  if (e != cudaSuccess) return dpg::fail(DPG_ERR_CUDA, std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e));
  const int grid = std::min(Lin->C, dpg::num_sms() * kc.per_sm);
  DpgLaunch L = *Lin;
  void* scratch = nullptr;
  cudaError_t ea = dpg::ws_alloc(&scratch, (size_t)grid * plan->scratch_per_cta * sizeof(double), stream);
  if (ea != cudaSuccess) {
    cudaGetLastError();
    return dpg::fail(DPG_ERR_OUT_OF_MEMORY, std::string("scratch allocation: ") + cudaGetErrorString(ea));
  }
  L.scratch = (double*)scratch;
  k<<<grid, kc.threads, (size_t)plan->sm_total * sizeof(double), stream>>>(*plan, L);
  e = cudaGetLastError();
  cudaFreeAsync(scratch, stream);
  if (e != cudaSuccess) return dpg::fail(DPG_ERR_CUDA, std::string("kernel launch: ") + cudaGetErrorString(e));
  return DPG_OK;
}
