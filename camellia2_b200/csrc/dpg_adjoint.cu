// dpg_adjoint.cu — the reverse mode's kernel instances and launch.
#include "dpg_phases.cuh"

#include <climits>

namespace {
#include "dpg_adjoint.cuh"
}  // namespace

static DpgKernelChoice choose_adjoint_kernel(const DpgPlanDev* plan, int C) {
  DpgKernelChoice c = dpg_small_kernel(plan, DPG_KIND_ADJOINT, C);
  if (!c.k) c = DpgKernelChoice{pick_adjoint_kernel(plan), NT, 1};
  return c;
}

int dpg_configure_adjoint(const DpgPlanDev* plan, int bytes) {
  for (int C : {1, INT_MAX}) {  // few cells, many cells (a small bucket's other kernel)
    if (C > 1 && !plan->small) break;
    const DpgKernelChoice kc = choose_adjoint_kernel(plan, C);
    KernelFn k = kc.k;
    if (!k) return DPG_OK;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess && kc.per_sm > 1)
      e = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return dpg::fail(DPG_ERR_CUDA, std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e));
  }
  return DPG_OK;
}

int dpg_launch_adjoint(const DpgPlanDev* plan, const DpgLaunch* Lin, cudaStream_t stream) {
  if (Lin->C <= 0) return DPG_OK;
  if (!plan->adj_ok) return dpg::fail(DPG_ERR_UNSUPPORTED, "reverse mode is not available for this bucket");
  const DpgKernelChoice kc = choose_adjoint_kernel(plan, Lin->C);
  KernelFn k = kc.k;
  if (!k) return dpg::fail(DPG_ERR_UNSUPPORTED, "no adjoint kernel instance for this bucket size");
  const int grid = std::min(Lin->C, dpg::num_sms() * kc.per_sm);
  DpgLaunch L = *Lin;
  void* scratch = nullptr;
  const size_t per = plan->scratch_per_cta;
  cudaError_t ea = dpg::ws_alloc(&scratch, (size_t)grid * per * 2 * sizeof(double), stream);
  if (ea != cudaSuccess) {
    cudaGetLastError();
    return dpg::fail(DPG_ERR_OUT_OF_MEMORY, std::string("scratch allocation: ") + cudaGetErrorString(ea));
  }
  L.scratch = (double*)scratch;
  L.scratch2 = L.scratch + (size_t)grid * per;
  size_t bytes = (size_t)plan->sm_total * sizeof(double);
  k<<<grid, kc.threads, bytes, stream>>>(*plan, L);
  cudaError_t e = cudaGetLastError();
  cudaFreeAsync(scratch, stream);
  if (e != cudaSuccess) return dpg::fail(DPG_ERR_CUDA, std::string("kernel launch: ") + cudaGetErrorString(e));
  return DPG_OK;
}
