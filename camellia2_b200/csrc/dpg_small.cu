// dpg_small.cu — the kernels of the small buckets: 8 warps per CTA, two CTAs per SM.
//
// A bucket of up to 14 test and 8 trial tiles leaves a 16-warp CTA waiting for most of its time: two or
// three tensor blocks per warp and phase between block barriers, and a chain of diagonal tiles that
// occupies one warp.  Two CTAs with their own cells fill each other's waits.  The phases, their sums and
// their order are those of the 16-warp kernels, so the results are the same bit for bit.
// B200, one CTA per SM -> two: 256 quads of k = 2 (72 test rows) 96 -> 66 us, 16,384 CDR quads of k = 3
// (104 test rows) 9.9 -> 8.1 ms, their reverse mode 28.3 -> 21.5 ms.
#define DPG_CTA_WARPS 8
#include "dpg_phases.cuh"

static_assert(DPG_CTA_WARPS == DPG_SMALL_WARPS, "warps of the small buckets");

namespace {
#include "dpg_cell.cuh"
#include "dpg_adjoint.cuh"
#include "dpg_energy.cuh"
}  // namespace

DpgKernelChoice dpg_small_kernel(const DpgPlanDev* plan, int kind, int C) {
  DpgKernelChoice c{nullptr, NT, CTAS_PER_SM};
  if (!plan->small) return c;
  // Up to as many cells as SMs: a cell has its SM to itself, so 16 warps finish it sooner.  1..148 CDR quads of
  // k = 3 (13 test tiles), 8 -> 16 warps: assembly 102 -> 83 us, parts 98 -> 70, DLS 100 -> 79, reverse mode
  // 317 -> 245; Poisson quads of k = 1 (4 tiles): assembly 36 -> 34 us, reverse mode 44.4 -> 44.4..46.  With one
  // cell more, 16 warps take a second wave: 122 against 160 us for 149 Poisson quads of k = 3 (13 tiles).
  if (C <= dpg::num_sms()) return c;
  switch (kind) {
    case DPG_KIND_ASSEMBLE: c.k = pick_kernel(plan); break;
    case DPG_KIND_ADJOINT: c.k = pick_adjoint_kernel(plan); break;
    case DPG_KIND_ENERGY: c.k = pick_energy_kernel(plan); break;
    case DPG_KIND_DLS: c.k = pick_dls_kernel(plan); break;
  }
  return c;
}
