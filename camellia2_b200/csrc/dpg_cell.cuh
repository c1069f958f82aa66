// dpg_cell.cuh — the assembly kernel: one persistent CTA walks cells through all phases
// (included inside the anonymous namespace of the translation units that instantiate it).

template <int NBTM, int GTM, int BTW>
__global__ void __launch_bounds__(NT, CTAS_PER_SM) dpg_cell_kernel(const __grid_constant__ DpgPlanDev P,
                                                                  const __grid_constant__ DpgLaunch L) {
  const int tid = threadIdx.x;
  double* const sm = dpg_smem;
  double* nodes_s = sm + P.sm_nodes;
  int* flag_s = reinterpret_cast<int*>(sm + P.sm_nodes + 24);
  int* tri_s = reinterpret_cast<int*>(sm + P.sm_nodes + 32);
  double* coef_s = sm + P.sm_coef;
  cta_setup(P);

  for (int cell = blockIdx.x; cell < L.C; cell += gridDim.x) {
    if (tid == 0) { flag_s[0] = 0; flag_s[1] = 0; flag_s[2] = 0; }
    if (!L.solve_only) {
      if (tid < P.nv * P.d) nodes_s[tid] = L.nodes[(size_t)cell * P.nv * P.d + tid];
      const int nco = P.nslots * P.Ptot;
      if (L.coeff)
        for (int i = tid; i < nco; i += NT) coef_s[i] = L.coeff[(size_t)cell * nco + i];
    }
    __syncthreads();
    double* GT = sm + P.sm_gt;
    if (L.solve_only) {
      const double* Gc = L.Gin + (size_t)cell * P.N * P.N;
      for (int e = tid; e < P.ngt * 64; e += NT) {
        int tau = e >> 6, idx = e & 63;
        int ij = tri_s[tau];
        int I = ij & 255, J = ij >> 8;
        int r = (idx >> 2) & 7, c = (idx >> 5) * 4 + (idx & 3);
        int gr = I * 8 + r, gc = J * 8 + c;
        double v = 0.0;
        if (gr < P.N && gc < P.N) v = Gc[(size_t)gr * P.N + gc];
        else if (gr == gc) v = 1.0;
        GT[e] = v;
      }
      __syncthreads();
    } else {
      phase_b<BTW>(P, L, cell);
      __syncthreads();
      phase_gram<GTM>(P, L, cell);
      if (L.parts) {
        __syncthreads();
        continue;
      }
    }
    phase_factor(P);
    phase_trsm<NBTM>(P, L, cell);
    phase_syrk_out(P, L, cell);
    __syncthreads();
    if (tid == 0 && L.info) {
      int f0 = flag_s[0], f1 = flag_s[1];
      int v = 0;
      if (flag_s[2]) {
        v = ERR_TIMEOUT_FLAG;
      } else if (f0 != 0) {
        int r = f0 - 1;
        int u = L.solve_only ? r : P.dev2user_test[r];
        v = (u >= 0 ? u : r) + 1;
      } else if (f1 != 0) {
        v = f1;
      }
      L.info[cell] = v;
    }
    __syncthreads();
  }
}

// Instances: register arrays sized for the test-tile count of the bucket.
#if DPG_CTA_WARPS == DPG_NWARPS
#define DPG_INSTANCES(X) \
  X(8, 3, 4) X(12, 5, 4) X(16, 6, 4) X(18, 8, 4) X(20, 8, 4) X(22, 9, 3) X(24, 12, 4) X(24, 12, 6)
#else
#define DPG_INSTANCES(X) X(9, 4, 4) X(12, 6, 6) X(14, 8, 6)
#endif

static KernelFn pick_kernel(const DpgPlanDev* plan) {
  const int per = (plan->ngb + NW - 1) / NW;
  int btw = 0;
  for (int s = 0; s < plan->nseg; s++) btw = std::max(btw, (plan->seg[s].ntile + NW - 1) / NW);
#define DPG_PICK(NB, GT, BT) \
  if (plan->NBT <= NB && per <= GT && btw <= BT) return dpg_cell_kernel<NB, GT, BT>;
  DPG_INSTANCES(DPG_PICK)
#undef DPG_PICK
  return nullptr;
}

