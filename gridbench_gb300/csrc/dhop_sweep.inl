// The sweep form's kernels for rows of SWEEP_TE slices: included by one unit per extent.
#include "dhop_sweep.cuh"

namespace gbdw {
namespace {

template <int DAG, int EPI, int TE, int EO>
int go_sweep(const DhopParams& p, const SweepParams& q, unsigned blocks) {
  auto kern = k_dhop_sweep<DAG, EPI, TE, EO>;
  static bool opted_in = false;  // one attribute call per instance
  if (!opted_in) {
    GBDW_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sweep_smem(TE))));
    opted_in = true;
  }
  launch_after(kern, blocks, (4 * TE + 31) / 32 * 32, sweep_smem(TE), p, q);
  GBDW_LAUNCHED();
  return GBDW_OK;
}

template <int TE, int EO>
int sweep_by_epi(const DhopParams& p, const SweepParams& q, unsigned blocks, int dag, int epi) {
  constexpr bool pow2 = (TE & (TE - 1)) == 0;
  switch (epi * 2 + dag) {
    case 0: return go_sweep<0, 0, TE, EO>(p, q, blocks);
    case 1: return go_sweep<1, 0, TE, EO>(p, q, blocks);
    case 2: return go_sweep<0, 1, TE, EO>(p, q, blocks);
    case 3: return go_sweep<1, 1, TE, EO>(p, q, blocks);
    case 5: return go_sweep<1, 2, TE, EO>(p, q, blocks);
    case 7: return go_sweep<1, 3, TE, EO>(p, q, blocks);
    case 10:
      if constexpr (EO) return go_sweep<0, 5, TE, EO>(p, q, blocks);
      break;
    case 11:
      if constexpr (EO) return go_sweep<1, 5, TE, EO>(p, q, blocks);
      break;
    case 12:
      if constexpr (pow2 && !EO) return go_sweep<0, 6, TE, EO>(p, q, blocks);
      break;
  }
  set_error("hopping kernel: epilogue not compiled for the sweep form");
  return GBDW_ERR_INVALID;
}

}  // namespace

#define GBDW_SWEEP_NAME2(TE) launch_dhop_sweep##TE
#define GBDW_SWEEP_NAME(TE) GBDW_SWEEP_NAME2(TE)
int GBDW_SWEEP_NAME(SWEEP_TE)(const DhopParams& p, const SweepParams& q, unsigned blocks, int dag, int epi) {
  return q.parity >= 0 ? sweep_by_epi<SWEEP_TE, 1>(p, q, blocks, dag, epi)
                       : sweep_by_epi<SWEEP_TE, 0>(p, q, blocks, dag, epi);
}

}  // namespace gbdw
