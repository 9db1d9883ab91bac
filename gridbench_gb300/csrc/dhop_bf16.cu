// FP16 spinors with 12-real BF16 links: the same kernels as dhop_f16.cu.
#include "dhop_launch.cuh"

namespace gbdw {
int launch_dhop_bf16(const DhopParams& p, int dag, int epi, DhopLaunch L) {
  return dispatch<GBDW_F16, GBDW_F16, GBDW_BF16, 2, 4>(p, dag, epi, L);
}
}  // namespace gbdw
