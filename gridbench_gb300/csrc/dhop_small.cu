// The FP32 hopping term on small lattices, where one chain of eight neighbour loads per thread is the
// time and most of the chip has nothing to do: the legs are spread over four warps.  A CTA takes 32
// (site, slice pair) items; warp d loads both neighbours of direction d at once (24 loads of 16 bytes
// in flight per thread), multiplies them by their links and leaves its 12 components in shared memory;
// warp s then adds the four parts of spin s and stores its three rows.
//
// Taken where every CTA has an SM to itself (run_dhop): 4^4 x 8 6.2 -> 4.2 us.  6^4 x 8, at the limit,
// 6.2 either way; 8^4 x 8 would take 8.2 in place of 6.2.  M gained nothing from it (6.1 against 6.2).
#include "dhop_sweep.cuh"

namespace gbdw {
namespace {

constexpr int SMALL_ITEMS = 32;

// both legs of direction D for one item
template <int D, int DAG>
__device__ __forceinline__ void small_direction(const DhopParams& p, unsigned site, int e0, cp2 (&acc)[12]) {
  const uint32_t* nb = p.nbr4 + size_t(site) * 8;
  const uint32_t n0 = nb[D], n1 = nb[D + 4];
  cpx<float> u0[3][3], u1[3][3];
  RawSpinor x0, x1;
  const uint32_t row_bytes = uint32_t(p.LsP) * 8;
  const char* in = reinterpret_cast<const char*>(p.in) + e0 * 8;
  sweep_issue(x0, in + int64_t(n0) * 12 * row_bytes, row_bytes);
  sweep_issue(x1, in + int64_t(n1) * 12 * row_bytes, row_bytes);
  LinkIO<GBDW_F32>::load(p.U, size_t(site) * 8 + D, u0);
  LinkIO<GBDW_F32>::load(p.U, size_t(site) * 8 + D + 4, u1);
  const MobLeg none{};
  sweep_leg<D, false>(u0, x0, DAG ? -1.f : 1.f, acc, none);
  sweep_leg<D, false>(u1, x1, DAG ? 1.f : -1.f, acc, none);
}

template <int DAG>
__global__ void __launch_bounds__(4 * SMALL_ITEMS) k_dhop_small(const DhopParams p) {
  dep_wait();
  __shared__ float4 parts[4][12][SMALL_ITEMS];
  const unsigned G = (unsigned(p.LsE) + 1) / 2;
  const unsigned item = sweep_block(DAG) * SMALL_ITEMS + (threadIdx.x & 31);
  const bool active = item < unsigned(p.nsite) * G;
  const unsigned site = active ? item / G : 0;
  const int e0 = int(item - site * G) * 2;
  const int w = threadIdx.x >> 5;
  if (active) {
    cp2 acc[12];
#pragma unroll
    for (int k = 0; k < 12; ++k) acc[k] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
    if (w == 0) small_direction<0, DAG>(p, site, e0, acc);
    else if (w == 1) small_direction<1, DAG>(p, site, e0, acc);
    else if (w == 2) small_direction<2, DAG>(p, site, e0, acc);
    else small_direction<3, DAG>(p, site, e0, acc);
#pragma unroll
    for (int k = 0; k < 12; ++k)
      parts[w][k][threadIdx.x & 31] = make_float4(acc[k].r.x, acc[k].r.y, acc[k].i.x, acc[k].i.y);
  }
  dep_release();
  __syncthreads();
  if (!active) return;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    cp2 a = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
    for (int d = 0; d < 4; ++d) {
      const float4 q = parts[d][w * 3 + c][threadIdx.x & 31];
      a = cadd2(a, {make_float2(q.x, q.y), make_float2(q.z, q.w)});
    }
    const cpx<float> o[2] = {{a.r.x, a.i.x}, {a.r.y, a.i.y}};
    Vec<GBDW_F32, 2>::store(p.out, int64_t(site) * 12 + w * 3 + c, e0, p.LsP, o);
  }
}

}  // namespace

int64_t small_blocks(const DhopParams& p) { return (p.nsite * ((p.LsE + 1) / 2) + SMALL_ITEMS - 1) / SMALL_ITEMS; }

int launch_dhop_small(const DhopParams& p, int dag) {
  const unsigned blocks = unsigned(small_blocks(p));
  if (dag) launch_after(k_dhop_small<1>, blocks, 4 * SMALL_ITEMS, 0, p);
  else launch_after(k_dhop_small<0>, blocks, 4 * SMALL_ITEMS, 0, p);
  GBDW_LAUNCHED();
  return GBDW_OK;
}

}  // namespace gbdw
