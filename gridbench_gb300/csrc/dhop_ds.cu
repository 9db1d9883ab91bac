// The FP64-accurate hopping operator in double-single arithmetic: FP64 fields and gauge, the
// spin/colour algebra on FP32 pairs (dsfloat.cuh).  GB300 runs FP64 at 1/64 of its FP32 rate, so
// the FP64 kernel is bound by the FP64 pipe, far from its memory roofline; this form moves the
// same bytes and computes on the FP32 pipe, at ~1e-14 relative accuracy.  It serves the solvers'
// FP64 operator (true residuals of the reliable updates, the FP64 CG) by default and any FP64
// operator call on request (gbdw_set_fp64_arith).
#include "dhop_kernel.cuh"
#include "dspairs.cuh"

namespace gbdw {

namespace {
int g_mode[2] = {GBDW_FP64_NATIVE, GBDW_FP64_DOUBLE_SINGLE};  // operators, solvers
thread_local int g_solver_depth = 0;
thread_local int g_forced = -1;  // Fp64ArithOverride

// one thread per link entry: FP64 complex -> (re h, re l, im h, im l)
__global__ void k_split_links(const double2* __restrict__ U, float4* __restrict__ out, int64_t n) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double2 a = U[i];
  const dsf r = ds_split(a.x), m = ds_split(a.y);
  out[i] = make_float4(r.h, r.l, m.h, m.l);
}
}  // namespace

SolverScope::SolverScope() { ++g_solver_depth; }
SolverScope::~SolverScope() { --g_solver_depth; }

Fp64ArithOverride::Fp64ArithOverride(int mode) : prev(g_forced) { g_forced = mode; }
Fp64ArithOverride::~Fp64ArithOverride() { g_forced = prev; }

bool fp64_double_single() {
  if (g_forced >= 0) return g_forced == GBDW_FP64_DOUBLE_SINGLE;
  return g_mode[g_solver_depth > 0 ? 1 : 0] == GBDW_FP64_DOUBLE_SINGLE;
}

int ds_links(const gbdw_gauge* g, const void** out) {
  if (g->prec != GBDW_F64) {
    set_error("double-single operator: needs an F64 gauge field");
    return GBDW_ERR_INVALID;
  }
  if (!g->d_ds) {
    const int64_t n = g->lat->nsite * 8 * 9;
    void* d = nullptr;
    cudaError_t e = object_alloc(&d, size_t(n) * sizeof(float4));
    if (e != cudaSuccess) return cuda_fail(e, "cudaMalloc(double-single links)");
    const int t = 256;
    k_split_links<<<unsigned((n + t - 1) / t), t, 0, stream()>>>((const double2*)g->d, (float4*)d, n);
    if ((e = cudaGetLastError()) != cudaSuccess) {
      object_free(d);
      return cuda_fail(e, "k_split_links");
    }
    count_launch();
    g->d_ds = d;
  }
  *out = g->d_ds;
  return GBDW_OK;
}

namespace {

// c y for a unit c known at run time: the components exchanged or not, times a pair of signs
struct Unit2 {
  bool swap;
  float2 sign;
};
__device__ __forceinline__ Unit2 unit_of(int code) {  // codes of LegSpin
  return {code >= 2, make_float2(code == 1 || code == 2 ? -1.f : 1.f, code == 1 || code == 3 ? -1.f : 1.f)};
}
__device__ __forceinline__ ds2 times(const Unit2& c, ds2 y) {
  return {mul2(c.swap ? swap2(y.h) : y.h, c.sign), mul2(c.swap ? swap2(y.l) : y.l, c.sign)};
}

// One leg, its direction and side known at run time (and the same for the whole CTA): spins 0 and 1
// take c0 and c1 times spins A and B.
__device__ __forceinline__ void ds_leg(const float4* u, const double2* in, int64_t row0,
                                       int LsE, int leg, ds2 (&acc)[12]) {
  const int d = leg & 3, back = leg >> 2;
  const int spin_a = d < 2 ? 3 : 2, spin_b = d < 2 ? 2 : 3;
  const int k0 = (d == 1 ? 0 : d == 3 ? 1 : 3) ^ back, k1 = (d == 0 ? 3 : d == 2 ? 2 : 1) ^ back;
  const Unit2 c0 = unit_of(k0), c1 = unit_of(k1);
  ds2 h0[3], h1[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    h0[c] = split2(in[(row0 + c) * LsE]) + times(c0, split2(in[(row0 + spin_a * 3 + c) * LsE]));
    h1[c] = split2(in[(row0 + 3 + c) * LsE]) + times(c1, split2(in[(row0 + spin_b * 3 + c) * LsE]));
  }
  const Unit2 q0 = unit_of(k0 >= 2 ? k0 ^ 1 : k0), q1 = unit_of(k1 >= 2 ? k1 ^ 1 : k1);
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    float2 s0 = make_float2(0.f, 0.f), e0 = s0, s1 = s0, e1 = s0;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const float4 a = u[r * 3 + c];  // re h, re l, im h, im l
      const float2 rh = make_float2(a.x, a.x), rl = make_float2(a.y, a.y);
      const float2 ih = make_float2(-a.z, a.z), il = make_float2(-a.w, a.w);
      dot2(rh, rl, h0[c], s0, e0);
      dot2(rh, rl, h1[c], s1, e1);
      dot2(ih, il, {swap2(h0[c].h), swap2(h0[c].l)}, s0, e0);
      dot2(ih, il, {swap2(h1[c].h), swap2(h1[c].l)}, s1, e1);
    }
    const ds2 u0 = join2(s0, e0), u1 = join2(s1, e1);
    acc[r] = acc[r] + u0;
    acc[3 + r] = acc[3 + r] + u1;
    const ds2 w0 = times(q0, u0), w1 = times(q1, u1);
    acc[6 + r] = acc[6 + r] + (d < 2 ? w1 : w0);
    acc[9 + r] = acc[9 + r] + (d < 2 ? w0 : w1);
  }
}

// One slice per thread, 128-thread CTAs with registers capped for MINB CTAs per SM.  What bounds the
// kernel is its instructions on the FP32 pipe; the epilogue (M's diagonal part and |.|^2) is FP64, on a
// pipe that is otherwise idle.  The legs are one loop: eight copies of a leg are 180 KB of code, more than
// the SM's instruction cache holds, and a quarter of the warps' time went into waiting for instructions;
// the units and spins that a leg then selects at run time are 5 % more of them.  Measured (ms; Dhop, M;
// scalar pairs -> packed pairs, legs unrolled -> this):
//   16^4 x 16  1.061, 1.45 -> 0.619, 0.717 -> 0.496, 0.516 (native FP64 1.63)
//   32^4 x 16  20.2, 22.9 -> 11.1, 11.5 -> 7.79, 8.07
//   half of 16^4 x 16  0.612, 0.975 -> 0.332, 0.466 -> 0.253, 0.270
// and 2.8e-15 from FP64 (4.0e-15 with scalar pairs).  Tried and slower: running some of the CTAs in native
// FP64 beside the others to use both pipes (2 of 16: 1.07 ms, 4 of 16: 1.20; they stay resident far longer
// than their share of the work).
template <int DAG, int EPI, int MINB>
__global__ void __launch_bounds__(DS_THREADS, MINB) k_dhop_ds(const DhopParams p) {
  dep_wait();
  const unsigned tid = sweep_block(DAG) * DS_THREADS + threadIdx.x;
  const unsigned LsE = unsigned(p.LsE);
  float part = 0.f;
  double dpart = 0.0;
  if (tid < unsigned(p.nsite) * LsE) {
    unsigned site = tid / LsE;
    const int s0 = int(tid - site * LsE);
    if (p.brick > 1) site = brick_site(p, site);
    ds2 acc[12];
#pragma unroll
    for (int k = 0; k < 12; ++k) acc[k] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
    const uint32_t* nb = p.nbr4 + size_t(site) * 8;
    const float4* u = (const float4*)p.U + size_t(site) * 72;
    const double2* in = (const double2*)p.in + s0;
#pragma unroll 1
    for (int k = 0; k < 8; ++k) {
      const int leg = (k >> 1) + 4 * (k & 1);
      ds_leg(u + 9 * leg, in, int64_t(nb[leg]) * 12, p.LsE, DAG ? leg ^ 4 : leg, acc);
    }
    cpx<double> v[1][12];
#pragma unroll
    for (int k = 0; k < 12; ++k)
      v[0][k] = {double(acc[k].h.x) + double(acc[k].l.x), double(acc[k].h.y) + double(acc[k].l.y)};
    finish_site<GBDW_F64, GBDW_F64, DAG, 1, EPI>(p, site, s0, p.LsE, p.LsP, v, part, dpart);
  }
  if (p.partials) {
    double v[1] = {dpart};
    block_partial<1>(v, p.partials);
  }
}

}  // namespace

// minb: the register cap, as CTAs per SM (4: 128 registers, 3: 168); the t-brick order comes in p.brick
int launch_dhop_ds(const DhopParams& p, int dag, int epi, int minb) {
  if (epi > 1 || (minb != 3 && minb != 4)) {
    set_error("double-single operator: Dhop and M, three or four CTAs per SM");
    return GBDW_ERR_INVALID;
  }
  const int64_t nthreads = p.nsite * p.LsE;
  const unsigned blocks = unsigned((nthreads + DS_THREADS - 1) / DS_THREADS);
#define GBDW_DSK(D, E, MB) launch_after(k_dhop_ds<D, E, MB>, blocks, DS_THREADS, 0, p)
  if (minb == 4) {
    if (dag) epi ? GBDW_DSK(1, 1, 4) : GBDW_DSK(1, 0, 4);
    else epi ? GBDW_DSK(0, 1, 4) : GBDW_DSK(0, 0, 4);
  } else {
    if (dag) epi ? GBDW_DSK(1, 1, 3) : GBDW_DSK(1, 0, 3);
    else epi ? GBDW_DSK(0, 1, 3) : GBDW_DSK(0, 0, 3);
  }
#undef GBDW_DSK
  GBDW_LAUNCHED();
  return GBDW_OK;
}

}  // namespace gbdw

using namespace gbdw;

extern "C" {

int gbdw_set_fp64_arith(int where, int mode) {
  if ((where != GBDW_FP64_OPERATORS && where != GBDW_FP64_SOLVERS) ||
      (mode != GBDW_FP64_NATIVE && mode != GBDW_FP64_DOUBLE_SINGLE)) {
    set_error("gbdw_set_fp64_arith: where GBDW_FP64_OPERATORS / GBDW_FP64_SOLVERS, mode GBDW_FP64_NATIVE / "
              "GBDW_FP64_DOUBLE_SINGLE");
    return GBDW_ERR_INVALID;
  }
  g_mode[where] = mode;
  return GBDW_OK;
}

int gbdw_get_fp64_arith(int where, int* mode) {
  if (!mode || (where != GBDW_FP64_OPERATORS && where != GBDW_FP64_SOLVERS)) return GBDW_ERR_INVALID;
  *mode = g_mode[where];
  return GBDW_OK;
}

}  // extern "C"
