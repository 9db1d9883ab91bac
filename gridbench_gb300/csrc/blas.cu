// BLAS-1 on spinor fields with FP64 global sums, and the fused vector updates of the
// conjugate-gradient solvers.  Each thread handles whole 5D entries (12 complex numbers of
// one (site, slice)), so F16 fields keep one norm per entry; consecutive threads take
// consecutive slices, so every component access of a warp is contiguous.  Sums accumulate
// each entry in the arithmetic precision and everything above an entry in FP64, followed by
// the fixed-order grid reduction of common.cuh.  FP32 and FP64 fields without padding slots run the
// flat forms further down.
#include "blas.h"
#include "common.cuh"
#include "dhop_kernel.cuh"
#include "layout.cuh"

#include <type_traits>

namespace gbdw {

namespace {

template <int P>
struct Calc {
  using T = float;
};
template <>
struct Calc<GBDW_F64> {
  using T = double;
};

template <int P, class T>
__device__ __forceinline__ void ld24(const void* d, const float* nrm, int64_t site, int e, int LsE, int LsP, T (&v)[24]) {
  const float n = (P == GBDW_F16) ? nrm[site * LsE + e] : 1.f;
#pragma unroll
  for (int k = 0; k < 12; ++k) {
    const auto a = Elem<P>::ld(d, site * 12 + k, e, LsP);
    v[2 * k] = (P == GBDW_F16) ? T(float(a.r) * n) : T(a.r);
    v[2 * k + 1] = (P == GBDW_F16) ? T(float(a.i) * n) : T(a.i);
  }
}

// Stores v and returns the entry's |.|^2 as stored.
template <int P, class T>
__device__ __forceinline__ T st24(void* d, float* nrm, int64_t site, int e, int LsE, int LsP, const T (&v)[24]) {
  T s = T(0);
  if constexpr (P == GBDW_F16) {
    float m = 0.f;
#pragma unroll
    for (int k = 0; k < 24; ++k) m = fmaxf(m, fabsf(float(v[k])));
    const float sc = m > 0.f ? 1.f / m : 0.f;
    nrm[site * LsE + e] = m;
#pragma unroll
    for (int k = 0; k < 12; ++k) {
      const float2 f = __half22float2(__floats2half2_rn(float(v[2 * k]) * sc, float(v[2 * k + 1]) * sc));
      Elem<GBDW_F16>::st(d, site * 12 + k, e, LsP, f.x, f.y);
      s += T((f.x * f.x + f.y * f.y) * m * m);
    }
  } else {
    using S = typename std::conditional<P == GBDW_F64, double, float>::type;
#pragma unroll
    for (int k = 0; k < 12; ++k) {
      const S re = S(v[2 * k]), im = S(v[2 * k + 1]);
      Elem<P>::st(d, site * 12 + k, e, LsP, re, im);
      s += T(re) * T(re) + T(im) * T(im);
    }
  }
  return s;
}

struct FieldRef {
  const void* d;
  const float* n;
  int LsP;
};
struct FieldOut {
  void* d;
  float* n;
  int LsP;
};

template <int P>
__global__ void k_norm2(FieldRef x, int64_t nsite, int LsE, Reduce red) {
  using T = typename Calc<P>::T;
  double acc[1] = {0.0};
  const int64_t n = nsite * LsE;
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
    const int64_t site = i / LsE;
    const int e = int(i - site * LsE);
    T v[24];
    ld24<P>(x.d, x.n, site, e, LsE, x.LsP, v);
    T s = T(0);
#pragma unroll
    for (int k = 0; k < 24; ++k) s += v[k] * v[k];
    acc[0] += double(s);
  }
  grid_sum<1>(acc, red.partials, red.counter, red.result);
}

template <int PX, int PY>
__global__ void k_dot(FieldRef x, FieldRef y, int64_t nsite, int LsE, Reduce red) {
  using T = typename Calc<(PX == GBDW_F64 || PY == GBDW_F64) ? GBDW_F64 : GBDW_F32>::T;
  double acc[2] = {0.0, 0.0};
  const int64_t n = nsite * LsE;
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
    const int64_t site = i / LsE;
    const int e = int(i - site * LsE);
    T a[24], b[24];
    ld24<PX>(x.d, x.n, site, e, LsE, x.LsP, a);
    ld24<PY>(y.d, y.n, site, e, LsE, y.LsP, b);
    T re = T(0), im = T(0);
#pragma unroll
    for (int k = 0; k < 12; ++k) {
      re += a[2 * k] * b[2 * k] + a[2 * k + 1] * b[2 * k + 1];
      im += a[2 * k] * b[2 * k + 1] - a[2 * k + 1] * b[2 * k];
    }
    acc[0] += double(re);
    acc[1] += double(im);
  }
  grid_sum<2>(acc, red.partials, red.counter, red.result);
}

constexpr int kThreads = 256;

// y = a x + b y (FP16: 64 registers; left alone the loads ahead of the stores take 72, and 24^4 x 12 174 us for 171)
template <int PX, int PY>
__global__ void __launch_bounds__(kThreads, PY == GBDW_F16 ? 4 : 0)
    k_axpby(double a, FieldRef x, double b, FieldOut y, int64_t nsite, int LsE) {
  using T = typename Calc<(PX == GBDW_F64 || PY == GBDW_F64) ? GBDW_F64 : GBDW_F32>::T;
  const int64_t n = nsite * LsE;
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
    const int64_t site = i / LsE;
    const int e = int(i - site * LsE);
    T u[24], v[24];
    ld24<PX>(x.d, x.n, site, e, LsE, x.LsP, u);
    ld24<PY>(y.d, y.n, site, e, LsE, y.LsP, v);
#pragma unroll
    for (int k = 0; k < 24; ++k) v[k] = T(a) * u[k] + T(b) * v[k];
    st24<PY>(y.d, y.n, site, e, LsE, y.LsP, v);
  }
}

// r = b - t, |r|^2
template <int PB, int PT, int PR>
__global__ void k_xmy_norm(FieldRef b, FieldRef t, FieldOut r, int64_t nsite, int LsE, Reduce red) {
  using T = typename Calc<(PB == GBDW_F64 || PT == GBDW_F64 || PR == GBDW_F64) ? GBDW_F64 : GBDW_F32>::T;
  double acc[1] = {0.0};
  const int64_t n = nsite * LsE;
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
    const int64_t site = i / LsE;
    const int e = int(i - site * LsE);
    T u[24], v[24];
    ld24<PB>(b.d, b.n, site, e, LsE, b.LsP, u);
    ld24<PT>(t.d, t.n, site, e, LsE, t.LsP, v);
#pragma unroll
    for (int k = 0; k < 24; ++k) u[k] -= v[k];
    acc[0] += double(st24<PR>(r.d, r.n, site, e, LsE, r.LsP, u));
  }
  grid_sum<1>(acc, red.partials, red.counter, red.result);
}

// r -= alpha Ap ; |r|^2
template <int PR, int PA>
__global__ void k_cg_r(double alpha, FieldOut r, FieldRef ap, int64_t nsite, int LsE, Reduce red) {
  using T = typename Calc<PR>::T;
  double acc[1] = {0.0};
  const int64_t n = nsite * LsE;
  const T al = T(alpha);
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
    const int64_t site = i / LsE;
    const int e = int(i - site * LsE);
    T u[24], v[24];
    ld24<PR>(r.d, r.n, site, e, LsE, r.LsP, u);
    ld24<PA>(ap.d, ap.n, site, e, LsE, ap.LsP, v);
#pragma unroll
    for (int k = 0; k < 24; ++k) u[k] -= al * v[k];
    acc[0] += double(st24<PR>(r.d, r.n, site, e, LsE, r.LsP, u));
  }
  grid_sum<1>(acc, red.partials, red.counter, red.result);
}

// alpha and beta of the vector update, from the host or from the fused step's device scalars
struct CgStep {
  double alpha, beta;
  const double* dev;
  __device__ __forceinline__ bool go() {
    if (!dev) return true;
    alpha = dev[CG_ALPHA];
    beta = dev[CG_BETA];
    return dev[CG_GO] != 0.0;
  }
};

// x += alpha p ; p = r + beta p (both with the old p) ; optionally q = p.  Two CTAs per SM: three fields' rows
// loaded ahead of the stores would take 168 registers
template <int PX, int PP, int PR, int PQ>
__global__ void __launch_bounds__(kThreads, 2)
    k_cg_xp(CgStep cg, FieldOut x, FieldOut p, FieldRef r, FieldOut q, int64_t nsite, int LsE) {
  using T = typename Calc<(PX == GBDW_F64 || PR == GBDW_F64) ? GBDW_F64 : GBDW_F32>::T;
  const int64_t n = nsite * LsE;
  if (!cg.go()) return;
  const T al = T(cg.alpha), be = T(cg.beta);
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
    const int64_t site = i / LsE;
    const int e = int(i - site * LsE);
    T u[24], v[24];
    ld24<PP>(p.d, p.n, site, e, LsE, p.LsP, v);
    ld24<PX>(x.d, x.n, site, e, LsE, x.LsP, u);
#pragma unroll
    for (int k = 0; k < 24; ++k) u[k] += al * v[k];
    st24<PX>(x.d, x.n, site, e, LsE, x.LsP, u);
    ld24<PR>(r.d, r.n, site, e, LsE, r.LsP, u);
#pragma unroll
    for (int k = 0; k < 24; ++k) v[k] = u[k] + be * v[k];
    st24<PP>(p.d, p.n, site, e, LsE, p.LsP, v);
    if (PQ >= 0) st24<PQ < 0 ? GBDW_F32 : PQ>(q.d, q.n, site, e, LsE, q.LsP, v);
  }
}

// p = r + beta p ; optionally q = p (a lower-precision copy that feeds the operator)
template <int PR, int PP, int PQ>
__global__ void k_cg_p(double beta, FieldRef r, FieldOut p, FieldOut q, int64_t nsite, int LsE) {
  using T = typename Calc<(PR == GBDW_F64 || PP == GBDW_F64) ? GBDW_F64 : GBDW_F32>::T;
  const int64_t n = nsite * LsE;
  const T be = T(beta);
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
    const int64_t site = i / LsE;
    const int e = int(i - site * LsE);
    T u[24], v[24];
    ld24<PR>(r.d, r.n, site, e, LsE, r.LsP, u);
    ld24<PP>(p.d, p.n, site, e, LsE, p.LsP, v);
#pragma unroll
    for (int k = 0; k < 24; ++k) v[k] = u[k] + be * v[k];
    st24<PP>(p.d, p.n, site, e, LsE, p.LsP, v);
    if (PQ >= 0) st24<PQ < 0 ? GBDW_F32 : PQ>(q.d, q.n, site, e, LsE, q.LsP, v);
  }
}

FieldRef ref(const gbdw_field* f) { return FieldRef{f->d, f->norm, f->LsP}; }
FieldOut out(gbdw_field* f) { return FieldOut{f->d, f->norm, f->LsP}; }

int64_t grid_for(const gbdw_field* f) {
  const int64_t n = f->lat->nsite * f->LsE;
  int64_t g = (n + kThreads - 1) / kThreads;
  const int64_t cap = int64_t(num_sms()) * 8;
  return g < cap ? (g > 0 ? g : 1) : cap;
}

bool same_shape(const gbdw_field* a, const gbdw_field* b) { return a && b && a->lat == b->lat && a->nrhs == b->nrhs; }

// ------------------------------------------------------------------ slice-pair forms
// The hot CG updates on FP32/FP16 fields with an even slice count: one thread per (site, slice
// pair), 128-bit (FP32) / 64-bit (FP16) loads and stores of the paired layout, one norm pair per
// FP16 access; FP32 arithmetic as in the element-wise forms.
template <int P>
__device__ __forceinline__ void ld_pair(const void* d, const float* nrm, int64_t site, int e0, int LsE, int LsP,
                                        cpx<float> (&v)[2][12]) {
#pragma unroll
  for (int k = 0; k < 12; ++k) {
    cpx<float> x[2];
    Vec<P, 2>::load(d, site * 12 + k, e0, LsP, x);
    v[0][k] = x[0];
    v[1][k] = x[1];
  }
  if constexpr (P == GBDW_F16) {
    float n[2];
    load_norms<2>(nrm, site * LsE + e0, n);
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int k = 0; k < 12; ++k) v[j][k] = {v[j][k].r * n[j], v[j][k].i * n[j]};
  }
}

template <int PX, int PP, int PR>
__global__ void __launch_bounds__(kThreads, 2) k_cg_xp_pairs(CgStep cg, FieldOut x, FieldOut p, FieldRef r, int64_t nsite, int LsE) {
  dep_wait();
  const int G = LsE / 2;
  const int64_t n = nsite * G;
  if (!cg.go()) return;
  const float al = float(cg.alpha), be = float(cg.beta);
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
    const int64_t site = i / G;
    const int e0 = int(i - site * G) * 2;
    cpx<float> u[2][12], v[2][12];
    ld_pair<PP>(p.d, p.n, site, e0, LsE, p.LsP, v);
    ld_pair<PX>(x.d, x.n, site, e0, LsE, x.LsP, u);
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int k = 0; k < 12; ++k) u[j][k] = {fmaf(al, v[j][k].r, u[j][k].r), fmaf(al, v[j][k].i, u[j][k].i)};
    store_spinor<PX, 2>(x.d, x.n, site, e0, LsE, x.LsP, u);
    ld_pair<PR>(r.d, r.n, site, e0, LsE, r.LsP, u);
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int k = 0; k < 12; ++k) v[j][k] = {fmaf(be, v[j][k].r, u[j][k].r), fmaf(be, v[j][k].i, u[j][k].i)};
    store_spinor<PP, 2>(p.d, p.n, site, e0, LsE, p.LsP, v);
  }
}

template <int PR, int PA>
__global__ void k_cg_r_pairs(double alpha, FieldOut r, FieldRef ap, int64_t nsite, int LsE, Reduce red) {
  double acc[1] = {0.0};
  const int G = LsE / 2;
  const int64_t n = nsite * G;
  const float al = float(alpha);
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
    const int64_t site = i / G;
    const int e0 = int(i - site * G) * 2;
    cpx<float> u[2][12], v[2][12];
    ld_pair<PR>(r.d, r.n, site, e0, LsE, r.LsP, u);
    ld_pair<PA>(ap.d, ap.n, site, e0, LsE, ap.LsP, v);
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int k = 0; k < 12; ++k) u[j][k] = {fmaf(-al, v[j][k].r, u[j][k].r), fmaf(-al, v[j][k].i, u[j][k].i)};
    acc[0] += double(store_spinor<PR, 2>(r.d, r.n, site, e0, LsE, r.LsP, u));
  }
  grid_sum<1>(acc, red.partials, red.counter, red.result);
}

// ------------------------------------------------------------------ flat forms
// FP32 and FP64 fields with as many stored slots as slices are plain arrays to an element-wise
// update or a sum: one thread takes kVec 16-byte vectors a grid stride apart per pass, loaded before
// the first is used.  The entry-wise kernels above load 24 scalars per thread, 64 bytes of a 128-byte
// line per access, and run at a quarter of the L2 rate on lattices that fit there.  At 12^4 x 8 FP32
// (16 MB a field, in L2), entry-wise -> flat: axpby 13.1 -> 6.3 us.  FP32 sums stay FP32 over one
// pass's vectors (8 complex entries; the entry-wise form sums 12) and are FP64 above that: a conversion
// and an FP64 add per vector, at 1/64 of the FP32 rate, would cost more than the loads.
constexpr int kVec = 4;

template <int P>
struct Flat {
  using V = float4;
};
template <>
struct Flat<GBDW_F64> {
  using V = double2;
};

__device__ __forceinline__ float4 axpby_v(float a, float4 x, float b, float4 y) {
  return make_float4(fmaf(a, x.x, b * y.x), fmaf(a, x.y, b * y.y), fmaf(a, x.z, b * y.z), fmaf(a, x.w, b * y.w));
}
__device__ __forceinline__ double2 axpby_v(double a, double2 x, double b, double2 y) {
  return make_double2(fma(a, x.x, b * y.x), fma(a, x.y, b * y.y));
}
__device__ __forceinline__ void norm_v(float4 x, float& s) {
  s = fmaf(x.x, x.x, fmaf(x.y, x.y, fmaf(x.z, x.z, fmaf(x.w, x.w, s))));
}
__device__ __forceinline__ void norm_v(double2 x, double& s) { s = fma(x.x, x.x, fma(x.y, x.y, s)); }
// conj(x) y: an FP32 vector holds (Re, Re, Im, Im) of two slices
__device__ __forceinline__ void dot_v(float4 x, float4 y, float& re, float& im) {
  re = fmaf(x.x, y.x, fmaf(x.z, y.z, fmaf(x.y, y.y, fmaf(x.w, y.w, re))));
  im = fmaf(x.x, y.z, fmaf(-x.z, y.x, fmaf(x.y, y.w, fmaf(-x.w, y.y, im))));
}
__device__ __forceinline__ void dot_v(double2 x, double2 y, double& re, double& im) {
  re = fma(x.x, y.x, fma(x.y, y.y, re));
  im = fma(x.x, y.y, fma(-x.y, y.x, im));
}

// f(i, k) for the vectors i of this thread, loads of V of them (load(i, k)) before the first f;
// done() after each pass of V
template <int V = kVec, class LOAD, class F, class DONE>
__device__ __forceinline__ void flat_loop(int64_t n, LOAD load, F f, DONE done) {
  const int64_t step = int64_t(gridDim.x) * blockDim.x;
  for (int64_t i0 = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i0 < n; i0 += V * step) {
#pragma unroll
    for (int k = 0; k < V; ++k)
      if (i0 + k * step < n) load(i0 + k * step, k);
#pragma unroll
    for (int k = 0; k < V; ++k)
      if (i0 + k * step < n) f(i0 + k * step, k);
    done();
  }
}

// The flat sums' grid: two CTAs of kSumThreads per SM, so all of them run at once, each thread looping.
// The threads' FP64 sums meet in shared memory, where one warp adds them: an FP64 add costs a scheduler
// some 90 clocks a warp, and five per warp in shuffles were most of a short sum's time.  The last CTA adds
// the CTA sums in their order.  12^4 x 8 FP32 norm 13.1 -> 6.1 us, FP64 17.6 -> 14.0.
constexpr int kSumThreads = 512;

template <int W>
__device__ __forceinline__ void block_sum_wide(double (&v)[W], double (&buf)[W][kSumThreads]) {
#pragma unroll
  for (int w = 0; w < W; ++w) buf[w][threadIdx.x] = v[w];
  __syncthreads();
  if (threadIdx.x >= 32) return;
#pragma unroll
  for (int w = 0; w < W; ++w) {
    double a = 0.0, b = 0.0;
#pragma unroll
    for (int k = 0; k < kSumThreads; k += 64) {
      a += buf[w][k + threadIdx.x];
      b += buf[w][k + 32 + threadIdx.x];
    }
    a += b;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    v[w] = a;
  }
}

template <int W>
__device__ __forceinline__ void grid_sum_wide(double (&v)[W], const Reduce& red) {
  __shared__ double buf[W][kSumThreads];
  __shared__ bool last;
  block_sum_wide<W>(v, buf);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int w = 0; w < W; ++w) red.partials[size_t(blockIdx.x) * W + w] = v[w];
    __threadfence();
    last = atomicAdd(red.counter, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
#pragma unroll
  for (int w = 0; w < W; ++w) {
    v[w] = 0.0;
    for (unsigned k = threadIdx.x; k < gridDim.x; k += kSumThreads) v[w] += __ldcg(red.partials + size_t(k) * W + w);
  }
  block_sum_wide<W>(v, buf);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int w = 0; w < W; ++w) red.result[w] = v[w];
    *red.counter = 0u;
  }
}

template <int P>
__global__ void k_axpby_flat(typename Arith<P>::T a, const void* x_, typename Arith<P>::T b, void* y_, int64_t n) {
  dep_wait();
  using V = typename Flat<P>::V;
  const V* x = (const V*)x_;
  V* y = (V*)y_;
  V u[kVec], v[kVec];
  flat_loop(n, [&](int64_t i, int k) { u[k] = x[i]; v[k] = y[i]; },
            [&](int64_t i, int k) { y[i] = axpby_v(a, u[k], b, v[k]); }, [] {});
}

template <int P>
__global__ void __launch_bounds__(kSumThreads, 2) k_norm2_flat(const void* x_, int64_t n, Reduce red) {
  dep_wait();
  using V = typename Flat<P>::V;
  const V* x = (const V*)x_;
  double acc[1] = {0.0};
  typename Arith<P>::T s[2] = {};
  V u[2 * kVec];
  flat_loop<2 * kVec>(n, [&](int64_t i, int k) { u[k] = x[i]; },
                      [&](int64_t, int k) { norm_v(u[k], s[k / kVec]); },
                      [&] {
                        acc[0] += double(s[0]);
                        acc[0] += double(s[1]);
                        s[0] = s[1] = 0;
                      });
  dep_release();
  grid_sum_wide<1>(acc, red);
}

template <int P>
__global__ void __launch_bounds__(kSumThreads, 2) k_dot_flat(const void* x_, const void* y_, int64_t n, Reduce red) {
  dep_wait();
  using V = typename Flat<P>::V;
  const V *x = (const V*)x_, *y = (const V*)y_;
  double acc[2] = {0.0, 0.0};
  typename Arith<P>::T re = 0, im = 0;
  V u[kVec], v[kVec];
  flat_loop(n, [&](int64_t i, int k) { u[k] = x[i]; v[k] = y[i]; },
            [&](int64_t, int k) { dot_v(u[k], v[k], re, im); },
            [&] {
              acc[0] += double(re);
              acc[1] += double(im);
              re = im = 0;
            });
  dep_release();
  grid_sum_wide<2>(acc, red);
}

// r = b - t, |r|^2 (FP64)
__global__ void __launch_bounds__(kSumThreads, 2)
    k_xmy_norm_flat(const double2* b, const double2* t, double2* r, int64_t n, Reduce red) {
  dep_wait();
  double acc[1] = {0.0};
  double2 u[2], v[2];
  flat_loop<2>(n, [&](int64_t i, int k) { u[k] = b[i]; v[k] = t[i]; },
            [&](int64_t i, int k) {
              const double2 d = make_double2(u[k].x - v[k].x, u[k].y - v[k].y);
              r[i] = d;
              norm_v(d, acc[0]);
            },
            [] {});
  dep_release();
  grid_sum_wide<1>(acc, red);
}

// x += alpha p ; p = r + beta p, all FP64, and q = p in the FP32 pair layout: one thread per slice
// pair of a row, which is two FP64 vectors side by side and one FP32 vector.  Bound by the FP64 pipe (8 FMAs
// and 4 conversions a pair).  A grid-stride loop of up to four pairs a thread took 30.8 us at 12^4 x 8 and 178
// at 16^4 x 16, one pair a thread 28.7 and 163.
__global__ void k_cg_xp_f64_pairs(CgStep cg, double2* x, double2* p, const double2* r, float4* q, int64_t npair) {
  dep_wait();
  if (!cg.go()) return;
  const double alpha = cg.alpha, beta = cg.beta;
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= npair) return;
  const double2 p0 = p[2 * i], p1 = p[2 * i + 1], x0 = x[2 * i], x1 = x[2 * i + 1];
  const double2 r0 = r[2 * i], r1 = r[2 * i + 1];
  const double2 n0 = make_double2(fma(beta, p0.x, r0.x), fma(beta, p0.y, r0.y));
  const double2 n1 = make_double2(fma(beta, p1.x, r1.x), fma(beta, p1.y, r1.y));
  x[2 * i] = make_double2(fma(alpha, p0.x, x0.x), fma(alpha, p0.y, x0.y));
  x[2 * i + 1] = make_double2(fma(alpha, p1.x, x1.x), fma(alpha, p1.y, x1.y));
  p[2 * i] = n0;
  p[2 * i + 1] = n1;
  if (q) q[i] = make_float4(float(n0.x), float(n1.x), float(n0.y), float(n1.y));
}

bool flat_ok(const gbdw_field* f) { return f->prec != GBDW_F16 && f->LsP == f->LsE; }
// 16-byte vectors of a field, and a grid whose threads take kVec of them (eight CTAs per SM at most)
int64_t vectors(const gbdw_field* f) { return f->lat->nsite * 12 * int64_t(f->LsP) / (f->prec == GBDW_F64 ? 1 : 2); }
int64_t grid_flat(int64_t n) {
  const int64_t g = (n + kThreads * kVec - 1) / (kThreads * kVec);
  const int64_t cap = int64_t(num_sms()) * 8;
  return g < cap ? (g > 0 ? g : 1) : cap;
}

int64_t grid_sums(int64_t n) {
  const int64_t g = (n + kSumThreads * kVec - 1) / (kSumThreads * kVec);
  const int64_t cap = int64_t(num_sms()) * 2;
  return g < cap ? (g > 0 ? g : 1) : cap;
}

bool pairs_ok(const gbdw_field* f) { return f->prec != GBDW_F64 && f->LsE % 2 == 0 && f->LsP == f->LsE; }

int64_t grid_pairs(const gbdw_field* f) {
  const int64_t n = f->lat->nsite * (f->LsE / 2);
  int64_t g = (n + kThreads - 1) / kThreads;
  const int64_t cap = int64_t(num_sms()) * 8;
  return g < cap ? (g > 0 ? g : 1) : cap;
}

}  // namespace

// ------------------------------------------------------------------ internal entry points

int blas_norm2(const gbdw_field* x, double* out, bool fetch) {
  if (flat_ok(x)) {
    const int64_t n = vectors(x), g = grid_sums(n);
    Reduce red;
    if (int st = reduce_scratch(g, 1, &red)) return st;
    if (x->prec == GBDW_F64) launch_after(k_norm2_flat<GBDW_F64>, unsigned(g), kSumThreads, 0, x->d, n, red);
    else launch_after(k_norm2_flat<GBDW_F32>, unsigned(g), kSumThreads, 0, x->d, n, red);
    GBDW_LAUNCHED();
    return fetch ? reduce_fetch(red, 1, out) : GBDW_OK;
  }
  const int64_t g = grid_for(x);
  Reduce red;
  if (int st = reduce_scratch(g, 1, &red)) return st;
  const int64_t ns = x->lat->nsite;
  const int L = x->LsE;
  switch (x->prec) {
    case GBDW_F64: k_norm2<GBDW_F64><<<unsigned(g), kThreads, 0, stream()>>>(ref(x), ns, L, red); break;
    case GBDW_F32: k_norm2<GBDW_F32><<<unsigned(g), kThreads, 0, stream()>>>(ref(x), ns, L, red); break;
    default: k_norm2<GBDW_F16><<<unsigned(g), kThreads, 0, stream()>>>(ref(x), ns, L, red); break;
  }
  GBDW_LAUNCHED();
  return fetch ? reduce_fetch(red, 1, out) : GBDW_OK;
}

int blas_xmy_norm(const gbdw_field* b, const gbdw_field* t, gbdw_field* r, double* rr) {
  if (b->prec != GBDW_F64 || r->prec != GBDW_F64 || (t->prec != GBDW_F64 && t->prec != GBDW_F32)) {
    set_error("blas_xmy_norm: b and r must be F64, t F64 or F32");
    return GBDW_ERR_INVALID;
  }
  if (t->prec == GBDW_F64 && b != r && t != r) {
    const int64_t n = vectors(r), g = grid_sums(n);
    Reduce red;
    if (int st = reduce_scratch(g, 1, &red)) return st;
    launch_after(k_xmy_norm_flat, unsigned(g), kSumThreads, 0, (const double2*)b->d, (const double2*)t->d, (double2*)r->d, n, red);
    GBDW_LAUNCHED();
    return reduce_fetch(red, 1, rr);
  }
  const int64_t g = grid_for(r);
  Reduce red;
  if (int st = reduce_scratch(g, 1, &red)) return st;
  const int64_t ns = r->lat->nsite;
  const int L = r->LsE;
  if (t->prec == GBDW_F64)
    k_xmy_norm<GBDW_F64, GBDW_F64, GBDW_F64><<<unsigned(g), kThreads, 0, stream()>>>(ref(b), ref(t), out(r), ns, L, red);
  else
    k_xmy_norm<GBDW_F64, GBDW_F32, GBDW_F64><<<unsigned(g), kThreads, 0, stream()>>>(ref(b), ref(t), out(r), ns, L, red);
  GBDW_LAUNCHED();
  return reduce_fetch(red, 1, rr);
}

int blas_cg_r(double alpha, gbdw_field* r, const gbdw_field* ap, double* rr) {
  const int64_t ns = r->lat->nsite;
  const int L = r->LsE;
  if (pairs_ok(r) && pairs_ok(ap)) {
    const int64_t g = grid_pairs(r);
    Reduce red;
    if (int st = reduce_scratch(g, 1, &red)) return st;
    const int key = r->prec * 4 + ap->prec;
    if (key == GBDW_F32 * 4 + GBDW_F32)
      k_cg_r_pairs<GBDW_F32, GBDW_F32><<<unsigned(g), kThreads, 0, stream()>>>(alpha, out(r), ref(ap), ns, L, red);
    else if (key == GBDW_F32 * 4 + GBDW_F16)
      k_cg_r_pairs<GBDW_F32, GBDW_F16><<<unsigned(g), kThreads, 0, stream()>>>(alpha, out(r), ref(ap), ns, L, red);
    else if (key == GBDW_F16 * 4 + GBDW_F16)
      k_cg_r_pairs<GBDW_F16, GBDW_F16><<<unsigned(g), kThreads, 0, stream()>>>(alpha, out(r), ref(ap), ns, L, red);
    else {
      set_error("blas_cg_r: unsupported precision combination");
      return GBDW_ERR_INVALID;
    }
    GBDW_LAUNCHED();
    return reduce_fetch(red, 1, rr);
  }
  const int64_t g = grid_for(r);
  Reduce red;
  if (int st = reduce_scratch(g, 1, &red)) return st;
  const int key = r->prec * 4 + ap->prec;
#define GBDW_R(PR, PA)                                                                                  \
  case PR * 4 + PA:                                                                                     \
    k_cg_r<PR, PA><<<unsigned(g), kThreads, 0, stream()>>>(alpha, out(r), ref(ap), ns, L, red);         \
    break;
  switch (key) {
    GBDW_R(GBDW_F64, GBDW_F64)  // FP64 solve
    GBDW_R(GBDW_F64, GBDW_F32)  // plain: FP64 vectors, FP32 operator
    GBDW_R(GBDW_F32, GBDW_F16)  // mixed, FP16 sloppy
    GBDW_R(GBDW_F32, GBDW_F32)  // mixed, FP32 sloppy
    GBDW_R(GBDW_F16, GBDW_F16)  // mixed, FP16 sloppy with an FP16 iterated residual
    default:
      set_error("blas_cg_r: unsupported precision combination");
      return GBDW_ERR_INVALID;
  }
#undef GBDW_R
  GBDW_LAUNCHED();
  return reduce_fetch(red, 1, rr);
}

int blas_cg_xp(double alpha, double beta, gbdw_field* x, gbdw_field* p, const gbdw_field* r, gbdw_field* q,
               const double* dev) {
  const int64_t ns = r->lat->nsite;
  const int L = r->LsE;
  const CgStep cg{alpha, beta, dev};
  if (!q && pairs_ok(x) && pairs_ok(p) && pairs_ok(r) && x->prec == GBDW_F32) {
    const unsigned g = unsigned(grid_pairs(r));
    if (p->prec == GBDW_F16 && r->prec == GBDW_F16)
      launch_after(k_cg_xp_pairs<GBDW_F32, GBDW_F16, GBDW_F16>, g, kThreads, 0, cg, out(x), out(p), ref(r), ns, L);
    else if (p->prec == GBDW_F16 && r->prec == GBDW_F32)
      launch_after(k_cg_xp_pairs<GBDW_F32, GBDW_F16, GBDW_F32>, g, kThreads, 0, cg, out(x), out(p), ref(r), ns, L);
    else if (p->prec == GBDW_F32 && r->prec == GBDW_F32)
      launch_after(k_cg_xp_pairs<GBDW_F32, GBDW_F32, GBDW_F32>, g, kThreads, 0, cg, out(x), out(p), ref(r), ns, L);
    else {
      set_error("blas_cg_xp: unsupported precision combination");
      return GBDW_ERR_INVALID;
    }
    GBDW_LAUNCHED();
    return GBDW_OK;
  }
  if (x->prec == GBDW_F64 && p->prec == GBDW_F64 && r->prec == GBDW_F64 && L % 2 == 0 && x != p && x != r && p != r &&
      (!q || q->prec == GBDW_F32)) {
    const int64_t npair = ns * 12 * int64_t(L / 2);
    launch_after(k_cg_xp_f64_pairs, unsigned((npair + kThreads - 1) / kThreads), kThreads, 0,
        cg, (double2*)x->d, (double2*)p->d, (const double2*)r->d, q ? (float4*)q->d : nullptr, npair);
    GBDW_LAUNCHED();
    return GBDW_OK;
  }
  const int64_t g = grid_for(r);
  const int qp = q ? q->prec : -1;
  FieldOut qo = q ? out(q) : FieldOut{nullptr, nullptr, 0};
  const int key = ((x->prec * 4 + p->prec) * 4 + r->prec) * 8 + (qp + 1);
#define GBDW_XP(PX, PP, PR, PQ)                                                                              \
  case ((PX * 4 + PP) * 4 + PR) * 8 + (PQ + 1):                                                              \
    k_cg_xp<PX, PP, PR, PQ><<<unsigned(g), kThreads, 0, stream()>>>(cg, out(x), out(p), ref(r), qo, ns, L); \
    break;
  switch (key) {
    GBDW_XP(GBDW_F64, GBDW_F64, GBDW_F64, -1)
    GBDW_XP(GBDW_F64, GBDW_F64, GBDW_F64, GBDW_F32)
    GBDW_XP(GBDW_F32, GBDW_F16, GBDW_F32, -1)
    GBDW_XP(GBDW_F32, GBDW_F32, GBDW_F32, -1)
    GBDW_XP(GBDW_F32, GBDW_F16, GBDW_F16, -1)
    default:
      set_error("blas_cg_xp: unsupported precision combination");
      return GBDW_ERR_INVALID;
  }
#undef GBDW_XP
  GBDW_LAUNCHED();
  return GBDW_OK;
}

int blas_cg_p(double beta, const gbdw_field* r, gbdw_field* p, gbdw_field* q) {
  const int64_t g = grid_for(r);
  const int64_t ns = r->lat->nsite;
  const int L = r->LsE;
  const int qp = q ? q->prec : -1;
  FieldOut qo = q ? out(q) : FieldOut{nullptr, nullptr, 0};
  const int key = (r->prec * 4 + p->prec) * 8 + (qp + 1);
#define GBDW_P(PR, PP, PQ)                                                                             \
  case (PR * 4 + PP) * 8 + (PQ + 1):                                                                   \
    k_cg_p<PR, PP, PQ><<<unsigned(g), kThreads, 0, stream()>>>(beta, ref(r), out(p), qo, ns, L);      \
    break;
  switch (key) {
    GBDW_P(GBDW_F64, GBDW_F64, -1)
    GBDW_P(GBDW_F64, GBDW_F64, GBDW_F32)
    GBDW_P(GBDW_F32, GBDW_F16, -1)
    GBDW_P(GBDW_F32, GBDW_F32, -1)
    GBDW_P(GBDW_F16, GBDW_F16, -1)
    default:
      set_error("blas_cg_p: unsupported precision combination");
      return GBDW_ERR_INVALID;
  }
#undef GBDW_P
  GBDW_LAUNCHED();
  return GBDW_OK;
}

int blas_axpby(double a, const gbdw_field* x, double b, gbdw_field* y) {
  if (x->prec == y->prec && flat_ok(x)) {
    const int64_t n = vectors(y);
    const unsigned g = unsigned(grid_flat(n));
    if (x->prec == GBDW_F64) launch_after(k_axpby_flat<GBDW_F64>, g, kThreads, 0, a, x->d, b, y->d, n);
    else launch_after(k_axpby_flat<GBDW_F32>, g, kThreads, 0, float(a), x->d, float(b), y->d, n);
    GBDW_LAUNCHED();
    return GBDW_OK;
  }
  const int64_t g = grid_for(y);
  const int64_t ns = y->lat->nsite;
  const int L = y->LsE;
  const int key = x->prec * 4 + y->prec;
#define GBDW_AX(PX, PY) \
  case PX * 4 + PY: k_axpby<PX, PY><<<unsigned(g), kThreads, 0, stream()>>>(a, ref(x), b, out(y), ns, L); break;
  switch (key) {
    GBDW_AX(GBDW_F64, GBDW_F64)
    GBDW_AX(GBDW_F32, GBDW_F64)
    GBDW_AX(GBDW_F16, GBDW_F64)
    GBDW_AX(GBDW_F64, GBDW_F32)
    GBDW_AX(GBDW_F32, GBDW_F32)
    GBDW_AX(GBDW_F16, GBDW_F32)
    GBDW_AX(GBDW_F32, GBDW_F16)
    GBDW_AX(GBDW_F16, GBDW_F16)
    default:
      set_error("axpby: unsupported precision combination");
      return GBDW_ERR_INVALID;
  }
#undef GBDW_AX
  GBDW_LAUNCHED();
  return GBDW_OK;
}

int blas_dot(const gbdw_field* x, const gbdw_field* y, double* re, double* im) {
  if (x->prec == y->prec && flat_ok(x)) {
    const int64_t n = vectors(x), g = grid_sums(n);
    Reduce red;
    if (int st = reduce_scratch(g, 2, &red)) return st;
    if (x->prec == GBDW_F64) launch_after(k_dot_flat<GBDW_F64>, unsigned(g), kSumThreads, 0, x->d, y->d, n, red);
    else launch_after(k_dot_flat<GBDW_F32>, unsigned(g), kSumThreads, 0, x->d, y->d, n, red);
    GBDW_LAUNCHED();
    double v[2];
    if (int st = reduce_fetch(red, 2, v)) return st;
    if (re) *re = v[0];
    if (im) *im = v[1];
    return GBDW_OK;
  }
  const int64_t g = grid_for(x);
  Reduce red;
  if (int st = reduce_scratch(g, 2, &red)) return st;
  const int64_t ns = x->lat->nsite;
  const int L = x->LsE;
  const int key = x->prec * 4 + y->prec;
#define GBDW_DOT(PX, PY) \
  case PX * 4 + PY: k_dot<PX, PY><<<unsigned(g), kThreads, 0, stream()>>>(ref(x), ref(y), ns, L, red); break;
  switch (key) {
    GBDW_DOT(GBDW_F64, GBDW_F64)
    GBDW_DOT(GBDW_F32, GBDW_F32)
    GBDW_DOT(GBDW_F16, GBDW_F16)
    GBDW_DOT(GBDW_F64, GBDW_F32)
    GBDW_DOT(GBDW_F32, GBDW_F64)
    default:
      set_error("dot: unsupported precision combination");
      return GBDW_ERR_INVALID;
  }
#undef GBDW_DOT
  GBDW_LAUNCHED();
  double v[2];
  if (int st = reduce_fetch(red, 2, v)) return st;
  if (re) *re = v[0];
  if (im) *im = v[1];
  return GBDW_OK;
}

}  // namespace gbdw

using namespace gbdw;

extern "C" {

int gbdw_norm2(const gbdw_field* x, double* out) {
  if (!x || !out) return GBDW_ERR_INVALID;
  if (int st = ensure_device()) return st;
  return blas_norm2(x, out, true);
}

int gbdw_dot(const gbdw_field* x, const gbdw_field* y, double* re, double* im) {
  if (!same_shape(x, y)) {
    set_error("gbdw_dot: fields must share lattice and nrhs");
    return GBDW_ERR_INVALID;
  }
  if (int st = ensure_device()) return st;
  return blas_dot(x, y, re, im);
}

int gbdw_axpby(double a, const gbdw_field* x, double b, gbdw_field* y) {
  if (!same_shape(x, y)) {
    set_error("gbdw_axpby: fields must share lattice and nrhs");
    return GBDW_ERR_INVALID;
  }
  if (int st = ensure_device()) return st;
  return blas_axpby(a, x, b, y);
}

}  // extern "C"
