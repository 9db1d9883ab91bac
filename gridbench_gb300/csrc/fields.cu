// Lattices, gauge fields and spinor fields on the device, and the conversions between the
// reference layout (dslash_simple.h:3-5, Nsimd lanes per bench.cc:105-139) and the GB300
// layout of common.cuh.
#include <algorithm>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "dhop_kernel.cuh"
#include "layout.cuh"

namespace gbdw {

bool is_device_ptr(const void* p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged;
}

bool is_pinned_host(const void* p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeHost;
}

// Makes `bytes` of src available on the device: returns src itself for device memory,
// otherwise a copy in scratch slot `slot` (a staging buffer of the current stream).
int stage_in(const void* src, size_t bytes, int slot, const void** dev) {
  if (is_device_ptr(src) || host_in_place(src)) {
    *dev = src;
    return GBDW_OK;
  }
  void* s = scratch(bytes, slot);
  if (!s) {
    set_error("staging buffer allocation failed");
    return GBDW_ERR_ALLOC;
  }
  GBDW_CUDA(cudaMemcpyAsync(s, src, bytes, cudaMemcpyHostToDevice, stream()));
  *dev = s;
  return GBDW_OK;
}

namespace {

__device__ __forceinline__ int lane_mask(int mu, int nsimd) { return nsimd >> (3 - (mu & 3) + 1); }

// Checks a reference table and derives the 4D table.  flags: bit0 out of range,
// bit1 not 4D-factorisable.
__global__ void k_table_check(const uint64_t* nbr, const uint8_t* prm, int64_t nouter, int Ls, int nsimd,
                              uint32_t* nbr4, unsigned* flags) {
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;  // (o, s, mu)
  if (i >= nouter * Ls * 8) return;
  const int mu = int(i & 7);
  const int64_t os = i >> 3;
  const int64_t o = os / Ls;
  const int s = int(os - o * Ls);
  const uint64_t n = nbr[i];
  const uint64_t n0 = nbr[(o * Ls) * 8 + mu];
  const unsigned p = prm ? prm[i] : 0u;
  const unsigned p0 = prm ? prm[(o * Ls) * 8 + mu] : 0u;
  if (n >= uint64_t(nouter) * uint64_t(Ls)) {
    atomicOr(flags, 1u);
    return;
  }
  if (n0 % uint64_t(Ls) != 0 || n != n0 + uint64_t(s) || p != p0) atomicOr(flags, 2u);
  if (s == 0 && nbr4) {
    const uint64_t no = n0 / uint64_t(Ls);
    for (int lane = 0; lane < nsimd; ++lane) {
      const int nl = p0 ? (lane ^ lane_mask(mu, nsimd)) : lane;
      nbr4[(o * nsimd + lane) * 8 + mu] = uint32_t(no * nsimd + nl);
    }
  }
}

__global__ void k_table_general(const uint64_t* nbr, const uint8_t* prm, int64_t nouter, int Ls, int nsimd,
                                uint32_t* nbr5) {
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= nouter * Ls * 8) return;
  const int mu = int(i & 7);
  const int64_t os = i >> 3;
  const int64_t o = os / Ls;
  const int s = int(os - o * Ls);
  const uint64_t n = nbr[i];
  const unsigned p = prm ? prm[i] : 0u;
  const uint64_t no = n / uint64_t(Ls), sn = n % uint64_t(Ls);
  for (int lane = 0; lane < nsimd; ++lane) {
    const int nl = p ? (lane ^ lane_mask(mu, nsimd)) : lane;
    nbr5[((o * nsimd + lane) * Ls + s) * 8 + mu] = uint32_t((no * nsimd + nl) * Ls + sn);
  }
}

__global__ void k_table_periodic(int4 L, uint32_t* nbr4) {
  const int64_t site = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  const int64_t V = int64_t(L.x) * L.y * L.z * L.w;
  if (site >= V) return;
  int x[4];
  int64_t r = site;
  const int Ld[4] = {L.x, L.y, L.z, L.w};
  for (int d = 0; d < 4; ++d) {
    x[d] = int(r % Ld[d]);
    r /= Ld[d];
  }
  for (int mu = 0; mu < 8; ++mu) {
    const int d = mu & 3;
    int y[4] = {x[0], x[1], x[2], x[3]};
    y[d] = mu < 4 ? (y[d] + 1) % Ld[d] : (y[d] + Ld[d] - 1) % Ld[d];
    nbr4[site * 8 + mu] = uint32_t(y[0] + int64_t(Ld[0]) * (y[1] + int64_t(Ld[1]) * (y[2] + int64_t(Ld[2]) * y[3])));
  }
}

// Reference gauge (complex SRC, nsimd lanes) -> device storage P.
template <class SRC, int P>
__global__ void k_gauge_import(const SRC* src, int64_t nsite, int nsimd, void* dst) {
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;  // (site, mu)
  if (i >= nsite * 8) return;
  const int64_t site = i >> 3;
  const int mu = int(i & 7);
  const int64_t o = site / nsimd;
  const int lane = int(site - o * nsimd);
  const int nrows = (P == GBDW_F16 || P == GBDW_BF16) ? 2 : 3;
  for (int k = 0; k < nrows * 3; ++k) {
    const int64_t j = ((o * 8 + mu) * 9 + k) * nsimd + lane;
    const double re = double(src[2 * j]), im = double(src[2 * j + 1]);
    if (P == GBDW_F64) {
      ((double2*)dst)[i * 9 + k] = make_double2(re, im);
    } else if (P == GBDW_F32) {
      ((float2*)dst)[i * 9 + k] = make_float2(float(re), float(im));
    } else if (P == GBDW_F16) {
      ((__half2*)dst)[i * 6 + k] = __floats2half2_rn(float(re), float(im));
    } else {
      ((__nv_bfloat162*)dst)[i * 6 + k] = __floats2bfloat162_rn(float(re), float(im));
    }
  }
}

// The same for one lane, where both sides keep the order of the entries: one thread per entry.
template <class SRC, int P>
__global__ void k_gauge_flat(const SRC* __restrict__ src, int64_t n, void* dst) {
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;  // stored entry
  if (i >= n) return;
  constexpr int per = (P == GBDW_F16 || P == GBDW_BF16) ? 6 : 9;
  using V = typename std::conditional<sizeof(SRC) == 8, double2, float2>::type;
  const V v = __ldg(reinterpret_cast<const V*>(src) + (per == 9 ? i : i / per * 9 + i % per));
  if (P == GBDW_F64) ((double2*)dst)[i] = make_double2(v.x, v.y);
  else if (P == GBDW_F32) ((float2*)dst)[i] = make_float2(float(v.x), float(v.y));
  else if (P == GBDW_F16) ((__half2*)dst)[i] = __floats2half2_rn(float(v.x), float(v.y));
  else ((__nv_bfloat162*)dst)[i] = __floats2bfloat162_rn(float(v.x), float(v.y));
}

// Reference spinor (complex SRC, nsimd lanes, Ls slices) -> right-hand side `rhs` of a field.
template <class SRC, int P>
__global__ void k_spinor_import(const SRC* src, int64_t nsite, int Ls, int nsimd, int nrhs, int rhs, void* dst,
                                float* norm, int LsP) {
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;  // (site, s)
  if (i >= nsite * Ls) return;
  const int64_t site = i / Ls;
  const int s = int(i - site * Ls);
  const int64_t o = site / nsimd;
  const int lane = int(site - o * nsimd);
  const int LsE = Ls * nrhs;
  const int e = rhs * Ls + s;
  double v[24];
  for (int k = 0; k < 12; ++k) {
    const int64_t j = ((o * Ls + s) * 12 + k) * nsimd + lane;
    v[2 * k] = double(src[2 * j]);
    v[2 * k + 1] = double(src[2 * j + 1]);
  }
  if (P == GBDW_F16) {
    float m = 0.f;
    for (int k = 0; k < 24; ++k) m = fmaxf(m, fabsf(float(v[k])));
    const float sc = m > 0.f ? 1.f / m : 0.f;
    norm[site * LsE + e] = m;
    for (int k = 0; k < 12; ++k) Elem<GBDW_F16>::st(dst, site * 12 + k, e, LsP, float(v[2 * k]) * sc, float(v[2 * k + 1]) * sc);
  } else {
    for (int k = 0; k < 12; ++k) Elem<P>::st(dst, site * 12 + k, e, LsP, v[2 * k], v[2 * k + 1]);
  }
}

template <int P>
__device__ __forceinline__ void read_entry(const void* d, const float* norm, int64_t row, int e, int LsP, int64_t nidx,
                                           double& re, double& im) {
  const auto a = Elem<P>::ld(d, row, e, LsP);
  if (P == GBDW_F16) {
    const float n = norm[nidx];
    re = double(float(a.r) * n);
    im = double(float(a.i) * n);
  } else {
    re = double(a.r);
    im = double(a.i);
  }
}

template <class DST, int P>
__global__ void k_spinor_export(const void* srcd, const float* norm, int64_t nsite, int Ls, int nsimd, int nrhs,
                                int rhs, DST* dst, int LsP) {
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= nsite * Ls) return;
  const int64_t site = i / Ls;
  const int s = int(i - site * Ls);
  const int64_t o = site / nsimd;
  const int lane = int(site - o * nsimd);
  const int LsE = Ls * nrhs;
  const int e = rhs * Ls + s;
  for (int k = 0; k < 12; ++k) {
    double re, im;
    read_entry<P>(srcd, norm, site * 12 + k, e, LsP, site * LsE + e, re, im);
    const int64_t j = ((o * Ls + s) * 12 + k) * nsimd + lane;
    dst[2 * j] = DST(re);
    dst[2 * j + 1] = DST(im);
  }
}

// Site-block conversions (Nsimd = 1): a site's spinor is one contiguous run in both layouts, so one
// warp per site moves it with whole 16-byte accesses and permutes it in shared memory.  Lanes run over
// (row, slice pair) on the field's side; SINGLE: over (row, slice), where a right-hand side's slices
// straddle the stored pairs (several right-hand sides of an odd Ls).  e0 is the right-hand side's
// first slice.  A slice's 24 reals take kTile reals of shared memory: the lanes of one row write 28
// floats apart, two to a bank where 24 put four, and keep 16-byte alignment.  Bound by DRAM.
// One of 12 right-hand sides of 24^4 x 12 FP32 (113 us of bytes): 147 us; with the right-hand
// sides interleaved slice by slice, and one thread per 5D site, it took 771 (684 with these kernels:
// reading every twelfth slice fetches all of the field).
template <class R>
constexpr int kTile = sizeof(R) == 4 ? 28 : 26;

template <class SRC, int P, bool SINGLE>
__global__ void k_import_sites(const SRC* __restrict__ src, int64_t nsite, int Ls, int LsE, int e0, void* dst,
                               float* norm, int LsP) {
  extern __shared__ __align__(16) unsigned char sm[];
  constexpr int TS = kTile<SRC>, V = 16 / sizeof(SRC);  // V reals per 16-byte vector
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t site = int64_t(blockIdx.x) * (blockDim.x >> 5) + warp;
  if (site >= nsite) return;
  SRC* buf = reinterpret_cast<SRC*>(sm) + size_t(warp) * TS * Ls;
  float* scale = reinterpret_cast<float*>(reinterpret_cast<SRC*>(sm) + size_t(blockDim.x >> 5) * TS * Ls) + warp * Ls;
  const uint4* s = reinterpret_cast<const uint4*>(src + site * 24 * Ls);
  constexpr int VE = 24 / V;  // vectors of one slice
  for (int i = lane; i < VE * Ls; i += 32) {
    const int e = i / VE;
    *reinterpret_cast<uint4*>(buf + e * TS + (i - e * VE) * V) = __ldg(s + i);
  }
  __syncwarp();
  if constexpr (P == GBDW_F16) {
    for (int e = lane; e < Ls; e += 32) {
      const SRC* v = buf + e * TS;
      float m = 0.f;
      for (int k = 0; k < 24; ++k) m = fmaxf(m, fabsf(float(v[k])));
      scale[e] = m > 0.f ? 1.f / m : 0.f;
      norm[site * LsE + e0 + e] = m;
    }
    __syncwarp();
  }
  if constexpr (P == GBDW_F64 || SINGLE) {
    for (int i = lane; i < 12 * Ls; i += 32) {
      const int row = i / Ls, e = i - row * Ls;
      const SRC* v = buf + e * TS + 2 * row;
      if constexpr (P == GBDW_F16) Elem<P>::st(dst, site * 12 + row, e0 + e, LsP, float(v[0]) * scale[e], float(v[1]) * scale[e]);
      else Elem<P>::st(dst, site * 12 + row, e0 + e, LsP, v[0], v[1]);
    }
  } else {
    const int Q = (Ls + 1) / 2;
    for (int i = lane; i < 12 * Q; i += 32) {
      const int row = i / Q, e = 2 * (i - row * Q);
      const SRC* v = buf + e * TS + 2 * row;
      float a[4] = {float(v[0]), 0.f, float(v[1]), 0.f};
      if (e + 1 < Ls) {  // an odd Ls leaves the last pair's second slot zero
        a[1] = float(v[TS]);
        a[3] = float(v[TS + 1]);
      }
      const int64_t g = ((site * 12 + row) * LsP + e0 + e) >> 1;
      if constexpr (P == GBDW_F16) {
        const float s0 = scale[e], s1 = e + 1 < Ls ? scale[e + 1] : 0.f;
        reinterpret_cast<uint2*>(dst)[g] = make_uint2(f2h(a[0] * s0, a[1] * s1), f2h(a[2] * s0, a[3] * s1));
      } else {
        reinterpret_cast<float4*>(dst)[g] = make_float4(a[0], a[1], a[2], a[3]);
      }
    }
  }
}

template <class DST, int P, bool SINGLE>
__global__ void k_export_sites(const void* srcd, const float* norm, int64_t nsite, int Ls, int LsE, int e0, DST* dst,
                               int LsP) {
  dep_wait();
  extern __shared__ __align__(16) unsigned char sm[];
  constexpr int TS = kTile<DST>, V = 16 / sizeof(DST);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t site = int64_t(blockIdx.x) * (blockDim.x >> 5) + warp;
  if (site >= nsite) return;
  DST* buf = reinterpret_cast<DST*>(sm) + size_t(warp) * TS * Ls;
  auto put = [&](int row, int s, float re, float im) {
    if constexpr (P == GBDW_F16) {
      const float n = norm[site * LsE + e0 + s];
      re *= n;
      im *= n;
    }
    DST* b = buf + s * TS + 2 * row;
    b[0] = DST(re);
    b[1] = DST(im);
  };
  if constexpr (P == GBDW_F64) {
    const double2* d = reinterpret_cast<const double2*>(srcd) + site * 12 * LsP;
    for (int i0 = lane; i0 < 12 * Ls; i0 += 128) {  // four loads ahead of the first use
      double2 a[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int i = i0 + 32 * j, row = i / Ls;
        if (i < 12 * Ls) a[j] = d[row * LsP + e0 + i - row * Ls];
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int i = i0 + 32 * j, row = i / Ls, s = i - row * Ls;
        if (i >= 12 * Ls) break;
        DST* b = buf + s * TS + 2 * row;
        b[0] = DST(a[j].x);
        b[1] = DST(a[j].y);
      }
    }
  } else {
    auto group = [&](int row, int e) -> float4 {  // (Re, Re, Im, Im) of the stored pair of slice e
      const int64_t g = ((site * 12 + row) * LsP + e) >> 1;
      if constexpr (P == GBDW_F16) {
        const uint2 h = reinterpret_cast<const uint2*>(srcd)[g];
        const float2 r = h2f(h.x), m = h2f(h.y);
        return make_float4(r.x, r.y, m.x, m.y);
      } else {
        return reinterpret_cast<const float4*>(srcd)[g];
      }
    };
    if constexpr (SINGLE) {
      for (int i = lane; i < 12 * Ls; i += 32) {
        const int row = i / Ls, s = i - row * Ls, e = e0 + s;
        const float4 a = group(row, e);
        put(row, s, e & 1 ? a.y : a.x, e & 1 ? a.w : a.z);
      }
    } else {
      const int Q = (Ls + 1) / 2;
      for (int i0 = lane; i0 < 12 * Q; i0 += 128) {  // four loads ahead of the first use
        float4 a[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int i = i0 + 32 * j, row = i / Q;
          if (i < 12 * Q) a[j] = group(row, e0 + 2 * (i - row * Q));
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int i = i0 + 32 * j, row = i / Q, q = i - row * Q;
          if (i >= 12 * Q) break;
          put(row, 2 * q, a[j].x, a[j].z);
          if (2 * q + 1 < Ls) put(row, 2 * q + 1, a[j].y, a[j].w);
        }
      }
    }
  }
  __syncwarp();
  dep_release();
  uint4* d = reinterpret_cast<uint4*>(dst + site * 24 * Ls);
  constexpr int VE = 24 / V;
  for (int i = lane; i < VE * Ls; i += 32) {
    const int e = i / VE;
    d[i] = *reinterpret_cast<const uint4*>(buf + e * TS + (i - e * VE) * V);
  }
}

// Field-to-field precision conversion, one thread per 5D entry (site, e).
template <int PS, int PD>
__global__ void k_field_convert(const void* src, const float* snorm, void* dst, float* dnorm, int64_t nsite, int LsE,
                                int LsPs, int LsPd) {
  dep_wait();
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= nsite * LsE) return;
  const int64_t site = i / LsE;
  const int e = int(i - site * LsE);
  double v[24];
  for (int k = 0; k < 12; ++k) read_entry<PS>(src, snorm, site * 12 + k, e, LsPs, i, v[2 * k], v[2 * k + 1]);
  if (PD == GBDW_F16) {
    float m = 0.f;
    for (int k = 0; k < 24; ++k) m = fmaxf(m, fabsf(float(v[k])));
    const float sc = m > 0.f ? 1.f / m : 0.f;
    dnorm[i] = m;
    for (int k = 0; k < 12; ++k) Elem<GBDW_F16>::st(dst, site * 12 + k, e, LsPd, float(v[2 * k]) * sc, float(v[2 * k + 1]) * sc);
  } else {
    for (int k = 0; k < 12; ++k) Elem<PD>::st(dst, site * 12 + k, e, LsPd, v[2 * k], v[2 * k + 1]);
  }
}

inline unsigned nblk(int64_t n, int t) { return unsigned((n + t - 1) / t); }

}  // namespace

int field_convert(gbdw_field* dst, const gbdw_field* src) {
  const int64_t n = src->lat->nsite * src->LsE;
  if (n == 0) return GBDW_OK;
  const int t = 256;
#define GBDW_CONV(PS, PD) \
  launch_after(k_field_convert<PS, PD>, nblk(n, t), t, 0, src->d, src->norm, dst->d, dst->norm, src->lat->nsite, src->LsE, \
                                                          src->LsP, dst->LsP)
  const int key = src->prec * 4 + dst->prec;
  switch (key) {
    case GBDW_F64 * 4 + GBDW_F32: GBDW_CONV(GBDW_F64, GBDW_F32); break;
    case GBDW_F64 * 4 + GBDW_F16: GBDW_CONV(GBDW_F64, GBDW_F16); break;
    case GBDW_F32 * 4 + GBDW_F64: GBDW_CONV(GBDW_F32, GBDW_F64); break;
    case GBDW_F32 * 4 + GBDW_F16: GBDW_CONV(GBDW_F32, GBDW_F16); break;
    case GBDW_F16 * 4 + GBDW_F64: GBDW_CONV(GBDW_F16, GBDW_F64); break;
    case GBDW_F16 * 4 + GBDW_F32: GBDW_CONV(GBDW_F16, GBDW_F32); break;
    case GBDW_F64 * 4 + GBDW_F64:
    case GBDW_F32 * 4 + GBDW_F32:
      GBDW_CUDA(cudaMemcpyAsync(dst->d, src->d, src->bytes, cudaMemcpyDeviceToDevice, stream()));
      return GBDW_OK;
    case GBDW_F16 * 4 + GBDW_F16:
      GBDW_CUDA(cudaMemcpyAsync(dst->d, src->d, src->bytes, cudaMemcpyDeviceToDevice, stream()));
      GBDW_CUDA(cudaMemcpyAsync(dst->norm, src->norm, size_t(n) * sizeof(float), cudaMemcpyDeviceToDevice, stream()));
      return GBDW_OK;
    default:
      set_error("unsupported field conversion");
      return GBDW_ERR_INVALID;
  }
#undef GBDW_CONV
  GBDW_LAUNCHED();
  return GBDW_OK;
}

int lattice_from_table_impl(gbdw_lattice** out, uint64_t nouter, int Ls, int nsimd, const uint64_t* nbr,
                            const uint8_t* prm, bool force_general) {
  if (!out || !nbr || nouter == 0 || Ls < 1 || !(nsimd == 1 || nsimd == 2 || nsimd == 4 || nsimd == 8 || nsimd == 16)) {
    set_error("gbdw_lattice_from_table: invalid arguments");
    return GBDW_ERR_INVALID;
  }
  if (double(nouter) * nsimd * Ls * 12 >= 2147483647.0) {
    set_error("gbdw_lattice_from_table: lattice too large for 32-bit site indexing");
    return GBDW_ERR_INVALID;
  }
  if (int st = ensure_device()) return st;
  const int64_t nent = int64_t(nouter) * Ls * 8;
  const void* dnbr = nullptr;
  const void* dprm = nullptr;
  if (int st = stage_in(nbr, size_t(nent) * 8, 2, &dnbr)) return st;
  if (prm)
    if (int st = stage_in(prm, size_t(nent), 3, &dprm)) return st;
  gbdw_lattice* L = new gbdw_lattice();
  L->nsite = int64_t(nouter) * nsimd;
  L->Ls = Ls;
  L->nsimd = nsimd;
  L->nbr4 = nullptr;
  L->nbr5 = nullptr;
  unsigned* dflags = (unsigned*)scratch(64, 4);
  if (!dflags) {
    delete L;
    set_error("flag allocation failed");
    return GBDW_ERR_ALLOC;
  }
  auto fail = [&](int st) {
    if (L->nbr4) object_free(L->nbr4);
    if (L->nbr5) object_free(L->nbr5);
    delete L;
    return st;
  };
  cudaError_t e = object_alloc((void**)&L->nbr4, size_t(L->nsite) * 8 * sizeof(uint32_t));
  if (e != cudaSuccess) return fail(cuda_fail(e, "cudaMalloc(nbr4)"));
  if ((e = cudaMemsetAsync(dflags, 0, sizeof(unsigned), stream())) != cudaSuccess) return fail(cuda_fail(e, "memset"));
  k_table_check<<<nblk(nent, 256), 256, 0, stream()>>>((const uint64_t*)dnbr, (const uint8_t*)dprm, int64_t(nouter), Ls,
                                                        nsimd, L->nbr4, dflags);
  if ((e = cudaGetLastError()) != cudaSuccess) return fail(cuda_fail(e, "k_table_check"));
  count_launch();
  unsigned flags = 0;
  if ((e = cudaMemcpyAsync(&flags, dflags, sizeof(unsigned), cudaMemcpyDeviceToHost, stream())) != cudaSuccess)
    return fail(cuda_fail(e, "flags"));
  if ((e = cudaStreamSynchronize(stream())) != cudaSuccess) return fail(cuda_fail(e, "sync"));
  if (flags & 1u) {
    set_error("neighbour table entry out of range (>= nsite*Ls)");
    return fail(GBDW_ERR_TABLE);
  }
  L->fast = !(flags & 2u) && !force_general;
  if (!L->fast) {
    e = object_alloc((void**)&L->nbr5, size_t(L->nsite) * Ls * 8 * sizeof(uint32_t));
    if (e != cudaSuccess) return fail(cuda_fail(e, "cudaMalloc(nbr5)"));
    k_table_general<<<nblk(nent, 256), 256, 0, stream()>>>((const uint64_t*)dnbr, (const uint8_t*)dprm, int64_t(nouter),
                                                            Ls, nsimd, L->nbr5);
    if ((e = cudaGetLastError()) != cudaSuccess) return fail(cuda_fail(e, "k_table_general"));
    count_launch();
  }
  for (int d = 0; d < 4; ++d) L->dims[d] = 0;
  *out = L;
  return GBDW_OK;
}

}  // namespace gbdw

using namespace gbdw;

extern "C" {

int gbdw_lattice_from_table(gbdw_lattice** lat, uint64_t nsite, int Ls, int nsimd, const uint64_t* nbr,
                            const uint8_t* prm) {
  return lattice_from_table_impl(lat, nsite, Ls, nsimd, nbr, prm, false);
}

int gbdw_lattice_create(gbdw_lattice** lat, const int dims[4], int Ls) {
  if (!lat || !dims || Ls < 1) {
    set_error("gbdw_lattice_create: invalid arguments");
    return GBDW_ERR_INVALID;
  }
  int64_t V = 1;
  for (int d = 0; d < 4; ++d) {
    if (dims[d] < 1) {
      set_error("gbdw_lattice_create: dims must be >= 1");
      return GBDW_ERR_INVALID;
    }
    V *= dims[d];
  }
  if (double(V) * Ls * 12 >= 2147483647.0) {
    set_error("gbdw_lattice_create: lattice too large for 32-bit site indexing");
    return GBDW_ERR_INVALID;
  }
  if (int st = ensure_device()) return st;
  gbdw_lattice* L = new gbdw_lattice();
  L->nsite = V;
  L->Ls = Ls;
  L->nsimd = 1;
  L->fast = true;
  L->nbr5 = nullptr;
  for (int d = 0; d < 4; ++d) L->dims[d] = dims[d];
  cudaError_t e = object_alloc((void**)&L->nbr4, size_t(V) * 8 * sizeof(uint32_t));
  if (e != cudaSuccess) {
    delete L;
    return cuda_fail(e, "cudaMalloc(nbr4)");
  }
  k_table_periodic<<<nblk(V, 256), 256, 0, stream()>>>(make_int4(dims[0], dims[1], dims[2], dims[3]), L->nbr4);
  if ((e = cudaGetLastError()) != cudaSuccess) {
    object_free(L->nbr4);
    delete L;
    return cuda_fail(e, "k_table_periodic");
  }
  count_launch();
  *lat = L;
  return GBDW_OK;
}

int gbdw_lattice_destroy(gbdw_lattice* lat) {
  if (!lat) return GBDW_OK;
  cudaStreamSynchronize(stream());
  if (lat->nbr4) object_free(lat->nbr4);
  if (lat->nbr5) object_free(lat->nbr5);
  if (lat->cbsite) object_free(lat->cbsite);
  delete lat;
  return GBDW_OK;
}

int gbdw_lattice_info(const gbdw_lattice* lat, int64_t info[4]) {
  if (!lat || !info) return GBDW_ERR_INVALID;
  info[0] = lat->nsite;
  info[1] = lat->Ls;
  info[2] = lat->nsimd;
  info[3] = lat->fast ? 1 : 0;
  return GBDW_OK;
}

int gbdw_gauge_create(gbdw_gauge** g, const gbdw_lattice* lat, int prec, const void* src, int src_prec) {
  if (!g || !lat || !src || prec < GBDW_F64 || prec > GBDW_BF16 || (src_prec != GBDW_F64 && src_prec != GBDW_F32)) {
    set_error("gbdw_gauge_create: invalid arguments");
    return GBDW_ERR_INVALID;
  }
  if (int st = ensure_device()) return st;
  const int64_t nlink = lat->nsite * 8;
  const size_t src_bytes = size_t(nlink) * 9 * (src_prec == GBDW_F64 ? 16 : 8);
  const void* dsrc = nullptr;
  if (int st = stage_in(src, src_bytes, 2, &dsrc)) return st;
  gbdw_gauge* G = new gbdw_gauge();
  G->lat = lat;
  G->prec = prec;
  G->bytes = size_t(nlink) * link_bytes(prec);
  cudaError_t e = object_alloc((void**)&G->d, G->bytes);
  if (e != cudaSuccess) {
    delete G;
    return cuda_fail(e, "cudaMalloc(gauge)");
  }
  const int t = 256;
  const int64_t nsite = lat->nsite;
  const int ns = lat->nsimd;
  const bool flat = ns == 1 && (uintptr_t(dsrc) & 15) == 0;
  const int64_t entries = nlink * (prec == GBDW_F16 || prec == GBDW_BF16 ? 6 : 9);
#define GBDW_GI(SRC, P)                                                                            \
  if (flat) k_gauge_flat<SRC, P><<<nblk(entries, t), t, 0, stream()>>>((const SRC*)dsrc, entries, G->d); \
  else k_gauge_import<SRC, P><<<nblk(nlink, t), t, 0, stream()>>>((const SRC*)dsrc, nsite, ns, G->d)
  if (src_prec == GBDW_F64) {
    switch (prec) {
      case GBDW_F64: GBDW_GI(double, GBDW_F64); break;
      case GBDW_F32: GBDW_GI(double, GBDW_F32); break;
      case GBDW_F16: GBDW_GI(double, GBDW_F16); break;
      default: GBDW_GI(double, GBDW_BF16); break;
    }
  } else {
    switch (prec) {
      case GBDW_F64: GBDW_GI(float, GBDW_F64); break;
      case GBDW_F32: GBDW_GI(float, GBDW_F32); break;
      case GBDW_F16: GBDW_GI(float, GBDW_F16); break;
      default: GBDW_GI(float, GBDW_BF16); break;
    }
  }
#undef GBDW_GI
  if ((e = cudaGetLastError()) != cudaSuccess) {
    object_free(G->d);
    delete G;
    return cuda_fail(e, "k_gauge_import");
  }
  count_launch();
  *g = G;
  return GBDW_OK;
}

int gbdw_gauge_destroy(gbdw_gauge* g) {
  if (!g) return GBDW_OK;
  cudaStreamSynchronize(stream());
  object_free(g->d);
  if (g->d_ds) object_free(g->d_ds);
  delete g;
  return GBDW_OK;
}

int gbdw_field_create(gbdw_field** f, const gbdw_lattice* lat, int prec, int nrhs) {
  if (!f || !lat || prec < GBDW_F64 || prec > GBDW_F16 || nrhs < 1) {
    set_error("gbdw_field_create: invalid arguments");
    return GBDW_ERR_INVALID;
  }
  if (double(lat->nsite) * lat->Ls * nrhs * 12 >= 2147483647.0) {
    set_error("gbdw_field_create: field too large for 32-bit indexing");
    return GBDW_ERR_INVALID;
  }
  if (int st = ensure_device()) return st;
  gbdw_field* F = new gbdw_field();
  F->lat = lat;
  F->prec = prec;
  F->nrhs = nrhs;
  F->LsE = lat->Ls * nrhs;
  F->LsP = padded_slices(prec, F->LsE);
  F->norm = nullptr;
  F->bytes = size_t(F->elems()) * spinor_elem_bytes(prec);
  cudaError_t e = object_alloc((void**)&F->d, F->bytes);
  if (e != cudaSuccess) {
    delete F;
    return cuda_fail(e, "cudaMalloc(field)");
  }
  if (prec == GBDW_F16) {
    e = object_alloc((void**)&F->norm, size_t(lat->nsite) * F->LsE * sizeof(float));
    if (e != cudaSuccess) {
      object_free(F->d);
      delete F;
      return cuda_fail(e, "cudaMalloc(norm)");
    }
  }
  *f = F;
  return gbdw_field_zero(F);
}

int gbdw_field_destroy(gbdw_field* f) {
  if (!f) return GBDW_OK;
  cudaStreamSynchronize(stream());
  object_free(f->d);
  if (f->norm) object_free(f->norm);
  delete f;
  return GBDW_OK;
}

int gbdw_field_zero(gbdw_field* f) {
  if (!f) return GBDW_ERR_INVALID;
  GBDW_CUDA(cudaMemsetAsync(f->d, 0, f->bytes, stream()));
  if (f->norm) GBDW_CUDA(cudaMemsetAsync(f->norm, 0, size_t(f->lat->nsite) * f->LsE * sizeof(float), stream()));
  return GBDW_OK;
}

int gbdw_field_import(gbdw_field* f, int rhs, const void* src, int src_prec) {
  if (!f || !src || rhs < 0 || rhs >= f->nrhs || (src_prec != GBDW_F64 && src_prec != GBDW_F32)) {
    set_error("gbdw_field_import: invalid arguments");
    return GBDW_ERR_INVALID;
  }
  const gbdw_lattice* L = f->lat;
  const int64_t n5 = L->nsite * L->Ls;
  const size_t bytes = size_t(n5) * 12 * (src_prec == GBDW_F64 ? 16 : 8);
  const int t = 256;
  // site blocks: up to 4 warps per CTA, the tile and the F16 scales of one site per warp
  const size_t warp_smem = size_t(L->Ls) * ((src_prec == GBDW_F64 ? kTile<double> * 8 : kTile<float> * 4) + 4);
  const int warps = int(std::min<size_t>(4, 48 * 1024 / warp_smem));
  const bool blocks = L->nsimd == 1 && warps > 0;
  const bool single = f->nrhs > 1 && L->Ls % 2;
  // host memory goes through a copy engine into the stream's staging buffer: the copy needs
  // no SMs, so copies of work queued on other streams overlap with it
  const void* dsrc = nullptr;
  if (int st = stage_in(src, bytes, 5, &dsrc)) return st;
  if (blocks && (uintptr_t(dsrc) & 15) == 0) {
    const unsigned nb = unsigned((L->nsite + warps - 1) / warps);
#define GBDW_IB(SRC, P)                                                                                       \
  (single ? k_import_sites<SRC, P, true> : k_import_sites<SRC, P, false>)<<<nb, 32 * warps, warps * warp_smem, stream()>>>( \
      (const SRC*)dsrc, L->nsite, L->Ls, f->LsE, rhs * L->Ls, f->d, f->norm, f->LsP)
    if (src_prec == GBDW_F64) {
      if (f->prec == GBDW_F64) GBDW_IB(double, GBDW_F64);
      else if (f->prec == GBDW_F32) GBDW_IB(double, GBDW_F32);
      else GBDW_IB(double, GBDW_F16);
    } else {
      if (f->prec == GBDW_F64) GBDW_IB(float, GBDW_F64);
      else if (f->prec == GBDW_F32) GBDW_IB(float, GBDW_F32);
      else GBDW_IB(float, GBDW_F16);
    }
#undef GBDW_IB
    GBDW_LAUNCHED();
    return GBDW_OK;
  }
#define GBDW_SI(SRC, P)                                                                                      \
  k_spinor_import<SRC, P><<<nblk(n5, t), t, 0, stream()>>>((const SRC*)dsrc, L->nsite, L->Ls, L->nsimd, f->nrhs, rhs, \
                                                          f->d, f->norm, f->LsP)
  if (src_prec == GBDW_F64) {
    if (f->prec == GBDW_F64) GBDW_SI(double, GBDW_F64);
    else if (f->prec == GBDW_F32) GBDW_SI(double, GBDW_F32);
    else GBDW_SI(double, GBDW_F16);
  } else {
    if (f->prec == GBDW_F64) GBDW_SI(float, GBDW_F64);
    else if (f->prec == GBDW_F32) GBDW_SI(float, GBDW_F32);
    else GBDW_SI(float, GBDW_F16);
  }
#undef GBDW_SI
  GBDW_LAUNCHED();
  return GBDW_OK;
}

static int field_export(const gbdw_field* f, int rhs, void* dst, int dst_prec, bool sync) {
  if (!f || !dst || rhs < 0 || rhs >= f->nrhs || (dst_prec != GBDW_F64 && dst_prec != GBDW_F32)) {
    set_error("gbdw_field_export: invalid arguments");
    return GBDW_ERR_INVALID;
  }
  const gbdw_lattice* L = f->lat;
  const int64_t n5 = L->nsite * L->Ls;
  const size_t bytes = size_t(n5) * 12 * (dst_prec == GBDW_F64 ? 16 : 8);
  const int t = 256;
  const size_t warp_smem = size_t(L->Ls) * (dst_prec == GBDW_F64 ? kTile<double> * 8 : kTile<float> * 4);
  const int warps = int(std::min<size_t>(4, 48 * 1024 / warp_smem));
  const bool blocks = L->nsimd == 1 && warps > 0;
  const bool single = f->nrhs > 1 && L->Ls % 2;
  const bool dev = is_device_ptr(dst);
  void* ddst = dst;
  if (!dev) {
    if (!sync && !is_pinned_host(dst)) {
      set_error("gbdw_field_export_async: the destination must be device or page-locked host memory");
      return GBDW_ERR_INVALID;
    }
    ddst = scratch(bytes, 6);
    if (!ddst) {
      set_error("staging buffer allocation failed");
      return GBDW_ERR_ALLOC;
    }
  }
  if (blocks && (uintptr_t(ddst) & 15) == 0) {
    const unsigned nb = unsigned((L->nsite + warps - 1) / warps);
#define GBDW_EB(DST, P)                                                                                       \
  launch_after(single ? k_export_sites<DST, P, true> : k_export_sites<DST, P, false>, nb, 32 * warps, warps * warp_smem, \
      f->d, f->norm, L->nsite, L->Ls, f->LsE, rhs * L->Ls, (DST*)ddst, f->LsP)
    if (dst_prec == GBDW_F64) {
      if (f->prec == GBDW_F64) GBDW_EB(double, GBDW_F64);
      else if (f->prec == GBDW_F32) GBDW_EB(double, GBDW_F32);
      else GBDW_EB(double, GBDW_F16);
    } else {
      if (f->prec == GBDW_F64) GBDW_EB(float, GBDW_F64);
      else if (f->prec == GBDW_F32) GBDW_EB(float, GBDW_F32);
      else GBDW_EB(float, GBDW_F16);
    }
#undef GBDW_EB
  } else {
#define GBDW_SE(DST, P) \
  k_spinor_export<DST, P><<<nblk(n5, t), t, 0, stream()>>>(f->d, f->norm, L->nsite, L->Ls, L->nsimd, f->nrhs, rhs, \
                                                           (DST*)ddst, f->LsP)
  if (dst_prec == GBDW_F64) {
    if (f->prec == GBDW_F64) GBDW_SE(double, GBDW_F64);
    else if (f->prec == GBDW_F32) GBDW_SE(double, GBDW_F32);
    else GBDW_SE(double, GBDW_F16);
  } else {
    if (f->prec == GBDW_F64) GBDW_SE(float, GBDW_F64);
    else if (f->prec == GBDW_F32) GBDW_SE(float, GBDW_F32);
    else GBDW_SE(float, GBDW_F16);
  }
#undef GBDW_SE
  }
  GBDW_LAUNCHED();
  if (!dev) GBDW_CUDA(cudaMemcpyAsync(dst, ddst, bytes, cudaMemcpyDeviceToHost, stream()));
  if (sync) GBDW_CUDA(cudaStreamSynchronize(stream()));
  return GBDW_OK;
}

int gbdw_field_export(const gbdw_field* f, int rhs, void* dst, int dst_prec) {
  return field_export(f, rhs, dst, dst_prec, true);
}

int gbdw_field_export_async(const gbdw_field* f, int rhs, void* dst, int dst_prec) {
  return field_export(f, rhs, dst, dst_prec, false);
}

int gbdw_field_copy(gbdw_field* dst, const gbdw_field* src) {
  if (!dst || !src || dst->lat != src->lat || dst->nrhs != src->nrhs) {
    set_error("gbdw_field_copy: fields must share lattice and nrhs");
    return GBDW_ERR_INVALID;
  }
  return field_convert(dst, src);
}

}  // extern "C"
