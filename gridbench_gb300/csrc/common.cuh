// Internal types shared by the libgbdw translation units.
//
// Device layout ("GB300 layout"), chosen so that consecutive threads read consecutive
// addresses and one 4D link serves every fifth-dimension slice of its site:
//   spinor  [site][sc = spin*3+colour][e = rhs*Ls + s]    complex (F64 16 B, F32 8 B, F16 4 B);
//           F32/F16 store slice pairs as (Re, Re, Im, Im) -- layout.cuh has the addressing --
//           and F16 adds norm[site][e] (FP32, max |re|,|im| over the 24 reals of that 5D site)
//   gauge   [site][mu][row][col] complex, 9 entries (F64/F32) or rows 0-1 only (F16/BF16)
//   nbr4    [site][mu] uint32 neighbour 4D site (fast path)
// "site" runs over 4D sites with SIMD lanes unrolled: site = outer_site*nsimd + lane, so a
// reference table with lane permutes maps onto a plain 4D table.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

#include "../../include/gbdw.h"

namespace gbdw {

void set_error(const std::string& msg);
int cuda_fail(cudaError_t e, const char* what);
cudaStream_t stream();
void count_launch(uint64_t n = 1);
// Device scratch owned by the library (grown on demand, kept until exit).
void* scratch(size_t bytes, int slot);
int ensure_device();
int num_sms();
// Device the library's stream belongs to (-1 before the first ensure_device()).
int library_device();
// cudaMalloc through the library's one allocation point (honours gbdw_debug_fail_allocs).
cudaError_t dev_alloc(void** p, size_t bytes);
// The memory of lattices, links and fields.  While an ArenaScope lives on this thread it comes from a
// buffer of the current stream's scratch (kept, at most kArenaMax bytes; cudaMalloc serves what does not
// fit) and object_free leaves it alone: for objects that live inside one call.
cudaError_t object_alloc(void** p, size_t bytes);
void object_free(void* p);
constexpr size_t kArenaMax = size_t(256) << 20;
struct ArenaScope {
  explicit ArenaScope(size_t bytes);
  ~ArenaScope();
  bool held;
};
// While alive on this thread, imports let the kernels read host memory in place where the GPU can (for
// a call that waits for the stream before it returns).
struct HostInPlace {
  HostInPlace();
  ~HostInPlace();
};
bool host_in_place(const void* p);  // p is 16-byte aligned and such a scope is open
unsigned* device_error_word();  // set by kernels whose bounded waits expired
size_t max_dynamic_smem();      // opt-in dynamic shared memory per CTA, minus room for static

#define GBDW_CUDA(call)                                       \
  do {                                                        \
    cudaError_t e_ = (call);                                  \
    if (e_ != cudaSuccess) return ::gbdw::cuda_fail(e_, #call); \
  } while (0)

// Back-to-back launches.  A kernel started with launch_after may be placed on the SMs while the launch
// before it on the stream still drains; its first statement is dep_wait(), which returns when that launch
// is complete and its writes are visible (and at once in a kernel started the ordinary way).  dep_release()
// lets the next such launch come up; it stands behind a kernel's dep_wait and behind its loads of anything
// it writes, so no line that an SM's L1 keeps across a release can be stale.  Such a kernel is resident while
// the launch before it still writes, so its loads are ordinary ones: a read-only load (__ldg, ld.global.nc, a
// pointer marked __restrict__) promises that nobody writes during the kernel's whole life, and the compiler may
// move it above the wait.  Here dep_wait's memory clobber holds them back.
// Hopping terms of 4^4 x 8 in a row 5.2 -> 2.7 us each; 16^4 x 16 57.5 -> 54; a Lanczos step's 38 launches at
// 12^4 x 8 569 -> 482.
__device__ __forceinline__ void dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void dep_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
template <class... P, class... A>
void launch_after(void (*kern)(P...), unsigned grid, unsigned threads, size_t smem, A&&... args) {
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream();
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kern, P(args)...);  // its status is read by GBDW_LAUNCHED
}

#define GBDW_LAUNCHED()                                                  \
  do {                                                                   \
    cudaError_t e_ = cudaGetLastError();                                 \
    if (e_ != cudaSuccess) return ::gbdw::cuda_fail(e_, "kernel launch"); \
    ::gbdw::count_launch();                                              \
  } while (0)

}  // namespace gbdw

struct gbdw_lattice {
  int64_t nsite;     // 4D sites, lanes unrolled
  int Ls;
  int nsimd;
  int dims[4];       // 0 when built from a table
  bool fast;         // 4D factorised table available
  uint32_t* nbr4;    // [nsite][8] (fast)
  uint32_t* nbr5;    // [nsite][Ls][8] neighbour (site*Ls+s) in device numbering (general)
  // Checkerboarded half lattice (even-odd): the sites of one 4D parity of a periodic parent,
  // numbered site = parent_site / 2.  nbr4 then holds neighbour indices into the partner
  // half (the other parity), and cbsite[site] the parent site.
  int parity = -1;                         // -1: not a half lattice
  const gbdw_lattice* parent = nullptr;
  const gbdw_lattice* partner = nullptr;   // the other parity of the same parent
  uint32_t* cbsite = nullptr;              // [nsite] parent site index
};

struct gbdw_gauge {
  const gbdw_lattice* lat;
  int prec;
  void* d;           // device storage
  size_t bytes;
  // F64 gauge: the links split into FP32 pairs (re h, re l, im h, im l per entry) for the
  // double-single operator, built on first use and freed with the gauge
  mutable void* d_ds = nullptr;
};

struct gbdw_field {
  const gbdw_lattice* lat;
  int prec;
  int nrhs;
  int LsE;           // Ls * nrhs, the innermost extent
  int LsP;           // stored slots per row: LsE, rounded up to even for F32/F16
  void* d;           // complex data
  float* norm;       // F16 only
  size_t bytes;
  int64_t elems() const { return lat->nsite * 12 * int64_t(LsP); }  // stored complex slots
};

namespace gbdw {

inline size_t spinor_elem_bytes(int prec) { return prec == GBDW_F64 ? 16 : prec == GBDW_F32 ? 8 : 4; }
inline size_t link_bytes(int prec) {
  return prec == GBDW_F64 ? 144 : prec == GBDW_F32 ? 72 : 24;
}

// ------------------------------------------------------------------ small complex helpers
template <class T>
struct cpx {
  T r, i;
};

template <class T>
__device__ __forceinline__ cpx<T> cmul(cpx<T> a, cpx<T> b) {
  return {a.r * b.r - a.i * b.i, a.r * b.i + a.i * b.r};
}
// acc += a*b
template <class T>
__device__ __forceinline__ void cmac(cpx<T>& acc, cpx<T> a, cpx<T> b) {
  acc.r = fma(a.r, b.r, acc.r);
  acc.r = fma(-a.i, b.i, acc.r);
  acc.i = fma(a.r, b.i, acc.i);
  acc.i = fma(a.i, b.r, acc.i);
}
// Multiply by a compile-time unit c in {+1, -1, +i, -i}: code 0:+1 1:-1 2:+i 3:-i
template <int C, class T>
__device__ __forceinline__ cpx<T> cunit(cpx<T> a) {
  if (C == 0) return a;
  if (C == 1) return {-a.r, -a.i};
  if (C == 2) return {-a.i, a.r};
  return {a.i, -a.r};
}
template <int C>
struct conj_unit {
  static constexpr int v = (C == 2) ? 3 : (C == 3) ? 2 : C;
};

// ------------------------------------------------------------------ device reductions
// Block-wide sums, then "last block finishes" passes over the per-block partials, so the sum
// order is fixed (deterministic) and no second launch is needed.
//
// grid_sum_flat: the last block sums all gridDim partials.  partials holds gridDim.x * W
// doubles, counter one unsigned that must be zero on entry and is left zero.
//
// grid_sum: two levels, so no single block walks thousands of partials after everyone else
// has finished: the last block of each group of kReduceGroup blocks sums its group (the sum
// replaces the group's first partial), and the last group to finish sums the group sums.
// counter holds 1 + ceil(gridDim.x / kReduceGroup) unsigned, zero on entry, left zero.
constexpr unsigned kReduceGroup = 128;

template <int W>
__device__ __forceinline__ void block_sum_to_thread0(double (&v)[W], double (&sh)[32][W]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int w = 0; w < W; ++w) {
    double x = v[w];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if (lane == 0) sh[warp][w] = x;
  }
  __syncthreads();
  const int nw = (blockDim.x + 31) >> 5;
  if (nw <= 4) {
    if (threadIdx.x == 0) {
#pragma unroll
      for (int w = 0; w < W; ++w) {
        double x = 0.0;
        for (int k = 0; k < nw; ++k) x += sh[k][w];
        v[w] = x;
      }
    }
  } else if (warp == 0) {  // up to 32 dependent FP64 adds by one thread take longer than five exchanges
#pragma unroll
    for (int w = 0; w < W; ++w) {
      double x = lane < nw ? sh[lane][w] : 0.0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
      v[w] = x;
    }
  }
}

// Sum of partials[(first + k*stride)*W + w] for k < n, by the whole block, into thread 0's v.
template <int W>
__device__ __forceinline__ void block_sum_of(const double* partials, unsigned first, unsigned stride, unsigned n,
                                             double (&v)[W], double (&sh)[32][W]) {
#pragma unroll
  for (int w = 0; w < W; ++w) {
    double x = 0.0;
    for (unsigned k = threadIdx.x; k < n; k += blockDim.x)
      x += __ldcg(&partials[size_t(first + k * stride) * W + w]);
    v[w] = x;
  }
  block_sum_to_thread0<W>(v, sh);
}

// Block partials only: thread 0 of every block writes the block's sum to partials[blockIdx];
// a separate one-CTA kernel (sum_partials) adds them up in a fixed order.  For grids of many
// short blocks, where a fence and an atomic per block would hold every block until its
// stores have landed.
template <int W>
__device__ __forceinline__ void block_partial(double (&v)[W], double* partials) {
  __shared__ double sh[32][W];
  block_sum_to_thread0<W>(v, sh);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int w = 0; w < W; ++w) partials[size_t(blockIdx.x) * W + w] = v[w];
  }
}

template <int W>
__device__ __forceinline__ void grid_sum_flat(double (&v)[W], double* partials, unsigned* counter,
                                              double* result) {
  __shared__ double sh[32][W];
  __shared__ bool last;
  block_sum_to_thread0<W>(v, sh);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int w = 0; w < W; ++w) partials[size_t(blockIdx.x) * W + w] = v[w];
    __threadfence();
    const unsigned prev = atomicAdd(counter, 1u);
    last = (prev == gridDim.x - 1);
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  block_sum_of<W>(partials, 0, 1, gridDim.x, v, sh);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int w = 0; w < W; ++w) result[w] = v[w];
    *counter = 0u;
  }
}

template <int W>
__device__ __forceinline__ void grid_sum(double (&v)[W], double* partials, unsigned* counter,
                                         double* result) {
  __shared__ double sh[32][W];
  __shared__ bool last;
  const unsigned g = blockIdx.x / kReduceGroup, g0 = g * kReduceGroup;
  const unsigned ng = (gridDim.x + kReduceGroup - 1) / kReduceGroup;
  const unsigned gsize = min(kReduceGroup, gridDim.x - g0);
  block_sum_to_thread0<W>(v, sh);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int w = 0; w < W; ++w) partials[size_t(blockIdx.x) * W + w] = v[w];
    __threadfence();
    const unsigned prev = atomicAdd(&counter[1 + g], 1u);
    last = (prev == gsize - 1);
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  block_sum_of<W>(partials, g0, 1, gsize, v, sh);  // this group, fixed order
  if (threadIdx.x == 0) {
#pragma unroll
    for (int w = 0; w < W; ++w) partials[size_t(g0) * W + w] = v[w];
    counter[1 + g] = 0u;
    __threadfence();
    const unsigned prev = atomicAdd(&counter[0], 1u);
    last = (prev == ng - 1);
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  block_sum_of<W>(partials, 0, kReduceGroup, ng, v, sh);  // the group sums, fixed order
  if (threadIdx.x == 0) {
#pragma unroll
    for (int w = 0; w < W; ++w) result[w] = v[w];
    counter[0] = 0u;
  }
}

// Scratch slots used for reductions: partial sums and a counter; result is page-locked host memory,
// valid once the stream has been waited for (reduce_fetch).
struct Reduce {
  double* partials;
  unsigned* counter;
  double* result;
};
int reduce_scratch(int64_t nblocks, int width, Reduce* r);
// One fused CG step's device scalars (cg_scalars): <p, A p>, alpha, |r|^2 after the update, beta, and
// whether the step goes on with the common vector update (1) or the host takes over (0).
enum { CG_PAP = 0, CG_ALPHA = 1, CG_RR = 2, CG_BETA = 3, CG_GO = 4, CG_SCALARS = 5 };
double* cg_scalars();
// The rule of that last scalar: the step's residual is finite, <p, A p> positive, and |r|^2 neither
// below `update` (a reliable update is due) nor at most `stop`; rr: |r|^2 before the step.
struct CgRule {
  double rr, update, stop;
};
// result[0] = sum of partials[0..n) in a fixed order (on the library stream); with alpha_out, also
// alpha_out[0] = num / result[0] (the CG step length, computed on the device); with rule, result is
// cg_scalars() + CG_RR, the scalars after it are set and all of them copied to the host
int sum_partials(const double* partials, int64_t n, double* result, double num = 0.0, double* alpha_out = nullptr,
                 const CgRule* rule = nullptr);
// the host's copy of a step's scalars in two halves, the first behind the step: work queued between
// them runs while the host waits
int cg_scalars_mark();
int cg_scalars_wait(double* host);
int reduce_fetch(const Reduce& r, int width, double* host);

}  // namespace gbdw
