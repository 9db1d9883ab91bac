// Drop-in replacement for GridBench's kernel seam
//   template<class Simd> double dslash_kernel(int nrep, Simd* Up, Simd* outp, Simd* inp,
//                                             uint64_t* nbr, uint64_t nsite, uint64_t Ls, uint8_t* prm)
// (WilsonKernelsHand.h:17-18,25-26; called from bench.cc:148-164).
//
// Same arguments and meaning: reference-layout gauge field, input and output spinors with
// Nsimd lanes, the TableGenerate neighbour/permute tables, nsite outer sites, nrep
// repetitions.  Buffers may live on the host or the device.  The table is validated and
// reduced to a 4D table, the fields are converted once into the GB300 layout, the hopping
// term runs nrep times, and the result is converted back once.  The returned time covers
// repetitions 1..nrep-1 as in WilsonKernelsHandCpu.h:407-450 (device time from CUDA events
// instead of a host clock).  Errors come back as a status; nothing exits the process
// (unlike Macros.h:47-51).
#include "common.cuh"

namespace gbdw {
int lattice_from_table_impl(gbdw_lattice** out, uint64_t nouter, int Ls, int nsimd, const uint64_t* nbr,
                            const uint8_t* prm, bool force_general);
}

using namespace gbdw;

namespace {
struct Owned {
  gbdw_lattice* lat = nullptr;
  gbdw_gauge* g = nullptr;
  gbdw_field* in = nullptr;
  gbdw_field* out = nullptr;
  ~Owned() {
    gbdw_field_destroy(out);
    gbdw_field_destroy(in);
    gbdw_gauge_destroy(g);
    gbdw_lattice_destroy(lat);
  }
};

thread_local cudaEvent_t g_begin = nullptr, g_end = nullptr;  // of the timed repetitions, kept between calls
}  // namespace

// What a call on host buffers costs beyond its hopping kernel (8^4 x 8 FP64: 588 us, the kernel 58): four
// allocations and their release, 250 us, now a kept arena; pageable inputs through the driver's staging
// copies at 31 GB/s, now read in place by the table and conversion kernels at 185 GB/s where the GPU shares
// the host's page tables.  227 us with both.  The result still goes out by a copy (51 us): a kernel's first
// write to a page that the caller has not touched yet would decide where that page lives.
extern "C" int gbdw_dslash_kernel(int nrep, int prec, int nsimd, const void* U, void* out, const void* in,
                                  const uint64_t* nbr, uint64_t nsite, uint64_t Ls, const uint8_t* prm, int dag,
                                  double* usec) {
  if (nrep < 1 || !U || !out || !in || !nbr || nsite == 0 || Ls == 0 || Ls > 4096 ||
      (prec != GBDW_F64 && prec != GBDW_F32)) {
    set_error("gbdw_dslash_kernel: invalid arguments (nrep >= 1, non-null buffers, prec F64 or F32)");
    return GBDW_ERR_INVALID;
  }
  if (int st = ensure_device()) return st;
  // neighbour table, links (FP64: also as pairs of floats) and both fields, with room for their alignment
  const size_t sites = size_t(nsite) * size_t(nsimd > 0 ? nsimd : 1), real = prec == GBDW_F64 ? 8 : 4;
  ArenaScope arena(sites * (32 + 2 * 144 * real + 2 * 24 * real * (size_t(Ls) + 1)) + 4096);
  HostInPlace in_place;
  Owned o;
  if (int st = lattice_from_table_impl(&o.lat, nsite, int(Ls), nsimd, nbr, prm, false)) return st;
  if (int st = gbdw_gauge_create(&o.g, o.lat, prec, U, prec)) return st;
  if (int st = gbdw_field_create(&o.in, o.lat, prec, 1)) return st;
  if (int st = gbdw_field_create(&o.out, o.lat, prec, 1)) return st;
  if (int st = gbdw_field_import(o.in, 0, in, prec)) return st;
  if (!g_begin) GBDW_CUDA(cudaEventCreate(&g_begin));
  if (!g_end) GBDW_CUDA(cudaEventCreate(&g_end));
  if (nrep == 1) GBDW_CUDA(cudaEventRecord(g_begin, stream()));
  for (int rep = 0; rep < nrep; ++rep) {
    if (rep == 1) GBDW_CUDA(cudaEventRecord(g_begin, stream()));
    if (int st = gbdw_dhop(o.g, o.out, o.in, dag)) return st;
  }
  GBDW_CUDA(cudaEventRecord(g_end, stream()));
  if (int st = gbdw_field_export(o.out, 0, out, prec)) return st;
  GBDW_CUDA(cudaEventSynchronize(g_end));
  float ms = 0.f;
  GBDW_CUDA(cudaEventElapsedTime(&ms, g_begin, g_end));
  if (usec) *usec = double(ms) * 1000.0;
  GBDW_CUDA(cudaStreamSynchronize(stream()));
  return GBDW_OK;
}
