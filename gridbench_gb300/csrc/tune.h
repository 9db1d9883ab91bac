// Launch-shape selection for the hopping kernel (threads per CTA, slices per thread).
#pragma once
#include "dhop_kernel.cuh"

namespace gbdw {
// The shape for these operands when no entry exists (the rules' reasons are with the code).
DhopLaunch untuned_launch(const gbdw_gauge* g, const gbdw_field* in, int epi);
void set_tuned_launch(int gprec, int sprec, int LsE, int epi, DhopLaunch L);
// Optional parts of a hopping launch used by the fused CG step.
struct DhopExtra {
  gbdw_field* r = nullptr;          // with epi 1: r -= (*alpha) M(in) instead of storing M(in)
  const double* alpha = nullptr;    // device
  double* sum_to = nullptr;         // device: where the fused |.|^2 goes (default: the reduce result, for norm2)
  double num = 0.0;                 // with alpha_to: alpha_to = num / sum
  double* alpha_to = nullptr;       // device
  const CgRule* rule = nullptr;     // with sum_to = cg_scalars() + CG_RR
  double c5 = 1.0;                  // the epilogue's 5th-dimension hopping coefficient
  // Mobius operator in one pass: A(mb, mc) on the loaded neighbours (dag 0, FP32) or A(mb, mc)^dag
  // on DhopDag in before the epilogue (dag 1); epi 1, where mobius_fusable
  bool mobius = false;
  double mb = 1.0, mc = 0.0;
  // D5^-1 of the hopping term (dag: D5^-dag) in one pass, with mb = 1 / a5 and mc = 1 / (a5 (1 + mf a5^-Ls));
  // epi 0 on a half lattice, where m5inv_fusable
  bool m5inv = false;
  // a tune-cache key to take the launch shape from when it holds one (else the epilogue's own)
  int tune_key = -1;
};
// tune-cache epilogue keys of the even-odd hopping term (half lattices) are offset by this; a half
// lattice without its own entry takes the full lattice's
constexpr int EO_KEY = 32;
// tune-cache key of the fused CG step (both passes of mdagm_residual) with a residual of precision rprec
inline int cg_step_key(int rprec) { return 16 + rprec; }
// the cached shape for the key, if one was tuned or pinned
// (a t-sweep that was timed on a lattice of another volume is none: its slices of t fill other waves)
bool find_tuned_launch(int gprec, int sprec, int LsE, int epi, int64_t sites, DhopLaunch* L);
// cen / khop: the M epilogue's diagonal field (default: in) and hopping coefficient (1/2)
int run_dhop(const gbdw_gauge* g, gbdw_field* out, const gbdw_field* in, int dag, int epi, double a5, double mf,
             double* norm2, bool fetch = true, const gbdw_field* cen = nullptr, double khop = 0.5,
             const DhopExtra* ex = nullptr);
// The two passes of M^dag M with the CG update of the second fused in, queued:
//   t = M p, <p, A p> = |t|^2, alpha = rule.rr / <p, A p>, r -= alpha M^dag t, |r|^2, and the rule's
// scalars, all in cg_scalars().
int mdagm_residual(const gbdw_gauge* g, gbdw_field* t, gbdw_field* r, const gbdw_field* p, double M5, double mf,
                   const CgRule& rule);
int check_operands(const gbdw_gauge* g, const gbdw_field* out, const gbdw_field* in, bool need_single_rhs);
DhopParams make_params(const gbdw_gauge* g, gbdw_field* out, const gbdw_field* in);
// spt slices per thread cut a row: whole groups, or pairs of an odd FP32 extent whose last one is half
// padding (direct forms, Dhop and M)
bool slices_ok(const gbdw_field* in, int epi, int spt, int form);
// form 3 (direct, registers capped for six or eight CTAs per SM) applies: slice pairs, FP32 or FP16
// with Ls*nrhs = 16
bool form3_ok(const gbdw_field* in, int epi, int spt);
// form 4 for FP16 (blocked site order) applies: Ls*nrhs = 16, periodic lattice, even extents
bool blocked_ok(const gbdw_lattice* lat, const gbdw_field* in);
// form 4 for FP32 (t-sweep over 2x2x2 columns) applies to these operands: slices per tile (16, 12 or 8; the
// whole row for M and its variants), or 0
int sweep_extent(const gbdw_gauge* g, const gbdw_field* in, int epi, int spt);
// slices per tile of a direct launch with L.split tiles per site, or 0 (one tile: the split does
// not divide the extent into whole slice groups, a staged or blocked form, or whole_sites)
int tile_extent(int LsE, const DhopLaunch& L, bool whole_sites);
// t-brick of a direct launch on a periodic lattice whose Lt it divides, or 0 (natural order)
int brick_extent(const gbdw_lattice* lat, const DhopLaunch& L);
// the Mobius operator (dag 0) or its adjoint (dag 1) can be fused into the hopping pass for these
// operands (DhopExtra::mobius)
bool m5inv_fusable(const gbdw_gauge* g, const gbdw_field* in);
// the shape run_dhop takes for epilogue key epi with this gauge field
DhopLaunch lookup(const gbdw_gauge* g, const gbdw_field* in, int epi);
bool mobius_fusable(const gbdw_gauge* g, const gbdw_field* in, int dag);
}  // namespace gbdw
