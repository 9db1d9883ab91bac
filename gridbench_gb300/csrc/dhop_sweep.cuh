// The t-sweep form of the FP32 hopping kernel (form 4).
//
// What bounds the other forms is the L2 -> SM path: each of a site's eight neighbour spinors comes
// from L2, 834 MB per launch at 16^4 x 16 where DRAM moves 239 MB.  Here a CTA owns a column of
// 2 x 2 x 2 sites (x, y, z) and walks along t with the planes t and t+1 of its own sites in shared
// memory (cp.async, one plane ahead).  The T legs are the thread's own rows of the neighbouring
// planes, and in each of x, y, z one of the two legs is the other site of the pair, so a site costs
// one plane copy and three loads from L2 in place of eight (470 MB per launch).  Those three loads
// are issued about two legs before they are used.  The links of a plane's sites are staged as well
// (their broadcast 64-bit loads are 43 % of the direct form's L1 wavefronts).
//
// 2 x 2 x 2 because each thread then has exactly one outside neighbour per direction, in every
// warp; four CTAs of 64 threads fit an SM (34 KB and, at 16 slices, 212 to 255 registers a thread).  Hopping term, us,
// this form / the best of the others (TMA warp rings or form 3, before launches overlapped) / all bytes once
// at the copy rate:
//   16^4 x 8    34 / 49 / 20      24^4 x 8   152 / 215 / 104     24^4 x 12  247 / 287 / 141
//   16^4 x 16   56 / 59 / 35      24^4 x 16  264 / 303 / 179     32^4 x 16  847 / 1016 / 565
//   24^4 x 32  521 / 618 / 329    half of 32^4 x 16  404 / 506 / 283
// With the planes, links and stores taken away the 32^4 case still takes 528 us: the FMA pipes are
// busy for 390 us of it, and two warps per scheduler don't hide all of the rest (37 % of the issue slots
// used; a third of the stalls wait for L2).  Three, at 168 registers with 24 to 64 bytes spilled, are slower
// at every size: the loads move back towards their use (16^4 x 16 62 us, 32^4 x 16 961).  Lattices of a few
// waves of CTAs (16^4 x 16) lose what they gain to the last wave; sweep_slices (tune.cu) looks for the
// cheapest waves.
// Tried and slower: 4 x 2 x 2 and 4 x 4 x 2 columns with 2.5 / 2 loads from L2 a site, waited for
// at once (72 / 80 us at 16^4); two threads per slice pair, one per spin pair (12 to 16 warps but
// 46 % more instructions: 64 us, 971 us at 32^4); one persistent CTA per slot (the columns drift
// apart in t and lose each other's planes in L2: 72 us, 1121 us).
#pragma once
#include "dhop_kernel.cuh"

namespace gbdw {

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  const unsigned d = unsigned(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

constexpr int SWEEP_LS = 592;  // bytes of one site's eight links in shared memory (576 + a bank offset)
// 12 rows of TE slices; the pad makes the next site's row continue the bank sequence
__host__ __device__ constexpr int sweep_site_bytes(int TE) { return 96 * TE + (((8 * TE - 96 * TE) % 128) + 128) % 128; }
constexpr size_t sweep_smem(int TE) { return 16 * (size_t(sweep_site_bytes(TE)) + SWEEP_LS); }

// a link from shared memory with 128-bit loads (72 bytes; ODD: at an 8-byte boundary)
template <bool ODD>
__device__ __forceinline__ void sweep_link(const char* p, cpx<float> (&u)[3][3]) {
  float v[18];
  constexpr int o = ODD ? 2 : 0, s = ODD ? 0 : 16;
  const float2 c = *reinterpret_cast<const float2*>(p + 4 * s);
  v[s] = c.x;
  v[s + 1] = c.y;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float4 a = *reinterpret_cast<const float4*>(p + 4 * o + 16 * k);
    v[o + 4 * k] = a.x;
    v[o + 1 + 4 * k] = a.y;
    v[o + 2 + 4 * k] = a.z;
    v[o + 3 + 4 * k] = a.w;
  }
#pragma unroll
  for (int k = 0; k < 9; ++k) u[k / 3][k % 3] = {v[2 * k], v[2 * k + 1]};
}

// a neighbour's 12 rows of one slice pair
struct RawSpinor {
  cp2 v[12];
};
// global loads issued in program order (ahead of their use)
__device__ __forceinline__ void sweep_issue(RawSpinor& w, const char* base, uint32_t stride) {
#pragma unroll
  for (int r = 0; r < 12; ++r)
    asm volatile("ld.global.v4.f32 {%0,%1,%2,%3}, [%4];"
                 : "=f"(w.v[r].r.x), "=f"(w.v[r].r.y), "=f"(w.v[r].i.x), "=f"(w.v[r].i.y)
                 : "l"(base + uint32_t(r) * stride));
}
template <int ROW>
__device__ __forceinline__ void sweep_take(RawSpinor& w, const char* rows) {
#pragma unroll
  for (int r = 0; r < 12; ++r) {
    const float4 a = *reinterpret_cast<const float4*>(rows + r * ROW);
    w.v[r] = {make_float2(a.x, a.y), make_float2(a.z, a.w)};
  }
}

// Leg of direction D with the sign of its side (+1: the forward leg's projector, -1: the backward
// leg's, whose unit coefficients are the opposite ones).  MOB: A(b, c) on the neighbour first.
template <int D, bool MOB>
__device__ __forceinline__ void sweep_leg(const cpx<float> (&u)[3][3], RawSpinor& w, float sgn, cp2 (&acc)[12],
                                          const MobLeg& ml) {
  using S = LegSpin<D>;
  if constexpr (MOB) {
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      mob_lower(w.v[k], ml);
      mob_upper(w.v[6 + k], ml);
    }
  }
  const float2 sg = make_float2(sgn, sgn), sn = make_float2(-sgn, -sgn);
  cp2 h0[3], h1[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    h0[c] = w.v[c];
    cacc2<S::C0>(h0[c], w.v[S::A * 3 + c], sg, sn);
    h1[c] = w.v[3 + c];
    cacc2<S::C1>(h1[c], w.v[S::B * 3 + c], sg, sn);
  }
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    const cp2 u0 = su3_row2(u[r], h0);
    const cp2 u1 = su3_row2(u[r], h1);
    acc[r] = cadd2(acc[r], u0);
    acc[3 + r] = cadd2(acc[3 + r], u1);
    cacc2<conj_unit<S::C0>::v>(acc[S::A * 3 + r], u0, sg, sn);
    cacc2<conj_unit<S::C1>::v>(acc[S::B * 3 + r], u1, sg, sn);
  }
}

// EO: half lattices.  An output site (xh, y, z, t) has x = 2 xh + odd, so of its two x-neighbours
// one has the same index xh (this thread's own rows of plane t) and the other index is one off.
template <int DAG, int EPI, int TE, int EO>
__global__ void __launch_bounds__((4 * TE + 31) / 32 * 32, 256 / ((4 * TE + 31) / 32 * 32))
    k_dhop_sweep(const DhopParams p, const SweepParams q) {
  dep_wait();
  constexpr int NS = 8, G = TE / 2, SS = sweep_site_bytes(TE), ROW = TE * 8;
  extern __shared__ __align__(16) char sw_smem[];
  // a site's slice pairs are lanes of one warp: eight sites of four pairs, four of six or eight
  constexpr int SPW = G <= 4 ? 8 : 4;
  const int lane = threadIdx.x & 31;
  const int sl = int(threadIdx.x >> 5) * SPW + lane / G, lg = lane % G;
  const int xl = sl & 1, yl = (sl >> 1) & 1, zl = sl >> 2;
  const int Lx = q.L[0], Ly = q.L[1], Lz = q.L[2], Lt = q.L[3];
  const int vol3 = Lx * Ly * Lz;
  const uint32_t row_bytes = uint32_t(p.LsP) * 8;
  const int64_t site_bytes = int64_t(12) * row_bytes, plane_bytes = site_bytes * vol3;
  unsigned b = sweep_block(DAG);
  // slice tiles of a column side by side, or a whole pass over the lattice per tile
  const unsigned per = gridDim.x / unsigned(q.ntile);
  const int tile = int(q.tile_pass ? b / per : b % unsigned(q.ntile));
  b = q.tile_pass ? b % per : b / unsigned(q.ntile);
  const int x = int(b % q.nbx) * 2 + xl;
  b /= q.nbx;
  const int y = int(b % q.nby) * 2 + yl;
  b /= q.nby;
  const int z = int(b % q.nbz) * 2 + zl;
  const int ta = int(b / q.nbz) * q.nt, tb = min(ta + q.nt, Lt);
  const bool active = lane < SPW * G;  // whole warps are launched
  constexpr unsigned lanes = 0xffffffffu >> (32 - SPW * G);  // the active ones, in every warp
  const int col = active ? x + Lx * (y + Ly * z) : 0;
  const int e0 = tile * TE + 2 * lg;
  const char* const gcol = reinterpret_cast<const char*>(p.in) + int64_t(e0) * 8 + col * site_bytes;
  char* const own = sw_smem + sl * SS + lg * 16;            // this thread's rows in plane slot 0
  char* const ulk = sw_smem + 2 * NS * SS + sl * SWEEP_LS;  // its site's links in buffer 0
  double dpart = 0.0;
  const float fl = DAG ? -1.f : 1.f;
  auto fetch_plane = [&](int t, int slot) {
    if (!active) return;
    const char* s = gcol + (t >= Lt ? t - Lt : t) * plane_bytes;
    char* d = own + slot * NS * SS;
#pragma unroll
    for (int r = 0; r < 12; ++r) cp_async16(d + r * ROW, s + r * row_bytes);
  };
  auto fetch_links = [&](int t, int buf) {
    // each site's threads copy its own links
    if (!active) return;
    const char* s = reinterpret_cast<const char*>(p.U) + (int64_t(t) * vol3 + col) * 576;
    char* d = ulk + buf * NS * SWEEP_LS;
#pragma unroll
    for (int i = 0; i < 36; i += G)
      if (36 % G == 0 || i + lg < 36) cp_async16(d + (i + lg) * 16, s + (i + lg) * 16);
  };
  // direction d: leg A is the neighbour inside the column, leg B the one outside
  auto outside = [](int v, int up, int L) { return (up ? (v + 1 < L ? 1 : 1 - L) : (v > 0 ? -1 : L - 1)); };
  const int64_t gBy = int64_t(outside(y, yl, Ly)) * Lx * site_bytes;
  const int64_t gBz = int64_t(outside(z, zl, Lz)) * Lx * Ly * site_bytes;
  // x: bd = 1 when the inside neighbour is the backward one; on a half lattice that alternates with t
  auto x_side = [&](int t) { return EO ? (q.parity + y + z + t) & 1 : xl; };
  auto x_outside = [&](int bd) { return int64_t(outside(x, bd, Lx)) * site_bytes; };

  MobLeg ml;
  if constexpr (EPI == 6) ml = make_mobleg<SPW * G == 32>(p.Ls, p.mb, p.mc, p.mf, e0);
  cpx<float> u[3][3];
  RawSpinor ra, rb;
  Acc<GBDW_F32, 2> acc;
  acc.zero();
  fetch_plane(ta, 0);
  fetch_links(ta, 0);
  cp_async_commit();
  fetch_plane(ta + 1, 1);
  cp_async_commit();
  if (active) {
    sweep_issue(ra, gcol + (ta == 0 ? Lt - 1 : ta - 1) * plane_bytes, row_bytes);
    sweep_issue(rb, gcol + int64_t(ta) * plane_bytes + x_outside(x_side(ta)), row_bytes);
  }
  cp_async_wait<1>();
  __syncthreads();
  if (active) {
    sweep_link<true>(ulk + 72 * 7, u);
    sweep_leg<3, EPI == 6>(u, ra, -fl, acc.v[0], ml);
  }
  int cur = 0, lb = 0;
  for (int t = ta; t < tb; ++t) {
    const bool more = t + 1 < tb;
    if (more) fetch_links(t + 1, lb ^ 1);
    cp_async_commit();
    const char* ul = ulk + lb * NS * SWEEP_LS;
    const char* sc = own + cur * NS * SS;
    const char* gplane = gcol + int64_t(t) * plane_bytes;
    const int bx = x_side(t);
    const float sx = bx ? -fl : fl, sy = yl ? -fl : fl, sz = zl ? -fl : fl;
    if (active) {
      // x inside, x outside, y inside, z inside, y outside, T+, z outside
      sweep_link<false>(ul + (bx ? 72 * 4 : 0), u);
      sweep_take<ROW>(ra, EO ? sc : sc + (xl ? -SS : SS));
      sweep_leg<0, EPI == 6>(u, ra, sx, acc.v[0], ml);
      sweep_link<false>(ul + (bx ? 0 : 72 * 4), u);
      sweep_leg<0, EPI == 6>(u, rb, -sx, acc.v[0], ml);
      sweep_issue(rb, gplane + gBy, row_bytes);
      sweep_link<true>(ul + (yl ? 72 * 5 : 72), u);
      sweep_take<ROW>(ra, sc + (yl ? -2 * SS : 2 * SS));
      sweep_leg<1, EPI == 6>(u, ra, sy, acc.v[0], ml);
      sweep_link<false>(ul + (zl ? 72 * 6 : 72 * 2), u);
      sweep_take<ROW>(ra, sc + (zl ? -4 * SS : 4 * SS));
      sweep_leg<2, EPI == 6>(u, ra, sz, acc.v[0], ml);
      sweep_link<true>(ul + (yl ? 72 : 72 * 5), u);
      sweep_leg<1, EPI == 6>(u, rb, -sy, acc.v[0], ml);
      sweep_issue(rb, gplane + gBz, row_bytes);
    }
    cp_async_wait<1>();  // this thread's rows of plane t + 1
    if (active) {
      sweep_link<true>(ul + 72 * 3, u);
      sweep_take<ROW>(ra, own + (cur ^ 1) * NS * SS);
      sweep_leg<3, EPI == 6>(u, ra, fl, acc.v[0], ml);
      sweep_link<false>(ul + (zl ? 72 * 2 : 72 * 6), u);
      sweep_leg<2, EPI == 6>(u, rb, -sz, acc.v[0], ml);
      if (more) sweep_issue(rb, gplane + plane_bytes + x_outside(x_side(t + 1)), row_bytes);
      cpx<float> v[2][12];
      acc.unpack(v);
      float pt = 0.f;
      double dt = 0.0;
      const int64_t site = int64_t(t) * vol3 + col;
      if ((EPI <= 1 || EPI >= 5) && !more) dep_release();
      if (!EO && EPI >= 1 && !p.cen)  // the diagonal part reads this site's plane t, in shared memory
        finish_site<GBDW_F32, GBDW_F32, DAG, 2, EPI, !EO && EPI >= 1>(p, site, e0, p.LsE, p.LsP, v, pt, dt, sc - lg * 16);
      else
        finish_site<GBDW_F32, GBDW_F32, DAG, 2, EPI>(p, site, e0, p.LsE, p.LsP, v, pt, dt, nullptr, lanes);
      // |M in|^2 is FP64 above one site's 48 squares, as in the other forms, however far this walk goes
      if (p.partials) dpart += (EPI >= 2 && EPI <= 4) ? dt : double(pt);
    }
    if (!more) break;
    cp_async_wait<0>();
    __syncthreads();  // plane t + 1 and the links of t + 1 are in, by every thread
    if (active) {     // T- of the next slice from this thread's own rows of plane t
      acc.zero();
      sweep_link<true>(ulk + (lb ^ 1) * NS * SWEEP_LS + 72 * 7, u);
      sweep_take<ROW>(ra, sc);
      sweep_leg<3, EPI == 6>(u, ra, -fl, acc.v[0], ml);
    }
    // over this thread's own rows of plane t, which nobody else reads after the barrier
    if (t + 2 <= tb) fetch_plane(t + 2, cur);
    cp_async_commit();
    cur ^= 1;
    lb ^= 1;
  }
  cp_async_wait<0>();
  if (p.partials) {
    double v[1] = {dpart};
    block_partial<1>(v, p.partials);
  }
}

}  // namespace gbdw
