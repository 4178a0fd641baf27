// lce_passes.cuh -- the update passes' device code, kernels and launches.
//
// The kernels are compiled in a module (a source file lce_passes_*.cu) per
// precision and place of the chains (Chains): the runtime loads a module as a
// whole when a context first uses one of its kernels.  In one module with the
// persistent sweep, a process's first context took 58 ms to create.
#pragma once
#include <algorithm>
#include <type_traits>

#include "lce_internal.hpp"

namespace lce {

// The reference evaluates cos(tpi*u) and sin(tpi*u) with tpi = 2 acos(-1)
// (f/heat_kpi.f:29, f/gauss.f:17); M<R>::cos2pi / sincos2pi take u itself
// (lce_common.cuh).

__device__ __forceinline__ int find_chain(const int* blk_begin, int n, int b) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (__ldg(blk_begin + mid) <= b) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// Field loads.  NC = true: the read-only (non-coherent) path, valid when no
// earlier writer runs in the same kernel (the per-pass form).  NC = false:
// L2 loads (ld.global.cg) for the persistent form, where fields written by
// other blocks before a grid barrier are read after it.  Ordinary cached
// loads are not enough there: measured on B200, lines an SM's L1 fetched
// before the barrier were still served after it (the persistent sweep then
// differs from the per-pass sweep), so L1 is bypassed.
//
// ONE not kTable (the chain in the parameter bank): a plane's base is one address in uniform registers and a load costs
// one multiply-add of the 32-bit site index.  Otherwise a link's plane and
// site are added first: a base per plane would take vector registers.
template <typename R, bool NC = true>
__device__ __forceinline__ R ldA(const R* A, int nh, int p, int k, int s) {
  const R* q = A + ((size_t)(p * 3 + k)) * nh + s;
  return NC ? __ldg(q) : __ldcg(q);
}

// A pass kernel's arguments, by where it finds the chain its block works on.
enum Chains : int { kTable = 0, kOne = 1, kMany = 2 };
template <int ONE>
using Args = std::conditional_t<ONE == kOne, PassArgsOne, std::conditional_t<ONE == kMany, PassArgsMany, PassArgs>>;
__device__ __forceinline__ const ChainDev& chain_of(const PassArgsOne& p, int) { return p.one; }
__device__ __forceinline__ const ChainDev& chain_of(const PassArgsMany& p, int c) { return p.ch[c]; }
__device__ __forceinline__ const ChainDev& chain_of(const PassArgs& p, int c) { return p.chains[c]; }
// the chain of a block's tile, and the tile's place among the chain's
__device__ __forceinline__ int find_tile(const PassArgsOne&, int&) { return 0; }
__device__ __forceinline__ int find_tile(const PassArgsMany& p, int& tile) {
  int lo = 0, hi = p.nchains - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (p.begin[mid] <= tile) lo = mid;
    else hi = mid - 1;
  }
  tile -= p.begin[lo];
  return lo;
}
__device__ __forceinline__ int find_tile(const PassArgs& p, int& tile) {
  const int c = p.nchains > 1 ? find_chain(p.blk_begin, p.nchains, tile) : 0;
  tile -= __ldg(p.blk_begin + c);
  return c;
}

// the couplings in the kernels' precision (FP32, ONE: converted on the host)
template <typename R, int ONE>
struct Cpl {
  const ChainDev& c;
  __device__ Cpl(const Args<ONE>&, const ChainDev& ch) : c(ch) {}
  __device__ R beta() const { return (R)c.beta; }
  __device__ R beta_a() const { return (R)c.beta_a; }
  __device__ R beta_2() const { return (R)c.beta_2; }
  __device__ R beta_4() const { return (R)c.beta_4; }
  __device__ R inv_beta2() const { return (R)c.inv_beta2; }
  __device__ R cxval0() const { return (R)c.cxval0; }
};
template <>
struct Cpl<float, kOne> {
  const PassArgsOne& a;
  __device__ Cpl(const PassArgsOne& p, const ChainDev&) : a(p) {}
  __device__ float beta() const { return a.beta; }
  __device__ float beta_a() const { return a.beta_a; }
  __device__ float beta_2() const { return a.beta_2; }
  __device__ float beta_4() const { return a.beta_4; }
  __device__ float inv_beta2() const { return a.inv_beta2; }
  __device__ float cxval0() const { return a.cxval0; }
};

template <typename R, bool NC = true, int ONE = kTable>
__device__ __forceinline__ su2<R> ldU(const ChainDev& ch, int mu, int p, int s) {
  if (ONE != kTable) {
    const void* plane = static_cast<const char*>(ch.u) + (size_t)(mu * 2 + p) * ch.nh * LinkIO<R>::kBytes;
    return NC ? LinkIO<R>::ld(plane, s) : LinkIO<R>::ld_cg(plane, s);
  }
  const size_t i = (size_t)(mu * 2 + p) * ch.nh + s;
  return NC ? LinkIO<R>::ld(ch.u, i) : LinkIO<R>::ld_cg(ch.u, i);
}

// f/staples.f:65-221: for each nu != mu (ascending),
//   upper  = U_nu(x+mu) [U_mu(x+nu)^+ U_nu(x)^+]          (NN of DD)
//   lower  = U_nu(x-nu+mu)^+ [U_mu(x-nu)^+ U_nu(x-nu)]    (DN of DN)
//   V      = (V + upper) + lower
template <typename R, int MU, int NU, bool NC, int ONE>
__device__ __forceinline__ void staple_add(const ChainDev& ch, int eo, const NbrOff& o, int s, su2<R>& V) {
  const int oe = 1 - eo;
  const int xpmu = s + o.p[MU], xpnu = s + o.p[NU], xmnu = s + o.m[NU];
  const int xmnupmu = xmnu + o.p[MU];
  su2<R> up1 = dd(ldU<R, NC, ONE>(ch, MU, oe, xpnu), ldU<R, NC, ONE>(ch, NU, eo, s));
  su2<R> up2 = nn(ldU<R, NC, ONE>(ch, NU, oe, xpmu), up1);
  su2<R> bt1 = dn(ldU<R, NC, ONE>(ch, MU, oe, xmnu), ldU<R, NC, ONE>(ch, NU, oe, xmnu));
  su2<R> bt2 = dn(ldU<R, NC, ONE>(ch, NU, eo, xmnupmu), bt1);
  V.a = (V.a + up2.a) + bt2.a;
  V.b = (V.b + up2.b) + bt2.b;
}

template <typename R, int MU, bool NC = true, int ONE = kTable>
__device__ __forceinline__ su2<R> staple(const ChainDev& ch, int eo, const NbrOff& o, int s) {
  su2<R> V{{(R)0, (R)0}, {(R)0, (R)0}};
  if (MU == 0) {
    staple_add<R, 0, 1, NC, ONE>(ch, eo, o, s, V);
    staple_add<R, 0, 2, NC, ONE>(ch, eo, o, s, V);
  } else if (MU == 1) {
    staple_add<R, 1, 0, NC, ONE>(ch, eo, o, s, V);
    staple_add<R, 1, 2, NC, ONE>(ch, eo, o, s, V);
  } else {
    staple_add<R, 2, 0, NC, ONE>(ch, eo, o, s, V);
    staple_add<R, 2, 1, NC, ONE>(ch, eo, o, s, V);
  }
  return V;
}

// f/a_force.f:54-110: F = sum_mu [U(x)(iA(x+mu))U(x)^+ + U(x-mu)^+(iA(x-mu))U(x-mu)],
// components F3 = Im(.)_a, F2 = Re(.)_b, F1 = Im(.)_b
template <typename R, int MU, bool NC, int ONE>
__device__ __forceinline__ void force_add(const ChainDev& ch, int eo, const NbrOff& o, int s, R& f1, R& f2,
                                          R& f3) {
  const int oe = 1 - eo, nh = ch.nh;
  const R* A = reinterpret_cast<const R*>(ch.a);
  const int xp = s + o.p[MU], xm = s + o.m[MU];
  su2<R> ux = ldU<R, NC, ONE>(ch, MU, eo, s);
  su2<R> ud = ldU<R, NC, ONE>(ch, MU, oe, xm);
  su2<R> t1 = nn(ux, ad(ldA<R, NC>(A, nh, oe, 0, xp), ldA<R, NC>(A, nh, oe, 1, xp), ldA<R, NC>(A, nh, oe, 2, xp), ux));
  su2<R> tb = dn(ud, an(ldA<R, NC>(A, nh, oe, 0, xm), ldA<R, NC>(A, nh, oe, 1, xm), ldA<R, NC>(A, nh, oe, 2, xm), ud));
  f3 = f3 + (t1.a.im + tb.a.im);
  f2 = f2 + (t1.b.re + tb.b.re);
  f1 = f1 + (t1.b.im + tb.b.im);
}

template <typename R, bool NC = true, int ONE = kTable>
__device__ __forceinline__ void higgs_force(const ChainDev& ch, int eo, const NbrOff& o, int s, R& f1, R& f2,
                                            R& f3) {
  f1 = f2 = f3 = (R)0;
  force_add<R, 0, NC, ONE>(ch, eo, o, s, f1, f2, f3);
  force_add<R, 1, NC, ONE>(ch, eo, o, s, f1, f2, f3);
  force_add<R, 2, NC, ONE>(ch, eo, o, s, f1, f2, f3);
}

// Set up the uniform source of this pass (of hit `hit` of a multi-hit pass:
// the next N*nh stream values, the next Philox pass).  Returns false (and
// flags the context) when the validation stream cannot cover the pass.
template <typename R, int N>
__device__ __forceinline__ bool setup_uniforms(const PassArgs& p, const ChainDev& ch, int s, int layout,
                                               Uniforms<R, N>& U, int hit = 0) {
  if (p.stream) {
    const int snh = p.stream_nh ? p.stream_nh : ch.nh;
    unsigned long long base = p.st->stream_pos + p.stream_off + (unsigned long long)hit * N * snh;
    if (base + (unsigned long long)N * snh > p.stream_n) {
      if (s == p.s_lo) atomicOr(&p.st->status, kStatusStreamExhausted);
      return false;
    }
    U.fill_stream(p.stream + base, snh, layout, s + p.site_off);
  } else {
    U.fill_philox(ch.key0, ch.key1, p.st->pass_ctr + p.pass_off + hit, s + p.site_off);
  }
  return true;
}

// ------------------------------------------------------------------ Higgs
// One tile (BS * SPT consecutive sites of one chain, BS threads) of a Higgs
// pass.  PDL: wait for the previous kernel, then let the next pass launch
// (per-pass form only).  Not before the wait: then the blocks of many waiting
// passes fill the SMs, and a pass's own blocks land together on the slots the
// last one left instead of one by one on all SMs.  24^3 24.3 -> 20.2 us per
// sweep, 32^3 24.8 -> 21.8, 48^3 33.4 -> 31.3, FP64 32^3 44.8 -> 37.2; from
// 56^3 on a pass fills the SMs by itself and nothing changes.
template <typename R, int MODE, bool PDL, int SPT = 1, int BS = kBlock, int ONE = kTable>
__device__ __forceinline__ void higgs_tile(const Args<ONE>& p, int tile) {
  // the chain table is written once at context creation: safe before pdl_wait
  int ctile = tile;
  const int c = find_tile(p, ctile);
  const ChainDev& ch = chain_of(p, c);
  const Cpl<R, ONE> cpl(p, ch);
  // a tile is BS * SPT consecutive sites; thread t takes t, t + BS, ...
  const int s0 = p.s_lo + ctile * BS * SPT + threadIdx.x;
  const int eo = p.eo, nh = ch.nh, s_hi = nh - p.s_lo;
  const Coord X0 = site_coord(eo, s0 < s_hi ? s0 : p.s_lo, ch.hx, ch.nxy, ch.dhx, ch.dnxy);
  unsigned acc[1] = {0u};
  double q[3] = {0.0, 0.0, 0.0};
  constexpr int NS = MODE == 0 ? 7 : (MODE == 1 ? 1 : 4);
  const int layout = MODE == 2 ? kTriple : kPlanar;
  // the first site's uniforms, drawn before the wait when the counters are settled
  Uniforms<R, NS> Un0;
  const bool early = PDL && SPT == 1 && p.rng_early && s0 < s_hi;
  const bool ok0 = early ? setup_uniforms<R, NS>(p, ch, s0, layout, Un0) : false;
  if (PDL) {
    pdl_wait();
    pdl_trigger();
  }
#pragma unroll 1
  for (int r = 0; r < SPT; ++r) {
    const int s = s0 + r * BS;
    if (s >= s_hi) break;
    const Coord X = r == 0 ? X0 : site_coord(eo, s, ch.hx, ch.nxy, ch.dhx, ch.dnxy);
    const NbrOff no = nbr_offsets(ch, X);
    Uniforms<R, NS> Un = Un0;
    if (r == 0 && early ? ok0 : setup_uniforms<R, NS>(p, ch, s, layout, Un)) {
      R f[3];
      higgs_force<R, PDL, ONE>(ch, eo, no, s, f[0], f[1], f[2]);
      R* A = reinterpret_cast<R*>(ch.a);
      R ao[3], an_[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        if (PDL) ao[k] = ONE ? (A + (size_t)(eo * 3 + k) * nh)[s] : A[((size_t)(eo * 3 + k)) * nh + s];
        else ao[k] = __ldcg(A + ((size_t)(eo * 3 + k)) * nh + s);
      }
      const R beta_a = cpl.beta_a(), beta_2 = cpl.beta_2(), beta_4 = cpl.beta_4();
      R alph = (R)0, sf_o = (R)0, sf_n = (R)0;
      if constexpr (MODE == 0 || MODE == 1) {
        // f/ahiggs2.f:52-77 width / cxval / alph
        R rr, cxval;
        if (ch.imode == 1) {
          R conf2 = (R)0;
#pragma unroll
          for (int i = 0; i < 3; ++i) conf2 = conf2 + beta_a * (f[i] * f[i]);
          R qq = beta_2 + beta_4 * conf2;
          alph = M<R>::div(beta_4 * conf2, (R)2 * (qq * qq));
          const R width = beta_2 + alph;
          rr = M<R>::div((R)1, width);
          cxval = M<R>::div(M<R>::div((R)1, (R)2), width);
        } else {
          rr = cpl.inv_beta2();      // 1/width, width = beta_2
          cxval = cpl.cxval0();      // 1/beta_2/2
        }
        if constexpr (MODE == 0) {
          // f/gauss.f:17-29: X = sqrt(-ln(W1)/R) cos(2 pi W2); f/ahiggs2.f:83-91
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            const R w1 = -(R)1 * rr * M<R>::log(Un.v[2 * i]);
            const R g = M<R>::sqrt(w1) * M<R>::cos2pi(Un.v[2 * i + 1]);
            an_[i] = g + beta_a * f[i] * cxval;
          }
        } else {
          // f/ahiggs3.f:83-87
#pragma unroll
          for (int i = 0; i < 3; ++i) an_[i] = -ao[i] + (R)2 * beta_a * f[i] * cxval;
        }
      } else {
        // f/ahiggs1.f:51-56 box proposal
        const R delta = (R)p.cst[c].delta;
#pragma unroll
        for (int i = 0; i < 3; ++i) an_[i] = ao[i] + (Un.v[i] - (R)0.5) * delta;
      }
      R rho_o = (R)0, rho_n = (R)0;
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        if (MODE == 2) {
          sf_o = sf_o + ao[i] * f[i];
          sf_n = sf_n + an_[i] * f[i];
        }
        rho_o = rho_o + ao[i] * ao[i];
        rho_n = rho_n + an_[i] * an_[i];
      }
      R boltz;
      if constexpr (MODE == 2) {
        // f/ahiggs1.f:77-78
        boltz = M<R>::exp(-beta_a * (sf_o - sf_n) + beta_2 * (rho_o - rho_n) +
                          beta_4 * (rho_o * rho_o - rho_n * rho_n));
      } else {
        // f/ahiggs2.f:108-109
        boltz = M<R>::exp(-alph * (rho_o - rho_n) + beta_4 * (rho_o * rho_o - rho_n * rho_n));
      }
      constexpr int acc_slot = MODE == 0 ? 6 : (MODE == 1 ? 0 : 3);
      if (boltz >= Un.v[acc_slot]) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          if (ONE) (A + (size_t)(eo * 3 + k) * nh)[s] = an_[k];
          else A[((size_t)(eo * 3 + k)) * nh + s] = an_[k];
          ao[k] = an_[k];
        }
        rho_o = rho_n;
        sf_o = sf_n;
        acc[0] += 1u;
      }
      if (p.part) {
        q[0] += (double)rho_o;
        q[1] += (double)rho_o * (double)rho_o;
        if (MODE == 2) q[2] += (double)sf_o;
        else if constexpr (sizeof(R) == 4) q[2] += (double)(ao[0] * f[0] + ao[1] * f[1] + ao[2] * f[2]);
        else q[2] += (double)ao[0] * f[0] + (double)ao[1] * f[1] + (double)ao[2] * f[2];
      }
    }
  }
  // partials {accepted, sum rho, sum rho^2, sum a.F}
  if (p.part) block_reduce_cs<1, 3, kNQ, !PDL>(acc, q, p.part + (size_t)tile * kNQ);
}

// ------------------------------------------------------------------ links
// NHIT = 3 is f/agauge1.f: the staple is built once and the heatbath +
// Metropolis hit is repeated on the updated link, each hit with its own
// uniforms (f/agauge1.f:95-198).
template <typename R, int MU, int OR, bool PDL, int NHIT = 1, int SPT = 1, int BS = kBlock, int ONE = kTable>
__device__ __forceinline__ void link_tile(const Args<ONE>& p, int tile) {
  int ctile = tile;
  const int c = find_tile(p, ctile);
  const ChainDev& ch = chain_of(p, c);
  const Cpl<R, ONE> cpl(p, ch);
  // a tile is BS * SPT consecutive sites; thread t takes t, t + BS, ...
  const int s0 = p.s_lo + ctile * BS * SPT + threadIdx.x;
  const int eo = p.eo, oe = 1 - eo, nh = ch.nh, s_hi = nh - p.s_lo;
  const Coord X0 = site_coord(eo, s0 < s_hi ? s0 : p.s_lo, ch.hx, ch.nxy, ch.dhx, ch.dnxy);
  unsigned cnt[2] = {0u, 0u};
  double pl[1] = {0.0};
  // the first site's uniforms (of the first hit), drawn before the wait when
  // the counters are settled
  Uniforms<R, OR ? 1 : 7> Un0;
  const bool early = PDL && SPT == 1 && p.rng_early && s0 < s_hi;
  const bool ok0 = early ? setup_uniforms<R, OR ? 1 : 7>(p, ch, s0, OR ? kPlanar : kTriple, Un0) : false;
  if (PDL) {
    pdl_wait();
    pdl_trigger();
  }
#pragma unroll 1
  for (int r = 0; r < SPT; ++r) {
    const int s = s0 + r * BS;
    if (s >= s_hi) break;
    const Coord X = r == 0 ? X0 : site_coord(eo, s, ch.hx, ch.nxy, ch.dhx, ch.dnxy);
    const NbrOff no = nbr_offsets(ch, X);
    Uniforms<R, OR ? 1 : 7> Un = Un0;
    if (r == 0 && early ? ok0 : setup_uniforms<R, OR ? 1 : 7>(p, ch, s, OR ? kPlanar : kTriple, Un)) {
      const su2<R> V = staple<R, MU, PDL, ONE>(ch, eo, no, s);
      // (kTable: the index formed once and kept for the store; formed again
      // there, the FP64 persistent sweep of 12^3 took 70.6 us instead of 69.0)
      const size_t li = (size_t)(MU * 2 + eo) * nh + s;
      su2<R> uo = ONE ? ldU<R, PDL, ONE>(ch, MU, eo, s) : (PDL ? LinkIO<R>::ld(ch.u, li) : LinkIO<R>::ld_cg(ch.u, li));
      // f/agauge.f:71-84: normalised staple, 1/(beta |V|), 1/2 Re Tr(U Vhat)
      const R tn = M<R>::rsqrt(norm2(V));
      const su2<R> vh{{tn * V.a.re, tn * V.a.im}, {tn * V.b.re, tn * V.b.im}};
      // f/agauge.f:126-174 hopping term beta_a Re[(iA(x) U)(iA(x+mu) U^+)]_11 and accept
      const R* A = reinterpret_cast<const R*>(ch.a);
      const int xp = s + no.p[MU];
      const R x1 = ldA<R, PDL>(A, nh, eo, 0, s), x2 = ldA<R, PDL>(A, nh, eo, 1, s), x3 = ldA<R, PDL>(A, nh, eo, 2, s);
      const R y1 = ldA<R, PDL>(A, nh, oe, 0, xp), y2 = ldA<R, PDL>(A, nh, oe, 1, xp), y3 = ldA<R, PDL>(A, nh, oe, 2, xp);
      const R beta_a = cpl.beta_a();
      bool changed = false;
#pragma unroll 1
      for (int hit = 0; hit < NHIT; ++hit) {
        if (hit > 0 && !setup_uniforms<R, OR ? 1 : 7>(p, ch, s, OR ? kPlanar : kTriple, Un, hit)) break;
        su2<R> hn;
        if constexpr (!OR) {
          const R t1 = M<R>::div(tn, cpl.beta());
          const R t2 = (uo.a * vh.a - uo.b * cj(vh.b)).re;
          // f/heat_kpi.f:33-98 single-trial Kennedy-Pendleton
          R a1 = Un.v[0], a2 = Un.v[1], a3 = Un.v[2];
          if (a1 == (R)0) a1 = (R)0.0000033;
          if (a2 == (R)0) a2 = (R)0.0000066;
          const R cc = M<R>::cos2pi(a3);
          R a0 = -(M<R>::log(a1) + M<R>::log(a2) * (cc * cc)) * t1;
          const R r4 = Un.v[3];
          const bool lacc = r4 * r4 <= ((R)1 - (R)0.5 * a0);
          a0 = lacc ? (R)1 - a0 : t2;
          cnt[0] += lacc ? 1u : 0u;
          R b1 = (R)1 - a0 * a0;
          b1 = b1 >= (R)0 ? M<R>::sqrt(b1) : (R)0;
          const R b2 = (R)2 * (Un.v[4] - (R)0.5);
          su2<R> Xk;
          Xk.a = mk<R>(a0, b1 * b2);
          R q0 = (R)1 - b2 * b2;
          q0 = q0 >= (R)0 ? b1 * M<R>::sqrt(q0) : (R)0;
          R sph, cph;
          M<R>::sincos2pi(Un.v[5], &sph, &cph);
          Xk.b = mk<R>(q0 * sph, q0 * cph);
          hn = nd(Xk, vh);  // f/agauge.f:98-99
        } else {
          // overrelaxation U' = (Vhat U Vhat)^+ leaves Re Tr(U V) unchanged
          const su2<R> w = nn(nn(vh, uo), vh);
          hn = su2<R>{cj(w.a), -w.b};
        }
        const R sa_old = beta_a * nn(an(x1, x2, x3, uo), ad(y1, y2, y3, uo)).a.re;
        const R sa_new = beta_a * nn(an(x1, x2, x3, hn), ad(y1, y2, y3, hn)).a.re;
        if (M<R>::exp(sa_old - sa_new) >= Un.v[OR ? 0 : 6]) {
          uo = hn;
          changed = true;
          cnt[OR ? 0 : 1] += 1u;
        }
      }
      if (changed) {
        const su2<R> un = p.fuse_renorm ? unitarise64(uo) : uo;
        if (ONE) LinkIO<R>::st(static_cast<char*>(ch.u) + (size_t)(MU * 2 + eo) * nh * LinkIO<R>::kBytes, s, un);
        else LinkIO<R>::st(ch.u, li, un);
      }
      // f/agauge.f:179-185 plaquette against the staple
      if (!OR && p.part) pl[0] += (double)nn(uo, V).a.re;
    }
  }
  // partials {KP accepted, Metropolis accepted, sum plaquette} / {OR accepted}
  if (p.part) {
    if constexpr (!OR) block_reduce_cs<2, 1, kNQ, !PDL>(cnt, pl, p.part + (size_t)tile * kNQ);
    else {
      unsigned c1[1] = {cnt[0]};
      double d0[1] = {0.0};
      block_reduce_cs<1, 0, kNQ, !PDL>(c1, d0, p.part + (size_t)tile * kNQ);
    }
  }
}

// ------------------------------------------------------------------ finalize
// The partial sums of a reduction slot (kNQ doubles per tile) are added in two
// fixed levels, so the order of every FP64 addition depends only on the tile
// table, never on which warp or block does the work (the per-pass and the
// persistent forms give the same bits):
//   level 1  chunk k of chain c = the chain's tiles [k*128, (k+1)*128); lane l
//            adds the tiles l, l+32, l+64, l+96 of the chunk in order and the
//            lanes are combined by a fixed shuffle tree;
//   level 2  a chain of several chunks: lane l adds the chunk sums l, l+32,
//            ... in order, same tree.  A one-chunk chain's level-1 sum is its
//            total.
// One (chunk, slot) or (chain, slot) item per warp; the loads of four tiles
// (or chunk sums) are issued together before their in-order adds.  In the
// per-pass form level 1 of a pass's slot is done by extra blocks of the next
// pass (reduce-behind), so the finalize kernel is left with level 1 of the
// last pass's slot, level 2 and the combine.
__device__ __forceinline__ void warp_tree(double (&v)[kNQ]) {
#pragma unroll
  for (int q = 0; q < kNQ; ++q) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_down_sync(0xffffffffu, v[q], o);
  }
}

// in-order sum over the strided elements e = e0 + lane, e0 + lane + 32, ...
// (e < e1) of an array of kNQ-double records with record stride `stride`
// (in double2), reading through L2
__device__ __forceinline__ void strided_sum(const double2* base, size_t stride, int e0, int e1, double (&v)[kNQ]) {
  static_assert(kNQ == 4, "a record is two double2");
  const int lane = threadIdx.x & 31;
  v[0] = v[1] = v[2] = v[3] = 0.0;
  constexpr int kBatch = 4;
  for (int b = e0 + lane; b < e1; b += 32 * kBatch) {
    double2 x[kBatch][2];
#pragma unroll
    for (int j = 0; j < kBatch; ++j) {
      const int e = b + 32 * j;
      x[j][0] = e < e1 ? __ldcg(base + (size_t)e * stride) : make_double2(0.0, 0.0);
      x[j][1] = e < e1 ? __ldcg(base + (size_t)e * stride + 1) : make_double2(0.0, 0.0);
    }
#pragma unroll
    for (int j = 0; j < kBatch; ++j) {
      if (b + 32 * j < e1) {
        v[0] += x[j][0].x;
        v[1] += x[j][0].y;
        v[2] += x[j][1].x;
        v[3] += x[j][1].y;
      }
    }
  }
  warp_tree(v);
}

// level 1 of slot i (partials at part_i), item g = chunk g over all chains:
// the chunk's sum goes to the chain's total when the chain is one chunk,
// else to chunks[g][i]
__device__ __forceinline__ void level1_item(const double* part_i, const int* blk_begin, const int* chunk_begin,
                                            int nchains, int g, int i, double* chunks, double* totals) {
  const int c = nchains > 1 ? find_chain(chunk_begin, nchains, g) : 0;
  const int t0 = __ldg(blk_begin + c) + (g - __ldg(chunk_begin + c)) * kChunkTiles;
  const int t1 = min(__ldg(blk_begin + c + 1), t0 + kChunkTiles);
  double v[kNQ];
  strided_sum(reinterpret_cast<const double2*>(part_i), 2, t0, t1, v);
  if ((threadIdx.x & 31) == 0) {
    const bool one = __ldg(chunk_begin + c + 1) - __ldg(chunk_begin + c) == 1;
    double* dst = one ? totals + ((size_t)c * kMaxSlots + i) * kNQ : chunks + ((size_t)g * kMaxSlots + i) * kNQ;
#pragma unroll
    for (int q = 0; q < kNQ; ++q) dst[q] = v[q];
  }
}

// level 1, item w = (chunk g over all chains, slot pre + w % (nslots - pre))
__device__ __forceinline__ void finalize_chunk_warp(const FinalizeArgs& f, int w) {
  const int nrem = f.nslots - f.pre;
  const int g = w / nrem, i = f.pre + w % nrem;
  level1_item(f.part + (size_t)i * f.slot_stride, f.blk_begin, f.chunk_begin, f.nchains, g, i, f.chunks, f.totals);
}

// The reduce-behind blocks of a per-pass launch (blockIdx.x >= p.ntiles):
// after the wait the previous pass has completed, and its slot's level-1
// items are spread over these blocks' warps.
__device__ __forceinline__ void reduce_behind(const PassArgs& p) {
  pdl_trigger();
  pdl_wait();
  const int nw = (int)(blockDim.x >> 5);
  const int nred = ((int)gridDim.x - p.ntiles) * nw;
  const CtxState& st = *p.st;
  const int slot = p.rb_slot & 0xff;
  const double* part = st.rb_part + (size_t)slot * st.rb_slot_stride;
  const int* chunk_begin = st.rb_chunk_begin[p.rb_slot >> 8];
  for (int g = ((int)blockIdx.x - p.ntiles) * nw + (int)(threadIdx.x >> 5); g < p.rb_nitems; g += nred)
    level1_item(part, p.blk_begin, chunk_begin, p.nchains, g, slot, st.rb_chunks, st.rb_totals);
}

// Reduce-behind blocks are compiled into the one-site-per-thread kernels:
// in the two-sites form, at its 64-register cap, the extra branch made the
// link kernels spill (56-76 bytes).
template <int SPT>
constexpr bool kReduceBehind = SPT == 1;

// Tile shape: BS threads per block, SPT sites per thread (1, or 2 for the
// LCE_SWEEP_PASSES2 form), and OCC resident threads per SM the register cap
// is set for: OCC = 0 keeps the cap of min_blocks<R>() blocks of kBlock
// threads (64 registers in FP32); OCC = 1152 is nine blocks of 128 (56).
template <typename R, int BS, int OCC>
constexpr int min_blocks_bs() {
  return OCC ? OCC / BS : (min_blocks<R>() * kBlock / BS > 0 ? min_blocks<R>() * kBlock / BS : 1);
}

// ONE, where a kernel finds its chain.  kOne: a single-chain context's chain
// in the parameter bank: its extents, plane addresses and couplings are
// uniform and need no loads, conversions or registers of their own.  Sweeps
// without measurements, the same tile: 16^3 22.1 -> 20.4 us, 64^3 38.6 ->
// 36.6, with 4 overrelaxations 125.0 -> 115.8, 128^3 301 -> 290, FP64 64^3
// 93.8 -> 88.8.  kMany: a batch's table in the parameter bank, found by the
// block's tile: 96 chains of 16^3-48^3 with two sites of 128 threads 829 -> 802
// us per measured sweep, one site 880 -> 817; 64 of 32^3 382 -> 366 and 402 ->
// 370, in FP64 772 -> 718.  kTable: the table in memory (kParamTiles).  The FP32
// passes of 64^3 and above are bound by instruction issue: at 128^3 a link
// heatbath takes 775 warp instructions per site, 309 of them FP32 adds,
// multiplies and multiply-adds, and 68% of the issue slots of an active SM.  The
// FP64 ones are not (64^3: issue 37%, FP64 pipe 28%): their 80 registers leave
// 18 warps per SM to hide the latency of the loads.
template <typename R, int MODE, int SPT, int BS, int OCC, int ONE>
__global__ void __launch_bounds__(BS, min_blocks_bs<R, BS, OCC>()) higgs_kernel(Args<ONE> p) {
  if (kReduceBehind<SPT> && p.rb_nitems && (int)blockIdx.x >= p.ntiles) reduce_behind(p);
  else higgs_tile<R, MODE, true, SPT, BS, ONE>(p, blockIdx.x);
}

template <typename R, int MU, int OR, int SPT, int BS, int OCC, int ONE>
__global__ void __launch_bounds__(BS, min_blocks_bs<R, BS, OCC>()) link_kernel(Args<ONE> p) {
  if (kReduceBehind<SPT> && p.rb_nitems && (int)blockIdx.x >= p.ntiles) reduce_behind(p);
  else link_tile<R, MU, OR, true, 1, SPT, BS, ONE>(p, blockIdx.x);
}

// f/agauge1.f (3 hits)
template <typename R, int MU, int SPT, int BS, int OCC, int ONE>
__global__ void __launch_bounds__(BS, min_blocks_bs<R, BS, OCC>()) link3_kernel(Args<ONE> p) {
  if (kReduceBehind<SPT> && p.rb_nitems && (int)blockIdx.x >= p.ntiles) reduce_behind(p);
  else link_tile<R, MU, 0, true, 3, SPT, BS, ONE>(p, blockIdx.x);
}

// level 2, item w = (chain c, slot i); nothing to do for a one-chunk chain
__device__ __forceinline__ void finalize_chain_warp(const FinalizeArgs& f, int w) {
  const int c = w / f.nslots, i = w % f.nslots;
  const int g0 = __ldg(f.chunk_begin + c), g1 = __ldg(f.chunk_begin + c + 1);
  if (g1 - g0 <= 1) return;
  double v[kNQ];
  strided_sum(reinterpret_cast<const double2*>(f.chunks + (size_t)i * kNQ), kMaxSlots * kNQ / 2, g0, g1, v);
  if ((threadIdx.x & 31) == 0) {
#pragma unroll
    for (int q = 0; q < kNQ; ++q) f.totals[((size_t)c * kMaxSlots + i) * kNQ + q] = v[q];
  }
}

// The combine's slot tables in shared memory, copied by the finalize kernels
// before their wait, while the previous pass still runs.
struct FinTables {
  unsigned char kinds[kMaxSlots], gid[kMaxSlots], gflags[kMaxSlots], gbeg[kMaxSlots], gend[kMaxSlots];
};
__device__ __forceinline__ void load_tables(const FinalizeArgs& f, FinTables& T) {
  for (int i = threadIdx.x; i < kMaxSlots; i += blockDim.x) {
    T.kinds[i] = f.kinds[i];
    T.gid[i] = f.gid[i];
    T.gflags[i] = f.gflags[i];
    T.gbeg[i] = f.gbeg[i];
    T.gend[i] = f.gend[i];
  }
}

// Per chain the reference's normalisations of the slot totals, then the RNG
// counters advance.  Run by one block after every total is complete, one
// warp per chain.  The routine groups (fin_groups) are independent: lane j
// sums the slots of groups j and j + 32 in slot order, and the divisions of
// the normalisations (up to four per group) run one per lane, lane 4 g' + d
// taking division d of group g = g' + 8 r, so that they overlap instead of
// following one another.  The additions and divisions are those of a scan
// over the slots in order, and each field is written by the last group that
// sets it.  Only the ahiggs1 step adaptation runs as a chain over the
// ahiggs1 groups in order.
// SM: a single chain whose totals are in shared memory (stot) instead of
// f.totals, with its volume, ahiggs1 step and RNG counters loaded at the
// kernel's start (pre = {2 nh, delta}, ctr = {pass_ctr, stream_pos}).
template <bool SM = false>
__device__ __forceinline__ void finalize_combine(const FinalizeArgs& f, const FinTables& T, const double* stot = nullptr,
                                                 const double* pre = nullptr, const unsigned long long* ctr = nullptr) {
  static_assert(kMaxSlots <= 64, "two slots (groups) per lane");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = (int)(blockDim.x >> 5);
  for (int c = warp; c < f.nchains; c += nwarps) {
    const double V = SM ? pre[0] : 2.0 * f.chains[c].nh;
    const double* base = SM ? stot : f.totals + (size_t)c * kMaxSlots * kNQ;
    double t0[kNQ], t1[kNQ];
    bool bad = false;
#pragma unroll
    for (int q = 0; q < kNQ; ++q) {
      const size_t i0 = (size_t)lane * kNQ + q, i1 = (size_t)(lane + 32) * kNQ + q;
      t0[q] = lane < f.nslots ? (SM ? base[i0] : __ldcg(base + i0)) : 0.0;
      t1[q] = lane + 32 < f.nslots ? (SM ? base[i1] : __ldcg(base + i1)) : 0.0;
      bad = bad || !isfinite(t0[q]) || !isfinite(t1[q]);
    }
    if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(&f.st->status, kStatusNaN);
    lce_meas& m = f.meas[c];
    // the group sums: lane j, groups j (hs[0]) and j + 32 (hs[1])
    double hs[2][kNQ] = {{0, 0, 0, 0}, {0, 0, 0, 0}};
    if (SM) {
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const int g = lane + 32 * s;
        if (g >= f.ngroups) continue;
        for (int i = T.gbeg[g]; i <= T.gend[g]; ++i) {
          if (T.gid[i] != g) continue;
#pragma unroll
          for (int q = 0; q < kNQ; ++q) hs[s][q] += stot[i * kNQ + q];
        }
      }
    } else {
      // warp-uniform scan: slot i's totals by shuffle, added by its group's lane
      for (int i = 0; i < f.nslots; ++i) {
        const int g = T.gid[i];
        double t[kNQ];
#pragma unroll
        for (int q = 0; q < kNQ; ++q) t[q] = __shfl_sync(0xffffffffu, i < 32 ? t0[q] : t1[q], i & 31);
        if (g == kNoGroup || lane != (g & 31)) continue;
#pragma unroll
        for (int q = 0; q < kNQ; ++q) {
          if (g < 32) hs[0][q] += t[q];
          else hs[1][q] += t[q];
        }
      }
    }
    // the normalisations, one division per lane
    for (int g0 = 0; g0 < f.ngroups; g0 += 8) {
      const int g = g0 + (lane >> 2), d = lane & 3;
      double h[kNQ];
#pragma unroll
      for (int q = 0; q < kNQ; ++q) {
        const double x0 = __shfl_sync(0xffffffffu, hs[0][q], g & 31), x1 = __shfl_sync(0xffffffffu, hs[1][q], g & 31);
        h[q] = g < 32 ? x0 : x1;
      }
      const int kind = g < f.ngroups ? (T.kinds[T.gend[g]] & 0x7f) : -1;
      const unsigned fl = g < f.ngroups ? T.gflags[g] : 0u;
      const bool higgs = kind >= 0 && kind <= kHiggsMetro, link = kind == kLinkHB || kind == kLinkHB3;
      // f/ahiggs2.f:142-147 (same in ahiggs1/3): a2 = h1/V, a4 = h2/V, akin = h3/(6V), acc = h0/V;
      // f/agauge.f:195-200: plaq = l2/(12V), acc = (l0/(3V)) (l1/(12V)); f/agauge1.f:227-232
      // divides the Metropolis factor by the 3 hits; link overrelaxation: l0/(3V)
      double num = 1.0, den = 1.0;
      if (higgs) {
        num = d == 0 ? h[1] : (d == 1 ? h[2] : (d == 2 ? h[3] : h[0]));
        den = d == 2 ? 6.0 * V : V;
      } else if (link) {
        num = d == 0 ? h[2] : (d == 1 ? h[0] : h[1]);
        den = d == 1 ? 3.0 * V : 12.0 * V;
      } else if (kind == kLinkOR) {
        num = h[0];
        den = 3.0 * V;
      }
      double r = num / den;
      if (kind == kLinkHB3 && d == 2) r = r / 3.0;
      const double r2 = __shfl_down_sync(0xffffffffu, r, 1);  // division d + 1 of the same group
      if (higgs) {
        if (fl & kGrpHiggsLast) {
          if (d == 0) m.a2 = r;
          if (d == 1) m.a4 = r;
          if (d == 2) m.akin = r;
        }
        if ((fl & kGrpKindLast) && d == 3) {
          if (kind == kHiggsHB) m.acc_hb = r;
          if (kind == kHiggsOR) m.acc_or = r;
        }
      } else if (link) {
        if (fl & kGrpKindLast) {
          if (d == 0) m.plaq = r;
          if (d == 1) m.acc_gauge = r * r2;
        }
      } else if (kind == kLinkOR) {
        if ((fl & kGrpKindLast) && d == 0) m.acc_link_or = r;
      }
    }
    // f/ahiggs1.f:113-123 step adaptation after each ahiggs1 group, in order,
    // in the build's precision
    double delta = SM ? pre[1] : f.cst[c].delta;
    if (f.nmetro) {
      for (int g = 0; g < f.ngroups; ++g) {
        if (!(T.gflags[g] & kGrpMetro)) continue;
        const double h0 = __shfl_sync(0xffffffffu, g < 32 ? hs[0][0] : hs[1][0], g & 31);
        if (f.single) {
          float a = (float)h0 / (float)V, dl = (float)delta;
          if (fabsf(a - 0.5f) > 0.1f) dl = (a > 0.5f) ? 1.1131241f * dl : 0.8989669f * dl;
          if (lane == 0 && (T.gflags[g] & kGrpKindLast)) m.acc_metro = a;
          delta = dl;
        } else {
          const double a = h0 / V;
          double dl = delta;
          if (fabs(a - 0.5) > 0.1) dl = (a > 0.5) ? 1.1131241 * dl : 0.8989669 * dl;
          if (lane == 0 && (T.gflags[g] & kGrpKindLast)) m.acc_metro = a;
          delta = dl;
        }
      }
      if (lane == 0) f.cst[c].delta = delta;
    }
    if (lane == 0) m.delta = delta;
  }
  __syncthreads();
  if (threadIdx.x == 0 && (f.npasses || f.nstream)) {
    if (SM) {
      f.st->pass_ctr = ctr[0] + f.npasses;
      f.st->stream_pos = ctr[1] + f.nstream;
    } else {
      f.st->pass_ctr += f.npasses;
      f.st->stream_pos += f.nstream;
    }
  }
}

// One block for a single chain of at most kSmallChunks chunks, everything
// after the wait in one global round trip: warp w < (nslots - pre) * nch
// sums chunk w % nch of slot pre + w / nch (level 1, to shared memory) while
// the block loads the chunk sums of the slots [0, pre) that the passes
// summed behind; level 2 per slot (lane k holds chunk k, the fixed tree) and
// the combine then read shared memory.  Same additions, same order as the
// two-level kernel below.
constexpr int kFinSmallWarps = 16;
constexpr int kSmallChunks = 8;
struct SmallFinSmem {
  double tot[kMaxSlots * kNQ];
  double ck[kMaxSlots * kSmallChunks * kNQ];  // [slot][chunk][q]
  double pre[2];
  unsigned long long ctr[2];
  FinTables T;
};
// The single-chain finalize, run by one block of any number of warps: the
// finalize_small_kernel block, or the block a sweep's first pass carries for
// the previous sweep (DEFERRED: called after the caller's wait; the RNG
// counters are then left alone when f.npasses and f.nstream are 0).
template <bool DEFERRED>
__device__ __forceinline__ void finalize_small_body(const FinalizeArgs& f, SmallFinSmem& S) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = (int)(blockDim.x >> 5);
  // the slot tables, and the combine's inputs other than the totals -- the
  // volume, and the ahiggs1 step and the RNG counters, which only an earlier
  // finalize writes (before the wait in the finalize kernel: that finalize
  // completed before this queue's first pass went past its wait)
  load_tables(f, S.T);
  if ((int)threadIdx.x == (int)blockDim.x - 1) {
    S.pre[0] = 2.0 * f.chains[0].nh;
    S.pre[1] = f.cst[0].delta;
    S.ctr[0] = f.st->pass_ctr;
    S.ctr[1] = f.st->stream_pos;
  }
  if (!DEFERRED) pdl_wait();
  const int nch = f.nchunks, b1 = f.ntiles0;  // chain 0's chunks and tiles, from the host
  // chunk sums summed behind: one chunk -> the total, else chunks[k][i]
  // (the slots [0, pre) of one chunk are pre * kNQ consecutive doubles, up to
  // 252: more than a block of 128 threads takes in one step)
  for (int e = threadIdx.x; e < f.pre * kNQ; e += blockDim.x) {
    const int i = e / kNQ, q = e % kNQ;
#pragma unroll
    for (int k = 0; k < kSmallChunks; ++k) {
      if (k < nch)
        S.ck[(i * kSmallChunks + k) * kNQ + q] =
            nch == 1 ? __ldcg(f.totals + e) : __ldcg(f.chunks + (size_t)k * kMaxSlots * kNQ + e);
    }
  }
  // level 1 of the remaining slots
  for (int w = warp; w < (f.nslots - f.pre) * nch; w += nwarps) {
    const int i = f.pre + w / nch, k = w % nch;
    const int t0 = k * kChunkTiles, t1 = min(b1, t0 + kChunkTiles);
    double v[kNQ];
    strided_sum(reinterpret_cast<const double2*>(f.part + (size_t)i * f.slot_stride), 2, t0, t1, v);
    if (lane == 0) {
#pragma unroll
      for (int q = 0; q < kNQ; ++q) S.ck[(i * kSmallChunks + k) * kNQ + q] = v[q];
    }
  }
  __syncthreads();
  // level 2: lane k adds chunk k to zero, then the tree (a one-chunk chain's
  // level-1 sum is its total)
  for (int i = warp; i < f.nslots; i += nwarps) {
    double v[kNQ];
#pragma unroll
    for (int q = 0; q < kNQ; ++q)
      v[q] = nch == 1 || lane < nch ? S.ck[(i * kSmallChunks + (nch == 1 ? 0 : lane)) * kNQ + q] : 0.0;
    if (nch > 1) {
#pragma unroll
      for (int q = 0; q < kNQ; ++q) v[q] = 0.0 + v[q];
      warp_tree(v);
    }
    if (lane == 0) {
#pragma unroll
      for (int q = 0; q < kNQ; ++q) {
        S.tot[i * kNQ + q] = v[q];
        f.totals[(size_t)i * kNQ + q] = v[q];
      }
    }
  }
  __syncthreads();
  finalize_combine<true>(f, S.T, S.tot, S.pre, S.ctr);
}

// The first pass (ahiggs2, eo 0) of a sweep inside a graph of several
// sweeps, with one extra block that runs the previous sweep's finalize (fp):
// its inputs -- the other slots' chunk sums and the last pass's partials --
// are not overwritten before this pass completes (the next pass's
// reduce-behind blocks write slot 0's chunk sums), and the RNG counters are
// not advanced inside such a graph (each sweep's passes take fixed offsets
// from its start; the graph's last finalize advances them), so the finalize
// runs beside this pass's tiles instead of between the sweeps.
template <typename R, int BS>
__global__ void __launch_bounds__(BS, min_blocks_bs<R, BS, 0>())
    higgs_fin_kernel(PassArgsOne p, const __grid_constant__ FinalizeArgs fp) {
  if ((int)blockIdx.x >= p.ntiles) {
    __shared__ SmallFinSmem S;
    pdl_wait();
    pdl_trigger();
    finalize_small_body<true>(fp, S);
  } else {
    higgs_tile<R, 0, true, 1, BS, kOne>(p, blockIdx.x);
  }
}

// ------------------------------------------------------------------ launches
// with programmatic dependent launch (lce_common.cuh: launch_pdl / pdl_wait)
template <typename R, int SPT, int BS, int OCC, int ONE>
void launch_higgs_k(int mode, const Args<ONE>& a, int nblocks, cudaStream_t s) {
  void (*k)(Args<ONE>) = mode == 0 ? higgs_kernel<R, 0, SPT, BS, OCC, ONE>
                                  : (mode == 1 ? higgs_kernel<R, 1, SPT, BS, OCC, ONE> : higgs_kernel<R, 2, SPT, BS, OCC, ONE>);
  (void)launch_pdl(k, nblocks, BS, 0, s, a);
}
template <typename R, int SPT, int BS, int OCC, int ONE>
void launch_link_k(int mode, int mu, const Args<ONE>& a, int nblocks, cudaStream_t s) {
  void (*k)(Args<ONE>);
  if (mode == 0)
    k = mu == 0 ? link_kernel<R, 0, 0, SPT, BS, OCC, ONE>
                : (mu == 1 ? link_kernel<R, 1, 0, SPT, BS, OCC, ONE> : link_kernel<R, 2, 0, SPT, BS, OCC, ONE>);
  else if (mode == 1)
    k = mu == 0 ? link_kernel<R, 0, 1, SPT, BS, OCC, ONE>
                : (mu == 1 ? link_kernel<R, 1, 1, SPT, BS, OCC, ONE> : link_kernel<R, 2, 1, SPT, BS, OCC, ONE>);
  else
    k = mu == 0 ? link3_kernel<R, 0, SPT, BS, OCC, ONE>
                : (mu == 1 ? link3_kernel<R, 1, SPT, BS, OCC, ONE> : link3_kernel<R, 2, SPT, BS, OCC, ONE>);
  (void)launch_pdl(k, nblocks, BS, 0, s, a);
}

// Tile shapes compiled: FP32 (BS, SPT) in {128, 256, 512} x {1} and
// {128, 256} x {2} at the 64-register cap, (448, 1) at two blocks per SM (72
// registers), and (128, 1) at 56 registers (a.occ = 1152); FP64 (256, 1),
// (256, 2) and (128, 1).  FP64 with 128 instead of 256 threads, us per sweep
// with measurements, in graphs of 8 sweeps and of one: 8^3 38.6 -> 35.2, 24^3
// 42.1 -> 38.7 and 47.2 -> 43.1 (few blocks: a pass is the latency of the SM
// with the most warps), 32^3 41.3 -> 42.0 and 47.2 -> 45.1, 40^3 51.6 -> 50.1
// and 51.3 -> 49.4, 48^3 63.8 -> 65.8 and 59.4 -> 55.4, 56^3 70.9 -> 72.2 (8),
// 64^3 96.5 -> 94.3 and 102.5 -> 98.6 (a finer last wave); a looser register cap
// (128) changed nothing.  The autotuner tells them apart, by graphs of one.
template <typename R, int ONE>
void pass_higgs(int mode, const Args<ONE>& a, int nblocks, cudaStream_t s) {
  if constexpr (sizeof(R) == 4) {
    if (a.bs == 128 && a.occ == 1152) {
      launch_higgs_k<R, 1, 128, 1152, ONE>(mode, a, nblocks, s);
      return;
    }
    if (a.bs == 128 && a.spt == 2) {
      launch_higgs_k<R, 2, 128, 0, ONE>(mode, a, nblocks, s);
      return;
    }
    if (a.bs == 512) {
      launch_higgs_k<R, 1, 512, 0, ONE>(mode, a, nblocks, s);
      return;
    }
    if (a.bs == 448) {
      launch_higgs_k<R, 1, 448, 0, ONE>(mode, a, nblocks, s);
      return;
    }
  }
  if (a.bs == 128) launch_higgs_k<R, 1, 128, 0, ONE>(mode, a, nblocks, s);
  else if (a.spt == 2) launch_higgs_k<R, 2, 256, 0, ONE>(mode, a, nblocks, s);
  else launch_higgs_k<R, 1, 256, 0, ONE>(mode, a, nblocks, s);
}

template <typename R, int ONE>
void pass_link(int mode, int mu, const Args<ONE>& a, int nblocks, cudaStream_t s) {
  if constexpr (sizeof(R) == 4) {
    if (a.bs == 128 && a.occ == 1152) {
      launch_link_k<R, 1, 128, 1152, ONE>(mode, mu, a, nblocks, s);
      return;
    }
    if (a.bs == 128 && a.spt == 2) {
      launch_link_k<R, 2, 128, 0, ONE>(mode, mu, a, nblocks, s);
      return;
    }
    if (a.bs == 512) {
      launch_link_k<R, 1, 512, 0, ONE>(mode, mu, a, nblocks, s);
      return;
    }
    if (a.bs == 448) {
      launch_link_k<R, 1, 448, 0, ONE>(mode, mu, a, nblocks, s);
      return;
    }
  }
  if (a.bs == 128) launch_link_k<R, 1, 128, 0, ONE>(mode, mu, a, nblocks, s);
  else if (a.spt == 2) launch_link_k<R, 2, 256, 0, ONE>(mode, mu, a, nblocks, s);
  else launch_link_k<R, 1, 256, 0, ONE>(mode, mu, a, nblocks, s);
}

// the first pass of a sweep carrying the previous sweep's finalize (one site
// per thread, 128 (64 registers in FP32) or 256 threads, in FP32 also 448 or 512)
template <typename R>
void pass_higgs_fin(const PassArgsOne& a, const FinalizeArgs& fp, int nblocks, cudaStream_t s) {
  if constexpr (sizeof(R) == 4) {
    if (a.bs == 448) {
      (void)launch_pdl(higgs_fin_kernel<R, 448>, nblocks, 448, 0, s, a, fp);
      return;
    }
    if (a.bs == 512) {
      (void)launch_pdl(higgs_fin_kernel<R, 512>, nblocks, 512, 0, s, a, fp);
      return;
    }
  }
  if (a.bs == 128) (void)launch_pdl(higgs_fin_kernel<R, 128>, nblocks, 128, 0, s, a, fp);
  else (void)launch_pdl(higgs_fin_kernel<R, 256>, nblocks, 256, 0, s, a, fp);
}

// a module's launches: LCE_PASSES(template, ..) defines them, (extern template, ..)
// declares them
#define LCE_PASSES(KIND, R, ONE)                                          \
  KIND void pass_higgs<R, ONE>(int, const Args<ONE>&, int, cudaStream_t); \
  KIND void pass_link<R, ONE>(int, int, const Args<ONE>&, int, cudaStream_t);
#define LCE_PASSES_FIN(KIND, R) \
  KIND void pass_higgs_fin<R>(const PassArgsOne&, const FinalizeArgs&, int, cudaStream_t);

}  // namespace lce
