// lce_gaugefix.cu -- overrelaxed Landau gauge fixing on the device, and the
// reference's iterative (steepest-descent) form, f/it_gauge_fixing.f.
//
// One iteration of f/or_gauge_fixing1.f:52-337 is two half-steps (eo = 0, 1).
// A half-step kernel gives one thread per site x of parity eo; the thread
//   * gathers w(x) = sum_mu c_mu [U_mu(x) + U_mu(x-mu)^+] (c_3 = alpha),
//   * on eo = 1 adds theta(x) = (Im w_a)^2 + |w_b|^2 to an FP64 partial sum,
//   * builds Omega = w/|w|, overrelaxes its angle by lambda,
//   * writes A_f(x) -> Omega A_f Omega^+, U_mu(x) -> Omega U_mu(x) and
//     U_mu(x-mu) -> U_mu(x-mu) Omega^+.
// Every link touched in a half-step belongs to exactly one thread, so the
// update is race free.  All links are rewritten in the eo = 1 half-step, so
// reunitarising there is exactly f/u_f_renorm.f after the iteration
// (f/landau_gauge.f:54-59).  The check sums the partials in a fixed order,
// counts the iteration and raises a device flag when theta <= limit_or (or
// the cap is reached): a one-block kernel after each iteration, or, while a
// block can add the partials itself (kGfMaxPartials), the blocks of the next
// half-step, with the kernel only at a batch's end.  Later kernels of a
// captured batch see the flag and return at once, so the host reads the
// state only once per batch.
#include <algorithm>

#include "lce_internal.hpp"

namespace lce {

template <typename R>
__device__ __forceinline__ su2<R> ldUf(const ChainDev& ch, int mu, int p, int s) {
  return LinkIO<R>::ld_cg(ch.uf, ((size_t)(mu * 2 + p)) * ch.nh + s);
}

// A value the compiler takes as new here.  The FP32 products of a value that
// was loaded in an earlier block are contracted otherwise than those of one
// loaded beside them; A_f, loaded early, keeps the bits it always had.
__device__ __forceinline__ void opaque(float& x) { asm volatile("" : "+f"(x)); }
__device__ __forceinline__ void opaque(double& x) { asm volatile("" : "+d"(x)); }

template <int MU>
__device__ __forceinline__ int nbr_dn(const ChainDev& ch, Coord X) {
  int x = X.x, y = X.y, z = X.z;
  if (MU == 0) x = wrap(x - 1, ch.L1);
  if (MU == 1) y = wrap(y - 1, ch.L2);
  if (MU == 2) z = wrap(z - 1, ch.L3);
  return site_index(x, y, z, ch.hx, ch.nxy);
}

// w sums in FP64: t1 = sum_mu c_mu U_mu(x), t2 = sum_mu c_mu U_mu(x-mu)
// (f/or_gauge_fixing1.f:97-142)
template <typename R>
__device__ __forceinline__ void gf_sums(const ChainDev& ch, const su2<R> (&um)[3], const su2<R> (&ud)[3],
                                        su2<double>& t1, su2<double>& t2) {
  const double al = ch.alpha;
  t1 = su2<double>{{0, 0}, {0, 0}};
  t2 = t1;
#pragma unroll
  for (int mu = 0; mu < 2; ++mu) {
    t1.a = t1.a + mk<double>(um[mu].a.re, um[mu].a.im);
    t1.b = t1.b + mk<double>(um[mu].b.re, um[mu].b.im);
  }
  t1.a = t1.a + mk<double>(al * um[2].a.re, al * um[2].a.im);
  t1.b = t1.b + mk<double>(al * um[2].b.re, al * um[2].b.im);
#pragma unroll
  for (int mu = 0; mu < 2; ++mu) {
    t2.a = t2.a + mk<double>(ud[mu].a.re, ud[mu].a.im);
    t2.b = t2.b + mk<double>(ud[mu].b.re, ud[mu].b.im);
  }
  t2.a = t2.a + mk<double>(al * ud[2].a.re, al * ud[2].a.im);
  t2.b = t2.b + mk<double>(al * ud[2].b.re, al * ud[2].b.im);
}

// The check of the previous iteration, made by every block of an iteration's
// first half-step for itself (nprev partials; 0: a check kernel follows every
// iteration), so that a batch needs no one-block kernel between iterations:
// the blocks add the partials in the same order and agree.  Block 0 records a
// stop.  gf_iters is counted by the second half-step, so it stands still here;
// 0: nothing to check yet.  A batch ends with gf_check_kernel, which gives the
// host the state of its last iteration.
__device__ __forceinline__ bool gf_stops(const ChainDev& ch, const ChainState* cst, double theta, int it) {
  return !(theta > ch.limit_or) || (cst->gf_cap > 0 && it >= cst->gf_cap);
}
template <int BS>
__device__ __forceinline__ bool gf_prev_stops(const ChainDev& ch, ChainState* cst, const double* part, int nprev) {
  const int it = cst->gf_iters;
  __shared__ double tot;
  double v[1] = {0.0};
#pragma unroll 4
  for (int b = threadIdx.x; b < nprev; b += BS) v[0] += __ldcg(part + b);
  block_reduce_store<1>(v, &tot);
  __syncthreads();
  const double theta = tot / ch.nh;
  if (it == 0 || !gf_stops(ch, cst, theta, it)) return false;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    cst->gf_theta = theta;
    cst->gf_done = 1;
  }
  return true;
}

// track != 0: also accumulate the gauge transform, G(x) -> Omega(x) G(x), so
// that U_f(x,mu) = G(x) U(x,mu) G(x+mu)^+ holds throughout.  FP32 is held to
// 64 registers (4 blocks per SM; 68 allowed 3): 8.5% less time per
// iteration at 128^3, the kernel being latency-bound.  s_lo: a z-slab's
// first visited site (its first and last planes are halos; sites
// [s_lo, nh - s_lo) are visited), 0 for a whole lattice.  last: the
// iteration's second half-step (the whole lattice's odd sites; a slab's
// local parity eo may be flipped), which sums theta and reunitarises.
// BS: threads per block (gf_block).  nprev: gf_prev_stops (first half-step).
template <typename R, int BS>
__global__ void __launch_bounds__(BS, sizeof(R) == 4 ? 4 * kBlock / BS : 1)
    gf_half_kernel(const ChainDev* chp, ChainState* cst, int eo, double* part, int track, int s_lo, int last,
                   int nprev) {
  const ChainDev& ch = *chp;
  const int s = s_lo + blockIdx.x * BS + threadIdx.x;
  const int oe = 1 - eo, nh = ch.nh, s_hi = nh - s_lo;
  const Coord X = site_coord(eo, s < s_hi ? s : s_lo, ch.hx, ch.nxy, ch.dhx, ch.dnxy);
  const int xm[3] = {nbr_dn<0>(ch, X), nbr_dn<1>(ch, X), nbr_dn<2>(ch, X)};
  pdl_wait();
  // every load of the half-step before the first branch on one: a chain of
  // round trips to L2 is what a small lattice's half-step waits for
  double th[1] = {0.0};
  su2<R> um[3], ud[3];
  R a1 = (R)0, a2 = (R)0, a3 = (R)0;
  R* Af = reinterpret_cast<R*>(ch.af);
  if (s < s_hi) {
#pragma unroll
    for (int mu = 0; mu < 3; ++mu) {
      um[mu] = ldUf<R>(ch, mu, eo, s);
      ud[mu] = ldUf<R>(ch, mu, oe, xm[mu]);
    }
    a1 = __ldcg(Af + ((size_t)(eo * 3 + 0)) * nh + s);
    a2 = __ldcg(Af + ((size_t)(eo * 3 + 1)) * nh + s);
    a3 = __ldcg(Af + ((size_t)(eo * 3 + 2)) * nh + s);
  }
  const int done = cst->gf_done;
  const bool stop = !last && nprev && gf_prev_stops<BS>(ch, cst, part, nprev);
  // Dependents may launch from here on.  Triggered at the kernel's start, the
  // blocks of many waiting half-steps filled the SMs and a half-step's own
  // blocks landed together on the few slots the last one left: 48 x 40 x 36
  // 12.0 us per iteration against 7.5.
  pdl_trigger();
  if (done || stop) return;
  if (last && nprev && blockIdx.x == 0 && threadIdx.x == 0) cst->gf_iters += 1;
  if (s < s_hi) {
    su2<double> t1, t2;
    gf_sums<R>(ch, um, ud, t1, t2);
    // (:145-146) w = first row of sum [U + U^+(x-mu)]
    const cpx<double> w1 = t1.a + cj(t2.a), w2 = t1.b - t2.b;
    if (last) {
      // (:153-158)
      const double d = t1.a.im - t2.a.im;
      th[0] = d * d + (w2.re * w2.re + w2.im * w2.im);
    }
    // (:162-184) Omega = w/|w| with its angle overrelaxed by lambda
    su2<R> o{{(R)w1.re, (R)w1.im}, {(R)w2.re, (R)w2.im}};
    const R sk = M<R>::sqrt(norm2(o));
    o = su2<R>{{M<R>::div(o.a.re, sk), M<R>::div(o.a.im, sk)}, {M<R>::div(o.b.re, sk), M<R>::div(o.b.im, sk)}};
    const R lam = (R)ch.lambda;
    if (ch.gf_angle == LCE_GF_ACOS) {
      // the reference's angle acos(Re Omega), clamped to the domain
      const R ca = o.a.re > (R)1 ? (R)1 : (o.a.re < (R)-1 ? (R)-1 : o.a.re);
      const R tht = acos(ca);
      if (tht != (R)0) {
        const R tho = lam * tht;
        const R q1 = cos(tho);
        const R q2 = sin(tho) / sin(tht) * o.a.im;
        const R f = -sin(tho) / sin(tht);
        o.a = mk<R>(q1, -q2);
        o.b = mk<R>(f * o.b.re, f * o.b.im);
      }
    } else {
      // same rotation, angle atan2(|vector part|, scalar part) of w: accurate
      // for the small angles that decide convergence below theta ~ 1e-7
      const double svd = sqrt(w1.im * w1.im + w2.re * w2.re + w2.im * w2.im);
      if (svd != 0.0) {
        const R sv = (R)svd;
        const R tho = lam * atan2(sv, (R)w1.re);
        R sn, cs;
        sincos(tho, &sn, &cs);
        const R f = sn / sv;
        o.a = mk<R>(cs, -f * (R)w1.im);
        o.b = mk<R>(-f * (R)w2.re, -f * (R)w2.im);
      }
    }
    // (:243-252) A_f(x) -> Omega (iA) Omega^+
    opaque(a1);
    opaque(a2);
    opaque(a3);
    const su2<R> ta = nn(o, ad(a1, a2, a3, o));
    Af[((size_t)(eo * 3 + 0)) * nh + s] = ta.b.im;
    Af[((size_t)(eo * 3 + 1)) * nh + s] = ta.b.re;
    Af[((size_t)(eo * 3 + 2)) * nh + s] = ta.a.im;
    // (:256-324) links at both ends; renormalise on the eo = 1 half-step
#pragma unroll
    for (int mu = 0; mu < 3; ++mu) {
      su2<R> a = nn(o, um[mu]);
      su2<R> b = nd(ud[mu], o);
      if (last) {
        a = unitarise64(a);
        b = unitarise64(b);
      }
      LinkIO<R>::st(ch.uf, ((size_t)(mu * 2 + eo)) * nh + s, a);
      LinkIO<R>::st(ch.uf, ((size_t)(mu * 2 + oe)) * nh + xm[mu], b);
    }
    if (track) {
      const size_t gi = (size_t)eo * nh + s;
      LinkIO<R>::st(ch.g, gi, unitarise64(nn(o, LinkIO<R>::ld_cg(ch.g, gi))));
    }
  }
  if (last) block_reduce_store<1>(th, part + blockIdx.x);
}

// One parity of f/it_gauge_fixing.f:52-206 (the reference's iterative gauge
// fixing): g = sum_mu (i Im a, b) of U_f(x,mu) minus the same of
// U_f(x-mu,mu) (:62-84), the second component as written g1(1) - g2(2)
// (:110) unless LCE_ITGF_FIX_COMPONENT; |g|^2 into the partial sums on the
// second parity (:116-120); Omega = exp(h), h = +-step g (:122-141); the
// transform of A_f and of the links at both ends (:143-210).  g, |g|^2 and
// Omega in FP64.  The step comes from the chain state (gf_step); renorm
// reunitarises the links on the second parity (u_f_renorm after the
// iteration, as f/landau_gauge.f:56-57 does for the overrelaxed form).
// s_lo and last as for gf_half_kernel (a z-slab's visited sites; the whole
// lattice's second half-step, which sums |g|^2 and reunitarises).
template <typename R, int BS>
__global__ void __launch_bounds__(BS) it_half_kernel(const ChainDev* chp, ChainState* cst, int eo, double* part,
                                                     int flags, int renorm, int s_lo, int last, int nprev) {
  const ChainDev& ch = *chp;
  const int s = s_lo + blockIdx.x * BS + threadIdx.x;
  const int oe = 1 - eo, nh = ch.nh, s_hi = nh - s_lo;
  const Coord X = site_coord(eo, s < s_hi ? s : s_lo, ch.hx, ch.nxy, ch.dhx, ch.dnxy);
  const int xm[3] = {nbr_dn<0>(ch, X), nbr_dn<1>(ch, X), nbr_dn<2>(ch, X)};
  pdl_wait();
  // every load of the half-step before the first branch on one: a chain of
  // round trips to L2 is what a small lattice's half-step waits for
  double th[1] = {0.0};
  su2<R> um[3], ud[3];
  R a1 = (R)0, a2 = (R)0, a3 = (R)0;
  R* Af = reinterpret_cast<R*>(ch.af);
  if (s < s_hi) {
#pragma unroll
    for (int mu = 0; mu < 3; ++mu) {
      um[mu] = ldUf<R>(ch, mu, eo, s);
      ud[mu] = ldUf<R>(ch, mu, oe, xm[mu]);
    }
    a1 = __ldcg(Af + ((size_t)(eo * 3 + 0)) * nh + s);
    a2 = __ldcg(Af + ((size_t)(eo * 3 + 1)) * nh + s);
    a3 = __ldcg(Af + ((size_t)(eo * 3 + 2)) * nh + s);
  }
  const int done = cst->gf_done;
  const bool stop = !last && nprev && gf_prev_stops<BS>(ch, cst, part, nprev);
  // Dependents may launch from here on.  Triggered at the kernel's start, the
  // blocks of many waiting half-steps filled the SMs and a half-step's own
  // blocks landed together on the few slots the last one left: 48 x 40 x 36
  // 12.0 us per iteration against 7.5.
  pdl_trigger();
  if (done || stop) return;
  if (last && nprev && blockIdx.x == 0 && threadIdx.x == 0) cst->gf_iters += 1;
  if (s < s_hi) {
    double g1a = 0, g1br = 0, g1bi = 0, g2a = 0, g2br = 0, g2bi = 0;
#pragma unroll
    for (int mu = 0; mu < 3; ++mu) {
      g1a += (double)um[mu].a.im;
      g1br += (double)um[mu].b.re;
      g1bi += (double)um[mu].b.im;
    }
#pragma unroll
    for (int mu = 0; mu < 3; ++mu) {
      g2a += (double)ud[mu].a.im;
      g2br += (double)ud[mu].b.re;
      g2bi += (double)ud[mu].b.im;
    }
    const bool fix = (flags & LCE_ITGF_FIX_COMPONENT) != 0;
    const double ga = g1a - g2a;
    const double gbr = fix ? g1br - g2br : -g2br;
    const double gbi = fix ? g1bi - g2bi : g1a - g2bi;
    if (last) th[0] = ga * ga + (gbr * gbr + gbi * gbi);
    const double st = (flags & LCE_ITGF_ASCEND) ? -cst->gf_step : cst->gf_step;
    const double ha = st * ga, hbr = st * gbr, hbi = st * gbi;
    const double t1 = sqrt(ha * ha + hbr * hbr + hbi * hbi);
    // the reference divides 0 by 0 where g = 0; the limit is 1
    const double t2 = t1 > 0.0 ? sin(t1) / t1 : 1.0;
    const su2<R> o{{(R)cos(t1), (R)(ha * t2)}, {(R)(hbr * t2), (R)(hbi * t2)}};
    opaque(a1);
    opaque(a2);
    opaque(a3);
    const su2<R> ta = nn(o, ad(a1, a2, a3, o));
    Af[((size_t)(eo * 3 + 0)) * nh + s] = ta.b.im;
    Af[((size_t)(eo * 3 + 1)) * nh + s] = ta.b.re;
    Af[((size_t)(eo * 3 + 2)) * nh + s] = ta.a.im;
#pragma unroll
    for (int mu = 0; mu < 3; ++mu) {
      su2<R> a = nn(o, um[mu]);
      su2<R> b = nd(ud[mu], o);
      if (renorm && last) {
        a = unitarise64(a);
        b = unitarise64(b);
      }
      LinkIO<R>::st(ch.uf, ((size_t)(mu * 2 + eo)) * nh + s, a);
      LinkIO<R>::st(ch.uf, ((size_t)(mu * 2 + oe)) * nh + xm[mu], b);
    }
    if (flags & LCE_ITGF_TRACK) {
      const size_t gi = (size_t)eo * nh + s;
      LinkIO<R>::st(ch.g, gi, unitarise64(nn(o, LinkIO<R>::ld_cg(ch.g, gi))));
    }
  }
  if (last) block_reduce_store<1>(th, part + blockIdx.x);
}

// U_f(x,mu) = G(x) U(x,mu) G(x+mu)^+ and A_f(x) -> G(x) A(x) G(x)^+, one
// thread per site; the parities' tiles in turn (both_parities_site), so that
// G is read from HBM once (256^3 FP32: 422 us, 5.4 TB/s; 447 us with one
// parity after the other)
template <typename R>
__global__ void __launch_bounds__(kBlock) gauge_apply_kernel(const ChainDev* chp) {
  const ChainDev& ch = *chp;
  const int nh = ch.nh;
  int eo, s;
  if (!both_parities_site(blockIdx.x, nh, eo, s)) return;
  const int oe = 1 - eo;
  const Coord X = site_coord(eo, s, ch.hx, ch.nxy, ch.dhx, ch.dnxy);
  const NbrOff o = nbr_offsets(ch, X);
  const su2<R> gx = LinkIO<R>::ld(ch.g, (size_t)eo * nh + s);
#pragma unroll
  for (int mu = 0; mu < 3; ++mu) {
    const su2<R> gp = LinkIO<R>::ld(ch.g, (size_t)oe * nh + (s + o.p[mu]));
    const size_t li = ((size_t)(mu * 2 + eo)) * nh + s;
    LinkIO<R>::st(ch.uf, li, unitarise64(nd(nn(gx, LinkIO<R>::ld(ch.u, li)), gp)));
  }
  const R* A = reinterpret_cast<const R*>(ch.a);
  R* Af = reinterpret_cast<R*>(ch.af);
  const su2<R> t = nn(gx, ad(A[((size_t)(eo * 3 + 0)) * nh + s], A[((size_t)(eo * 3 + 1)) * nh + s],
                             A[((size_t)(eo * 3 + 2)) * nh + s], gx));
  Af[((size_t)(eo * 3 + 0)) * nh + s] = t.b.im;
  Af[((size_t)(eo * 3 + 1)) * nh + s] = t.b.re;
  Af[((size_t)(eo * 3 + 2)) * nh + s] = t.a.im;
}

template <typename R>
__global__ void transform_identity_kernel(void* g, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    LinkIO<R>::st(g, i, su2<R>{{(R)1, (R)0}, {(R)0, (R)0}});
}

// sum the theta partials in block order, count the iteration (unless the
// second half-step has), test convergence
__global__ void __launch_bounds__(1024) gf_check_kernel(const ChainDev* chp, ChainState* cst, const double* part,
                                                        int nblocks, int count) {
  pdl_trigger();
  pdl_wait();
  if (cst->gf_done) return;
  double v[1] = {0.0};
#pragma unroll 8
  for (int b = threadIdx.x; b < nblocks; b += blockDim.x) v[0] += part[b];
  __shared__ double tot;
  block_reduce_store<1>(v, &tot);
  __syncthreads();
  if (threadIdx.x == 0) {
    const double theta = tot / chp->nh;
    const int it = cst->gf_iters + count;
    cst->gf_iters = it;
    cst->gf_theta = theta;
    if (gf_stops(*chp, cst, theta, it)) cst->gf_done = 1;
  }
}

// the same test for a lattice split into z-slabs: the slabs' theta sums (in
// slab order) over the whole lattice's nh odd sites, counted into slab 0's
// chain state, which the host copies to the other slabs
// fa: the Fourier-accelerated iteration's check (stop at gf_limit; fa = 1
// also shortens the step after an overshoot, as fa_check_kernel, which the
// conjugate-gradient form, fa = 2, does not); fa = 0: the overrelaxed
// iteration's (stop at limit_or)
__global__ void gf_check_slabs_kernel(const ChainDev* chp, ChainState* cst, const double* sums, int nslabs,
                                      double nh, int fa) {
  if (cst->gf_done) return;
  double tot = 0.0;
  for (int j = 0; j < nslabs; ++j) tot += sums[j];
  const double theta = tot / nh;
  const int it = cst->gf_iters + 1;
  if (fa == 1 && it > 1 && theta > 2.0 * cst->gf_theta) cst->gf_step = fmax(0.1, 0.7 * cst->gf_step);
  cst->gf_iters = it;
  cst->gf_theta = theta;
  const double limit = fa ? cst->gf_limit : chp->limit_or;
  if (!(theta > limit) || (cst->gf_cap > 0 && it >= cst->gf_cap)) cst->gf_done = 1;
}

// theta of the current U_f without updating (odd sites)
template <typename R>
__global__ void __launch_bounds__(kBlock) gf_theta_kernel(const ChainDev* chp, double* part) {
  const ChainDev& ch = *chp;
  const int s = blockIdx.x * kBlock + threadIdx.x;
  double th[1] = {0.0};
  if (s < ch.nh) {
    const Coord X = site_coord(1, s, ch.hx, ch.nxy, ch.dhx, ch.dnxy);
    const int xm[3] = {nbr_dn<0>(ch, X), nbr_dn<1>(ch, X), nbr_dn<2>(ch, X)};
    su2<R> um[3], ud[3];
#pragma unroll
    for (int mu = 0; mu < 3; ++mu) {
      um[mu] = ldUf<R>(ch, mu, 1, s);
      ud[mu] = ldUf<R>(ch, mu, 0, xm[mu]);
    }
    su2<double> t1, t2;
    gf_sums<R>(ch, um, ud, t1, t2);
    const cpx<double> w2 = t1.b - t2.b;
    const double d = t1.a.im - t2.a.im;
    th[0] = d * d + (w2.re * w2.re + w2.im * w2.im);
  }
  block_reduce_store<1>(th, part + blockIdx.x);
}

// One block; eight records in flight per thread before their in-order adds
// (one at a time, 65,536 records took 28 us at 256^3)
template <int NQ>
__global__ void __launch_bounds__(1024) sum_partials_kernel(const double* part, int nblocks, double* out) {
  double v[NQ];
#pragma unroll
  for (int q = 0; q < NQ; ++q) v[q] = 0.0;
#pragma unroll 8
  for (int b = threadIdx.x; b < nblocks; b += blockDim.x) {
#pragma unroll
    for (int q = 0; q < NQ; ++q) v[q] += part[(size_t)b * NQ + q];
  }
  block_reduce_store<NQ>(v, out);
}

// Threads per block of an undecomposed lattice's half-steps, and whether an
// iteration's check is made by the next one's first half-step (gf_prev_stops).
// 128 threads up to 8192 sites per parity, where blocks of 256 leave most of
// the chip idle (16^3 6.97 -> 6.52 us per iteration, FP64 6.67 -> 5.45; at 48 x
// 40 x 36 256 is better, 12.00 against 12.27).  Up to 512 partials every block
// can add them (us per iteration with a check kernel against the fold: 16^3
// 8.0 / 6.8, FP64 9.3 / 8.1; 48 x 40 x 36 9.3 / 7.6, FP64 12.5 / 11.2; 64^3, 512
// of them, 14.1 / 13.2, FP64 27.6 / 27.8).  Beyond that the blocks' adds cost more
// than the kernel: 64 x 64 x 80, 640 partials, 16.9 / 16.7 and in FP64 31.6 /
// 33.8, 64 x 64 x 116, 928, 20.2 / 20.6 and 39.5 / 43.7.
constexpr int kGfSmallBlock = 128, kGfSmallSites = 8192, kGfMaxPartials = 512;
int gf_block(int nh) { return nh <= kGfSmallSites ? kGfSmallBlock : kBlock; }
int gf_folds(int nh) {
  const int nb = ceil_div(nh, gf_block(nh));
  return nb <= kGfMaxPartials ? nb : 0;
}

// programmatic dependent launch: each kernel waits in griddepcontrol.wait
template <typename R>
void gf_half(const ChainDev* ch, ChainState* cst, int eo, double* part, int track, int nh, cudaStream_t s) {
  const int bs = gf_block(nh), nb = ceil_div(nh, bs);
  auto* k = bs == kGfSmallBlock ? gf_half_kernel<R, kGfSmallBlock> : gf_half_kernel<R, kBlock>;
  (void)launch_pdl(k, nb, bs, 0, s, ch, cst, eo, part, track, 0, eo, gf_folds(nh));
}
template <typename R>
void it_half(const ChainDev* ch, ChainState* cst, int eo, double* part, int flags, int renorm, int nh, int nprev,
             cudaStream_t s) {
  const int bs = gf_block(nh), nb = ceil_div(nh, bs);
  auto* k = bs == kGfSmallBlock ? it_half_kernel<R, kGfSmallBlock> : it_half_kernel<R, kBlock>;
  (void)launch_pdl(k, nb, bs, 0, s, ch, cst, eo, part, flags, renorm, 0, eo, nprev);
}
void gf_check(const ChainDev* ch, ChainState* cst, const double* part, int nh, int count, cudaStream_t s) {
  (void)launch_pdl(gf_check_kernel, 1, 1024, 0, s, ch, cst, part, ceil_div(nh, gf_block(nh)), count);
}

template <typename R>
void launch_gf_batch(const ChainDev* ch, ChainState* cst, int track, int it_flags, double* part, int nh, int n,
                     cudaStream_t s) {
  const int folds = gf_folds(nh);
  for (int k = 0; k < n; ++k) {
    for (int eo = 0; eo < 2; ++eo) {
      if (it_flags >= 0) it_half<R>(ch, cst, eo, part, it_flags, 1, nh, folds, s);
      else gf_half<R>(ch, cst, eo, part, track, nh, s);
    }
    if (!folds) gf_check(ch, cst, part, nh, 1, s);
  }
  if (folds) gf_check(ch, cst, part, nh, 0, s);
}

template <typename R>
int launch_gf_half(const ChainDev* ch, ChainState* cst, int eo, int last, double* part, int nh, int s_lo, int track,
                   cudaStream_t s) {
  const int nb = ceil_div(nh - 2 * s_lo, kBlock);
  (void)launch_pdl(gf_half_kernel<R, kBlock>, nb, kBlock, 0, s, ch, cst, eo, part, track, s_lo, last, 0);
  return nb;
}

void launch_gf_check_slabs(const ChainDev* ch, ChainState* cst, const double* sums, int nslabs, double nh,
                           cudaStream_t s, int fa) {
  gf_check_slabs_kernel<<<1, 1, 0, s>>>(ch, cst, sums, nslabs, nh, fa);
}

template <typename R>
void launch_it_iteration(const ChainDev* ch, ChainState* cst, int flags, double* part, int nh, cudaStream_t s) {
  for (int eo = 0; eo < 2; ++eo) it_half<R>(ch, cst, eo, part, flags, 0, nh, 0, s);
  gf_check(ch, cst, part, nh, 1, s);
}

template <typename R>
void launch_gauge_apply(const ChainDev* ch, int nh, cudaStream_t s) {
  gauge_apply_kernel<R><<<2 * ceil_div(nh, kBlock), kBlock, 0, s>>>(ch);
}

template <typename R>
void launch_transform_identity(void* g, int nh, cudaStream_t s) {
  transform_identity_kernel<R><<<ceil_div(2L * nh, 256), 256, 0, s>>>(g, (size_t)2 * nh);
}

template void launch_gauge_apply<float>(const ChainDev*, int, cudaStream_t);
template void launch_gauge_apply<double>(const ChainDev*, int, cudaStream_t);
template void launch_transform_identity<float>(void*, int, cudaStream_t);
template void launch_transform_identity<double>(void*, int, cudaStream_t);

template <typename R>
int launch_gf_theta(const ChainDev* ch, double* part, int nh, cudaStream_t s) {
  const int nb = ceil_div(nh, kBlock);
  gf_theta_kernel<R><<<nb, kBlock, 0, s>>>(ch, part);
  return nb;
}

void launch_sum_partials(const double* part, int nblocks, int nq, double* out, cudaStream_t s) {
  if (nq == 1) sum_partials_kernel<1><<<1, 1024, 0, s>>>(part, nblocks, out);
  else if (nq == 2) sum_partials_kernel<2><<<1, 1024, 0, s>>>(part, nblocks, out);
  else if (nq == 3) sum_partials_kernel<3><<<1, 1024, 0, s>>>(part, nblocks, out);
  else sum_partials_kernel<4><<<1, 1024, 0, s>>>(part, nblocks, out);
}

template void launch_gf_batch<float>(const ChainDev*, ChainState*, int, int, double*, int, int, cudaStream_t);
template void launch_gf_batch<double>(const ChainDev*, ChainState*, int, int, double*, int, int, cudaStream_t);
template int launch_gf_half<float>(const ChainDev*, ChainState*, int, int, double*, int, int, int, cudaStream_t);
template int launch_gf_half<double>(const ChainDev*, ChainState*, int, int, double*, int, int, int, cudaStream_t);
template <typename R>
int launch_it_half(const ChainDev* ch, ChainState* cst, int eo, int last, double* part, int nh, int s_lo, int flags,
                   cudaStream_t s) {
  const int nb = ceil_div(nh - 2 * s_lo, kBlock);
  (void)launch_pdl(it_half_kernel<R, kBlock>, nb, kBlock, 0, s, ch, cst, eo, part, flags, 1, s_lo, last, 0);
  return nb;
}
template int launch_it_half<float>(const ChainDev*, ChainState*, int, int, double*, int, int, int, cudaStream_t);
template int launch_it_half<double>(const ChainDev*, ChainState*, int, int, double*, int, int, int, cudaStream_t);

template void launch_it_iteration<float>(const ChainDev*, ChainState*, int, double*, int, cudaStream_t);
template void launch_it_iteration<double>(const ChainDev*, ChainState*, int, double*, int, cudaStream_t);
template int launch_gf_theta<float>(const ChainDev*, double*, int, cudaStream_t);
template int launch_gf_theta<double>(const ChainDev*, double*, int, cudaStream_t);

}  // namespace lce
