// lce_meas.cu -- device reductions for the measurements.
//
// Slice quantities, summed per z slice over both parities in FP64 (the
// reference accumulates them per slice):
//   0..2   A_f                        f/correlator.f:58-59
//   3..11  per mu: Im a, Im b, -Re b  of U_f  (Im a and -i b, :61-74)
//   12     cos(4 |A|) on the un-fixed A     f/polyakov.f:52-55
//   13     |A|^2 on the un-fixed A          f/scalarcorr.f:48-51
// A measurement sums only the quantities it reports (SliceGroup): the
// correlators read U_f and A_f (60 bytes per FP32 site), the Polyakov loop
// and the scalar correlator A alone (12 bytes).  slice_sums_kernel gives a
// slice's sites to several blocks, slice_fold_kernel adds their partial sums
// in segment order, and correlators_kernel forms the periodic z
// autocorrelations of f/correlator.f:139-164, f/polyakov.f:100-108 and
// f/scalarcorr.f:96-104 (all z = 0..L3-1, as the reference writes them) and
// the meas2a average.
#include <algorithm>

#include "lce_internal.hpp"

namespace lce {

constexpr int kSliceQ = 14;
constexpr int kSliceThreads = 256;

// the quantities [q0, q0 + nq) of a group
template <int GROUP>
struct SliceCols {
  static constexpr int q0 = GROUP == kSliceFixed ? 0 : (GROUP == kSlicePolyakov ? 12 : 13);
  static constexpr int nq = GROUP == kSliceFixed ? 12 : 1;
};

// Sites of a slice one block sums: 1024 (4 per thread) up to 128 x 128
// slices, so that 128^3 gives 2048 blocks and 64^3 256; 4096 for larger
// slices, where there are blocks enough and the 12-quantity block reduction
// (~200 warp instructions) is spread over more sites.  It depends on the
// slice alone, so a z-slab adds a slice in the order of the whole lattice.
__host__ __device__ constexpr int slice_seg_sites(int nxy) { return 2 * nxy <= 16384 ? 1024 : 4096; }
int slice_segments(int nxy) { return ceil_div(2L * nxy, slice_seg_sites(nxy)); }

// One block per (segment, slice).  Bound by HBM where the fields exceed L2;
// the loads of four sites are in flight per thread.  At 256^3 in FP32 (ncu):
// U_f and A_f 190 us (5.3 TB/s), cos 4|A| 53 us, |A|^2 36 us, against 706 us
// for all quantities on every call with one block per slice, which left most
// of the chip without work; at 128^3 33 / 12 / 9 against 175 us.
template <typename R, int GROUP>
__global__ void __launch_bounds__(kSliceThreads) slice_sums_kernel(const ChainDev* chp, double* part) {
  const ChainDev& ch = *chp;
  const int nh = ch.nh, nxy = ch.nxy, z = blockIdx.y;
  constexpr int NQ = SliceCols<GROUP>::nq;
  double v[NQ];
#pragma unroll
  for (int q = 0; q < NQ; ++q) v[q] = 0.0;
  const int seg = slice_seg_sites(nxy), i0 = blockIdx.x * seg, i1 = min(2 * nxy, i0 + seg);
#pragma unroll 4
  for (int i = i0 + (int)threadIdx.x; i < i1; i += kSliceThreads) {
    const int eo = i >= nxy ? 1 : 0;
    const int s = z * nxy + (i - eo * nxy);
    const R* A = reinterpret_cast<const R*>(GROUP == kSliceFixed ? ch.af : ch.a) + (size_t)eo * 3 * nh + s;
    const R a1 = __ldg(A), a2 = __ldg(A + nh), a3 = __ldg(A + 2 * (size_t)nh);
    if constexpr (GROUP == kSliceFixed) {
      v[0] += (double)a1;
      v[1] += (double)a2;
      v[2] += (double)a3;
#pragma unroll
      for (int mu = 0; mu < 3; ++mu) {
        const su2<R> u = LinkIO<R>::ld(ch.uf, ((size_t)(mu * 2 + eo)) * nh + s);
        v[3 + 3 * mu] += (double)u.a.im;
        v[4 + 3 * mu] += (double)u.b.im;
        v[5 + 3 * mu] += -(double)u.b.re;
      }
    } else if constexpr (GROUP == kSlicePolyakov) {
      const R r2 = a1 * a1 + a2 * a2 + a3 * a3;
      v[0] += (double)cos((R)4 * sqrt(r2));
    } else {
      v[0] += (double)a1 * a1 + (double)a2 * a2 + (double)a3 * a3;
    }
  }
  block_reduce_store<NQ>(v, part + ((size_t)z * gridDim.x + blockIdx.x) * NQ);
}

// slice z's quantities from its segments' partial sums: one warp per
// quantity, lane l adds the segments l, l + 32, ... in order, then the tree
__global__ void __launch_bounds__(kSliceThreads) slice_fold_kernel(const double* part, int nseg, int nq, int q0,
                                                                   double* slices) {
  pdl_wait();
  const int z = blockIdx.x, lane = threadIdx.x & 31;
  for (int q = threadIdx.x >> 5; q < nq; q += kSliceThreads / 32) {
    double v = 0.0;
    for (int k = lane; k < nseg; k += 32) v += part[((size_t)z * nseg + k) * nq + q];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) slices[(size_t)z * kSliceQ + q0 + q] = v;
  }
}

// out: corr_a[L3], corr_u[L3], corr_3[L3], pol_slice[L3], pol_corr[L3],
//      sc_slice[L3], sc_corr[L3], af[3], pol_mean2, sc_mean; a group writes
// its own parts.  One warp per displacement z (8 per block), its lanes over
// the slices x0; every block holds all slice means in shared memory.
constexpr int kCorrThreads = 256;
template <int GROUP>
__global__ void __launch_bounds__(kCorrThreads) correlators_kernel(const double* slices, int L1, int L2, int L3,
                                                                   double* out) {
  extern __shared__ double sh[];  // [nq][L3], normalised by L1*L2
  constexpr int q0 = SliceCols<GROUP>::q0, NQ = SliceCols<GROUP>::nq;
  const double norm = 1.0 / ((double)L1 * (double)L2);
  pdl_wait();
  for (int i = threadIdx.x; i < L3 * NQ; i += kCorrThreads) {
    const int z = i / NQ, q = i - z * NQ;
    sh[q * L3 + z] = slices[(size_t)z * kSliceQ + q0 + q] * norm;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, z = blockIdx.x * (kCorrThreads / 32) + warp;
  double* tail = out + 7 * L3;
  constexpr int NC = GROUP == kSliceFixed ? 3 : 1;
  if (z < L3) {
    double c[NC];
#pragma unroll
    for (int k = 0; k < NC; ++k) c[k] = 0.0;
    for (int x0 = lane; x0 < L3; x0 += 32) {
      const int x1 = x0 + z < L3 ? x0 + z : x0 + z - L3;
      auto pq = [&](int q) { return sh[q * L3 + x0] * sh[q * L3 + x1]; };
      if constexpr (GROUP == kSliceFixed) {
        c[0] += pq(0) + pq(1) + pq(2);
        // Re[s1 s1' + s2 conj(s2')], s1 = sum Im a (real), s2 = sum -i b
        c[1] += pq(3) + (pq(4) + pq(5));
        c[1] += pq(6) + (pq(7) + pq(8));
        c[2] += pq(9) + (pq(10) + pq(11));
      } else {
        c[0] += pq(0);
      }
    }
#pragma unroll
    for (int k = 0; k < NC; ++k) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) c[k] += __shfl_down_sync(0xffffffffu, c[k], o);
    }
    if (lane == 0) {
      if constexpr (GROUP == kSliceFixed) {
        out[z] = c[0] / L3;
        out[L3 + z] = c[1] / (L3 * 2.0);
        out[2 * L3 + z] = c[2] / L3;
      } else {
        double* d = out + (GROUP == kSlicePolyakov ? 3 : 5) * L3;
        d[z] = sh[z];
        d[L3 + z] = c[0] / L3;
      }
    }
  }
  // the averages over all slices
  if (blockIdx.x == 0 && warp < (GROUP == kSliceFixed ? 3 : 1)) {
    double m = 0.0;
    for (int k = lane; k < L3; k += 32) m += sh[warp * L3 + k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m += __shfl_down_sync(0xffffffffu, m, o);
    if (lane == 0) {
      if (GROUP == kSliceFixed) tail[warp] = m / L3;
      else if (GROUP == kSlicePolyakov) tail[3] = (m / L3) * (m / L3);
      else tail[4] = m / L3;
    }
  }
}

// plaquette 1/2 Re Tr U_mu(x) U_nu(x+mu) U_mu(x+nu)^+ U_nu(x)^+ over both
// parities, each link read from HBM once (256^3 FP32: 210 us, 283 us with one
// parity after the other).  A block sums several tiles, at most kSumBlocks
// blocks in all, so that their partial sums are few.
template <typename R>
__global__ void __launch_bounds__(kBlock) plaquette_kernel(const ChainDev* chp, double* part) {
  const ChainDev& ch = *chp;
  const int nh = ch.nh, ntiles = 2 * ((nh + kBlock - 1) / kBlock);
  double v[1] = {0.0};
  for (int b = blockIdx.x; b < ntiles; b += gridDim.x) {
    int eo, s;
    if (!both_parities_site(b, nh, eo, s)) continue;
    const int oe = 1 - eo;
    const Coord X = site_coord(eo, s, ch.hx, ch.nxy, ch.dhx, ch.dnxy);
    const NbrOff o = nbr_offsets(ch, X);
#pragma unroll
    for (int mu = 0; mu < 3; ++mu)
#pragma unroll
      for (int nu = mu + 1; nu < 3; ++nu) {
        const su2<R> p = LinkIO<R>::ld(ch.u, ((size_t)(mu * 2 + eo)) * nh + s);
        const su2<R> q = LinkIO<R>::ld(ch.u, ((size_t)(nu * 2 + oe)) * nh + (s + o.p[mu]));
        const su2<R> t = LinkIO<R>::ld(ch.u, ((size_t)(mu * 2 + oe)) * nh + (s + o.p[nu]));
        const su2<R> e = LinkIO<R>::ld(ch.u, ((size_t)(nu * 2 + eo)) * nh + s);
        v[0] += (double)nn(nn(p, q), dd(t, e)).a.re;
      }
  }
  block_reduce_store<1>(v, part + blockIdx.x);
}

// Landau functional: sum over links of U_f of c_mu Re a
template <typename R>
__global__ void __launch_bounds__(kBlock) functional_kernel(const ChainDev* chp, double* part) {
  const ChainDev& ch = *chp;
  const int n = 2 * ch.nh;
  double v[1] = {0.0};
#pragma unroll 2
  for (int i = blockIdx.x * kBlock + (int)threadIdx.x; i < n; i += gridDim.x * kBlock) {
#pragma unroll
    for (int mu = 0; mu < 3; ++mu) {
      const double w = mu == 2 ? ch.alpha : 1.0;
      su2<R> u = LinkIO<R>::ld(ch.uf, (size_t)mu * n + i);
      v[0] += w * (double)u.a.re;
    }
  }
  block_reduce_store<1>(v, part + blockIdx.x);
}

template <typename R, int GROUP>
void slice_group(const ChainDev* ch, int nxy, int L3, double* part, double* slices, cudaStream_t s) {
  const int nseg = slice_segments(nxy);
  slice_sums_kernel<R, GROUP><<<dim3(nseg, L3), kSliceThreads, 0, s>>>(ch, part);
  (void)launch_pdl(slice_fold_kernel, L3, kSliceThreads, 0, s, (const double*)part, nseg, SliceCols<GROUP>::nq,
                   SliceCols<GROUP>::q0, slices);
}
template <typename R>
void launch_slice_sums(const ChainDev* ch, int group, int nxy, int L3, double* part, double* slices, cudaStream_t s) {
  if (group == kSliceFixed) slice_group<R, kSliceFixed>(ch, nxy, L3, part, slices, s);
  else if (group == kSlicePolyakov) slice_group<R, kSlicePolyakov>(ch, nxy, L3, part, slices, s);
  else slice_group<R, kSliceScalar>(ch, nxy, L3, part, slices, s);
}
size_t slice_part_doubles(int nxy, int L3) { return (size_t)slice_segments(nxy) * L3 * SliceCols<kSliceFixed>::nq; }

template <int GROUP>
void corr_group(const double* slices, int L1, int L2, int L3, double* out, cudaStream_t s) {
  const size_t smem = (size_t)L3 * SliceCols<GROUP>::nq * sizeof(double);
  if (smem > 48 * 1024)
    cudaFuncSetAttribute(correlators_kernel<GROUP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  (void)launch_pdl(correlators_kernel<GROUP>, ceil_div(L3, kCorrThreads / 32), kCorrThreads, smem, s, slices, L1, L2,
                   L3, out);
}
void launch_correlators(const double* slices, int group, int L1, int L2, int L3, double* out, cudaStream_t s) {
  if (group == kSliceFixed) corr_group<kSliceFixed>(slices, L1, L2, L3, out, s);
  else if (group == kSlicePolyakov) corr_group<kSlicePolyakov>(slices, L1, L2, L3, out, s);
  else corr_group<kSliceScalar>(slices, L1, L2, L3, out, s);
}
template <typename R>
int launch_plaquette(const ChainDev* ch, double* part, int nh, cudaStream_t s) {
  const int nb = std::min(kSumBlocks, 2 * ceil_div(nh, kBlock));
  plaquette_kernel<R><<<nb, kBlock, 0, s>>>(ch, part);
  return nb;
}
template <typename R>
int launch_functional(const ChainDev* ch, double* part, int nh, cudaStream_t s) {
  const int nb = std::min(kSumBlocks, ceil_div(2L * nh, kBlock));
  functional_kernel<R><<<nb, kBlock, 0, s>>>(ch, part);
  return nb;
}

template void launch_slice_sums<float>(const ChainDev*, int, int, int, double*, double*, cudaStream_t);
template void launch_slice_sums<double>(const ChainDev*, int, int, int, double*, double*, cudaStream_t);
template int launch_plaquette<float>(const ChainDev*, double*, int, cudaStream_t);
template int launch_plaquette<double>(const ChainDev*, double*, int, cudaStream_t);
template int launch_functional<float>(const ChainDev*, double*, int, cudaStream_t);
template int launch_functional<double>(const ChainDev*, double*, int, cudaStream_t);

}  // namespace lce
