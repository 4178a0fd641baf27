// lce_update.cu -- checkerboard Monte Carlo update kernels.
//
// One pass = one routine over one parity (and one mu for links), one thread
// per site (or two), sites grouped in tiles of consecutive sites of one chain
// (the tile shape -- threads per block and sites per thread -- is chosen per
// context; the persistent form uses kBlock threads and one site per thread).
// The per-tile bodies fuse what the reference does as a chain of whole-lattice
// array passes (multall*, halo exchanges, temporaries): neighbour gathers, the
// SU(2) algebra, the random proposal, the accept/reject and the FP64 partial
// sums of the measurements, so every field element is read from HBM once per
// pass.
//
//   higgs_tile<R, MODE>    f/a_force.f + f/ahiggs2.f (MODE 0, heatbath),
//                          f/ahiggs3.f (MODE 1, overrelaxation),
//                          f/ahiggs1.f (MODE 2, Metropolis)
//   link_tile<R, MU, OR>   f/staples.f + f/agauge.f + f/heat_kpi.f (OR = 0);
//                          link overrelaxation (OR = 1, no reference)
//   finalize_sum/combine   deterministic FP64 reduction of the per-tile
//                          partials into /aver_loc/-style results (f/meas1.f)
//
// Two execution forms share these bodies:
//   * one kernel per pass (higgs_kernel, link_kernel, finalize_kernel),
//     chained with programmatic dependent launch and captured in a graph;
//   * sweep_persistent_kernel: one cooperative launch per sweep whose blocks
//     loop over the tile work list of every pass, with a bounded grid barrier
//     between passes (no kernel boundaries inside the sweep).
//
// Random numbers: Philox4x32-10 keyed by the chain seed with counter
// (site, call, pass), or, in validation mode, the host-supplied stream indexed
// in the reference's consumption order (slot layouts in lce_common.cuh).
//
// The tile bodies and the pass kernels are in lce_passes.cuh; here are the
// finalize kernels, the persistent sweep and the dispatch.
#include "lce_passes.cuh"

namespace lce {

LCE_PASSES(extern template, float, kOne)
LCE_PASSES(extern template, float, kMany)
LCE_PASSES(extern template, float, kTable)
LCE_PASSES(extern template, double, kOne)
LCE_PASSES(extern template, double, kMany)
LCE_PASSES(extern template, double, kTable)
LCE_PASSES_FIN(extern template, float)
LCE_PASSES_FIN(extern template, double)

__global__ void __launch_bounds__(kFinSmallWarps * 32) finalize_small_kernel(FinalizeArgs f) {
  __shared__ SmallFinSmem S;
  pdl_trigger();
  finalize_small_body<false>(f, S);
}

// kFinWarps warps per block, one level-1 item per warp.  One block: level 2
// and the combine follow in the same block (its own global writes are
// visible to it after the barrier).  Several blocks: the last block to finish
// level 1, by an atomic ticket, does level 2 and the combine.
constexpr int kFinWarps = 32;
__global__ void __launch_bounds__(kFinWarps * 32) finalize_kernel(FinalizeArgs f) {
  __shared__ FinTables T;
  pdl_trigger();
  load_tables(f, T);
  pdl_wait();
  const int warp = (int)(threadIdx.x >> 5);
  const int n1 = f.nchunks * (f.nslots - f.pre);
  for (int w = blockIdx.x * kFinWarps + warp; w < n1; w += gridDim.x * kFinWarps) finalize_chunk_warp(f, w);
  if (gridDim.x > 1) {
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned int t = atomicAdd(&f.st->ticket, 1u);
      last = (t == gridDim.x - 1);
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
  } else {
    __syncthreads();
  }
  if (f.nchunks > f.nchains) {
    for (int w = warp; w < f.nchains * f.nslots; w += kFinWarps) finalize_chain_warp(f, w);
    __syncthreads();
  }
  finalize_combine(f, T);
  if (gridDim.x > 1 && threadIdx.x == 0) f.st->ticket = 0;
}

// ------------------------------------------------------------------ persistent sweep
// Grid barrier for a cooperative launch (every block resident).  The arrival
// counter only grows: barrier k of a launch waits for count >= base +
// (k+1)*nblocks, where base (the count when the launch began) is stored in
// device memory by block 0 at the end of the previous launch.  Thread 0 of
// each block makes the block's writes visible (acq_rel fence after the block
// barrier), arrives with a non-returning release add, and polls the count
// with acquire loads and a bounded number of short sleeps.  On timeout the
// block records the status bit and the kernel returns instead of spinning on.
__device__ __forceinline__ void fence_acq_rel_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
__device__ __forceinline__ void red_release_add(unsigned* p, unsigned v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ bool grid_sync(GridBar* bar, unsigned nblocks, unsigned& target, unsigned* status) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    int ok = 1;
    fence_acq_rel_gpu();
    red_release_add(&bar->count, 1u);
    target += nblocks;
    unsigned spins = 0;
    while ((int)(ld_acquire(&bar->count) - target) < 0) {
      if (++spins > kBarrierSpinLimit) {
        ok = 0;
        atomicOr(status, kStatusBarrierTimeout);
        break;
      }
      __nanosleep(20);
    }
    fence_acq_rel_gpu();
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

template <typename R>
__device__ __forceinline__ void persistent_pass(const PersistArgs& a, const PassArgs& p, const PlanEntry& e) {
  const int nt = a.ntiles;
  switch (e.kind) {
    case kHiggsHB:
      for (int t = blockIdx.x; t < nt; t += gridDim.x) higgs_tile<R, 0, false>(p, t);
      break;
    case kHiggsOR:
      for (int t = blockIdx.x; t < nt; t += gridDim.x) higgs_tile<R, 1, false>(p, t);
      break;
    case kHiggsMetro:
      for (int t = blockIdx.x; t < nt; t += gridDim.x) higgs_tile<R, 2, false>(p, t);
      break;
    case kLinkHB:
      if (e.mu == 0) for (int t = blockIdx.x; t < nt; t += gridDim.x) link_tile<R, 0, 0, false>(p, t);
      else if (e.mu == 1) for (int t = blockIdx.x; t < nt; t += gridDim.x) link_tile<R, 1, 0, false>(p, t);
      else for (int t = blockIdx.x; t < nt; t += gridDim.x) link_tile<R, 2, 0, false>(p, t);
      break;
    case kLinkHB3:
      if (e.mu == 0) for (int t = blockIdx.x; t < nt; t += gridDim.x) link_tile<R, 0, 0, false, 3>(p, t);
      else if (e.mu == 1) for (int t = blockIdx.x; t < nt; t += gridDim.x) link_tile<R, 1, 0, false, 3>(p, t);
      else for (int t = blockIdx.x; t < nt; t += gridDim.x) link_tile<R, 2, 0, false, 3>(p, t);
      break;
    default:
      if (e.mu == 0) for (int t = blockIdx.x; t < nt; t += gridDim.x) link_tile<R, 0, 1, false>(p, t);
      else if (e.mu == 1) for (int t = blockIdx.x; t < nt; t += gridDim.x) link_tile<R, 1, 1, false>(p, t);
      else for (int t = blockIdx.x; t < nt; t += gridDim.x) link_tile<R, 2, 1, false>(p, t);
      break;
  }
}

// One sweep: every pass over the (chain, tile) work list, a grid barrier
// between passes, then the finalize reduction -- a single cooperative launch.
template <typename R>
__global__ void __launch_bounds__(kBlock, kPersistMinBlocks) sweep_persistent_kernel(PersistArgs a) {
  // only thread 0 of each block tracks the barrier target
  unsigned target = 0;
  if (threadIdx.x == 0) target = *(volatile unsigned*)&a.bar->base;
  PassArgs p = a.base;
  for (int i = 0; i < a.npasses; ++i) {
    const PlanEntry e = a.plan[i];
    p.eo = e.eo;
    p.pass_off = a.pass_off[i];
    p.stream_off = a.stream_off[i];
    p.part = e.slot == kNoSlot ? nullptr : const_cast<double*>(a.fin.part) + (size_t)e.slot * a.fin.slot_stride;
    persistent_pass<R>(a, p, e);
    if (!grid_sync(a.bar, gridDim.x, target, &a.base.st->status)) return;
  }
  {
    const int nw = (int)(blockDim.x >> 5), w0 = blockIdx.x * nw + (int)(threadIdx.x >> 5);
    for (int w = w0; w < a.fin.nchunks * a.fin.nslots; w += gridDim.x * nw) finalize_chunk_warp(a.fin, w);
    if (!grid_sync(a.bar, gridDim.x, target, &a.base.st->status)) return;
    if (a.fin.nchunks > a.fin.nchains)
      for (int w = w0; w < a.fin.nchains * a.fin.nslots; w += gridDim.x * nw) finalize_chain_warp(a.fin, w);
  }
  if (!grid_sync(a.bar, gridDim.x, target, &a.base.st->status)) return;
  if (blockIdx.x == 0) {
    __shared__ FinTables T;
    load_tables(a.fin, T);
    __syncthreads();
    finalize_combine(a.fin, T);
    // every block has passed the last barrier: record where the count stands
    if (threadIdx.x == 0) *(volatile unsigned*)&a.bar->base = target;
  }
}

// ------------------------------------------------------------------ renorm
// f/renorm.f:24-34, in FP64 arithmetic for FP32 links
template <typename R>
__global__ void renorm_kernel(void* u, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    LinkIO<R>::st(u, i, unitarise64(LinkIO<R>::ld_cg(u, i)));
}

// ------------------------------------------------------------------ debug
template <typename R, int MU>
__global__ void debug_staple_kernel(const ChainDev* chp, int eo, double* out) {
  const ChainDev& ch = *chp;
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= ch.nh) return;
  Coord X = site_coord(eo, s, ch.hx, ch.nxy, ch.dhx, ch.dnxy);
  su2<R> V = staple<R, MU>(ch, eo, nbr_offsets(ch, X), s);
  out[(size_t)s * 4 + 0] = V.a.re;
  out[(size_t)s * 4 + 1] = V.a.im;
  out[(size_t)s * 4 + 2] = V.b.re;
  out[(size_t)s * 4 + 3] = V.b.im;
}

template <typename R>
__global__ void debug_force_kernel(const ChainDev* chp, int eo, double* out) {
  const ChainDev& ch = *chp;
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= ch.nh) return;
  Coord X = site_coord(eo, s, ch.hx, ch.nxy, ch.dhx, ch.dnxy);
  R f1, f2, f3;
  higgs_force<R>(ch, eo, nbr_offsets(ch, X), s, f1, f2, f3);
  out[(size_t)s * 3 + 0] = f1;
  out[(size_t)s * 3 + 1] = f2;
  out[(size_t)s * 3 + 2] = f3;
}

// ------------------------------------------------------------------ launchers
// the single-chain kernels' arguments: the batch's first chain
PassArgsOne one_of(const PassArgsMany& a) {
  PassArgsOne o;
  static_cast<PassArgs&>(o) = a;
  const ChainDev& d = o.one = a.ch[0];
  o.beta = (float)d.beta;
  o.beta_a = (float)d.beta_a;
  o.beta_2 = (float)d.beta_2;
  o.beta_4 = (float)d.beta_4;
  o.inv_beta2 = (float)d.inv_beta2;
  o.cxval0 = (float)d.cxval0;
  return o;
}

template <typename R>
void launch_higgs(int mode, const PassArgsMany& a, int nblocks, cudaStream_t s) {
  if (a.nchains == 1) pass_higgs<R, kOne>(mode, one_of(a), nblocks, s);
  else if (a.many) pass_higgs<R, kMany>(mode, a, nblocks, s);
  else pass_higgs<R, kTable>(mode, a, nblocks, s);
}

template <typename R>
void launch_link(int mode, int mu, const PassArgsMany& a, int nblocks, cudaStream_t s) {
  if (a.nchains == 1) pass_link<R, kOne>(mode, mu, one_of(a), nblocks, s);
  else if (a.many) pass_link<R, kMany>(mode, mu, a, nblocks, s);
  else pass_link<R, kTable>(mode, mu, a, nblocks, s);
}

template <typename R>
void launch_higgs_fin(const PassArgsMany& a, const FinalizeArgs& fp, int nblocks, cudaStream_t s) {
  pass_higgs_fin<R>(one_of(a), fp, nblocks, s);
}
template void launch_higgs_fin<float>(const PassArgsMany&, const FinalizeArgs&, int, cudaStream_t);
template void launch_higgs_fin<double>(const PassArgsMany&, const FinalizeArgs&, int, cudaStream_t);

void launch_finalize(const FinalizeArgs& f, cudaStream_t s) {
  if (f.nchains == 1 && f.nchunks <= kSmallChunks) {
    (void)launch_pdl(finalize_small_kernel, 1, kFinSmallWarps * 32, 0, s, f);
    return;
  }
  // one block for up to four level-1 items per warp (no ticket); beyond
  // that one item per warp, all loads in flight at once
  const int n1 = f.nchunks * f.nslots;
  int grid = n1 <= 4 * kFinWarps ? 1 : (n1 + kFinWarps - 1) / kFinWarps;
  if (grid < 1) grid = 1;
  (void)launch_pdl(finalize_kernel, grid, kFinWarps * 32, 0, s, f);
}

template <typename R>
int persistent_grid() {
  int dev = 0, nsm = 0, per = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  if (cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, sweep_persistent_kernel<R>, kBlock, 0) != cudaSuccess)
    return 0;
  return per * nsm;
}

template <typename R>
cudaError_t launch_persistent(const PersistArgs& a, int grid, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = kBlock;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, sweep_persistent_kernel<R>, a);
}

template <typename R>
void launch_renorm(void* u, size_t nlinks, cudaStream_t s) {
  int grid = (int)std::min<size_t>((nlinks + 255) / 256, 148 * 16);
  renorm_kernel<R><<<grid, 256, 0, s>>>(u, nlinks);
}

template <typename R>
void launch_debug_staple(const ChainDev* ch, int eo, int mu, double* out, int nh, cudaStream_t s) {
  int grid = ceil_div(nh, 128);
  if (mu == 0) debug_staple_kernel<R, 0><<<grid, 128, 0, s>>>(ch, eo, out);
  else if (mu == 1) debug_staple_kernel<R, 1><<<grid, 128, 0, s>>>(ch, eo, out);
  else debug_staple_kernel<R, 2><<<grid, 128, 0, s>>>(ch, eo, out);
}

template <typename R>
void launch_debug_force(const ChainDev* ch, int eo, double* out, int nh, cudaStream_t s) {
  debug_force_kernel<R><<<ceil_div(nh, 128), 128, 0, s>>>(ch, eo, out);
}

#define LCE_INST(R)                                                                          \
  template void launch_higgs<R>(int, const PassArgsMany&, int, cudaStream_t);                  \
  template void launch_link<R>(int, int, const PassArgsMany&, int, cudaStream_t);              \
  template int persistent_grid<R>();                                                         \
  template cudaError_t launch_persistent<R>(const PersistArgs&, int, cudaStream_t);          \
  template void launch_renorm<R>(void*, size_t, cudaStream_t);                             \
  template void launch_debug_staple<R>(const ChainDev*, int, int, double*, int, cudaStream_t); \
  template void launch_debug_force<R>(const ChainDev*, int, double*, int, cudaStream_t);
LCE_INST(float)
LCE_INST(double)
#undef LCE_INST

}  // namespace lce
