// lce_net.cu -- learned warm start for Landau gauge fixing (no reference
// counterpart).
//
// A 3D convolutional network, 4 layers x 16 channels x 3^3 kernels, periodic
// boundaries, on the parity-split lattice (site i = eo*nh + s, the fields'
// order).  Inputs (16 channels): the 12 link components of U_f = U^G_prev and
// the 3 components of A_f, i.e. the configuration in the gauge of the previous
// measurement's converged transform G_prev.  Output: 4 channels, normalised
// to a unit quaternion Omega(x); the warm start is G = Omega G_prev.  Trained
// on (configuration in G_prev gauge, converged relative transform
// G_new G_prev^+) pairs recorded from the plain overrelaxed gauge fixing, with
// the loss 1 - Omega . T per site.
//
// Arithmetic: BF16 weights and activations, FP32 accumulation, on the tensor
// cores.  When L1 is a multiple of 128 all three contractions (forward, input
// gradient, weight gradient) run on tcgen05 with tensor-memory accumulators
// (conv_tc_kernel, wgrad_tc_kernel below); other extents use mma.sync.m16n8k16
// (bf16 x bf16 -> f32), which this paragraph describes.  A convolution is 27
// shifted 16x16 products: a warp owns 16 sites x 16 output channels (two
// m16n8 tiles), gathers the 16 neighbour rows of each offset straight into
// A fragments and takes the offset's weights (B) from shared memory.  The
// input gradient is the same kernel with the flipped, transposed weights; the
// weight gradient contracts over sites (M = out channel, N = in channel,
// K = 16 sites per step) into per-chunk partials summed in a fixed order.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "lce_internal.hpp"

namespace lce {
namespace {

constexpr int kC = 16;            // channels (inputs padded to 16)
constexpr int kK = 27;            // kernel offsets
constexpr int kLayers = 4;
constexpr int kOut = 4;           // output channels used (quaternion)
constexpr int kWl = kK * kC * kC;  // weights per layer [k][co][ci]
constexpr int kPl = kWl + kC;      // + bias
constexpr int kNParam = kLayers * kPl;
constexpr int kConvWarps = 4;
constexpr int kChunk = 4096;       // sites per weight-gradient block

struct NetGeom {
  int L1, L2, L3, hx, nxy, nh;
  FastDiv dhx, dnxy;
};

__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t pack2(__nv_bfloat16 lo, __nv_bfloat16 hi) {
  return (uint32_t)__bfloat16_as_ushort(lo) | ((uint32_t)__bfloat16_as_ushort(hi) << 16);
}

// two floats rounded to a BF16 pair, and a pair's two values
__device__ __forceinline__ uint32_t pack2f(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return pack2(v.x, v.y);
}
__device__ __forceinline__ float bf_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }

// flat index of the neighbour at offset (dx, dy, dz) of flat site i
__device__ __forceinline__ int nbr3(const NetGeom& g, int i, int dx, int dy, int dz) {
  const int eo = i >= g.nh ? 1 : 0, s = i - eo * g.nh;
  const Coord X = site_coord(eo, s, g.hx, g.nxy, g.dhx, g.dnxy);
  const int x = wrap(X.x + dx, g.L1), y = wrap(X.y + dy, g.L2), z = wrap(X.z + dz, g.L3);
  return ((eo + dx + dy + dz) & 1) * g.nh + site_index(x, y, z, g.hx, g.nxy);
}

// out[i][co] = act( bias[co] + sum_k sum_ci in[nbr_k(i)][ci] W[k][co][ci] ) (* mask)
// MODE 0: hidden layer (ReLU, BF16 out); 1: output layer (FP32 out, first 8
// channels); 2: input gradient (BF16 out times (mask_src > 0), no bias)
template <int MODE>
__global__ void __launch_bounds__(32 * kConvWarps) conv_kernel(const __nv_bfloat16* __restrict__ in,
                                                               const __nv_bfloat16* __restrict__ W,
                                                               const float* __restrict__ bias,
                                                               __nv_bfloat16* __restrict__ out16,
                                                               float* __restrict__ out32,
                                                               const __nv_bfloat16* __restrict__ mask_src, NetGeom g) {
  __shared__ uint32_t sw[kK * kC * kC / 2];  // W as bf16 pairs [k][co][ci/2]
  const uint32_t* W32 = reinterpret_cast<const uint32_t*>(W);
  for (int j = threadIdx.x; j < kK * kC * kC / 2; j += blockDim.x) sw[j] = W32[j];
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, gr = lane >> 2, tq = lane & 3;
  const int nsites = 2 * g.nh, ntiles = (nsites + 15) / 16;
  const uint32_t* in32 = reinterpret_cast<const uint32_t*>(in);
  for (int tile = blockIdx.x * kConvWarps + warp; tile < ntiles; tile += gridDim.x * kConvWarps) {
    const int r0 = tile * 16 + gr, r1 = r0 + 8;
    const bool v0 = r0 < nsites, v1 = r1 < nsites;
    float acc[2][4] = {{0, 0, 0, 0}, {0, 0, 0, 0}};
#pragma unroll 1
    for (int k = 0; k < kK; ++k) {
      const int dx = k / 9 - 1, dy = (k / 3) % 3 - 1, dz = k % 3 - 1;
      const int i0 = v0 ? nbr3(g, r0, dx, dy, dz) : 0, i1 = v1 ? nbr3(g, r1, dx, dy, dz) : 0;
      uint32_t a[4];
      a[0] = v0 ? __ldg(in32 + (size_t)i0 * 8 + tq) : 0u;
      a[1] = v1 ? __ldg(in32 + (size_t)i1 * 8 + tq) : 0u;
      a[2] = v0 ? __ldg(in32 + (size_t)i0 * 8 + tq + 4) : 0u;
      a[3] = v1 ? __ldg(in32 + (size_t)i1 * 8 + tq + 4) : 0u;
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const uint32_t* wk = sw + (k * kC + 8 * j + gr) * (kC / 2);
        mma16816(acc[j], a, wk[tq], wk[tq + 4]);
      }
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int c = 8 * j + 2 * tq;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = h ? r1 : r0;
        if (!(h ? v1 : v0)) continue;
        float x0 = acc[j][2 * h], x1 = acc[j][2 * h + 1];
        if (MODE != 2) {
          x0 += bias[c];
          x1 += bias[c + 1];
        }
        if (MODE == 0) {
          x0 = fmaxf(x0, 0.f);
          x1 = fmaxf(x1, 0.f);
          reinterpret_cast<uint32_t*>(out16)[(size_t)r * 8 + c / 2] =
              pack2(__float2bfloat16_rn(x0), __float2bfloat16_rn(x1));
        } else if (MODE == 1) {
          if (j == 0) {
            out32[(size_t)r * 8 + c] = x0;
            out32[(size_t)r * 8 + c + 1] = x1;
          }
        } else {
          const __nv_bfloat16* m = mask_src + (size_t)r * kC + c;
          if (!(__bfloat162float(m[0]) > 0.f)) x0 = 0.f;
          if (!(__bfloat162float(m[1]) > 0.f)) x1 = 0.f;
          reinterpret_cast<uint32_t*>(out16)[(size_t)r * 8 + c / 2] =
              pack2(__float2bfloat16_rn(x0), __float2bfloat16_rn(x1));
        }
      }
    }
  }
}

// ------------------------------------------------------------------ tcgen05 path
// The same convolution on the 5th-generation tensor cores when L1 is a
// multiple of 128.  A tile is 128 consecutive sites j = x0 .. x0+127 of one
// x-line (y, z).  Moving the x offset out of the operand,
//   P_dx[j][co] = sum_{(dy,dz)} sum_ci in[(j, y+dy, z+dz)][ci] W[dx,dy,dz][co][ci]
//   out[i][co]  = P_-1[i-1][co] + P_0[i][co] + P_+1[i+1][co],
// makes the tile one GEMM: M = 128 sites, K = 9 lines x 16 channels,
// N = 3 dx x 16 output channels -- 9 tcgen05.mma of M 128, N 48, K 16 (BF16
// in, FP32 accumulate in 48 tensor-memory columns) instead of 27 of N 16.
// The 9 (dy, dz) lines sit in shared memory as channel planes (channels 0-7
// and 8-15, 16-byte rows): the canonical K-major layout without swizzle
// (8-row core matrices of 128 B, the second K chunk one plane further); the
// weights, staged once per CTA, in the same layout with N = 48 rows per line.
// The epilogue reads each warp's 32 rows out of tensor memory and forms the
// x-shifted sum with warp shuffles; the rows across warp boundaries go
// through shared memory, and the two rows outside the tile (P_-1 at x0-1,
// P_+1 at x0+128) are computed on the CUDA cores from staged halo sites.
// A CTA takes a contiguous range of the tiles in the order (x segment, y, z)
// and walks each column (x0, y) along z: a tile shares the lines of two of its
// three planes with the tile before, so the planes go through a ring of four
// slots of three dy lines, one plane copied per tile instead of three (at
// 128^3 a convolution moves 218 MB from L2 to the SMs; staging all nine lines
// per tile moved 655 MB).  Two accumulators of 48 columns take turns: while
// the tensor core works on tile i + 1 and the copy of tile i + 2's plane is in
// flight, warps 0-3 run the epilogue of tile i.  Warp 4 issues the MMAs and
// warp 5 computes the rows outside the tile ahead of the epilogue (in the
// epilogue's warps, or both in one, they lengthen the chain of a tile).
// At 128^3 (ncu): hidden layer 87 us, input gradient 89, output layer 75,
// against 121 / 148 / 112 with nine lines staged, multiplied and written in
// turn per tile; bound now by a tile's chain of waits at 18 warps per SM
// (~3000 cycles; the MMAs take 24 cycles each, 9 per tile, of the tensor pipe).
constexpr int kTcRows = 128;                          // sites per tile
constexpr int kTcThreads = kTcRows + 64;
constexpr int kTcN = 3 * kC;                          // N: 3 dx x 16 output channels
constexpr int kTcSlots = 4;                           // ring of z planes
constexpr int kTcLineBytes = 2 * kTcRows * 16;        // one line: 2 channel planes
constexpr int kTcActBytes = kTcSlots * 3 * kTcLineBytes;
constexpr int kTcWtBytes = 9 * 2 * kTcN * 16;         // 9 lines x 2 planes x 48 rows
constexpr int kTcHaloBytes = kTcSlots * 3 * 2 * 2 * 16;  // x0-1 and x0+128: [slot][dy][side][plane]
constexpr int kTcXchBytes = (2 * 4 + 4) * kC * 4;     // warp-boundary rows, two sets of edge rows (FP32)
constexpr int kTcSmem = kTcActBytes + kTcWtBytes + kTcHaloBytes + kTcXchBytes + 16;
constexpr int kTcCtasPerSm = 3;
constexpr int kTcCols = 128;                          // tensor-memory columns: 2 accumulators, 64 apart
static_assert(kTcCtasPerSm * (kTcSmem + 1024) <= 228 * 1024, "conv CTAs per SM");
static_assert(kTcCtasPerSm * kTcCols <= 512, "tensor memory of the conv CTAs");
constexpr unsigned kTcSpin = 1u << 24;                // mbarrier polls before giving up

// tcgen05.mma instruction descriptor: BF16 A and B (K-major), FP32 D, M 128, N 48
constexpr uint32_t kTcIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((kTcN >> 3) << 17) | ((128u >> 4) << 24);

// shared-memory matrix descriptor, no swizzle: start address, leading-dimension
// byte offset (between the two K chunks), stride-dimension byte offset
// (between 8-row core matrices), all in 16 B units; version 1
__device__ __forceinline__ uint64_t tc_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)((lbo >> 4) & 0x3FFF) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFF) << 32) | (1ull << 46);
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// 16-byte asynchronous global -> shared copy (L2 only): a thread issues all of
// its staging copies before waiting once, instead of one load round trip each
__device__ __forceinline__ void cp16(void* dst_smem, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst_smem)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_wait_all() {
  asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ bool tc_try_wait(uint32_t mbar, uint32_t phase) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred P1;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, P1;\n\t}"
      : "=r"(ok)
      : "r"(mbar), "r"(phase)
      : "memory");
  return ok != 0;
}

__device__ __forceinline__ bool tc_wait(uint32_t mbar, uint32_t phase) {
  for (unsigned i = 0; i < kTcSpin; ++i)
    if (tc_try_wait(mbar, phase)) return true;
  return false;
}

// flat (parity-split) index of site (x, y, z), coordinates in range
__device__ __forceinline__ int tc_flat(const NetGeom& g, int x, int y, int z) {
  return ((x + y + z) & 1) * g.nh + site_index(x, y, z, g.hx, g.nxy);
}

// the tiles of CTA b of n: [first, last) of the order (x segment, y, z)
__device__ __forceinline__ void tc_range(int ntiles, int& first, int& last) {
  first = (int)((long long)ntiles * blockIdx.x / gridDim.x);
  last = (int)((long long)ntiles * (blockIdx.x + 1) / gridDim.x);
}

template <int MODE>
__global__ void __launch_bounds__(kTcThreads, kTcCtasPerSm) conv_tc_kernel(const __nv_bfloat16* __restrict__ in,
                                                      const __nv_bfloat16* __restrict__ W,
                                                      const float* __restrict__ bias,
                                                      __nv_bfloat16* __restrict__ out16, float* __restrict__ out32,
                                                      const __nv_bfloat16* __restrict__ mask_src, NetGeom g,
                                                      unsigned* status) {
  extern __shared__ __align__(1024) uint8_t tc_sm[];
  uint8_t* act = tc_sm;                                      // [slot][dy][plane][row] 16 B
  uint8_t* wts = act + kTcActBytes;
  uint8_t* halo = wts + kTcWtBytes;                          // [slot][dy][side][plane] 16 B
  float* xch = reinterpret_cast<float*>(halo + kTcHaloBytes);  // [0..3] P_-1 of lane 31, [4..7] P_+1 of lane 0, [8 + 2 (i % 2) + side] edges of tile i
  uint64_t* mbar = reinterpret_cast<uint64_t*>(xch + (2 * 4 + 4) * kC);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(mbar + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool epi = warp < 4;

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)), "r"(kTcCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(mbar)), "r"(1) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // weights once per CTA: line s, plane c, row n = dx_index * 16 + o holds
  // inputs 8c .. 8c+7 of output o at offset k = dx_index * 9 + s
  const uint4* W4 = reinterpret_cast<const uint4*>(W);
  for (int e = tid; e < 9 * 2 * kTcN; e += blockDim.x) {
    const int sg = e / (2 * kTcN), c = (e / kTcN) & 1, n = e % kTcN;
    const int k = (n >> 4) * 9 + sg, o = n & 15;
    cp16(reinterpret_cast<uint4*>(wts) + e, W4 + (k * kC + o) * 2 + c);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tslot;
  const uint4* in4 = reinterpret_cast<const uint4*>(in);
  uint32_t phase = 0;
  const int side = lane >> 4;  // warp 5: lane (side, output) of the rows outside the tile
  float bs[kC];
#pragma unroll
  for (int c = 0; c < kC; ++c) bs[c] = MODE != 2 ? __ldg(bias + c) : 0.f;

  int t, tend;
  tc_range((g.L1 >> 7) * g.L2 * g.L3, t, tend);
  bool ok = true;
  while (ok && t < tend) {
    // one column: tiles z0 .. z0 + n - 1; plane p of the run is z0 - 1 + p, in slot p % 4
    const int col = t / g.L3, z0 = t - col * g.L3, n = min(g.L3 - z0, tend - t);
    const int x0 = (col / g.L2) << 7, y = col % g.L2;
    t += n;
    auto load_plane = [&](int p) {
      const int slot = p & (kTcSlots - 1);
      int zz = z0 - 1 + p;
      zz = zz < 0 ? zz + g.L3 : (zz >= g.L3 ? zz - g.L3 : zz);
      if (epi) {
        uint4* d = reinterpret_cast<uint4*>(act + slot * 3 * kTcLineBytes);
#pragma unroll
        for (int dy = 0; dy < 3; ++dy) {
          const size_t f = (size_t)tc_flat(g, x0 + tid, wrap(y + dy - 1, g.L2), zz) * 2;
          cp16(d + (dy * 2) * kTcRows + tid, in4 + f);
          cp16(d + (dy * 2 + 1) * kTcRows + tid, in4 + f + 1);
        }
      } else if (warp == 5 && lane < 12) {
        // the halo sites, copied and read by warp 5 alone
        const int dy = lane >> 2, sd = (lane >> 1) & 1, c = lane & 1;
        const int xx = wrap(sd ? x0 + kTcRows : x0 - 1, g.L1);
        cp16(reinterpret_cast<uint4*>(halo) + slot * 12 + lane,
             in4 + (size_t)tc_flat(g, xx, wrap(y + dy - 1, g.L2), zz) * 2 + c);
      }
    };
    // tile i's nine MMAs in the order (dy, dz), into accumulator i & 1
    auto issue = [&](int i) {
      const uint32_t a0 = smem_u32(act), dst = tmem + (uint32_t)((i & 1) * 64);
      uint64_t ad[3];
#pragma unroll
      for (int dz = 0; dz < 3; ++dz)
        ad[dz] = tc_desc(a0 + ((i + dz) & (kTcSlots - 1)) * 3 * kTcLineBytes, kTcRows * 16, 128);
      const uint64_t bd = tc_desc(smem_u32(wts), kTcN * 16, 128);
#pragma unroll
      for (int sg = 0; sg < 9; ++sg) {
        // (the address fields, in 16-byte units, do not carry out of their 14 bits)
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(dst), "l"(ad[sg % 3] + (uint64_t)(sg / 3 * (kTcLineBytes / 16))), "l"(bd + (uint64_t)(sg * 2 * kTcN)),
              "r"(kTcIdesc), "r"(sg > 0 ? 1u : 0u)
            : "memory");
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                       smem_u32(mbar))
                   : "memory");
    };
    load_plane(0);
    load_plane(1);
    load_plane(2);
    cp_commit();
    if (n > 1) load_plane(3);
    cp_commit();
    cp_wait<1>();
    // generic-proxy shared-memory writes -> visible to the tensor core (async proxy)
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (tid == kTcRows) issue(0);

    for (int i = 0; i < n; ++i) {
      const int f = epi ? tc_flat(g, x0 + tid, y, z0 + i) : 0;
      uint4 m0, m1;  // MODE 2: the activation whose sign masks the gradient
      if (MODE == 2 && epi) {
        const uint4* m = reinterpret_cast<const uint4*>(mask_src) + (size_t)f * 2;
        m0 = __ldg(m);
        m1 = __ldg(m + 1);
      }
      if (warp == 5) {
        // the rows outside tile i on the CUDA cores: lanes 0-15 P_-1[x0-1][o],
        // lanes 16-31 P_+1[x0+128][o] (the tile's planes were waited for before its MMAs)
        float v = 0.f;
#pragma unroll
        for (int sg = 0; sg < 9; ++sg) {
          const int slot = (i + sg % 3) & (kTcSlots - 1);
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const uint4 x = reinterpret_cast<const uint4*>(halo)[((slot * 3 + sg / 3) * 2 + side) * 2 + c];
            const uint4 w = reinterpret_cast<const uint4*>(wts)[(sg * 2 + c) * kTcN + side * 2 * kC + (lane & 15)];
            const uint32_t xw[4] = {x.x, x.y, x.z, x.w}, ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              v = fmaf(bf_lo(xw[q]), bf_lo(ww[q]), v);
              v = fmaf(bf_hi(xw[q]), bf_hi(ww[q]), v);
            }
          }
        }
        xch[(8 + 2 * (i & 1) + side) * kC + (lane & 15)] = v;
        __syncwarp();
      }
      const uint32_t ph = phase;
      phase ^= 1u;
      const bool done = tc_wait(smem_u32(mbar), ph);
      // tile i's MMAs have read slot i % 4 (plane i) for the last time
      if (done && i + 2 < n) load_plane(i + 4);
      cp_commit();
      cp_wait<1>();  // the planes of tile i + 1
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      if (__syncthreads_or(!done)) {
        // record the failure, give the MMAs a second bounded wait, then stop
        if (!done) {
          if (lane == 0) atomicOr(status, 1u);
          tc_wait(smem_u32(mbar), ph);
        }
        ok = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (!epi) {
        if (tid == kTcRows && i + 1 < n) issue(i + 1);
        __syncwarp();
        continue;
      }
      // row j = 32 warp + lane: P_-1[j] (columns 0-15), P_0[j] (16-31), P_+1[j] (32-47)
      uint32_t vm[16], v0[16], vp[16];
      const uint32_t ta = tmem + (uint32_t)((i & 1) * 64) + ((uint32_t)(warp * 32) << 16);
#define LCE_TC_LD16(dst, col)                                                                                   \
  asm volatile(                                                                                                 \
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, " \
      "%15}, [%16];"                                                                                            \
      : "=r"(dst[0]), "=r"(dst[1]), "=r"(dst[2]), "=r"(dst[3]), "=r"(dst[4]), "=r"(dst[5]), "=r"(dst[6]),       \
        "=r"(dst[7]), "=r"(dst[8]), "=r"(dst[9]), "=r"(dst[10]), "=r"(dst[11]), "=r"(dst[12]), "=r"(dst[13]),   \
        "=r"(dst[14]), "=r"(dst[15])                                                                            \
      : "r"(ta + (col)))
      LCE_TC_LD16(vm, 0);
      LCE_TC_LD16(v0, 16);
      LCE_TC_LD16(vp, 32);
#undef LCE_TC_LD16
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      // rows across warp boundaries
      if (lane == 31 || lane == 0) {
        uint4* d = reinterpret_cast<uint4*>(xch + (lane ? warp : 4 + warp) * kC);
#pragma unroll
        for (int c = 0; c < 4; ++c)
          d[c] = lane ? make_uint4(vm[4 * c], vm[4 * c + 1], vm[4 * c + 2], vm[4 * c + 3])
                      : make_uint4(vp[4 * c], vp[4 * c + 1], vp[4 * c + 2], vp[4 * c + 3]);
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      asm volatile("bar.sync 1, %0;" ::"n"(kTcRows) : "memory");  // warps 0-3
      float o[kC];
#pragma unroll
      for (int c = 0; c < kC; ++c) {
        float pm = __shfl_up_sync(0xffffffffu, __uint_as_float(vm[c]), 1);
        float pp = __shfl_down_sync(0xffffffffu, __uint_as_float(vp[c]), 1);
        vm[c] = __float_as_uint(pm);
        vp[c] = __float_as_uint(pp);
      }
      if (lane == 31 || lane == 0) {
        const int edge = 8 + 2 * (i & 1);
        const uint4* e = reinterpret_cast<const uint4*>(
            xch + (lane == 0 ? (warp == 0 ? edge : warp - 1) : (warp == 3 ? edge + 1 : 4 + warp + 1)) * kC);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const uint4 r = e[c];
          if (lane == 0) vm[4 * c] = r.x, vm[4 * c + 1] = r.y, vm[4 * c + 2] = r.z, vm[4 * c + 3] = r.w;
          else vp[4 * c] = r.x, vp[4 * c + 1] = r.y, vp[4 * c + 2] = r.z, vp[4 * c + 3] = r.w;
        }
      }
#pragma unroll
      for (int c = 0; c < kC; ++c)
        o[c] = __uint_as_float(vm[c]) + __uint_as_float(v0[c]) + __uint_as_float(vp[c]) + (MODE != 2 ? bs[c] : 0.f);
      if (MODE == 1) {
        float4* d = reinterpret_cast<float4*>(out32 + (size_t)f * 8);
        d[0] = make_float4(o[0], o[1], o[2], o[3]);
        d[1] = make_float4(o[4], o[5], o[6], o[7]);
      } else {
        if (MODE == 0) {
#pragma unroll
          for (int c = 0; c < kC; ++c) o[c] = fmaxf(o[c], 0.f);
        } else {
          const uint32_t mw[8] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w};
#pragma unroll
          for (int c = 0; c < kC; ++c)
            if (!((c & 1 ? bf_hi(mw[c >> 1]) : bf_lo(mw[c >> 1])) > 0.f)) o[c] = 0.f;
        }
        const uint4 w0 = make_uint4(pack2f(o[0], o[1]), pack2f(o[2], o[3]), pack2f(o[4], o[5]), pack2f(o[6], o[7]));
        const uint4 w1 =
            make_uint4(pack2f(o[8], o[9]), pack2f(o[10], o[11]), pack2f(o[12], o[13]), pack2f(o[14], o[15]));
        uint4* d = reinterpret_cast<uint4*>(out16) + (size_t)f * 2;
        d[0] = w0;
        d[1] = w1;
      }
    }
  }
  cp_wait<0>();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTcCols) : "memory");
  }
}

// ------------------------------------------------------------------ tcgen05 weight gradient
// gW[k][co][ci] = sum_i gz[i][co] x[i + d_k][ci], d_k = (dx, dy, dz), when L1
// is a multiple of 128.  Substituting j = i + dx e_x turns every x offset into
// a shift of gz: gW = sum_j x[j + (0, dy, dz)][ci] gz[j - dx e_x][co].  A tile
// is 128 consecutive sites j of one x-line; a CTA (at most 4 per SM, each with
// 128 tensor-memory columns) loops over tiles and accumulates in tensor
// memory:
//   A (M 128 = 8 (dy, dz) lines x 16 ci, K = 128 sites), MN-major: the 9 lines
//     of x staged as 18 channel planes of 128 rows (16 B each); M groups of 8
//     channels are one plane apart.  M = 128 covers lines 0-7; lines 1-8 form
//     the second accumulator, of which only line 8's 16 rows are used;
//   B (K = 128 sites, N 48 = 3 dx x 16 co), MN-major: gz staged three times,
//     shifted by -dx, as 6 channel planes of 128 rows;
//   2 accumulators x 48 FP32 columns, 8 K steps of 16 sites: 16 MMAs per tile.
// The partial sums of each CTA go to part[k][cta][co][ci] (bias: sum of gz)
// and are reduced in a fixed order by wgrad_sum_kernel.
constexpr int kTgRows = 128;                            // sites per tile
constexpr int kTgActBytes = 18 * kTgRows * 16;          // 9 lines x 2 planes
constexpr int kTgGzBytes = 6 * kTgRows * 16;            // 3 shifts x 2 planes
constexpr int kTgSmem = 52 * 1024;  // padded so that at most 4 CTAs (4 x 128 columns) share an SM
static_assert(kTgActBytes + kTgGzBytes + 16 + 16 + 8 * kC * 4 <= kTgSmem, "wgrad shared memory");
constexpr int kTgMaxCtasPerSm = 4;
// BF16 A and B, both MN-major, FP32 D, M 128, N 48
constexpr uint32_t kTgIdesc =
    (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) | ((48u >> 3) << 17) | ((128u >> 4) << 24);

__global__ void __launch_bounds__(128) wgrad_tc_kernel(const __nv_bfloat16* __restrict__ gz,
                                                       const __nv_bfloat16* __restrict__ x, float* __restrict__ part,
                                                       int nchunk, NetGeom g, unsigned* status) {
  extern __shared__ __align__(1024) uint8_t tg_sm[];
  uint8_t* act = tg_sm;
  uint8_t* gzs = tg_sm + kTgActBytes;
  uint64_t* mbar = reinterpret_cast<uint64_t*>(gzs + kTgGzBytes);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(mbar + 1);
  float* bred = reinterpret_cast<float*>(tslot + 4);  // [8][16]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int segs = g.L1 >> 7, ntiles = segs * g.L2 * g.L3;

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)), "r"(128)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(mbar)), "r"(1) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tslot;

  const uint4* x4 = reinterpret_cast<const uint4*>(x);
  const uint4* gz4 = reinterpret_cast<const uint4*>(gz);
  const int bco = tid & 15, brow = tid >> 4;  // bias: channel, row group
  float bsum = 0.f;
  uint32_t phase = 0;
  bool ok = true;
  int ndone = 0;
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const int x0 = (t % segs) << 7, y = (t / segs) % g.L2, z = (t / segs) / g.L2;
    // x: line (dy, dz) = seg, plane c, row r = site x0 + r
#pragma unroll
    for (int seg = 0; seg < 9; ++seg) {
      const int yy = wrap(y + seg / 3 - 1, g.L2), zz = wrap(z + seg % 3 - 1, g.L3);
      const int f = tc_flat(g, x0 + tid, yy, zz);
      cp16(reinterpret_cast<uint4*>(act) + (seg * 2) * kTgRows + tid, x4 + (size_t)f * 2);
      cp16(reinterpret_cast<uint4*>(act) + (seg * 2 + 1) * kTgRows + tid, x4 + (size_t)f * 2 + 1);
    }
    // gz: shift s = dx + 1, plane c, row r = site x0 + r - dx
#pragma unroll
    for (int sh = 0; sh < 3; ++sh) {
      const int f = tc_flat(g, wrap(x0 + tid - (sh - 1), g.L1), y, z);
      cp16(reinterpret_cast<uint4*>(gzs) + (sh * 2) * kTgRows + tid, gz4 + (size_t)f * 2);
      cp16(reinterpret_cast<uint4*>(gzs) + (sh * 2 + 1) * kTgRows + tid, gz4 + (size_t)f * 2 + 1);
    }
    cp_wait_all();
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (tid == 0) {
      const uint32_t a0 = smem_u32(act), b0 = smem_u32(gzs);
#pragma unroll 1
      for (int kk = 0; kk < kTgRows / 16; ++kk) {
        const uint64_t bd = tc_desc(b0 + kk * 16 * 16, 128, kTgRows * 16);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint64_t ad = tc_desc(a0 + ((2 * h) * kTgRows + kk * 16) * 16, 128, kTgRows * 16);
          const uint32_t acc = (ndone > 0 || kk > 0) ? 1u : 0u;
          asm volatile(
              "{\n\t.reg .pred p;\n\t"
              "setp.ne.b32 p, %4, 0;\n\t"
              "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
              ::"r"(tmem + (uint32_t)(h * 48)), "l"(ad), "l"(bd), "r"(kTgIdesc), "r"(acc)
              : "memory");
        }
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(mbar))
                   : "memory");
    }
    // bias gradient from the unshifted gz planes (generic reads beside the MMAs)
    {
      const __nv_bfloat16* p = reinterpret_cast<const __nv_bfloat16*>(gzs) + (size_t)(2 + (bco >> 3)) * kTgRows * 8;
#pragma unroll
      for (int j = 0; j < 16; ++j) bsum += __bfloat162float(p[(brow + 8 * j) * 8 + (bco & 7)]);
    }
    const uint32_t ph = phase;
    phase ^= 1u;
    const bool done = tc_wait(smem_u32(mbar), ph);
    ++ndone;
    if (__syncthreads_or(!done)) {
      // record the failure, give the MMAs a second bounded wait, then stop
      if (!done) {
        if (lane == 0) atomicOr(status, 1u);
        tc_wait(smem_u32(mbar), ph);
      }
      ok = false;
      break;
    }
  }
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

  // epilogue: warp w reads tensor-memory lanes 32w .. 32w+31 (M rows)
  const int m = warp * 32 + lane, ci = m & 15;
  const bool valid = ok && ndone > 0;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    if (h == 1 && warp != 3) continue;  // second accumulator: only line 8 (rows 112-127)
#pragma unroll
    for (int sh = 0; sh < 3; ++sh) {
      uint32_t v[16];
      asm volatile(
          "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
          "%15}, [%16];"
          : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
            "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
          : "r"(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(h * 48 + sh * 16)));
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      const int seg = h + (m >> 4);
      if (h == 0 || m >= 112) {
        const int k = sh * 9 + seg;
        float* d = part + ((size_t)k * nchunk + blockIdx.x) * kC * kC + ci;
#pragma unroll
        for (int co = 0; co < kC; ++co) d[co * kC] = valid ? __uint_as_float(v[co]) : 0.f;
      }
    }
  }
  bred[brow * kC + bco] = bsum;
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (tid < kC) {
    float b = 0.f;
#pragma unroll
    for (int q = 0; q < 8; ++q) b += bred[q * kC + tid];
    part[(size_t)kK * nchunk * kC * kC + (size_t)blockIdx.x * kC + tid] = valid ? b : 0.f;
  }
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(128) : "memory");
  }
}

// partial[k][chunk][co][ci] = sum over the chunk's sites of gz[i][co] x[nbr_k(i)][ci]
__global__ void __launch_bounds__(128) wgrad_kernel(const __nv_bfloat16* __restrict__ gz,
                                                    const __nv_bfloat16* __restrict__ x, float* __restrict__ part,
                                                    int nchunk, NetGeom g) {
  const int chunk = blockIdx.x, k = blockIdx.y;
  const int dx = k / 9 - 1, dy = (k / 3) % 3 - 1, dz = k % 3 - 1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, gr = lane >> 2, tq = lane & 3;
  const int nsites = 2 * g.nh;
  const __nv_bfloat16 zero = __float2bfloat16_rn(0.f);
  float acc[2][4] = {{0, 0, 0, 0}, {0, 0, 0, 0}};
  const int base = chunk * kChunk + warp * (kChunk / 4);
  for (int s0 = base; s0 < base + kChunk / 4 && s0 < nsites; s0 += 16) {
    const int sa = s0 + 2 * tq, sb = sa + 1, sc = sa + 8, sd = sa + 9;
    auto gzv = [&](int s, int co) { return s < nsites ? gz[(size_t)s * kC + co] : zero; };
    uint32_t a[4];
    a[0] = pack2(gzv(sa, gr), gzv(sb, gr));
    a[1] = pack2(gzv(sa, gr + 8), gzv(sb, gr + 8));
    a[2] = pack2(gzv(sc, gr), gzv(sd, gr));
    a[3] = pack2(gzv(sc, gr + 8), gzv(sd, gr + 8));
    const int na = sa < nsites ? nbr3(g, sa, dx, dy, dz) : -1, nb = sb < nsites ? nbr3(g, sb, dx, dy, dz) : -1;
    const int nc = sc < nsites ? nbr3(g, sc, dx, dy, dz) : -1, nd = sd < nsites ? nbr3(g, sd, dx, dy, dz) : -1;
    auto xv = [&](int n, int ci) { return n >= 0 ? x[(size_t)n * kC + ci] : zero; };
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int ci = 8 * j + gr;
      mma16816(acc[j], a, pack2(xv(na, ci), xv(nb, ci)), pack2(xv(nc, ci), xv(nd, ci)));
    }
  }
  __shared__ float red[4][kC * kC];
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    red[warp][gr * kC + 8 * j + 2 * tq] = acc[j][0];
    red[warp][gr * kC + 8 * j + 2 * tq + 1] = acc[j][1];
    red[warp][(gr + 8) * kC + 8 * j + 2 * tq] = acc[j][2];
    red[warp][(gr + 8) * kC + 8 * j + 2 * tq + 1] = acc[j][3];
  }
  if (k == 0) {
    // bias partial of the chunk: bpart[chunk][co] = sum_i gz[i][co]
    float b = 0.f;
    const int co = threadIdx.x & 15, grp = threadIdx.x >> 4;  // 8 groups
    for (int s = chunk * kChunk + grp; s < (chunk + 1) * kChunk && s < nsites; s += 8)
      b += __bfloat162float(gz[(size_t)s * kC + co]);
    __shared__ float bred[8][kC];
    bred[grp][co] = b;
    __syncthreads();
    if (threadIdx.x < kC) {
      float t = 0.f;
      for (int q = 0; q < 8; ++q) t += bred[q][threadIdx.x];
      part[(size_t)kK * nchunk * kC * kC + (size_t)chunk * kC + threadIdx.x] = t;
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < kC * kC; e += blockDim.x)
    part[((size_t)k * nchunk + chunk) * kC * kC + e] = red[0][e] + red[1][e] + red[2][e] + red[3][e];
}

// grad W[k][co][ci] = sum over chunks of part (blocks 0..26); grad b[co]
// (block 27) -- fixed summation order, so the gradient is deterministic.
// A round trip to L2 per batch of loads sets its time: 32 loads in flight
// before their in-order adds, one warp per block over the whole chip (17 us
// for 592 partials; 27 us with 28 blocks of 256 threads).
__device__ __forceinline__ float chunk_sum(const float* p, int stride, int nchunk) {
  constexpr int kBatch = 32;
  float s = 0.f;
  for (int c = 0; c < nchunk; c += kBatch) {
    float v[kBatch];
#pragma unroll
    for (int j = 0; j < kBatch; ++j) v[j] = c + j < nchunk ? __ldg(p + (size_t)(c + j) * stride) : 0.f;
#pragma unroll
    for (int j = 0; j < kBatch; ++j)
      if (c + j < nchunk) s += v[j];
  }
  return s;
}
__global__ void __launch_bounds__(32) wgrad_sum_kernel(const float* part, int nchunk, float* gW) {
  const int k = blockIdx.x, e = blockIdx.y * 32 + threadIdx.x;
  if (k < kK) {
    gW[(size_t)k * kC * kC + e] = chunk_sum(part + (size_t)k * nchunk * kC * kC + e, kC * kC, nchunk);
  } else if (e < kC) {
    gW[(size_t)kK * kC * kC + e] = chunk_sum(part + (size_t)kK * nchunk * kC * kC + e, kC, nchunk);
  }
}

// loss 1 - q . t per site, q = o/|o|; gz = dL/do = -(t - (q.t) q) / (|o| N).
// One 16-byte access per record (o: the first half of its 32 bytes, t; gz two):
// 23 us at 128^3, 51 us with 4-byte accesses.
__global__ void loss_kernel(const float* out, const float* target, int nsites, __nv_bfloat16* gz, double* part) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double l[1] = {0.0};
  if (i < nsites) {
    const float4 o4 = __ldg(reinterpret_cast<const float4*>(out) + 2 * (size_t)i);
    const float4 t4 = __ldg(reinterpret_cast<const float4*>(target) + i);
    const float o[4] = {o4.x, o4.y, o4.z, o4.w}, t[4] = {t4.x, t4.y, t4.z, t4.w};
    const float n = sqrtf(o[0] * o[0] + o[1] * o[1] + o[2] * o[2] + o[3] * o[3]) + 1e-12f;
    float q[4], qt = 0.f;
    for (int c = 0; c < 4; ++c) {
      q[c] = o[c] / n;
      qt += q[c] * t[c];
    }
    l[0] = 1.0 - qt;
    const float sc = -1.0f / (n * (float)nsites);
    uint4* g4 = reinterpret_cast<uint4*>(gz) + 2 * (size_t)i;
    g4[0] = make_uint4(pack2f(sc * (t[0] - qt * q[0]), sc * (t[1] - qt * q[1])),
                       pack2f(sc * (t[2] - qt * q[2]), sc * (t[3] - qt * q[3])), 0u, 0u);
    g4[1] = make_uint4(0u, 0u, 0u, 0u);
  }
  block_reduce_store<1>(l, part + blockIdx.x);
}

// W16 = bf16(W32), WT16[k'][ci][co] = bf16(W32[26-k'][co][ci]); output-layer
// rows co >= kOut and their biases are kept at zero
__global__ void refresh_kernel(float* w32, __nv_bfloat16* w16, __nv_bfloat16* wt16) {
  const int l = blockIdx.x;
  float* W = w32 + (size_t)l * kPl;
  for (int e = blockIdx.y * blockDim.x + threadIdx.x; e < kWl; e += gridDim.y * blockDim.x) {
    const int k = e / (kC * kC), co = (e / kC) % kC, ci = e % kC;
    if (l == kLayers - 1 && co >= kOut) W[e] = 0.f;
    w16[(size_t)l * kWl + e] = __float2bfloat16_rn(W[e]);
    wt16[(size_t)l * kWl + ((size_t)(kK - 1 - k) * kC + ci) * kC + co] = __float2bfloat16_rn(W[e]);
  }
  if (blockIdx.y == 0 && l == kLayers - 1 && threadIdx.x >= kOut && threadIdx.x < kC) W[kWl + threadIdx.x] = 0.f;
}

__global__ void adam_kernel(float* w, float* m, float* v, const float* grad, int n, float lr, float b1, float b2,
                            float eps, float c1, float c2) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float gi = grad[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi, vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    w[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  }
}

// features: 12 link components of U_f and 3 of A_f per site (channel 15 = 0)
template <typename R>
__global__ void features_kernel(const ChainDev* chp, __nv_bfloat16* feat) {
  const ChainDev& ch = *chp;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 2 * ch.nh) return;
  const int eo = i >= ch.nh ? 1 : 0, s = i - eo * ch.nh, nh = ch.nh;
  float f[kC];
#pragma unroll
  for (int mu = 0; mu < 3; ++mu) {
    const su2<R> u = LinkIO<R>::ld(ch.uf, ((size_t)(mu * 2 + eo)) * nh + s);
    f[4 * mu + 0] = (float)u.a.re;
    f[4 * mu + 1] = (float)u.a.im;
    f[4 * mu + 2] = (float)u.b.re;
    f[4 * mu + 3] = (float)u.b.im;
  }
  const R* Af = reinterpret_cast<const R*>(ch.af);
#pragma unroll
  for (int k = 0; k < 3; ++k) f[12 + k] = (float)Af[((size_t)(eo * 3 + k)) * nh + s];
  f[15] = 0.f;
  uint32_t* o = reinterpret_cast<uint32_t*>(feat) + (size_t)i * 8;
#pragma unroll
  for (int w = 0; w < 8; ++w) o[w] = pack2(__float2bfloat16_rn(f[2 * w]), __float2bfloat16_rn(f[2 * w + 1]));
}

// G(x) = (o/|o|) G_prev(x) with o the network output as a first row
template <typename R>
__global__ void compose_kernel(const float* out, const void* gprev, void* g, int nsites) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nsites) return;
  const float* o = out + (size_t)i * 8;
  const float n = rsqrtf(o[0] * o[0] + o[1] * o[1] + o[2] * o[2] + o[3] * o[3] + 1e-30f);
  const su2<R> om{{(R)(o[0] * n), (R)(o[1] * n)}, {(R)(o[2] * n), (R)(o[3] * n)}};
  LinkIO<R>::st(g, i, unitarise64(nn(om, LinkIO<R>::ld(gprev, i))));
}

// T(x) = G_new(x) G_prev(x)^+ as a quaternion target
template <typename R>
__global__ void target_kernel(const void* gnew, const void* gprev, float* t, int nsites) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nsites) return;
  const su2<R> r = nd(LinkIO<R>::ld(gnew, i), LinkIO<R>::ld(gprev, i));
  t[(size_t)i * 4 + 0] = (float)r.a.re;
  t[(size_t)i * 4 + 1] = (float)r.a.im;
  t[(size_t)i * 4 + 2] = (float)r.b.re;
  t[(size_t)i * 4 + 3] = (float)r.b.im;
}

__global__ void init_params_kernel(float* w, uint32_t k0, uint32_t k1) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kNParam; i += gridDim.x * blockDim.x) {
    const int l = i / kPl, e = i % kPl;
    uint32_t c[4] = {(uint32_t)i, 0x4e4554u, 0u, 0u};
    philox4x32_10(c, k0, k1);
    const float u1 = u01(c[0]), u2 = u01(c[1]);
    const float gauss = sqrtf(-2.f * logf(u1)) * cospif(2.f * u2);
    float v;
    if (e >= kWl) v = (l == kLayers - 1 && e - kWl == 0) ? 1.f : 0.f;       // output bias: identity
    else if (l == kLayers - 1) v = 0.f;  // output = bias: the untrained network predicts Omega = 1
    else v = gauss * sqrtf(2.f / (kK * kC));                                   // He
    w[i] = v;
  }
}

NetGeom make_geom(int L1, int L2, int L3) {
  NetGeom g;
  g.L1 = L1;
  g.L2 = L2;
  g.L3 = L3;
  g.hx = L1 / 2;
  g.nxy = L1 * L2 / 2;
  g.nh = g.nxy * L3;
  g.dhx = make_fastdiv((uint32_t)g.hx);
  g.dnxy = make_fastdiv((uint32_t)g.nxy);
  return g;
}

}  // namespace
}  // namespace lce

using namespace lce;

struct lce_net {
  int device = 0;
  cudaStream_t stream = nullptr;
  float *w32 = nullptr, *m = nullptr, *v = nullptr, *grad = nullptr;
  __nv_bfloat16 *w16 = nullptr, *wt16 = nullptr;
  int step = 0;
  // work buffers for the current volume
  long nsites = 0;
  __nv_bfloat16* act[kLayers] = {nullptr, nullptr, nullptr, nullptr};
  __nv_bfloat16 *gz = nullptr, *gy = nullptr;
  float* out = nullptr;
  float* target = nullptr;
  double* part = nullptr;
  float* wpart = nullptr;
  int nchunk = 0;
  int tg_grid = 0;   // CTAs of the tcgen05 weight gradient
  unsigned* flag = nullptr;  // set on the device when a tensor-core wait gave up
  // recorded training pairs
  struct Pair {
    NetGeom g;
    __nv_bfloat16* feat;
    float* target;
  };
  std::vector<Pair> pairs;
  std::string err;
};

namespace {

int net_fail(lce_net* n, int code, const std::string& m) {
  if (n) n->err = m;
  set_thread_error(m);
  return code;
}
#define NCK(call)                                                                         \
  do {                                                                                    \
    cudaError_t e_ = (call);                                                              \
    if (e_ != cudaSuccess) return net_fail(n, LCE_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
  } while (0)

// CTAs of the tcgen05 weight gradient: 4 per SM, all resident (4 x 53 KB of
// shared memory; tensor memory: 4 x 128 columns).  The runtime's occupancy
// query reported 1 per SM for this kernel where the launch itself holds 4.
static_assert(kTgMaxCtasPerSm * (kTgSmem + 1024) <= 228 * 1024, "wgrad CTAs per SM");
template <typename K>
void tc_attributes(K kernel, int smem) {
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  // all of the unified L1 / shared memory as shared memory
  cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
}

// the grid of the persistent tcgen05 kernels; the first call for a network
// (on its device) also sets their shared-memory attributes there
int wgrad_tc_grid(lce_net* n) {
  if (n->tg_grid > 0) return n->tg_grid;
  int nsm = 0;
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, n->device);
  tc_attributes(wgrad_tc_kernel, kTgSmem);
  tc_attributes(conv_tc_kernel<0>, kTcSmem);
  tc_attributes(conv_tc_kernel<1>, kTcSmem);
  tc_attributes(conv_tc_kernel<2>, kTcSmem);
  n->tg_grid = std::max(1, nsm) * kTgMaxCtasPerSm;
  return n->tg_grid;
}

int net_buffers(lce_net* n, long nsites) {
  if (n->nsites == nsites) return LCE_OK;
  // the buffers may still be in use by work queued on a context's stream
  NCK(cudaDeviceSynchronize());
  n->nsites = 0;
  for (auto& a : n->act) {
    if (a) cudaFree(a);
    a = nullptr;
  }
  void* ptrs[] = {n->gz, n->gy, n->out, n->target, n->part, n->wpart};
  for (void* q : ptrs)
    if (q) cudaFree(q);
  n->gz = n->gy = nullptr;
  n->out = n->target = nullptr;
  n->part = nullptr;
  n->wpart = nullptr;
  for (auto& a : n->act) NCK(cudaMalloc(&a, (size_t)nsites * kC * sizeof(__nv_bfloat16)));
  NCK(cudaMalloc(&n->gz, (size_t)nsites * kC * sizeof(__nv_bfloat16)));
  NCK(cudaMalloc(&n->gy, (size_t)nsites * kC * sizeof(__nv_bfloat16)));
  NCK(cudaMalloc(&n->out, (size_t)nsites * 8 * sizeof(float)));
  NCK(cudaMalloc(&n->target, (size_t)nsites * 4 * sizeof(float)));
  NCK(cudaMalloc(&n->part, (size_t)ceil_div(nsites, 256) * sizeof(double) + 64));
  n->nchunk = ceil_div(nsites, kChunk);
  // partial sums of the mma.sync (per chunk) or the tcgen05 (per CTA) weight gradient
  const size_t nparts = std::max(n->nchunk, wgrad_tc_grid(n));
  NCK(cudaMalloc(&n->wpart, ((size_t)kK * nparts * kC * kC + nparts * kC) * sizeof(float)));
  n->nsites = nsites;
  return LCE_OK;
}

int conv_grid(long nsites) {
  const int ntiles = ceil_div(nsites, 16);
  return std::max(1, std::min(ceil_div(ntiles, kConvWarps), 148 * 8));
}

// forward through all layers from x (act[0], or a recorded pair's features); output in n->out
// one convolution: the tcgen05 kernel when L1 is a multiple of 128, else the
// mma.sync kernel
template <int MODE>
void launch_conv(lce_net* n, const __nv_bfloat16* in, const __nv_bfloat16* W, const float* bias,
                 __nv_bfloat16* out16, float* out32, const __nv_bfloat16* mask, const NetGeom& g, cudaStream_t s) {
  if (g.L1 % 128 == 0) {
    // persistent CTAs, kTcCtasPerSm per SM
    const int grid = std::min(wgrad_tc_grid(n) / kTgMaxCtasPerSm * kTcCtasPerSm, (g.L1 / 128) * g.L2 * g.L3);
    conv_tc_kernel<MODE><<<grid, kTcThreads, kTcSmem, s>>>(in, W, bias, out16, out32, mask, g, n->flag);
  } else {
    conv_kernel<MODE><<<conv_grid(2L * g.nh), 32 * kConvWarps, 0, s>>>(in, W, bias, out16, out32, mask, g);
  }
}

void net_forward(lce_net* n, const __nv_bfloat16* x, const NetGeom& g, cudaStream_t s) {
  for (int l = 0; l < kLayers; ++l) {
    const __nv_bfloat16* W = n->w16 + (size_t)l * kWl;
    const float* b = n->w32 + (size_t)l * kPl + kWl;
    const __nv_bfloat16* in = l ? n->act[l] : x;
    if (l < kLayers - 1) launch_conv<0>(n, in, W, b, n->act[l + 1], nullptr, nullptr, g, s);
    else launch_conv<1>(n, in, W, b, nullptr, n->out, nullptr, g, s);
  }
}

// loss and gradients (into n->grad) for the input x and the target t; returns
// the loss through part (device) -- caller sums
void net_backward(lce_net* n, const __nv_bfloat16* x, const float* t, const NetGeom& g, cudaStream_t s) {
  const long ns = 2L * g.nh;
  loss_kernel<<<ceil_div(ns, 256), 256, 0, s>>>(n->out, t, (int)ns, n->gz, n->part);
  __nv_bfloat16* gz = n->gz;   // gradient at the output of layer l (pre-activation)
  __nv_bfloat16* gy = n->gy;
  for (int l = kLayers - 1; l >= 0; --l) {
    float* gW = n->grad + (size_t)l * kPl;
    const __nv_bfloat16* in = l ? n->act[l] : x;
    if (g.L1 % 128 == 0) {
      const int grid = std::min(wgrad_tc_grid(n), (g.L1 / 128) * g.L2 * g.L3);
      wgrad_tc_kernel<<<grid, 128, kTgSmem, s>>>(gz, in, n->wpart, grid, g, n->flag);
      wgrad_sum_kernel<<<dim3(kK + 1, kC * kC / 32), 32, 0, s>>>(n->wpart, grid, gW);
    } else {
      wgrad_kernel<<<dim3(n->nchunk, kK), 128, 0, s>>>(gz, in, n->wpart, n->nchunk, g);
      wgrad_sum_kernel<<<dim3(kK + 1, kC * kC / 32), 32, 0, s>>>(n->wpart, n->nchunk, gW);
    }
    if (l > 0) {
      // gradient w.r.t. act[l] = conv_T(gz, W_l), times relu'(layer l-1) = (act[l] > 0)
      launch_conv<2>(n, gz, n->wt16 + (size_t)l * kWl, nullptr, gy, nullptr, n->act[l], g, s);
      std::swap(gz, gy);
    }
  }
}

void net_refresh(lce_net* n, cudaStream_t s) { refresh_kernel<<<dim3(kLayers, kWl / 256), 256, 0, s>>>(n->w32, n->w16, n->wt16); }

}  // namespace

// the device flag of the tensor-core kernels (a wait that gave up), read and
// cleared; the work of the network's stream and of the caller's stream must
// have completed
int lce::net_status(lce_net* n) {
  unsigned f = 0;
  NCK(cudaMemcpy(&f, n->flag, sizeof(f), cudaMemcpyDeviceToHost));
  if (!f) return LCE_OK;
  NCK(cudaMemset(n->flag, 0, sizeof(unsigned)));
  return net_fail(n, LCE_ERR_CUDA, "warm-start network: a tensor-core completion wait timed out");
}

namespace {

}  // namespace

extern "C" {

lce_net* lce_net_create(int device, unsigned long long seed) {
  DeviceScope ds_(device);
  lce_net* n = new lce_net();
  n->device = device;
  auto bad = [&](cudaError_t e, const char* w) -> lce_net* {
    set_thread_error(std::string("lce_net_create: ") + w + ": " + cudaGetErrorString(e));
    lce_net_destroy(n);
    return nullptr;
  };
  cudaError_t e;
  if ((e = cudaSetDevice(device)) != cudaSuccess) return bad(e, "cudaSetDevice");
  if ((e = cudaStreamCreateWithFlags(&n->stream, cudaStreamNonBlocking)) != cudaSuccess) return bad(e, "stream");
  if ((e = cudaMalloc(&n->w32, sizeof(float) * kNParam)) != cudaSuccess) return bad(e, "cudaMalloc");
  if ((e = cudaMalloc(&n->m, sizeof(float) * kNParam)) != cudaSuccess) return bad(e, "cudaMalloc");
  if ((e = cudaMalloc(&n->v, sizeof(float) * kNParam)) != cudaSuccess) return bad(e, "cudaMalloc");
  if ((e = cudaMalloc(&n->grad, sizeof(float) * kNParam)) != cudaSuccess) return bad(e, "cudaMalloc");
  if ((e = cudaMalloc(&n->w16, sizeof(__nv_bfloat16) * kLayers * kWl)) != cudaSuccess) return bad(e, "cudaMalloc");
  if ((e = cudaMalloc(&n->wt16, sizeof(__nv_bfloat16) * kLayers * kWl)) != cudaSuccess) return bad(e, "cudaMalloc");
  if ((e = cudaMalloc(&n->flag, sizeof(unsigned))) != cudaSuccess) return bad(e, "cudaMalloc");
  cudaMemsetAsync(n->flag, 0, sizeof(unsigned), n->stream);
  cudaMemsetAsync(n->m, 0, sizeof(float) * kNParam, n->stream);
  cudaMemsetAsync(n->v, 0, sizeof(float) * kNParam, n->stream);
  init_params_kernel<<<64, 256, 0, n->stream>>>(n->w32, (uint32_t)seed, (uint32_t)(seed >> 32));
  net_refresh(n, n->stream);
  if ((e = cudaStreamSynchronize(n->stream)) != cudaSuccess) return bad(e, "init");
  return n;
}

void lce_net_destroy(lce_net* n) {
  DeviceScope ds_(n ? n->device : -1);
  if (!n) return;
  cudaSetDevice(n->device);
  if (n->stream) cudaStreamSynchronize(n->stream);
  for (auto& p : n->pairs) {
    cudaFree(p.feat);
    cudaFree(p.target);
  }
  for (auto& a : n->act)
    if (a) cudaFree(a);
  void* ptrs[] = {n->w32, n->m, n->v, n->grad, n->w16, n->wt16, n->gz, n->gy, n->out, n->target, n->part, n->wpart,
                  n->flag};
  for (void* q : ptrs)
    if (q) cudaFree(q);
  if (n->stream) cudaStreamDestroy(n->stream);
  delete n;
}

int lce_net_num_params(lce_net* n) { return n ? kNParam : LCE_ERR_INVALID; }

int lce_net_get_params(lce_net* n, float* w) {
  DeviceScope ds_(n ? n->device : -1);
  if (!n || !w) return LCE_ERR_INVALID;
  NCK(cudaMemcpyAsync(w, n->w32, sizeof(float) * kNParam, cudaMemcpyDeviceToHost, n->stream));
  NCK(cudaStreamSynchronize(n->stream));
  return LCE_OK;
}

int lce_net_set_params(lce_net* n, const float* w) {
  DeviceScope ds_(n ? n->device : -1);
  if (!n || !w) return LCE_ERR_INVALID;
  NCK(cudaMemcpyAsync(n->w32, w, sizeof(float) * kNParam, cudaMemcpyHostToDevice, n->stream));
  net_refresh(n, n->stream);
  NCK(cudaStreamSynchronize(n->stream));
  return LCE_OK;
}

int lce_net_save(lce_net* n, const char* path) {
  DeviceScope ds_(n ? n->device : -1);
  std::vector<float> w(kNParam);
  int rc = lce_net_get_params(n, w.data());
  if (rc) return rc;
  FILE* f = std::fopen(path, "wb");
  if (!f) return net_fail(n, LCE_ERR_INVALID, std::string("lce_net_save: cannot open ") + path);
  const char magic[8] = {'L', 'C', 'E', 'N', 'E', 'T', '0', '1'};
  bool ok = std::fwrite(magic, 1, 8, f) == 8 && std::fwrite(w.data(), sizeof(float), w.size(), f) == w.size();
  ok = std::fclose(f) == 0 && ok;
  return ok ? LCE_OK : net_fail(n, LCE_ERR_INVALID, "lce_net_save: write failed");
}

int lce_net_load(lce_net* n, const char* path) {
  DeviceScope ds_(n ? n->device : -1);
  if (!n || !path) return LCE_ERR_INVALID;
  FILE* f = std::fopen(path, "rb");
  if (!f) return net_fail(n, LCE_ERR_INVALID, std::string("lce_net_load: cannot open ") + path);
  char magic[8];
  std::vector<float> w(kNParam);
  bool ok = std::fread(magic, 1, 8, f) == 8 && std::memcmp(magic, "LCENET01", 8) == 0 &&
            std::fread(w.data(), sizeof(float), w.size(), f) == w.size();
  std::fclose(f);
  if (!ok) return net_fail(n, LCE_ERR_INVALID, "lce_net_load: not a network file of this format");
  return lce_net_set_params(n, w.data());
}

// forward, loss and gradients on caller data (no update): feat [2][nh][16]
// float (rounded to BF16 here), target [2][nh][4]; out [2][nh][4] and grad
// [nparam] may be NULL
int lce_net_eval(lce_net* n, int L1, int L2, int L3, const float* feat, const float* target, float* out, float* grad,
                 double* loss) {
  DeviceScope ds_(n ? n->device : -1);
  if (!n || !feat || !target || L1 < 2 || L2 < 2 || L3 < 2 || ((L1 | L2 | L3) & 1)) return LCE_ERR_INVALID;
  const NetGeom g = make_geom(L1, L2, L3);
  const long ns = 2L * g.nh;
  int rc = net_buffers(n, ns);
  if (rc) return rc;
  std::vector<uint16_t> fb((size_t)ns * kC);
  for (size_t i = 0; i < fb.size(); ++i) fb[i] = __bfloat16_as_ushort(__float2bfloat16_rn(feat[i]));
  NCK(cudaMemcpyAsync(n->act[0], fb.data(), fb.size() * 2, cudaMemcpyHostToDevice, n->stream));
  NCK(cudaMemcpyAsync(n->target, target, sizeof(float) * ns * 4, cudaMemcpyHostToDevice, n->stream));
  net_forward(n, n->act[0], g, n->stream);
  net_backward(n, n->act[0], n->target, g, n->stream);
  NCK(cudaGetLastError());
  std::vector<double> lp(ceil_div(ns, 256));
  NCK(cudaMemcpyAsync(lp.data(), n->part, lp.size() * sizeof(double), cudaMemcpyDeviceToHost, n->stream));
  if (out) {
    std::vector<float> o((size_t)ns * 8);
    NCK(cudaMemcpyAsync(o.data(), n->out, o.size() * sizeof(float), cudaMemcpyDeviceToHost, n->stream));
    NCK(cudaStreamSynchronize(n->stream));
    for (long i = 0; i < ns; ++i)
      for (int c = 0; c < 4; ++c) out[i * 4 + c] = o[(size_t)i * 8 + c];
  }
  if (grad) NCK(cudaMemcpyAsync(grad, n->grad, sizeof(float) * kNParam, cudaMemcpyDeviceToHost, n->stream));
  NCK(cudaStreamSynchronize(n->stream));
  double l = 0;
  for (double x : lp) l += x;
  if (loss) *loss = l / ns;
  if (int rc = lce::net_status(n)) return rc;
  return LCE_OK;
}

int lce_net_num_pairs(lce_net* n) { return n ? (int)n->pairs.size() : LCE_ERR_INVALID; }

int lce_net_clear_pairs(lce_net* n) {
  DeviceScope ds_(n ? n->device : -1);
  if (!n) return LCE_ERR_INVALID;
  NCK(cudaStreamSynchronize(n->stream));
  for (auto& p : n->pairs) {
    cudaFree(p.feat);
    cudaFree(p.target);
  }
  n->pairs.clear();
  return LCE_OK;
}

// Adam over the recorded pairs, `epochs` passes in an order shuffled per epoch
int lce_net_train(lce_net* n, int epochs, double lr, double* mean_loss) {
  DeviceScope ds_(n ? n->device : -1);
  if (!n || epochs < 0 || n->pairs.empty()) return LCE_ERR_INVALID;
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  std::vector<int> order(n->pairs.size());
  for (size_t i = 0; i < order.size(); ++i) order[i] = (int)i;
  uint32_t rs = 0x12345u;
  double last_epoch = 0.0;
  for (int ep = 0; ep < epochs; ++ep) {
    for (size_t i = order.size(); i > 1; --i) {
      rs = rs * 1664525u + 1013904223u;
      std::swap(order[i - 1], order[rs % i]);
    }
    double tot = 0.0;
    for (int idx : order) {
      const auto& p = n->pairs[idx];
      const long ns = 2L * p.g.nh;
      int rc = net_buffers(n, ns);
      if (rc) return rc;
      net_forward(n, p.feat, p.g, n->stream);
      net_backward(n, p.feat, p.target, p.g, n->stream);
      ++n->step;
      const float c1 = 1.f - std::pow(b1, (float)n->step), c2 = 1.f - std::pow(b2, (float)n->step);
      adam_kernel<<<64, 256, 0, n->stream>>>(n->w32, n->m, n->v, n->grad, kNParam, (float)lr, b1, b2, eps, c1, c2);
      net_refresh(n, n->stream);
      NCK(cudaGetLastError());
      std::vector<double> lp(ceil_div(ns, 256));
      NCK(cudaMemcpyAsync(lp.data(), n->part, lp.size() * sizeof(double), cudaMemcpyDeviceToHost, n->stream));
      NCK(cudaStreamSynchronize(n->stream));
      double l = 0;
      for (double x : lp) l += x;
      tot += l / ns;
    }
    last_epoch = tot / order.size();
  }
  if (mean_loss) *mean_loss = last_epoch;
  if (int rc = lce::net_status(n)) return rc;
  return LCE_OK;
}

}  // extern "C"

// ---- used by the gauge-fixing warm start in lce_capi.cu
namespace lce {

int net_features(lce_net* n, const ChainDev* chd, const ChainDev& ch, bool f64, cudaStream_t s) {
  const long ns = 2L * ch.nh;
  int rc = net_buffers(n, ns);
  if (rc) return rc;
  if (f64) features_kernel<double><<<ceil_div(ns, 256), 256, 0, s>>>(chd, n->act[0]);
  else features_kernel<float><<<ceil_div(ns, 256), 256, 0, s>>>(chd, n->act[0]);
  return cudaGetLastError() == cudaSuccess ? LCE_OK : LCE_ERR_CUDA;
}

void net_predict(lce_net* n, const ChainDev& ch, cudaStream_t s) {
  net_forward(n, n->act[0], make_geom(ch.L1, ch.L2, ch.L3), s);
}

// ch.g = Omega G_prev from the last net_predict
int net_compose(lce_net* n, const ChainDev& ch, const void* gprev, bool f64, cudaStream_t s) {
  const long ns = 2L * ch.nh;
  if (f64) compose_kernel<double><<<ceil_div(ns, 256), 256, 0, s>>>(n->out, gprev, ch.g, (int)ns);
  else compose_kernel<float><<<ceil_div(ns, 256), 256, 0, s>>>(n->out, gprev, ch.g, (int)ns);
  return cudaGetLastError() == cudaSuccess ? LCE_OK : LCE_ERR_CUDA;
}

int net_device(lce_net* n) { return n->device; }

// store (current features, T = G_new G_prev^+) as a training pair
int net_record(lce_net* n, const ChainDev& ch, const void* gprev, bool f64, cudaStream_t s) {
  const long ns = 2L * ch.nh;
  lce_net::Pair p;
  p.g = make_geom(ch.L1, ch.L2, ch.L3);
  if (cudaMalloc(&p.feat, (size_t)ns * kC * 2) != cudaSuccess) return LCE_ERR_NOMEM;
  if (cudaMalloc(&p.target, (size_t)ns * 16) != cudaSuccess) {
    cudaFree(p.feat);
    return LCE_ERR_NOMEM;
  }
  cudaMemcpyAsync(p.feat, n->act[0], (size_t)ns * kC * 2, cudaMemcpyDeviceToDevice, s);
  if (f64) target_kernel<double><<<ceil_div(ns, 256), 256, 0, s>>>(ch.g, gprev, p.target, (int)ns);
  else target_kernel<float><<<ceil_div(ns, 256), 256, 0, s>>>(ch.g, gprev, p.target, (int)ns);
  if (cudaGetLastError() != cudaSuccess) return LCE_ERR_CUDA;
  n->pairs.push_back(p);
  return LCE_OK;
}

}  // namespace lce
