// The learned 3D CNN on the tensor cores: implicit-GEMM convolution with
// tcgen05 (BF16 operands in shared memory, FP32 accumulators in tensor
// memory), weight gradients, loss, Adam and the C ABI of include/msbg_cnn.h.
// No counterpart in the reference.
//
// Convolution as an implicit GEMM.  A layer's input is up to 18 padded z planes
// of two channel halves, each an [y][x] array of 18^2 cells x 16 bytes (8 bf16
// channels), in shared memory.  An M = 128 block of output cells is 8
// consecutive x by the 16 y rows of one z plane; its A operand for the
// in-plane tap (ky, kx) is the input plane read from a start address shifted by
// the tap: 8 rows (x) of 16 bytes form a core matrix, the 16 y rows are
// core-matrix groups 18 cells apart (SBO) and the two channel halves are the
// two K halves (LBO).  An input plane contributes to three output planes, one
// per kz: their accumulators sit side by side in tensor memory, so one
// tcgen05.mma of M = 128, N = 48 (3 planes x 16 channels), K = 16 serves the
// three kz of a tap straight from the activations, with no im2col copy.
//
// Backward: the data gradient of a "same" convolution is a "same"
// convolution of the output gradient with the flipped, transposed kernel, so
// it runs through the same kernel (weight image `bwd`) with the ReLU mask of
// the layer input applied in the epilogue.  The weight gradient, a
// 432 x 16 result reduced over all cells, has no 64-row operand for tcgen05; it runs on
// warp-level mma.sync with per-CTA partials reduced in a fixed order (deterministic).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstring>
#include <random>
#include <string>
#include <type_traits>
#include <vector>

#include "cnn.cuh"
#include "cnn_tc.cuh"
#include "common.cuh"
#include "msbg_cnn.h"

namespace msbg {
namespace cnn {

// ---------------------------------------------------------------------------
// weight images
// ---------------------------------------------------------------------------
// One B operand (N x K, K-major, no swizzle) per in-plane tap q = 3 ky + kx: its
// 48 rows are the 16 channels n of kz = 2, 1, 0 (the order of the output planes
// an input plane reaches).  Image element (q, kz, n, k):
// q*768 + (k>>3)*384 + ((2-kz)*16 + n)*8 + (k&7).  Forward: n = cout, k = cin,
// W[n][k][tap].  Backward-data: n = cin, k = cout, W[k][n][26 - tap].  Unused
// rows/columns (cin = 4 of layer 1, cout = 1 of layer 4) are zero.
__global__ void k_pack(const float* __restrict__ w, __nv_bfloat16* __restrict__ fwd,
                       __nv_bfloat16* __restrict__ bwd) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= NLAYER * WIMG) return;
  const int l = i / WIMG, e = i % WIMG;
  const int r = e % 768, row = (r % 384) / 8, n = row % 16, k = (r / 384) * 8 + (r % 8);
  const int tap = (2 - row / 16) * 9 + e / 768;
  const int cin = layer_cin(l), cout = layer_cout(l);
  const float* W = w + layer_off(l);
  float f = 0.f, b = 0.f;
  if (n < cout && k < cin) f = W[((size_t)n * cin + k) * 27 + tap];
  if (n < cin && k < cout) b = W[((size_t)k * cin + n) * 27 + (26 - tap)];
  fwd[i] = __float2bfloat16_rn(f);
  bwd[i] = __float2bfloat16_rn(b);
}

__device__ __forceinline__ uint32_t pack_bf2(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}

// ---------------------------------------------------------------------------
// convolution (tcgen05)
// ---------------------------------------------------------------------------
// A chain of up to 4 layers per tile, one CTA per SM walking its tiles; the
// activations of the layers in between never leave the SM.
//   * An input plane is read by MMAs once, for all three output planes that it
//     reaches, so output plane z takes the place of input plane z in `act` (16
//     planes, halo cells zero; the zero planes beyond both ends are not multiplied).
//     The first layer's planes have halos of their own and arrive in a ring.
//   * Warps 17-20 fill the ring, plane by plane: FP32 features packed to bf16, or
//     a bf16 gradient.  Channels 8-15 of either are zero: one zero plane stands
//     for that half of every ring plane.
//   * Warp 16 issues the MMAs, per plane 10 for each x half (tap 0 in two parts,
//     since it starts an output plane while it adds to two others), and the copies
//     of the weight images, one layer ahead.  The accumulators of the 16 output
//     planes x 2 x halves take the whole tensor memory (512 columns).
//   * Warps 0-7 drain the even planes z, 8-15 the odd ones, once input plane z + 1
//     is done: warp w reads TMEM lanes 32*(w%4).. of x half w/4 % 2, applies the
//     epilogue and writes the cells.  (8 warps for all planes took longer per
//     plane than its MMAs: 60 us per tile.)
// A tcgen05.mma of this shape costs about 45 cycles for every N <= 64 (measured; the
// A operand's 4 KB alone are 32 cycles of shared-memory reads), so the 27 taps cost
// 10 instead of 27 instructions per plane and x half, with the products added in
// the same order (kz, ky, kx): the same bits.  That bounds a tile to 30 us for 4
// layers; measured 50 us.  Forward pass of 4096 tiles on a B200: 3.40 ms with a launch
// per layer, N = 16 and the activations through global memory, 1.39 ms now.  (An MMA
// issued by a divergent thread costs over 100 cycles, its operands moving to uniform
// registers one by one: 2.43 ms.)  Every wait is bounded.
__global__ void __launch_bounds__(CONV_THREADS, 1) k_conv3_tc(const __grid_constant__ ConvChain a) {
  extern __shared__ __align__(1024) uint8_t sm[];
  uint8_t* act = sm;                                   // [TS] planes of both halves
  uint8_t* wts = act + TS * 2 * PLANE_BYTES;           // [2] weight images
  uint8_t* ring = wts + 2 * WIMG * 2;                  // [CONV_SLOTS] planes of half 0, a zero plane
  uint64_t* done = reinterpret_cast<uint64_t*>(ring + (CONV_SLOTS + 1) * PLANE_BYTES);
  // done[PD]: the plane's MMAs are complete (each used one once per pass); stored[TS]:
  // output plane drained, and in act; full, taken [CONV_SLOTS]: ring; wfull[2]
  uint64_t* stored = done + PD;
  uint64_t* full = stored + TS;
  uint64_t* taken = full + CONV_SLOTS;
  uint64_t* wfull = taken + CONV_SLOTS;
  uint32_t* tslot = reinterpret_cast<uint32_t*>(wfull + 2);
  volatile int* abort = reinterpret_cast<volatile int*>(tslot + 1);
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // uniform
  const int G = gridDim.x;
  if ((int)blockIdx.x >= a.n) return;

  for (int i = tid; i < (int)(TS * 2 * PLANE_BYTES / 16); i += CONV_THREADS)
    reinterpret_cast<uint4*>(act)[i] = make_uint4(0, 0, 0, 0);
  for (int i = tid; i < PLANE; i += CONV_THREADS)
    reinterpret_cast<uint4*>(ring + CONV_SLOTS * PLANE_BYTES)[i] = make_uint4(0, 0, 0, 0);
  if (tid == 0) {
    for (int b = 0; b < PD; b++) mbar_init(&done[b], 1);
    for (int b = 0; b < TS; b++) mbar_init(&stored[b], 8);
    for (int b = 0; b < 2 * CONV_SLOTS + 2; b++) mbar_init(&full[b], 1);
    fence_mbar_init();
    *abort = 0;
  }
  if (warp == 0) {
    tmem_alloc(tslot, 512);
    tmem_relinquish();
  }
  fence_proxy_async();  // the zeros (generic writes) -> tensor core
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = *tslot;
  const int nTiles = (a.n - (int)blockIdx.x + G - 1) / G;
  const int passes = nTiles * a.nl;  // pass p: layer p % nl of this CTA's tile p / nl

  if (warp == EPI_WARPS) {
    // the whole warp runs this loop on uniform values (an MMA takes its operands
    // from uniform registers); one lane issues
    const uint32_t zero = smem_addr(ring) + CONV_SLOTS * PLANE_BYTES;
    const uint64_t a0 = smem_desc(smem_addr(act), PLANE_BYTES, PD * 16);
    const uint64_t b0 = smem_desc(smem_addr(wts), 768, 128);
    auto wait = [&](uint64_t* b, uint32_t parity) -> bool {
      return __all_sync(0xffffffffu, mbar_wait_abort(b, parity, abort));
    };
    auto load_weights = [&](int p, int l) {
      if (elect_one()) {
        mbar_expect_tx(&wfull[p & 1], WIMG * 2);
        bulk_g2s(wts + (p & 1) * (WIMG * 2), a.L[l].wimg, WIMG * 2, &wfull[p & 1]);
      }
    };
    int wl = 0, wlL = 0;  // weight images asked for, the next one's layer
    for (; wl < 2 && wl < passes; wl++) {
      load_weights(wl, wlL);
      wlL = wlL + 1 == a.nl ? 0 : wlL + 1;
    }
    int slot = 0;          // ring plane
    uint32_t slotPar = 0;  // and the parity of its fill
    // what plane zi of pass p (layer l) waits for: its weights and its input, and
    // that the last pass has drained the accumulators of the output plane that it
    // starts (stored implies drained; input plane zi >= 1 of a later layer is
    // stored[zi - 1], waited for one plane before)
    auto ready = [&](int p, int l, int zi) -> bool {
      const uint32_t before = (uint32_t)((p - 1) & 1);
      bool ok = true;
      if (zi == (l > 0)) {
        ok = wait(&wfull[p & 1], (uint32_t)((p >> 1) & 1));
        if (ok && l > 0) ok = wait(&stored[0], before);
      }
      if (ok && p > 0 && zi < TS) ok = wait(&stored[zi], before);
      if (ok && l == 0) ok = wait(&full[slot], slotPar);
      return ok;
    };
    int p = 0, zi = 0, l = 0;
    bool ok = ready(0, 0, 0);
    while (ok) {
      tc_fence_after();
      // output planes reached lo..hi, of which nOld started before
      const int lo = max(zi - 2, 0), hi = min(zi, TS - 1);
      const int nOld = l > 0 && zi == 1 ? 0 : min(zi, TS) - lo;
      const int first = lo + nOld;
      const int row0 = 16 * (lo - (zi - 2));  // first row of B used
      const uint32_t one = 1u << 18;          // 16 more columns
      const uint32_t idAll = idesc_bf16_f32(128, 16) + (uint32_t)(hi - lo) * one;
      const uint32_t idOld = idesc_bf16_f32(128, 16) + (uint32_t)(nOld - 1) * one;
      const uint32_t idNew = idesc_bf16_f32(128, 16) + (uint32_t)(hi - first) * one;
      const uint32_t at = smem_addr(ring) + slot * PLANE_BYTES;
      const uint64_t az = l > 0 ? a0 + (uint64_t)((zi - 1) * (int)(2 * PLANE_BYTES / 16))
                                : smem_desc(at, zero - at, PD * 16);
      const uint64_t bz = b0 + (uint64_t)((p & 1) * (WIMG * 2 / 16) + row0);
      const uint32_t c = tbase + (uint32_t)(16 * lo);
      // (the x halves alternate: neighbouring MMAs add to different accumulators)
      auto taps = [&](auto t0, auto t1) {
#pragma unroll
        for (int t = decltype(t0)::value; t < decltype(t1)::value; t++)
#pragma unroll
          for (int xh = 0; xh < 2; xh++)
            mma_bf16(c + (uint32_t)(256 * xh), az + (uint64_t)((t / 3) * PD + 8 * xh + t % 3),
                     bz + (uint64_t)(t * 96), idAll, 1u);
      };
      // the next plane, and a first look at its barriers: the answer comes while the
      // MMAs below are issued
      const int pz = zi, pl = l, pslot = slot;
      if (l == 0 && ++slot == CONV_SLOTS) {
        slot = 0;
        slotPar ^= 1u;
      }
      int np = p, nl = l, nz = zi + 1;
      if (nz > (l > 0 ? TS : TS + 1)) {
        np++;
        nl = l + 1 == a.nl ? 0 : l + 1;
        nz = nl > 0;
      }
      const bool more = np < passes, inside = np == p;
      bool seen = inside;
      if (inside && p > 0 && nz < TS) seen = mbar_test(&stored[nz], (uint32_t)((p - 1) & 1));
      if (inside && l == 0) seen = mbar_test(&full[slot], slotPar) && seen;
      if (elect_one()) {
#pragma unroll
        for (int xh = 0; xh < 2; xh++)
          if (nOld > 0)
            mma_bf16(c + (uint32_t)(256 * xh), az + (uint64_t)(8 * xh), bz, idOld, 1u);
#pragma unroll
        for (int xh = 0; xh < 2; xh++)
          if (first <= hi)
            mma_bf16(c + (uint32_t)(256 * xh + 16 * nOld), az + (uint64_t)(8 * xh),
                     bz + (uint64_t)(16 * nOld), idNew, 0u);
        taps(std::integral_constant<int, 1>{}, std::integral_constant<int, 5>{});
      }
      __syncwarp();
      // the previous pass is done with its weights: those of the next one
      if (pz == 6 && p > 0 && wl < passes) {
        if (!(ok = wait(&done[PD - 1], (uint32_t)((p - 1) & 1)))) break;
        load_weights(wl++, wlL);
        wlL = wlL + 1 == a.nl ? 0 : wlL + 1;
      }
      p = np;
      l = nl;
      zi = nz;
      if (!__all_sync(0xffffffffu, seen) && more && !(ok = ready(p, l, zi))) break;
      if (elect_one()) {
        taps(std::integral_constant<int, 5>{}, std::integral_constant<int, 9>{});
        if (pz > 1) mma_commit(&done[pz]);  // (no output plane completes before)
        if (pl > 0 && pz == TS) mma_commit(&done[PD - 1]);  // (its last plane is zero)
        if (pl == 0) mma_commit(&taken[pslot]);
      }
      __syncwarp();
      if (!more) break;
    }
    if (!ok) {
      // a wait gave up: flag it, give the work in flight one more bounded wait
      *abort = 1;
      if (lane == 0) atomicExch(a.err, 1);
      if (elect_one()) mma_commit(&done[0]);  // (nothing else waits on done[0])
      __syncwarp();
      mbar_wait(&done[0], 0);
      for (int w = p; w < wl; w++)
        mbar_wait(&wfull[w & 1], (uint32_t)((w >> 1) & 1));
    }
  } else if (warp > EPI_WARPS) {
    // every fourth ring plane: loaded into registers before the slot
    // is free
    constexpr int PER = (PLANE + 31) / 32;
    const int total = nTiles * PD;
    for (int q = warp - EPI_WARPS - 1; q < total; q += CONV_THREADS / 32 - EPI_WARPS - 1) {
      const size_t t = blockIdx.x + (size_t)(q / PD) * G;
      const int zi = q % PD, slot = q % CONV_SLOTS, use = q / CONV_SLOTS;
      uint4 v[PER];
      if (a.feat) {
        const float* f = a.feat + t * NFEAT * NPAD + zi * PLANE;
#pragma unroll
        for (int i = 0; i < PER; i++) {
          const int c = min(lane + 32 * i, PLANE - 1);
          v[i] = make_uint4(pack_bf2(f[c], f[NPAD + c]), pack_bf2(f[2 * NPAD + c], f[3 * NPAD + c]),
                            0u, 0u);
        }
      } else {
        const uint4* f = a.in + t * 2 * NPAD + zi * PLANE;
#pragma unroll
        for (int i = 0; i < PER; i++) v[i] = f[min(lane + 32 * i, PLANE - 1)];
      }
      if (use && !mbar_wait_abort(&taken[slot], (uint32_t)((use - 1) & 1), abort)) {
        *abort = 1;
        if (lane == 0) atomicExch(a.err, 1);
        break;
      }
      uint4* d = reinterpret_cast<uint4*>(ring + slot * PLANE_BYTES);
#pragma unroll
      for (int i = 0; i < PER; i++)
        if (lane + 32 * i < PLANE) {
          d[lane + 32 * i] = v[i];
          if (a.x0) a.x0[t * 2 * NPAD + zi * PLANE + lane + 32 * i] = v[i];
        }
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(&full[slot]);
    }
  } else {
    const int xh = (warp >> 2) & 1, quarter = warp & 3;
    const int r = 32 * quarter + lane;
    const int x = 8 * xh + (r & 7), y = r >> 3;
    bool ok = true;
    for (int p = 0; p < passes && ok; p++) {
      const ConvLayer& Ly = a.L[p % a.nl];
      const bool last = p % a.nl == a.nl - 1;
      const size_t t = blockIdx.x + (size_t)(p / a.nl) * G;
      const int epi = Ly.epi;
      const float s = epi == EPI_OUT0 && a.outScale ? a.outScale[t] : 1.f;
      const int64_t base = epi == EPI_OUT0 ? (a.outOff ? a.outOff[t] : (int64_t)t * NCELL) : 0;
      uint4* out = Ly.out ? Ly.out + t * 2 * NPAD : nullptr;
      const uint4* mask = epi == EPI_MASK ? Ly.mask + t * 2 * NPAD : nullptr;
      for (int z = warp >> 3; z < TS; z += EPI_WARPS / 8) {
        const int cell = x + TS * (y + TS * z), pc = pad_index(cell);
        uint4 m2[2];
        if (epi == EPI_MASK) {  // in flight while the MMAs finish
          m2[0] = mask[pc];
          m2[1] = mask[NPAD + pc];
        }
        if (!(ok = mbar_wait_abort(&done[z + 2], (uint32_t)(p & 1), abort))) break;
        tc_fence_after();
        float v[16];
        tmem_ld16(tbase + ((uint32_t)(32 * quarter) << 16) + (uint32_t)(256 * xh + 16 * z), v);
        tc_fence_before();
        if (epi == EPI_OUT0) {
          __syncwarp();
          if (lane == 0) mbar_arrive(&stored[z]);  // drained
          a.out0[base + cell] = v[0] * s;
          continue;
        }
        if (epi == EPI_MASK) {
          const __nv_bfloat16* mb = reinterpret_cast<const __nv_bfloat16*>(m2);
#pragma unroll
          for (int c = 0; c < 16; c++)
            if (!(__bfloat162float(mb[c]) > 0.f)) v[c] = 0.f;
        } else {
#pragma unroll
          for (int c = 0; c < 16; c++) v[c] = fmaxf(v[c], 0.f);
        }
        uint4 q0, q1;
        q0.x = pack_bf2(v[0], v[1]);
        q0.y = pack_bf2(v[2], v[3]);
        q0.z = pack_bf2(v[4], v[5]);
        q0.w = pack_bf2(v[6], v[7]);
        q1.x = pack_bf2(v[8], v[9]);
        q1.y = pack_bf2(v[10], v[11]);
        q1.z = pack_bf2(v[12], v[13]);
        q1.w = pack_bf2(v[14], v[15]);
        if (!last) {
          uint4* d = reinterpret_cast<uint4*>(act + z * 2 * PLANE_BYTES) + (x + 1) + PD * (y + 1);
          d[0] = q0;
          d[PLANE] = q1;
          fence_proxy_async();
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&stored[z]);
        if (out) {
          out[pc] = q0;
          out[NPAD + pc] = q1;
        }
      }
    }
    if (!ok) {
      *abort = 1;
      if (lane == 0) atomicExch(a.err, 1);
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0) tmem_dealloc(tbase, 512);
}

// ---------------------------------------------------------------------------
// weight gradient (mma.sync)
// ---------------------------------------------------------------------------
// partial[layer][blockIdx.x][co][ci][tap] = sum over this CTA's slabs and their
// cells o of dz[o][co] * X[o + tap][ci], X the layer input on the padded box and dz
// the output gradient (both in the padded bf16 layout, as the forward pass
// reads them).  All four layers in one launch (blockIdx.y), two CTAs per SM; a
// unit of work is a slab of 4 output planes of a tile, brought in by four bulk
// copies of contiguous planes.
// Per x row of 16 cells a warp's dz (16 co x 16 cells) times the row of X (16 cells
// x 16 ci) at one of 27 shifts are two m16n8k16 products with bf16 operands (exact)
// and FP32 sums; warp (kz, ky) keeps the 3 kx.  Both operands come from the
// [cell][8 channels] halves by ldmatrix.trans without bank conflicts (8 cells are 128
// contiguous bytes).  The sums of a plane are added to the warp's FP32 totals with
// round-to-nearest, so what the tensor core's own additions lose stays within 16 of them.
// With FP32 CUDA cores, one thread per (co, ci) and 27 shared-memory reads per cell and
// thread, a training step of 128 tiles took 2.92 ms on a B200; now 0.34 ms.
constexpr int WG_SLAB = 4;  // output planes per unit
constexpr int WG_THREADS = 9 * 32;
constexpr uint32_t WG_XB = (WG_SLAB + 2) * PLANE_BYTES, WG_DB = WG_SLAB * PLANE_BYTES;
constexpr size_t WG_SMEM = 2 * (size_t)(WG_XB + WG_DB);

struct WgradArgs {
  int n;
  const uint4* X[NLAYER];
  const uint4* dz[NLAYER];
  float* partial;
  int* err;
};

__device__ __forceinline__ void ldmatrix4_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
__device__ __forceinline__ void mma_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0,
                                          uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// The same sums where a product with a zero gradient is left out, one thread per
// (co, ci): what counts when an input is not finite (0 * inf).
__device__ __noinline__ void wgrad_skip_zeros(const WgradArgs& a, int layer, float* p) {
  const int tid = threadIdx.x, co = tid >> 4, ci = tid & 15;
  if (tid >= 256) return;
  float acc[27];
#pragma unroll
  for (int k = 0; k < 27; k++) acc[k] = 0.f;
  for (int u = blockIdx.x; u < a.n * (TS / WG_SLAB); u += gridDim.x) {
    const size_t t = (size_t)(u / (TS / WG_SLAB)) * 2 * NPAD;
    const int z0 = u % (TS / WG_SLAB) * WG_SLAB;
    const __nv_bfloat16* X =
        reinterpret_cast<const __nv_bfloat16*>(a.X[layer] + t + (ci >> 3) * NPAD) + (ci & 7);
    const __nv_bfloat16* D =
        reinterpret_cast<const __nv_bfloat16*>(a.dz[layer] + t + (co >> 3) * NPAD) + (co & 7);
    for (int o = z0 * TS * TS; o < (z0 + WG_SLAB) * TS * TS; o++) {
      const int pc = pad_index(o), c0 = pc - 1 - PD - PLANE;
      const float d = __bfloat162float(D[(size_t)pc * 8]);
      if (d == 0.f) continue;
#pragma unroll
      for (int k = 0; k < 27; k++)
        acc[k] = fmaf(d, __bfloat162float(X[(size_t)(c0 + k % 3 + PD * (k / 3 % 3) + PLANE * (k / 9)) * 8]),
                      acc[k]);
    }
  }
#pragma unroll
  for (int k = 0; k < 27; k++) p[(co * NC + ci) * 27 + k] = acc[k];
}

__global__ void __launch_bounds__(WG_THREADS, 2) k_wgrad(const __grid_constant__ WgradArgs a) {
  extern __shared__ __align__(128) uint8_t smw[];
  __shared__ __align__(8) uint64_t bar;
  uint8_t* Xs = smw;              // [2] halves of WG_SLAB + 2 planes
  uint8_t* Ds = smw + 2 * WG_XB;  // [2] halves of WG_SLAB planes
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, layer = blockIdx.y;
  const int kz = warp / 3, ky = warp % 3;
  if (tid == 0) {
    mbar_init(&bar, 1);
    fence_mbar_init();
  }
  __syncthreads();
  // this lane's row of the 8x8 matrices: cells 0-7 or 8-15, channels 0-7 or 8-15.  dz
  // as A (co x cells): {cells lo, co lo}, {lo, hi}, {hi, lo}, {hi, hi}; X as B (cells x
  // ci): {lo, ci lo}, {hi, ci lo}, {lo, ci hi}, {hi, ci hi}
  const int m = lane >> 3;
  const uint32_t da = smem_addr(Ds) + (m & 1) * WG_DB + ((m >> 1) * 8 + (lane & 7) + 1) * 16;
  const uint32_t xa = smem_addr(Xs) + (m >> 1) * WG_XB + ((m & 1) * 8 + (lane & 7)) * 16;
  float tot[3][2][4];
#pragma unroll
  for (int i = 0; i < 24; i++) tot[i / 8][i / 4 % 2][i % 4] = 0.f;
  bool ok = true;
  uint32_t par = 0;
  for (int u = blockIdx.x; u < a.n * (TS / WG_SLAB); u += gridDim.x, par ^= 1u) {
    const size_t t = (size_t)(u / (TS / WG_SLAB)) * 2 * NPAD;
    const int z0 = u % (TS / WG_SLAB) * WG_SLAB;
    if (tid == 0) {
      mbar_expect_tx(&bar, WG_SMEM);
      for (int h = 0; h < 2; h++) {
        bulk_g2s(Xs + h * WG_XB, a.X[layer] + t + h * NPAD + z0 * PLANE, WG_XB, &bar);
        bulk_g2s(Ds + h * WG_DB, a.dz[layer] + t + h * NPAD + (z0 + 1) * PLANE, WG_DB, &bar);
      }
    }
    if (!__syncthreads_and(mbar_wait(&bar, par))) {
      ok = false;
      break;
    }
    for (int z = 0; z < WG_SLAB; z++) {
      float c[3][2][4];
#pragma unroll
      for (int i = 0; i < 24; i++) c[i / 8][i / 4 % 2][i % 4] = 0.f;
      const uint32_t dp = da + (z * PLANE + PD) * 16;
      const uint32_t xp = xa + ((z + kz) * PLANE + ky * PD) * 16;
#pragma unroll 4
      for (int y = 0; y < TS; y++) {
        uint32_t A[4];
        ldmatrix4_trans(A, dp + y * PD * 16);
#pragma unroll
        for (int kx = 0; kx < 3; kx++) {
          uint32_t B[4];
          ldmatrix4_trans(B, xp + (y * PD + kx) * 16);
          mma_16816(c[kx][0], A, B[0], B[1]);
          mma_16816(c[kx][1], A, B[2], B[3]);
        }
      }
#pragma unroll
      for (int i = 0; i < 24; i++) tot[i / 8][i / 4 % 2][i % 4] += c[i / 8][i / 4 % 2][i % 4];
    }
    __syncthreads();  // the slab is read: the next one may land
  }
  float* p = a.partial + ((size_t)layer * gridDim.x + blockIdx.x) * NC * NC * 27;
  bool fin = true;
#pragma unroll
  for (int i = 0; i < 24; i++) {
    const int kx = i / 8, nt = i / 4 % 2, j = i % 4;
    const int co = (lane >> 2) + 8 * (j >> 1), ci = 8 * nt + 2 * (lane & 3) + (j & 1);
    const float v = tot[kx][nt][j];
    fin = fin && isfinite(v);
    p[(co * NC + ci) * 27 + warp * 3 + kx] = v;
  }
  if (!ok) {
    if (tid == 0) {
      atomicExch(a.err, 1);
      mbar_wait(&bar, par);  // bounded: the copies in flight
    }
    return;
  }
  if (__syncthreads_or(!fin)) wgrad_skip_zeros(a, layer, p);
}

// grad = sum over the CTA partials of its layer, fixed order, FP64.
__global__ void k_wgrad_reduce(const float* __restrict__ partial, int nPart,
                               float* __restrict__ g) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= NPARAM) return;
  int l = 0;
  while (l + 1 < NLAYER && i >= layer_off(l + 1)) l++;
  const int cin = layer_cin(l), e = i - layer_off(l);
  const int co = e / (cin * 27), ci = (e / 27) % cin, k = e % 27;
  const float* p = partial + (size_t)l * nPart * NC * NC * 27 + (co * NC + ci) * 27 + k;
  double s = 0;
#pragma unroll 8
  for (int q = 0; q < nPart; q++) s += p[(size_t)q * NC * NC * 27];
  g[i] = (float)s;
}

// ---------------------------------------------------------------------------
// loss, Adam
// ---------------------------------------------------------------------------
// loss = sum m (y - t)^2 / count; dy = 2 m (y - t) / count into channel 0 of
// a padded-layout bf16 gradient (all other values stay 0).  Per-CTA partial.
constexpr int LOSS_GRID = 148 * 2;
__global__ void __launch_bounds__(512) k_loss(int64_t nc, const float* __restrict__ y,
                                              const float* __restrict__ tgt,
                                              const float* __restrict__ m, float invCount,
                                              __nv_bfloat16* __restrict__ dy,
                                              double* __restrict__ partial) {
  // dy: padded layout, channel 0 of half 0 at the interior cells
  __shared__ double ws[16];
  double acc = 0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nc;
       i += (int64_t)gridDim.x * blockDim.x) {
    const float d = m[i] > 0.f ? y[i] - tgt[i] : 0.f;
    acc += (double)d * d;
    if (dy) {
      const int64_t t = i / NCELL;
      dy[((size_t)t * 2 * NPAD + pad_index((int)(i % NCELL))) * 8] =
          __float2bfloat16_rn(2.f * d * invCount);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) s += ws[w];
    partial[blockIdx.x] = s * invCount;
  }
}

__global__ void k_adam(float* __restrict__ w, float* __restrict__ m, float* __restrict__ v,
                       const float* __restrict__ g, int n, float lr, float b1, float b2,
                       float eps, float c1, float c2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = g[i];
  const float mi = b1 * m[i] + (1.f - b1) * gi;
  const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  w[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

// Gather of training / inference samples lives in cnn_features.cu.

}  // namespace cnn
}  // namespace msbg

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
using namespace msbg;
using namespace msbg::cnn;

struct msbg_cnn {
  int device = 0;
  cudaStream_t stream = nullptr;
  std::string lastError;
  DeviceBuffer w, m, v, g;       // FP32 [NPARAM]
  DeviceBuffer imgF, imgB;       // bf16 [NLAYER][WIMG]
  DeviceBuffer err;              // int
  int step = 0;
  int numSMs = 148;
  // activations and gradients of the largest batch so far
  DeviceBuffer x0, a1, a2, a3, y, dy, dz3, dz2, dz1, part, lossPart;  // padded layout
};

namespace {

int cnn_error(msbg_cnn* n, int code, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  if (n) n->lastError = buf;
  return code;
}

#define CNN_TRY(net, expr)                                                                 \
  do {                                                                                     \
    cudaError_t _e = (expr);                                                               \
    if (_e != cudaSuccess)                                                                 \
      return cnn_error((net), _e == cudaErrorMemoryAllocation ? MSBG_ENOMEM : MSBG_ERROR, \
                       "%s: %s (%s:%d)", #expr, cudaGetErrorString(_e), __FILE__, __LINE__); \
  } while (0)

// The limits are attributes of the kernels on the current device: set for every network.
cudaError_t set_attrs() {
  const cudaError_t e = cudaFuncSetAttribute(
      k_conv3_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CONV_SMEM);
  return e != cudaSuccess ? e
                          : cudaFuncSetAttribute(
                                k_wgrad, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)WG_SMEM);
}

const __nv_bfloat16* image(msbg_cnn* net, int layer, bool backward) {
  return (backward ? net->imgB : net->imgF).as<__nv_bfloat16>() + (size_t)layer * WIMG;
}

void conv(msbg_cnn* net, ConvChain& a, int n, cudaStream_t st) {
  a.n = n;
  a.err = net->err.as<int>();
  k_conv3_tc<<<std::min(n, net->numSMs), CONV_THREADS, CONV_SMEM, st>>>(a);
}

// CTAs of the weight gradient per layer: two per SM over the four layers.
int wgrad_ctas(const msbg_cnn* net, int n) {
  return std::max(1, std::min(n * (TS / WG_SLAB), net->numSMs * 2 / NLAYER));
}

// Activations of n tiles, zeroed when allocated (the halos stay zero).
int ensure_act(msbg_cnn* net, DeviceBuffer& b, int n) {
  const size_t bytes = (size_t)n * ACT_BYTES;
  if (b.p && b.bytes >= bytes) return MSBG_OK;
  CNN_TRY(net, b.ensure(bytes));
  CNN_TRY(net, cudaMemsetAsync(b.p, 0, bytes, net->stream));
  return MSBG_OK;
}

int ensure_train(msbg_cnn* net, int n) {
  for (DeviceBuffer* b : {&net->x0, &net->a1, &net->a2, &net->a3, &net->dz3, &net->dz2, &net->dz1,
                          &net->dy}) {
    int rc = ensure_act(net, *b, n);
    if (rc) return rc;
  }
  CNN_TRY(net, net->y.ensure((size_t)n * NCELL * sizeof(float)));
  CNN_TRY(net, net->part.ensure((size_t)NLAYER * wgrad_ctas(net, n) * NC * NC * 27 *
                                sizeof(float)));
  CNN_TRY(net, net->lossPart.ensure(LOSS_GRID * sizeof(double)));
  return MSBG_OK;
}

int pack(msbg_cnn* net) {
  k_pack<<<(NLAYER * WIMG + 255) / 256, 256, 0, net->stream>>>(
      net->w.as<float>(), net->imgF.as<__nv_bfloat16>(), net->imgB.as<__nv_bfloat16>());
  CNN_TRY(net, cudaGetLastError());
  return MSBG_OK;
}

int check_err(msbg_cnn* net) {
  int e = 0;
  CNN_TRY(net, cudaMemcpyAsync(&e, net->err.p, sizeof(int), cudaMemcpyDeviceToHost, net->stream));
  CNN_TRY(net, cudaStreamSynchronize(net->stream));
  if (e) {
    cudaMemsetAsync(net->err.p, 0, sizeof(int), net->stream);
    return cnn_error(net, MSBG_ETIMEOUT, "a tensor-core wait gave up");
  }
  return MSBG_OK;
}

}  // namespace

namespace msbg {
namespace cnn {
// Forward pass into out0 (see msbg_cnn_forward); used by the pressure solver.
int forward(msbg_cnn* net, const float* feat, float* out0, const int64_t* outOff,
            const float* outScale, int n, cudaStream_t st) {
  if (n <= 0) return MSBG_OK;
  ConvChain a{};
  a.nl = NLAYER;
  a.feat = feat;
  for (int l = 0; l < NLAYER; l++)
    a.L[l] = ConvLayer{nullptr, nullptr, image(net, l, false), l < NLAYER - 1 ? EPI_RELU : EPI_OUT0};
  a.out0 = out0;
  a.outOff = outOff;
  a.outScale = outScale;
  conv(net, a, n, st);
  return cudaGetLastError() == cudaSuccess ? MSBG_OK : MSBG_ERROR;
}

int take_error(msbg_cnn* net, cudaStream_t st) {
  int e = 0;
  if (cudaMemcpyAsync(&e, net->err.p, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return MSBG_ERROR;
  if (e) cudaMemsetAsync(net->err.p, 0, sizeof(int), st);
  return e ? MSBG_ETIMEOUT : MSBG_OK;
}
}  // namespace cnn
}  // namespace msbg

extern "C" int msbg_cnn_create(int device, msbg_cnn** out) {
  if (!out) return MSBG_EINVARG;
  *out = nullptr;
  int nd = 0;
  if (cudaGetDeviceCount(&nd) != cudaSuccess || device < 0 || device >= nd) return MSBG_ENODEV;
  cudaSetDevice(device);
  auto* net = new msbg_cnn();
  net->device = device;
  cudaDeviceGetAttribute(&net->numSMs, cudaDevAttrMultiProcessorCount, device);
  if (set_attrs() != cudaSuccess) {
    delete net;
    return MSBG_ERROR;
  }
  if (cudaStreamCreateWithFlags(&net->stream, cudaStreamNonBlocking) != cudaSuccess ||
      net->w.ensure(NPARAM * sizeof(float)) != cudaSuccess ||
      net->m.ensure(NPARAM * sizeof(float)) != cudaSuccess ||
      net->v.ensure(NPARAM * sizeof(float)) != cudaSuccess ||
      net->g.ensure(NPARAM * sizeof(float)) != cudaSuccess ||
      net->imgF.ensure(NLAYER * WIMG * 2) != cudaSuccess ||
      net->imgB.ensure(NLAYER * WIMG * 2) != cudaSuccess ||
      net->err.ensure(sizeof(int)) != cudaSuccess) {
    if (net->stream) cudaStreamDestroy(net->stream);
    delete net;
    return MSBG_ENOMEM;
  }
  cudaMemsetAsync(net->err.p, 0, sizeof(int), net->stream);
  cudaMemsetAsync(net->m.p, 0, NPARAM * sizeof(float), net->stream);
  cudaMemsetAsync(net->v.p, 0, NPARAM * sizeof(float), net->stream);
  // He-uniform initial weights from a fixed seed
  std::vector<float> w(NPARAM);
  std::mt19937_64 rng(12345);
  for (int l = 0; l < NLAYER; l++) {
    const float b = std::sqrt(6.0f / (27.0f * layer_cin(l)));
    std::uniform_real_distribution<float> U(-b, b);
    for (int i = 0; i < layer_cout(l) * layer_cin(l) * 27; i++) w[layer_off(l) + i] = U(rng);
  }
  cudaMemcpyAsync(net->w.p, w.data(), NPARAM * sizeof(float), cudaMemcpyHostToDevice, net->stream);
  if (pack(net) != MSBG_OK || cudaStreamSynchronize(net->stream) != cudaSuccess) {
    cudaStreamDestroy(net->stream);
    delete net;
    return MSBG_ERROR;
  }
  *out = net;
  return MSBG_OK;
}

extern "C" int msbg_cnn_destroy(msbg_cnn* net) {
  if (!net) return MSBG_EINVARG;
  cudaSetDevice(net->device);
  cudaStreamSynchronize(net->stream);
  cudaStreamDestroy(net->stream);
  delete net;
  return MSBG_OK;
}

extern "C" const char* msbg_cnn_last_error(msbg_cnn* net) {
  return net ? net->lastError.c_str() : "null network";
}

extern "C" int msbg_cnn_num_params(void) { return NPARAM; }

extern "C" int msbg_cnn_set_weights(msbg_cnn* net, const float* w, int64_t n) {
  if (!net || !w || n != NPARAM) return cnn_error(net, MSBG_EINVARG, "expected %d weights", NPARAM);
  cudaSetDevice(net->device);
  CNN_TRY(net, cudaMemcpyAsync(net->w.p, w, NPARAM * sizeof(float), cudaMemcpyHostToDevice, net->stream));
  CNN_TRY(net, cudaMemsetAsync(net->m.p, 0, NPARAM * sizeof(float), net->stream));
  CNN_TRY(net, cudaMemsetAsync(net->v.p, 0, NPARAM * sizeof(float), net->stream));
  net->step = 0;
  int rc = pack(net);
  if (rc) return rc;
  CNN_TRY(net, cudaStreamSynchronize(net->stream));
  return MSBG_OK;
}

extern "C" int msbg_cnn_get_weights(msbg_cnn* net, float* w, int64_t n) {
  if (!net || !w || n != NPARAM) return cnn_error(net, MSBG_EINVARG, "expected %d weights", NPARAM);
  cudaSetDevice(net->device);
  CNN_TRY(net, cudaMemcpyAsync(w, net->w.p, NPARAM * sizeof(float), cudaMemcpyDeviceToHost, net->stream));
  CNN_TRY(net, cudaStreamSynchronize(net->stream));
  return MSBG_OK;
}

extern "C" int msbg_cnn_forward(msbg_cnn* net, const float* feat, float* out, int n) {
  if (!net || n < 0 || (n > 0 && (!feat || !out))) return cnn_error(net, MSBG_EINVARG, "bad arguments");
  if (n == 0) return MSBG_OK;
  cudaSetDevice(net->device);
  int rc = forward(net, feat, out, nullptr, nullptr, n, net->stream);
  if (rc) return cnn_error(net, rc, "forward launch failed: %s", cudaGetErrorString(cudaGetLastError()));
  return check_err(net);
}

// Loss and gradient of a batch (device inputs); the gradient stays on the
// device (and is copied to gradHost when given).
extern "C" int msbg_cnn_loss_grad(msbg_cnn* net, const float* feat, const float* target,
                                  const float* mask, int n, double count, double* loss,
                                  float* gradHost) {
  if (!net || n <= 0 || !feat || !target || !mask || !(count > 0))
    return cnn_error(net, MSBG_EINVARG, "bad arguments");
  cudaSetDevice(net->device);
  int rc = ensure_train(net, n);
  if (rc) return rc;
  cudaStream_t st = net->stream;
  uint4* x0 = net->x0.as<uint4>();
  uint4* a1 = net->a1.as<uint4>();
  uint4* a2 = net->a2.as<uint4>();
  uint4* a3 = net->a3.as<uint4>();
  uint4* dy = net->dy.as<uint4>();
  uint4* dz3 = net->dz3.as<uint4>();
  uint4* dz2 = net->dz2.as<uint4>();
  uint4* dz1 = net->dz1.as<uint4>();
  float* y = net->y.as<float>();
  // forward, keeping the activations
  ConvChain f{};
  f.nl = NLAYER;
  f.feat = feat;
  f.x0 = x0;
  f.L[0] = ConvLayer{a1, nullptr, image(net, 0, false), EPI_RELU};
  f.L[1] = ConvLayer{a2, nullptr, image(net, 1, false), EPI_RELU};
  f.L[2] = ConvLayer{a3, nullptr, image(net, 2, false), EPI_RELU};
  f.L[3] = ConvLayer{nullptr, nullptr, image(net, 3, false), EPI_OUT0};
  f.out0 = y;
  conv(net, f, n, st);
  // loss and dL/dy
  k_loss<<<LOSS_GRID, 512, 0, st>>>((int64_t)n * NCELL, y, target, mask, (float)(1.0 / count),
                                    reinterpret_cast<__nv_bfloat16*>(dy), net->lossPart.as<double>());
  // backward-data through layers 4, 3, 2 (ReLU masks of their inputs)
  ConvChain d{};
  d.nl = 3;
  d.in = dy;
  d.L[0] = ConvLayer{dz3, a3, image(net, 3, true), EPI_MASK};
  d.L[1] = ConvLayer{dz2, a2, image(net, 2, true), EPI_MASK};
  d.L[2] = ConvLayer{dz1, a1, image(net, 1, true), EPI_MASK};
  conv(net, d, n, st);
  // weight gradients
  const int ctas = wgrad_ctas(net, n);
  float* g = net->g.as<float>();
  const WgradArgs wg{n, {x0, a1, a2, a3}, {dz1, dz2, dz3, dy}, net->part.as<float>(),
                     net->err.as<int>()};
  k_wgrad<<<dim3(ctas, NLAYER), WG_THREADS, WG_SMEM, st>>>(wg);
  k_wgrad_reduce<<<(NPARAM + 127) / 128, 128, 0, st>>>(net->part.as<float>(), ctas, g);
  CNN_TRY(net, cudaGetLastError());
  std::vector<double> lp(LOSS_GRID);
  CNN_TRY(net, cudaMemcpyAsync(lp.data(), net->lossPart.p, LOSS_GRID * sizeof(double),
                               cudaMemcpyDeviceToHost, st));
  if (gradHost)
    CNN_TRY(net, cudaMemcpyAsync(gradHost, g, NPARAM * sizeof(float), cudaMemcpyDeviceToHost, st));
  rc = check_err(net);
  if (rc) return rc;
  if (loss) {
    double s = 0;
    for (double v : lp) s += v;
    *loss = s;
  }
  return MSBG_OK;
}

extern "C" int msbg_cnn_adam_step(msbg_cnn* net, float lr, float beta1, float beta2, float eps) {
  if (!net || !(lr > 0)) return cnn_error(net, MSBG_EINVARG, "bad arguments");
  cudaSetDevice(net->device);
  net->step++;
  const float c1 = 1.f - std::pow(beta1, (float)net->step);
  const float c2 = 1.f - std::pow(beta2, (float)net->step);
  k_adam<<<(NPARAM + 255) / 256, 256, 0, net->stream>>>(net->w.as<float>(), net->m.as<float>(),
                                                       net->v.as<float>(), net->g.as<float>(),
                                                       NPARAM, lr, beta1, beta2, eps, c1, c2);
  int rc = pack(net);
  if (rc) return rc;
  CNN_TRY(net, cudaStreamSynchronize(net->stream));
  return MSBG_OK;
}
