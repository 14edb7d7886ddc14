// G2P on mixed-resolution grids: the MAC velocity interpolation of
// interpVec3MSBG / interpCompMSBG (src/flip_sim.cpp:1354-1525) inside
// gridToParticle (src/flip_sim.cpp:1526-1545), and the fine/coarse distance
// channel it blends with (CH_DIST_FINECOARSE, built by setRefinementMap,
// src/msbg.cpp:1700-1723, 1887-1960, 1994-2029):
//   msbg_gpu_flip_mr_dist        the distance channel, built on the GPU
//   msbg_gpu_flip_mr_channel     the velocity channels in/out
//   msbg_gpu_flip_g2p_mr(_device) the particle update
//   msbg_gpu_flip_downsample_velocity  downsampleVelocity (src/msbg4.cpp:2035),
//                                the velocity restricted to the next MG level
//
// Layout (the packed layout of the pressure channels): for every block in
// ascending bid, its (bsx0 >> level)^3 voxels at its own level, vid = x +
// y*bs + z*bs^2.  A voxel of a level's grid inside a block of another level
// has no data there and reads 0, as a NULL block of that level's sparse grid
// does in the reference.  Vector channels hold the lower-face MAC values (u,
// v, w) per voxel.
//
// Per particle and component, one sample geometry serves both channels (vel
// and velOld) and the distance lookup; the arithmetic is the reference's, in
// its order, with no contraction into FMAs, and MtLinstep in double
// (src/mtool.c:200-208).
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstdint>
#include <map>
#include <memory>
#include <vector>

#include "common.cuh"

namespace msbg {
namespace {

#include "particle_bins.cuh"

// The reference's transition width: MultiresSparseGrid::create fixes
// _dTransRes at 6 whatever it is passed (src/msbg.cpp:198-201, 290).
constexpr int kDTransRes = 6;

constexpr int MR_LEVELS = 4;  // resolution levels at most

struct MrState {
  int sx = 0, sy = 0, sz = 0, bsx0 = 0, nLevels = 0;
  std::vector<int> levels;
  int64_t n = 0;  // packed voxels
  bool distBuilt = false;
  DeviceBuffer level, off, fc, kind, key, dist, parts;
  DeviceBuffer vel;      // [3n] (vel, velOld) side by side: a gather reads both in one load
  DeviceBuffer scratch;  // pieces of a channel on its way in or out; the visiting order of G2P
  DeviceBuffer dsOffA, dsOffB, dsFlags, dsSrc, dsDst;  // downsampleVelocity
};

std::map<msbg_gpu_ctx*, std::unique_ptr<MrState>>& states() {
  static std::map<msbg_gpu_ctx*, std::unique_ptr<MrState>> m;
  return m;
}

struct MrGrid {
  int sx, sy, sz, sh0, nbx, nby, nbz, nl;
  const int8_t* __restrict__ level;
  const int64_t* __restrict__ off;
  const int8_t* __restrict__ kind;  // [nl][nb]: 0 empty, 1 value, 2 full
  const uint16_t* __restrict__ dist;
  const uint64_t* __restrict__ key;  // level, kinds and offset of a block
};

// BLK_FINE_COARSE per block: a block of a coarser level among its 26
// neighbours (src/msbg.cpp:1700-1723).
__global__ void k_mr_fine_coarse(const int8_t* __restrict__ level, int nbx, int nby, int nbz,
                                 int8_t* __restrict__ fc) {
  const int64_t nb = (int64_t)nbx * nby * nbz;
  for (int64_t b = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; b < nb;
       b += (int64_t)gridDim.x * blockDim.x) {
    const int bx = (int)(b % nbx), by = (int)((b / nbx) % nby), bz = (int)(b / ((int64_t)nbx * nby));
    const int lv = level[b];
    int8_t f = 0;
    for (int d = 0; d < 27; d++) {
      const int x = bx + d % 3 - 1, y = by + (d / 3) % 3 - 1, z = bz + d / 9 - 1;
      if (d == 13 || x < 0 || y < 0 || z < 0 || x >= nbx || y >= nby || z >= nbz) continue;
      if (level[x + (int64_t)nbx * (y + (int64_t)nby * z)] > lv) f = 1;
    }
    fc[b] = f;
  }
}

// Block kinds of the distance channel of every level: value blocks are the
// BLK_FINE_COARSE blocks of that level; a block of level l or l-1 with a
// BLK_FINE_COARSE neighbour of level l is a full block of value
// dTransRes*1024 in the channel of level l (src/msbg.cpp:1994-2029).
__global__ void k_mr_kind(const int8_t* __restrict__ level, const int8_t* __restrict__ fc,
                          int nbx, int nby, int nbz, int nl, int8_t* __restrict__ kind) {
  const int64_t nb = (int64_t)nbx * nby * nbz;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nb * nl;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int l = (int)(i / nb);
    const int64_t b = i - (int64_t)l * nb;
    const int lv = level[b];
    int8_t k = 0;
    if (lv == l && fc[b]) {
      k = 1;
    } else if (lv == l || lv == l - 1) {
      const int bx = (int)(b % nbx), by = (int)((b / nbx) % nby),
                bz = (int)(b / ((int64_t)nbx * nby));
      for (int d = 0; d < 27; d++) {
        const int x = bx + d % 3 - 1, y = by + (d / 3) % 3 - 1, z = bz + d / 9 - 1;
        if (d == 13 || x < 0 || y < 0 || z < 0 || x >= nbx || y >= nby || z >= nbz) continue;
        const int64_t b2 = x + (int64_t)nbx * (y + (int64_t)nby * z);
        if (level[b2] == l && fc[b2]) k = 2;
      }
    }
    kind[i] = k;
  }
}

// The distance values: one CTA per block (grid-stride over blocks).  A
// BLK_FINE_COARSE block stores per voxel of its level the distance from the
// voxel centre to the nearest coarser neighbour's box (src/msbg.h:3936-3948),
// capped at dTransRes, as (uint16)(dist*1024); every other block stores 0.
// The squared distances are sums of squares of half-integers, exact in FP32,
// and __fsqrt_rn rounds as the host's sqrtf does.
__global__ void __launch_bounds__(256) k_mr_dist(MrGrid g, const int8_t* __restrict__ fc,
                                                 uint16_t* __restrict__ dist) {
  __shared__ int act[26][3];
  __shared__ int nAct;
  const int64_t nb = (int64_t)g.nbx * g.nby * g.nbz;
  for (int64_t b = blockIdx.x; b < nb; b += gridDim.x) {
    const int lv = g.level[b], sh = g.sh0 - lv, bs = 1 << sh;
    const int bx = (int)(b % g.nbx), by = (int)((b / g.nbx) % g.nby),
              bz = (int)(b / ((int64_t)g.nbx * g.nby));
    __syncthreads();  // the previous block's readers are done with act
    if (threadIdx.x == 0) {
      int n = 0;
      if (fc[b])
        for (int d = 0; d < 27; d++) {
          const int x = bx + d % 3 - 1, y = by + (d / 3) % 3 - 1, z = bz + d / 9 - 1;
          if (d == 13 || x < 0 || y < 0 || z < 0 || x >= g.nbx || y >= g.nby || z >= g.nbz)
            continue;
          if (g.level[x + (int64_t)g.nbx * (y + (int64_t)g.nby * z)] <= lv) continue;
          act[n][0] = x;
          act[n][1] = y;
          act[n][2] = z;
          n++;
        }
      nAct = n;
    }
    __syncthreads();
    const int na = nAct, nv = bs * bs * bs;
    uint16_t* out = dist + g.off[b];
    for (int v = threadIdx.x; v < nv; v += blockDim.x) {
      if (!na) {
        out[v] = 0;
        continue;
      }
      const float p[3] = {(float)(bx * bs + (v & (bs - 1))) + 0.5f,
                          (float)(by * bs + ((v >> sh) & (bs - 1))) + 0.5f,
                          (float)(bz * bs + (v >> (2 * sh))) + 0.5f};
      float d2 = 1e20f;
      for (int i = 0; i < na; i++) {
        float s = 0.f;
#pragma unroll
        for (int c = 0; c < 3; c++) {
          const float lo = (float)(act[i][c] * bs), hi = (float)((act[i][c] + 1) * bs);
          float e = fmaxf(__fsub_rn(lo, p[c]), 0.f);
          e = fmaxf(e, __fsub_rn(p[c], hi));
          s = __fadd_rn(s, __fmul_rn(e, e));
        }
        d2 = fminf(d2, s);
      }
      float d = __fsqrt_rn(d2);
      if (d > (float)kDTransRes) d = (float)kDTransRes;
      out[v] = (uint16_t)__fmul_rn(d, 1024.f);
    }
  }
}

// What a gather asks of a block, in one load: its level, its kinds in the distance channels
// and its offset.
constexpr int KEY_KIND = 4, KEY_OFF = KEY_KIND + 2 * MR_LEVELS;
__device__ __forceinline__ int key_level(uint64_t k) { return (int)(k & 15); }
__device__ __forceinline__ int key_kind(uint64_t k, int lv) {
  return (int)(k >> (KEY_KIND + 2 * lv)) & 3;
}

__global__ void __launch_bounds__(256) k_mr_key(MrGrid g, uint64_t* __restrict__ key) {
  const int64_t nb = (int64_t)g.nbx * g.nby * g.nbz;
  for (int64_t b = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; b < nb;
       b += (int64_t)gridDim.x * blockDim.x) {
    uint64_t k = (uint64_t)g.off[b] << KEY_OFF | (uint64_t)g.level[b];
    for (int l = 0; l < g.nl; l++) k |= (uint64_t)g.kind[l * nb + b] << (KEY_KIND + 2 * l);
    key[b] = k;
  }
}

// The gathers are shared by a pair of lanes, of which one (side 0) loads the values at x and
// the other those at x + 1: the two are next to each other in memory, so a pair asks for
// one line per row of its window.  The pair then trades what the other needs.
__device__ __forceinline__ float pair_trade(float v) { return __shfl_xor_sync(0xffffffffu, v, 1); }

// A lane's half of a 2x2x2 window at level lv: column x, rows y[0..1], planes z[0..1] (in the
// grid), by shares of the block index and of the voxel's place in its block.
struct MrWindow {
  int sh, bx, lx, by[2], ly[2], bz[2], lz[2];
  __device__ __forceinline__ MrWindow(const MrGrid& g, int lv, int x, int y0, int y1, int z0, int z1)
      : sh(g.sh0 - lv) {
    const int m = (1 << sh) - 1;
    bx = x >> sh;
    lx = x & m;
    by[0] = (y0 >> sh) * g.nbx;
    by[1] = (y1 >> sh) * g.nbx;
    ly[0] = (y0 & m) << sh;
    ly[1] = (y1 & m) << sh;
    bz[0] = (z0 >> sh) * (g.nbx * g.nby);
    bz[1] = (z1 >> sh) * (g.nbx * g.nby);
    lz[0] = (z0 & m) << (2 * sh);
    lz[1] = (z1 & m) << (2 * sh);
  }
  __device__ __forceinline__ int block(int c) const { return bx + by[c & 1] + bz[c >> 1]; }
  __device__ __forceinline__ int voxel(int c) const { return lx + ly[c & 1] + lz[c >> 1]; }
};

// SparseGrid<uint16_t>::interpolateToFloat<IP_LINEAR> with OPT_IPBC_NEUMAN
// (src/sbg.h:1386, 2936-2941, 3111-3420) on the distance channel of level
// lv: cell-centred, the 2x2x2 window clamped to the grid, value blocks read
// their data, full blocks dTransRes*1024, the others 0; p1*t + p0*(1-t)
// along x, then y, then z.
// All lanes of a warp call it; `on` is the same in both lanes of a pair.
__device__ __forceinline__ float dist_interp(const MrGrid& g, int lv, bool on, int side, float px,
                                             float py, float pz) {
  const float x = __fsub_rn(px, 0.5f), y = __fsub_rn(py, 0.5f), z = __fsub_rn(pz, 0.5f);
  const int ix = (int)floorf(x), iy = (int)floorf(y), iz = (int)floorf(z);
  const float u = __fsub_rn(x, (float)ix), v = __fsub_rn(y, (float)iy),
              w = __fsub_rn(z, (float)iz);
  float c[4] = {0.f, 0.f, 0.f, 0.f};
  if (on) {
    const int nx = g.sx >> lv, ny = g.sy >> lv, nz = g.sz >> lv;
    const MrWindow win(g, lv, min(max(ix + side, 0), nx - 1), min(max(iy, 0), ny - 1),
                       min(max(iy + 1, 0), ny - 1), min(max(iz, 0), nz - 1),
                       min(max(iz + 1, 0), nz - 1));
    uint64_t key[4];
#pragma unroll
    for (int k = 0; k < 4; k++) key[k] = g.key[win.block(k)];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const int kd = key_kind(key[k], lv);
      if (kd == 1) c[k] = (float)g.dist[(int64_t)(key[k] >> KEY_OFF) + win.voxel(k)];
      if (kd == 2) c[k] = (float)(kDTransRes * 1024);
    }
  }
  const float u1 = __fsub_rn(1.0f, u), v1 = __fsub_rn(1.0f, v), w1 = __fsub_rn(1.0f, w);
  float e[4], f[2];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const float mine = __fmul_rn(c[k], side ? u : u1), other = pair_trade(mine);
    e[k] = __fadd_rn(mine, other);  // the same in either order
  }
#pragma unroll
  for (int k = 0; k < 2; k++) f[k] = __fadd_rn(__fmul_rn(e[2 * k + 1], v), __fmul_rn(e[2 * k], v1));
  return __fadd_rn(__fmul_rn(f[1], w), __fmul_rn(f[0], w1));
}

__device__ __constant__ float kMrOff[3][3] = {{0.f, 0.5f, 0.5f}, {0.5f, 0.f, 0.5f},
                                              {0.5f, 0.5f, 0.f}};

// Trilinear sum of component d at level lv, from the sample origin (ix0, iy0, iz0) and
// fractions (fx, fy, fz): that of vel in side 0, that of velOld in side 1.  Outside the
// grid, and in a block of another level, every value reads 0.  All lanes of a warp call
// it; `on` is the same in both lanes of a pair.
__device__ __forceinline__ float trilinear_pair(const MrGrid& g, int lv, bool on, int side,
                                                const float2* __restrict__ vel, int d, int ix0,
                                                int iy0, int iz0, float fx, float fy, float fz) {
  float2 v[4];
#pragma unroll
  for (int c = 0; c < 4; c++) v[c] = make_float2(0.f, 0.f);
  const int x = ix0 + side, nx = g.sx >> lv, ny = g.sy >> lv, nz = g.sz >> lv;
  if (on && (unsigned)x < (unsigned)nx) {
    const MrWindow win(g, lv, x, iy0, iy0 + 1, iz0, iz0 + 1);
    bool in[4];
    uint64_t key[4];
#pragma unroll
    for (int c = 0; c < 4; c++) {
      in[c] = (unsigned)(iy0 + (c & 1)) < (unsigned)ny && (unsigned)(iz0 + (c >> 1)) < (unsigned)nz;
      key[c] = in[c] ? g.key[win.block(c)] : 15;
    }
#pragma unroll
    for (int c = 0; c < 4; c++)
      if (key_level(key[c]) == lv)
        v[c] = vel[3 * ((int64_t)(key[c] >> KEY_OFF) + win.voxel(c)) + d];
  }
  const float wx = side ? fx : __fsub_rn(1.f, fx), gy = __fsub_rn(1.f, fy), gz = __fsub_rn(1.f, fz);
  float s = 0.f;
#pragma unroll
  for (int c = 0; c < 4; c++) {
    const float w = __fmul_rn(__fmul_rn(wx, c & 1 ? fy : gy), c >> 1 ? fz : gz);
    const float a = __fmul_rn(w, v[c].x), b = __fmul_rn(w, v[c].y);
    const float mine = side ? b : a, other = pair_trade(side ? a : b);
    s = __fadd_rn(s, side ? other : mine);  // x, then x + 1
    s = __fadd_rn(s, side ? mine : other);
  }
  return s;
}

// gridToParticle with interpCompMSBG per component (interpVec3MSBG yields the
// same per component: its shared path, taken when the three staggered
// samples share a block, computes exactly interpCompMSBG's expressions).
// la, lb: MtLinstep's bounds as the reference forms them in float.
// Bound by the gather: 16 M particles in no order over 57 M voxels (512^3, 3 levels,
// B200) took 9.8 ms as they came, every sector a miss; visited block by block, with the
// channels side by side, 3.5 ms, of which the order takes 0.4.  That was 2000
// instructions for 16 particles, most for windows that cross blocks, of which every warp
// has some: with a pair of lanes per particle 3.26 ms, and with one look-up of a block's key
// per corner, the same for all windows, 1.94 ms.  The same bits.
__global__ void __launch_bounds__(256) k_g2p_mr(msbg_flip_particle* __restrict__ p, int64_t np,
                                                MrGrid g, const float2* __restrict__ vel,
                                                BinsOrder order, float alpha, double la,
                                                double lb) {
  const int* perm = order.get();
  const int side = threadIdx.x & 1;
  const int64_t n0 = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 1;
  const int lane2 = (threadIdx.x & 31) >> 1;
  // the bound is the warp's: its lanes stay together for the trades
  for (int64_t n = n0; n - lane2 < np; n += ((int64_t)gridDim.x * blockDim.x) >> 1) {
    const bool valid = n < np;
    const int64_t k = valid ? (perm ? perm[n] : n) : 0;
    const msbg_flip_particle q = p[k];
    const bool finite = valid && isfinite(q.pos[0]) && isfinite(q.pos[1]) && isfinite(q.pos[2]);
    float out[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const float gx = __fsub_rn(q.pos[0], kMrOff[d][0]), gy = __fsub_rn(q.pos[1], kMrOff[d][1]),
                  gz = __fsub_rn(q.pos[2], kMrOff[d][2]);
      const int ix0 = (int)floorf(gx), iy0 = (int)floorf(gy), iz0 = (int)floorf(gz);
      const float fx = __fsub_rn(gx, (float)ix0), fy = __fsub_rn(gy, (float)iy0),
                  fz = __fsub_rn(gz, (float)iz0);
      int lv = 0;
      if (finite) {
        const int cx = min(max(ix0, 0), g.sx - 1), cy = min(max(iy0, 0), g.sy - 1),
                  cz = min(max(iz0, 0), g.sz - 1);
        lv = key_level(g.key[(cx >> g.sh0) + g.nbx * ((cy >> g.sh0) + g.nby * (cz >> g.sh0))]);
      }
      // pic in side 0, the old value in side 1
      float s = trilinear_pair(g, 0, finite, side, vel, d, ix0, iy0, iz0, fx, fy, fz);
      if (__any_sync(0xffffffffu, lv > 0)) {
        const bool on = lv > 0;
        const float scale = 1.f / (float)(1 << lv);  // a power of two: exact
        const float cgx = __fmul_rn(gx, scale), cgy = __fmul_rn(gy, scale),
                    cgz = __fmul_rn(gz, scale);
        const int cix0 = (int)floorf(cgx), ciy0 = (int)floorf(cgy), ciz0 = (int)floorf(cgz);
        const float c = trilinear_pair(g, lv, on, side, vel, d, cix0, ciy0, ciz0,
                                       __fsub_rn(cgx, (float)cix0), __fsub_rn(cgy, (float)ciy0),
                                       __fsub_rn(cgz, (float)ciz0));
        const float dist =
            __fmul_rn(dist_interp(g, lv, on, side, cgx, cgy, cgz), 1.0f / 1024.0f);
        if (on) {
          const double x = (double)dist;
          const float af = x < la ? 0.f : x >= lb ? 1.f : (float)((x - la) / (lb - la));
          s = __fadd_rn(__fmul_rn(af, s), __fmul_rn(__fsub_rn(1.f, af), c));
        }
      }
      if (!finite) s = 0.f;  // no cell for a particle without a finite position
      const float t = pair_trade(s), pic = side ? t : s, old = side ? s : t;
      out[d] = __fadd_rn(__fmul_rn(__fsub_rn(1.f, alpha), pic),
                         __fmul_rn(alpha, __fadd_rn(q.vel[d], __fsub_rn(pic, old))));
    }
    if (!valid) continue;
    if (side) {
      p[k].vel[2] = out[2];
    } else {
      p[k].vel[0] = out[0];
      p[k].vel[1] = out[1];
    }
  }
}

// downsampleVelocity (src/msbg4.cpp:2035-2270), MG level m-1 -> m, one CTA
// per block (grid-stride), its threads over the block's voxels.  Block b sits
// at level max(level0[b], m - 1) at MG level m-1 (offA) and max(level0[b], m)
// at MG level m (offB).  A block already at level >= m is copied (0 in SOLID
// or VOID cells); a block coarsened at this MG level takes per non-SOLID cell
// the 4x4x4 (1,3,3,1)^3/512 sum over the level-(m-1) cells 2x-1 .. 2x+2
// clamped to that level's grid, each from the level-(m-1) block where it is
// one at MG level m-1, else the level-m value at (x2/2, y2/2, z2/2), summed in
// the reference's order k, j, i without contraction.
__global__ void __launch_bounds__(256)
    k_downsample_velocity(int sx, int sy, int sz, int sh0, int nbx, int nby, int nbz, int m,
                          const int8_t* __restrict__ level0, const int64_t* __restrict__ offA,
                          const int64_t* __restrict__ offB, const uint16_t* __restrict__ flags,
                          const float* __restrict__ src, float* __restrict__ dst) {
  const int64_t nb = (int64_t)nbx * nby * nbz;
  const int fs = m - 1, nsx = sx >> fs, nsy = sy >> fs, nsz = sz >> fs, shA = sh0 - fs;
  for (int64_t b = blockIdx.x; b < nb; b += gridDim.x) {
    const int l0 = level0[b], lv = max(l0, m), sh = sh0 - lv, bs = 1 << sh;
    const int bx = (int)(b % nbx), by = (int)((b / nbx) % nby), bz = (int)(b / ((int64_t)nbx * nby));
    const int nv = bs * bs * bs;
    for (int v = threadIdx.x; v < nv; v += blockDim.x) {
      const uint16_t fl = flags[offB[b] + v];
      float* out = dst + 3 * (offB[b] + v);
      if (l0 >= m) {
        const float* in = src + 3 * (offA[b] + v);
        const bool zero = (fl & (0x1 | 0x1000)) != 0;  // CELL_SOLID | CELL_VOID
        out[0] = zero ? 0.f : in[0];
        out[1] = zero ? 0.f : in[1];
        out[2] = zero ? 0.f : in[2];
        continue;
      }
      float v0 = 0.f, v1 = 0.f, v2 = 0.f;
      if (!(fl & 0x1)) {
        const int x = bx * bs + (v & (bs - 1)), y = by * bs + ((v >> sh) & (bs - 1)),
                  z = bz * bs + (v >> (2 * sh));
        for (int k = 0; k < 4; k++) {
          const int z2 = min(max(2 * z - 1 + k, 0), nsz - 1);
          for (int j = 0; j < 4; j++) {
            const int y2 = min(max(2 * y - 1 + j, 0), nsy - 1);
#pragma unroll
            for (int i = 0; i < 4; i++) {
              const int x2 = min(max(2 * x - 1 + i, 0), nsx - 1);
              const int64_t b2 = (x2 >> shA) + (int64_t)nbx * ((y2 >> shA) + (int64_t)nby * (z2 >> shA));
              const int l2 = max((int)level0[b2], fs);  // its level at MG level m-1
              int64_t q = -1;
              if (l2 == fs) {
                const int mk = (1 << shA) - 1;
                q = offA[b2] + (x2 & mk) + ((int64_t)(y2 & mk) << shA) +
                    ((int64_t)(z2 & mk) << (2 * shA));
              } else if (l2 == fs + 1) {
                const int s2 = shA - 1, mk = (1 << s2) - 1;
                q = offA[b2] + ((x2 >> 1) & mk) + ((int64_t)((y2 >> 1) & mk) << s2) +
                    ((int64_t)((z2 >> 1) & mk) << (2 * s2));
              }
              const float w = (float)((i == 0 || i == 3 ? 1 : 3) * (j == 0 || j == 3 ? 1 : 3) *
                                      (k == 0 || k == 3 ? 1 : 3)) * (1.0f / 512.0f);
              const float f0 = q < 0 ? 0.f : src[3 * q], f1 = q < 0 ? 0.f : src[3 * q + 1],
                          f2 = q < 0 ? 0.f : src[3 * q + 2];
              v0 = __fadd_rn(v0, __fmul_rn(f0, w));
              v1 = __fadd_rn(v1, __fmul_rn(f1, w));
              v2 = __fadd_rn(v2, __fmul_rn(f2, w));
            }
          }
        }
      }
      out[0] = v0;
      out[1] = v1;
      out[2] = v2;
    }
  }
}

int grid_blocks(int64_t n) { return (int)std::min<int64_t>((n + 255) / 256, 148 * 32); }

// From how many particles on G2P looks whether it should order them.  As they come and ordered
// (512^3, 3 levels, 16^3 blocks, in no order, B200): 1 M 193 and 206 us, 4 M 658 and 575.
constexpr int64_t MR_BINS_MIN = 1 << 21;

// Floats of a channel that are on the device at a time on their way in or out (16 MB).
constexpr int64_t MR_PIECE = 4 << 20;

// One of the two interleaved channels: into it (get = 0) or out of it.
__global__ void __launch_bounds__(256) k_mr_channel(float2* __restrict__ vel, int which,
                                                    float* __restrict__ data, int64_t n, int get) {
  float* v = reinterpret_cast<float*>(vel) + which;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    if (get)
      data[i] = v[2 * i];
    else
      v[2 * i] = data[i];
  }
}

// The state of a context for its current topology (rebuilt when it changed).
// The reference asserts that 26-neighbour blocks differ by at most one level
// (src/msbg.cpp:1718-1719); such a map is rejected here.
int mr_state(msbg_gpu_ctx* ctx, MrState** out, MrGrid& g) {
  if (!ctx->bsx0 || ctx->nLevels < 1)
    return set_error(ctx, MSBG_EINVARG, "msbg_gpu_sync_topology not called");
  auto& sp = states()[ctx];
  if (!sp || sp->sx != ctx->sx || sp->sy != ctx->sy || sp->sz != ctx->sz ||
      sp->bsx0 != ctx->bsx0 || sp->nLevels != ctx->nLevels || sp->levels != ctx->blockLevel) {
    const int64_t nb = ctx->nb();
    for (int64_t b = 0; b < nb; b++) {
      const int bx = (int)(b % ctx->nbx), by = (int)((b / ctx->nbx) % ctx->nby),
                bz = (int)(b / ((int64_t)ctx->nbx * ctx->nby));
      for (int d = 0; d < 27; d++) {
        const int x = bx + d % 3 - 1, y = by + (d / 3) % 3 - 1, z = bz + d / 9 - 1;
        if (x < 0 || y < 0 || z < 0 || x >= ctx->nbx || y >= ctx->nby || z >= ctx->nbz) continue;
        const int l2 = ctx->blockLevel[x + (int64_t)ctx->nbx * (y + (int64_t)ctx->nby * z)];
        if (std::abs(l2 - ctx->blockLevel[b]) > 1)
          return set_error(ctx, MSBG_EINVARG,
                           "blocks %lld and a neighbour differ by more than one level",
                           (long long)b);
      }
    }
    std::unique_ptr<MrState> s(new MrState());
    s->sx = ctx->sx;
    s->sy = ctx->sy;
    s->sz = ctx->sz;
    s->bsx0 = ctx->bsx0;
    s->nLevels = ctx->nLevels;
    s->levels = ctx->blockLevel;
    std::vector<int8_t> lv8(nb);
    std::vector<int64_t> off(nb);
    int64_t o = 0;
    for (int64_t b = 0; b < nb; b++) {
      lv8[b] = (int8_t)ctx->blockLevel[b];
      off[b] = o;
      const int64_t bs = ctx->bsx0 >> ctx->blockLevel[b];
      o += bs * bs * bs;
    }
    s->n = o;
    cudaStream_t st = ctx->stream;
    MSBG_CUDA_TRY(ctx, s->level.ensure(nb));
    MSBG_CUDA_TRY(ctx, s->off.ensure(8 * nb));
    MSBG_CUDA_TRY(ctx, s->fc.ensure(nb));
    MSBG_CUDA_TRY(ctx, s->kind.ensure((size_t)nb * ctx->nLevels));
    MSBG_CUDA_TRY(ctx, s->key.ensure(8 * nb));
    MSBG_CUDA_TRY(ctx, s->dist.ensure(2 * (size_t)o));
    MSBG_CUDA_TRY(ctx, s->vel.ensure(24 * (size_t)o));
    MSBG_CUDA_TRY(ctx, cudaMemcpyAsync(s->level.p, lv8.data(), nb, cudaMemcpyHostToDevice, st));
    MSBG_CUDA_TRY(ctx, cudaMemcpyAsync(s->off.p, off.data(), 8 * nb, cudaMemcpyHostToDevice, st));
    MSBG_CUDA_TRY(ctx, cudaMemsetAsync(s->vel.p, 0, s->vel.bytes, st));
    // the host vectors are read by the copies above before they go out of scope
    MSBG_CUDA_TRY(ctx, cudaStreamSynchronize(st));
    sp = std::move(s);
  }
  MrState& S = *sp;
  int sh = 0;
  while ((1 << sh) < ctx->bsx0) sh++;
  g = MrGrid{S.sx, S.sy, S.sz, sh, ctx->nbx, ctx->nby, ctx->nbz, S.nLevels,
             S.level.as<int8_t>(), S.off.as<int64_t>(), S.kind.as<int8_t>(),
             S.dist.as<uint16_t>(), S.key.as<uint64_t>()};
  *out = sp.get();
  return MSBG_OK;
}

int mr_build_dist(msbg_gpu_ctx* ctx, MrState* S, const MrGrid& g) {
  if (S->distBuilt) return MSBG_OK;
  const int64_t nb = ctx->nb();
  cudaStream_t st = ctx->stream;
  k_mr_fine_coarse<<<grid_blocks(nb), 256, 0, st>>>(S->level.as<int8_t>(), ctx->nbx, ctx->nby,
                                                     ctx->nbz, S->fc.as<int8_t>());
  k_mr_kind<<<grid_blocks(nb * S->nLevels), 256, 0, st>>>(S->level.as<int8_t>(),
                                                           S->fc.as<int8_t>(), ctx->nbx, ctx->nby,
                                                           ctx->nbz, S->nLevels,
                                                           S->kind.as<int8_t>());
  k_mr_dist<<<(int)std::min<int64_t>(nb, 148 * 16), 256, 0, st>>>(g, S->fc.as<int8_t>(),
                                                                   S->dist.as<uint16_t>());
  k_mr_key<<<grid_blocks(nb), 256, 0, st>>>(g, S->key.as<uint64_t>());
  MSBG_CUDA_TRY(ctx, cudaGetLastError());
  S->distBuilt = true;
  return MSBG_OK;
}

}  // namespace

void flip_mr_release(msbg_gpu_ctx* ctx) { states().erase(ctx); }

}  // namespace msbg

using namespace msbg;

extern "C" int msbg_gpu_flip_mr_dist(msbg_gpu_ctx* ctx, uint16_t* dist, int64_t n, int8_t* kind,
                                     int64_t nk) {
  if (!ctx) return MSBG_EINVARG;
  cudaSetDevice(ctx->device);
  MrState* S = nullptr;
  MrGrid g;
  int rc = mr_state(ctx, &S, g);
  if (rc) return rc;
  if (dist && n != S->n)
    return set_error(ctx, MSBG_EINVARG, "distance channel holds %lld voxels, not %lld",
                     (long long)S->n, (long long)n);
  if (kind && nk != ctx->nb() * S->nLevels)
    return set_error(ctx, MSBG_EINVARG, "block kinds: %lld entries, not %lld",
                     (long long)(ctx->nb() * S->nLevels), (long long)nk);
  rc = mr_build_dist(ctx, S, g);
  if (rc) return rc;
  if (dist)
    MSBG_CUDA_TRY(ctx, cudaMemcpyAsync(dist, S->dist.p, 2 * (size_t)n, cudaMemcpyDeviceToHost,
                                       ctx->stream));
  if (kind)
    MSBG_CUDA_TRY(ctx, cudaMemcpyAsync(kind, S->kind.p, (size_t)nk, cudaMemcpyDeviceToHost,
                                       ctx->stream));
  return msbg_gpu_sync(ctx);
}

extern "C" int msbg_gpu_flip_mr_channel(msbg_gpu_ctx* ctx, int which, float* data, int64_t n,
                                        int get) {
  if (!ctx || !data) return MSBG_EINVARG;
  cudaSetDevice(ctx->device);
  MrState* S = nullptr;
  MrGrid g;
  int rc = mr_state(ctx, &S, g);
  if (rc) return rc;
  if (which != MSBG_FLIP_VEL && which != MSBG_FLIP_VEL_OLD)
    return set_error(ctx, MSBG_EINVARG, "mixed-resolution channel %d unknown", which);
  if (n != 3 * S->n)
    return set_error(ctx, MSBG_EINVARG, "mixed-resolution channel holds %lld floats, not %lld",
                     (long long)(3 * S->n), (long long)n);
  const int w = which == MSBG_FLIP_VEL ? 0 : 1;
  cudaStream_t st = ctx->stream;
  if (S->scratch.ensure(sizeof(float) * std::min(n, MR_PIECE)) != cudaSuccess) {
    cudaGetLastError();  // no room for a piece: value by value
    float* v = S->vel.as<float>() + w;
    MSBG_CUDA_TRY(ctx, get ? cudaMemcpy2DAsync(data, 4, v, 8, 4, n, cudaMemcpyDeviceToHost, st)
                           : cudaMemcpy2DAsync(v, 8, data, 4, 4, n, cudaMemcpyHostToDevice, st));
    return msbg_gpu_sync(ctx);
  }
  float* piece = S->scratch.as<float>();
  for (int64_t o = 0; o < n; o += MR_PIECE) {
    const int64_t m = std::min(n - o, MR_PIECE);
    if (!get)
      MSBG_CUDA_TRY(ctx, cudaMemcpyAsync(piece, data + o, sizeof(float) * m,
                                         cudaMemcpyHostToDevice, st));
    k_mr_channel<<<grid_blocks(m), 256, 0, st>>>(S->vel.as<float2>() + o, w, piece, m, get);
    MSBG_CUDA_TRY(ctx, cudaGetLastError());
    if (get)
      MSBG_CUDA_TRY(ctx, cudaMemcpyAsync(data + o, piece, sizeof(float) * m,
                                         cudaMemcpyDeviceToHost, st));
  }
  return msbg_gpu_sync(ctx);
}

namespace {
int flip_g2p_mr(msbg_gpu_ctx* ctx, msbg_flip_particle* particles, int64_t np, float flipAlpha,
                bool onDevice) {
  if (!ctx || (!particles && np) || np < 0) return MSBG_EINVARG;
  cudaSetDevice(ctx->device);
  MrState* S = nullptr;
  MrGrid g;
  int rc = mr_state(ctx, &S, g);
  if (rc) return rc;
  rc = mr_build_dist(ctx, S, g);
  if (rc) return rc;
  if (!np) return msbg_gpu_sync(ctx);
  cudaStream_t st = ctx->stream;
  msbg_flip_particle* dp = particles;
  if (!onDevice) {
    MSBG_CUDA_TRY(ctx, S->parts.ensure(sizeof(msbg_flip_particle) * (size_t)np));
    MSBG_CUDA_TRY(ctx, cudaMemcpyAsync(S->parts.p, particles, sizeof(msbg_flip_particle) * np,
                                       cudaMemcpyHostToDevice, st));
    dp = S->parts.as<msbg_flip_particle>();
  }
  // MtLinstep's bounds as interpCompMSBG forms them, in float
  // (src/flip_sim.cpp:1514-1521): stenWidth 2, MT_SQRT3F
  const float sqrt3 = 1.73205080756887f;
  const float la = (1.0f * sqrt3) * 1.01f, lb = (0.99f * ((float)kDTransRes + 2.f)) / sqrt3;
  BinsOrder order;
  if (np >= MR_BINS_MIN)
    MSBG_CUDA_TRY(ctx, bins_build(S->scratch, dp, np, BinsGrid{g.sx, g.sy, g.sz, g.sh0, g.nbx, g.nby},
                                  ctx->nb(), 26.0 * (double)S->n / (double)ctx->nb(), st, order));
  k_g2p_mr<<<grid_blocks(2 * np), 256, 0, st>>>(dp, np, g, S->vel.as<float2>(), order, flipAlpha,
                                            (double)la, (double)lb);
  MSBG_CUDA_TRY(ctx, cudaGetLastError());
  if (!onDevice)
    MSBG_CUDA_TRY(ctx, cudaMemcpyAsync(particles, dp, sizeof(msbg_flip_particle) * np,
                                       cudaMemcpyDeviceToHost, st));
  return msbg_gpu_sync(ctx);
}
}  // namespace

extern "C" int msbg_gpu_flip_g2p_mr(msbg_gpu_ctx* ctx, msbg_flip_particle* particles, int64_t np,
                                    float flipAlpha) {
  return flip_g2p_mr(ctx, particles, np, flipAlpha, false);
}

extern "C" int msbg_gpu_flip_g2p_mr_device(msbg_gpu_ctx* ctx, msbg_flip_particle* particles,
                                           int64_t np, float flipAlpha) {
  return flip_g2p_mr(ctx, particles, np, flipAlpha, true);
}

extern "C" int msbg_gpu_flip_downsample_velocity(msbg_gpu_ctx* ctx, int levelMg,
                                                 const uint16_t* flags, const float* src,
                                                 int64_t nSrc, float* dst, int64_t nDst) {
  if (!ctx || !flags || !src || !dst) return MSBG_EINVARG;
  cudaSetDevice(ctx->device);
  MrState* S = nullptr;
  MrGrid g;
  int rc = mr_state(ctx, &S, g);
  if (rc) return rc;
  if (levelMg < 1 || levelMg >= ctx->nLevels)
    return set_error(ctx, MSBG_EINVARG, "levelMg=%d: the sparse MG levels are 1..%d", levelMg,
                     ctx->nLevels - 1);
  const int64_t nb = ctx->nb();
  std::vector<int64_t> offA(nb), offB(nb);
  int64_t nA = 0, nB = 0;
  for (int64_t b = 0; b < nb; b++) {
    const int l0 = ctx->blockLevel[b];
    const int64_t bsA = ctx->bsx0 >> std::max(l0, levelMg - 1), bsB = ctx->bsx0 >> std::max(l0, levelMg);
    offA[b] = nA;
    offB[b] = nB;
    nA += bsA * bsA * bsA;
    nB += bsB * bsB * bsB;
  }
  if (nSrc != 3 * nA || nDst != 3 * nB)
    return set_error(ctx, MSBG_EINVARG,
                     "MG levels %d / %d hold %lld / %lld floats, not %lld / %lld", levelMg - 1,
                     levelMg, (long long)(3 * nA), (long long)(3 * nB), (long long)nSrc,
                     (long long)nDst);
  cudaStream_t st = ctx->stream;
  MSBG_CUDA_TRY(ctx, S->dsOffA.ensure(8 * nb));
  MSBG_CUDA_TRY(ctx, S->dsOffB.ensure(8 * nb));
  MSBG_CUDA_TRY(ctx, S->dsFlags.ensure(2 * (size_t)nB));
  MSBG_CUDA_TRY(ctx, S->dsSrc.ensure(12 * (size_t)nA));
  MSBG_CUDA_TRY(ctx, S->dsDst.ensure(12 * (size_t)nB));
  MSBG_CUDA_TRY(ctx, cudaMemcpyAsync(S->dsOffA.p, offA.data(), 8 * nb, cudaMemcpyHostToDevice, st));
  MSBG_CUDA_TRY(ctx, cudaMemcpyAsync(S->dsOffB.p, offB.data(), 8 * nb, cudaMemcpyHostToDevice, st));
  MSBG_CUDA_TRY(ctx, cudaMemcpyAsync(S->dsFlags.p, flags, 2 * nB, cudaMemcpyHostToDevice, st));
  MSBG_CUDA_TRY(ctx, cudaMemcpyAsync(S->dsSrc.p, src, 12 * nA, cudaMemcpyHostToDevice, st));
  k_downsample_velocity<<<(int)std::min<int64_t>(nb, 148 * 16), 256, 0, st>>>(
      ctx->sx, ctx->sy, ctx->sz, g.sh0, ctx->nbx, ctx->nby, ctx->nbz, levelMg,
      S->level.as<int8_t>(), S->dsOffA.as<int64_t>(), S->dsOffB.as<int64_t>(),
      S->dsFlags.as<uint16_t>(), S->dsSrc.as<float>(), S->dsDst.as<float>());
  MSBG_CUDA_TRY(ctx, cudaGetLastError());
  MSBG_CUDA_TRY(ctx, cudaMemcpyAsync(dst, S->dsDst.p, 12 * nB, cudaMemcpyDeviceToHost, st));
  // the offset vectors are read by the copies above before they go out of scope
  return msbg_gpu_sync(ctx);
}
