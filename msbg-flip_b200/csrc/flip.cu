// FLIP transfers around the pressure solve, on the context's single-level
// grid (every block at level 0, all blocks present), device-resident grid
// channels in the block layout (blocks in bid order, bsx^3 voxels, vid =
// x + y*bsx + z*bsx^2; vector channels hold the lower-face u, v, w of each
// voxel):
//   msbg_gpu_flip_p2g              FlipSimulation::particleToGrid
//                                  (src/flip_sim.cpp:579-831)
//   msbg_gpu_flip_gravity          applyGravity (src/flip_sim.cpp:832-857)
//   msbg_gpu_flip_pressure_gradient the pressure-gradient update of
//                                  pressureProjection (src/flip_sim.cpp:1316-1349)
//   msbg_gpu_flip_g2p              gridToParticle with the level-0 branch of
//                                  interpVec3MSBG (src/flip_sim.cpp:1354-1395, 1526-1545)
// The scatter of P2G sums in an order that varies from run to run (as the
// reference's thread-local merge does); every other step is one thread per voxel face
// or per particle, with the reference's expressions in its order and no contraction
// into FMAs.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdint>
#include <map>
#include <memory>
#include <type_traits>
#include <vector>

#include "common.cuh"

namespace msbg {
namespace {

#include "particle_bins.cuh"

struct FlipState {
  int sx = 0, sy = 0, sz = 0, bsx = 0;
  int64_t n = 0;
  DeviceBuffer vel, velOld, beta, mass, liq, acc, active, parts;
  // P2G cell by cell: the particles' ranks and the list; G2P's visiting order.
  // (acc also takes G2P's side-by-side copy of vel and velOld.)
  DeviceBuffer lists;
};

std::map<msbg_gpu_ctx*, std::unique_ptr<FlipState>>& states() {
  static std::map<msbg_gpu_ctx*, std::unique_ptr<FlipState>> m;
  return m;
}

struct GridF {
  int sx, sy, sz, sh, nbx, nby;
  // voxel index in the block layout, or -1 outside the grid
  __device__ __forceinline__ int64_t idx(int x, int y, int z) const {
    if (x < 0 || y < 0 || z < 0 || x >= sx || y >= sy || z >= sz) return -1;
    const int m = (1 << sh) - 1;
    // (block ids are ints: 64 bits only for the voxel)
    const int bid = (x >> sh) + nbx * ((y >> sh) + nby * (z >> sh));
    return ((int64_t)bid << (3 * sh)) + ((x & m) + ((y & m) << sh) + ((z & m) << (2 * sh)));
  }
  // voxel coordinates of block-layout index i
  __device__ __forceinline__ void coords(int64_t i, int& x, int& y, int& z) const {
    const int m = (1 << sh) - 1;
    const unsigned bid = (unsigned)(i >> (3 * sh));
    const int v = (int)(i & ((1 << (3 * sh)) - 1));
    const unsigned row = bid / (unsigned)nbx, bz = row / (unsigned)nby;
    x = (int)(bid - row * nbx) * (1 << sh) + (v & m);
    y = (int)(row - bz * nby) * (1 << sh) + ((v >> sh) & m);
    z = (int)bz * (1 << sh) + (v >> (2 * sh));
  }
};

__device__ __constant__ float kOff[3][3] = {{0.f, 0.5f, 0.5f}, {0.5f, 0.f, 0.5f},
                                            {0.5f, 0.5f, 0.f}};

// The trilinear face weights of one particle, scattered with float atomics.
// acc: [vx vy vz wu wv ww ru rv rw][n].
__device__ __forceinline__ void scatter_faces(const msbg_flip_particle& q, const GridF& g,
                                              int64_t n, float mp, float* __restrict__ acc) {
#pragma unroll
  for (int d = 0; d < 3; d++) {
    const float gx = __fsub_rn(q.pos[0], kOff[d][0]), gy = __fsub_rn(q.pos[1], kOff[d][1]),
                gz = __fsub_rn(q.pos[2], kOff[d][2]);
    const int ix0 = (int)floorf(gx), iy0 = (int)floorf(gy), iz0 = (int)floorf(gz);
    const float fx = __fsub_rn(gx, (float)ix0), fy = __fsub_rn(gy, (float)iy0),
                fz = __fsub_rn(gz, (float)iz0);
#pragma unroll
    for (int c = 0; c < 8; c++) {
      const int dx = c & 1, dy = (c >> 1) & 1, dz = c >> 2;
      const float w = __fmul_rn(__fmul_rn(dx ? fx : __fsub_rn(1.f, fx), dy ? fy : __fsub_rn(1.f, fy)),
                                dz ? fz : __fsub_rn(1.f, fz));
      const int64_t i = g.idx(ix0 + dx, iy0 + dy, iz0 + dz);
      if (i < 0) continue;
      atomicAdd(&acc[(size_t)d * n + i], __fmul_rn(q.vel[d], w));
      atomicAdd(&acc[(size_t)(3 + d) * n + i], w);
      atomicAdd(&acc[(size_t)(6 + d) * n + i], __fmul_rn(mp, w));
    }
  }
}

__device__ __forceinline__ bool finite_pos(const msbg_flip_particle& q) {
  return isfinite(q.pos[0]) && isfinite(q.pos[1]) && isfinite(q.pos[2]);
}

// The particles' cell mass and face weights (particleToGrid's scatter loop), particle by
// particle: for few particles.
__global__ void k_p2g_scatter(const msbg_flip_particle* __restrict__ p, int64_t np, GridF g,
                              int64_t n, float rhoL, float rhoG, float* __restrict__ acc,
                              float* __restrict__ mass, int* __restrict__ liq) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < np;
       k += (int64_t)gridDim.x * blockDim.x) {
    const msbg_flip_particle q = p[k];
    // a particle without a finite position reaches no cell
    if (!finite_pos(q)) continue;
    const int64_t ci = g.idx((int)floorf(q.pos[0]), (int)floorf(q.pos[1]), (int)floorf(q.pos[2]));
    if (ci >= 0) {
      atomicAdd(&mass[ci], 1.f);
      if (q.phase == 0) atomicAdd(&liq[ci], 1);
    }
    scatter_faces(q, g, n, q.phase == 0 ? rhoL : rhoG, acc);
  }
}

// Many particles, where they lie close: cell by cell.  Scattering them one by one costs 72 float
// atomics each, at 400 G atomics/s the bound of the pass (13.3 M particles on 160^3 cells, B200:
// 2.2 of P2G's 2.5 ms).  Here, for boxes of 8 x 8 x 4 cells,
//   k_p2g_sample counts one particle of 32 of each box and lists the boxes that count as
//                crowded;
//   k_p2g_count  gives each particle of a crowded box its cell and its rank there, and counts the
//                cells' particles.  The others are scattered here: particles of other boxes,
//                those that a cell has beyond P2G_CELL_MAX, and those outside the grid, which
//                reach its boundary faces alone;
//   k_p2g_start, k_p2g_place  list the particles of crowded boxes cell by cell (indices; the
//                particles stay where they are);
//   k_p2g_cells  a CTA per crowded box, a thread per cell: a cell's particles reach 2 x 3 x
//                3 faces per direction, whose three sums the thread keeps in registers;
//                they go to the CTA's faces in shared memory one neighbour
//                offset at a time, in which no two threads meet, and from there to the
//                grid with one float atomic per face and sum.  A box whose particles lie in
//                few of its cells is scattered after all.
constexpr int SUB = 8, SUB_Z = 4, SUB_T = SUB * SUB * SUB_Z;

// A box counts as crowded from P2G_CROWDED sampled particles on.
constexpr int P2G_SAMPLE = 32, P2G_CROWDED = 8;

// Scattering a box's particles takes 27 ns each of an SM's share of the atomics; summing them
// takes its CTA, one of three on the SM, 54 barriers (5 us) and 1.2 us for each particle of
// its fullest cell.
__device__ __forceinline__ bool box_pays(int particles, int fullest) {
  return particles >= 64 + 16 * fullest;
}

// A cell's particles that its thread sums: a chain of dependent loads, 0.4 us each, that its
// CTA waits for; a clump of any size ends there.
constexpr int P2G_CELL_MAX = 32;

// The cell of a particle with a finite position, -1 outside the grid, and its box.
__device__ __forceinline__ int64_t cell_of(const msbg_flip_particle& q, const GridF& g, int& box) {
  const int x = (int)floorf(q.pos[0]), y = (int)floorf(q.pos[1]), z = (int)floorf(q.pos[2]);
  const int64_t ci = g.idx(x, y, z);
  box = ci < 0 ? 0 : x / SUB + g.sx / SUB * (y / SUB + g.sy / SUB * (z / SUB_Z));
  return ci;
}

struct P2GBoxes {
  int* cnt;      // [boxes] sampled particles
  int* n;        // crowded boxes, then the cursor of the particles' list
  int* crowded;  // [boxes] their ids
  int* start;    // [n] first entry of a cell of a crowded box
};

__global__ void __launch_bounds__(256) k_p2g_sample(const msbg_flip_particle* __restrict__ p,
                                                    int64_t np, GridF g, P2GBoxes B) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < np / P2G_SAMPLE;
       i += (int64_t)gridDim.x * blockDim.x) {
    // one of 32, no fixed one: programs lay particles out with strides of their own
    const msbg_flip_particle& q = p[i * P2G_SAMPLE + (((unsigned)i * 0x9e3779b1u) >> 27)];
    if (!finite_pos(q)) continue;
    int box;
    if (cell_of(q, g, box) >= 0 && atomicAdd(&B.cnt[box], 1) == P2G_CROWDED - 1)
      B.crowded[atomicAdd(&B.n[0], 1)] = box;
  }
}

// mass counts in float where a box is not crowded, in int where it is; liq leaves the listed
// particles to k_p2g_cells, which turns mass into floats too.
__global__ void __launch_bounds__(256) k_p2g_count(const msbg_flip_particle* __restrict__ p,
                                                   int64_t np, GridF g, int64_t n, float rhoL,
                                                   float rhoG, P2GBoxes B, float* __restrict__ mass,
                                                   int* __restrict__ liq, int2* __restrict__ place,
                                                   float* __restrict__ acc) {
  const bool any = B.n[0] > 0;
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < np;
       k += (int64_t)gridDim.x * blockDim.x) {
    const msbg_flip_particle& q = p[k];
    const bool finite = finite_pos(q);
    int box = 0;
    const int64_t ci = finite ? cell_of(q, g, box) : -1;
    int2 at = make_int2(-1, 0);
    if (ci >= 0) {
      if (B.cnt[box] >= P2G_CROWDED) {
        at.y = atomicAdd(reinterpret_cast<int*>(mass) + ci, 1);
        if ((unsigned)at.y < P2G_CELL_MAX) at.x = (int)ci;
      } else {
        atomicAdd(&mass[ci], 1.f);
      }
      if (q.phase == 0 && at.x < 0) atomicAdd(&liq[ci], 1);
    }
    if (any) place[k] = at;
    if (finite && at.x < 0) scatter_faces(q, g, n, q.phase == 0 ? rhoL : rhoG, acc);
  }
}

// Cell of thread t in a box, and its place in the block layout.
__device__ __forceinline__ int64_t box_cell(const GridF& g, int box, int t, int& bx, int& by, int& bz,
                                            int& x, int& y, int& z) {
  const int nsx = g.sx / SUB, nsy = g.sy / SUB;
  bx = box % nsx * SUB;
  by = box / nsx % nsy * SUB;
  bz = box / (nsx * nsy) * SUB_Z;
  x = bx + t % SUB;
  y = by + t / SUB % SUB;
  z = bz + t / (SUB * SUB);
  return g.idx(x, y, z);
}

// First entries of the cells of the crowded boxes in perm, box by box in any order.
__global__ void __launch_bounds__(SUB_T) k_p2g_start(GridF g, P2GBoxes B,
                                                     const float* __restrict__ mass) {
  __shared__ int sum[SUB_T / 32], base;
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  for (int i = blockIdx.x; i < B.n[0]; i += gridDim.x) {
    int bx, by, bz, x, y, z;
    const int64_t c = box_cell(g, B.crowded[i], t, bx, by, bz, x, y, z);
    const int v = min(reinterpret_cast<const int*>(mass)[c], P2G_CELL_MAX);
    int s = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += u;
    }
    if (lane == 31) sum[w] = s;
    __syncthreads();
    int before = 0;
    for (int k = 0; k < w; k++) before += sum[k];
    if (t == SUB_T - 1) base = atomicAdd(&B.n[1], before + s);
    __syncthreads();
    B.start[c] = base + before + s - v;
    __syncthreads();  // sum and base are read
  }
}

__global__ void __launch_bounds__(256) k_p2g_place(int64_t np, const int2* __restrict__ place,
                                                   P2GBoxes B, int* __restrict__ perm) {
  if (B.n[0] == 0) return;  // place is not written
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < np;
       k += (int64_t)gridDim.x * blockDim.x) {
    const int2 at = place[k];
    if (at.x >= 0) perm[B.start[at.x] + at.y] = (int)k;
  }
}

// A thread needs 54 sums and so close to 80 registers: three CTAs of this size share an SM, of
// 8^3 cells it holds one, which waits out its loads and barriers alone (0.66 ms for 13.3 M
// particles on 160^3 cells; 0.56 this way).
constexpr int FACE_ROW = SUB + 2, FACES = FACE_ROW * FACE_ROW * (SUB_Z + 2);

// Direction D: faces of cell (x, y, z) at offset 0, 1 along D and -1, 0, 1 along the others.
// Returns the number of liquid particles.
template <int D>
__device__ __forceinline__ int p2g_direction(const msbg_flip_particle* __restrict__ p,
                                              const int* __restrict__ list, int cnt, int x, int y,
                                              int z, int at, float rhoL, float rhoG,
                                              float (*sums)[FACES]) {
  constexpr int NX = D == 0 ? 2 : 3, NY = D == 1 ? 2 : 3, NZ = D == 2 ? 2 : 3;
  constexpr int X0 = D == 0 ? 0 : -1, Y0 = D == 1 ? 0 : -1, Z0 = D == 2 ? 0 : -1;
  float v[NX * NY * NZ], w[NX * NY * NZ], r[NX * NY * NZ];
#pragma unroll
  for (int i = 0; i < NX * NY * NZ; i++) v[i] = w[i] = r[i] = 0.f;
  int liquid = 0;
  for (int m = 0; m < cnt; m++) {
    const msbg_flip_particle& q = p[list[m]];
    liquid += q.phase == 0;
    const float mp = q.phase == 0 ? rhoL : rhoG, u = q.vel[D];
    // the weights along an axis: of the particle's two faces, 0 for a third
    auto axis = [](float pos, float off, int cell, int i0, int ni, float* out) -> int {
      const float gp = __fsub_rn(pos, off);
      const int b = (int)floorf(gp);
      const float f = __fsub_rn(gp, (float)b), e = __fsub_rn(1.f, f);
      const int lo = b - cell - i0;  // place of the lower face
#pragma unroll
      for (int i = 0; i < 3; i++)
        if (i < ni) out[i] = i == lo ? e : i == lo + 1 ? f : 0.f;
      return lo;
    };
    float wx[3], wy[3], wz[3];
    const int lx = axis(q.pos[0], D == 0 ? 0.f : 0.5f, x, X0, NX, wx);
    const int ly = axis(q.pos[1], D == 1 ? 0.f : 0.5f, y, Y0, NY, wy);
    const int lz = axis(q.pos[2], D == 2 ? 0.f : 0.5f, z, Z0, NZ, wz);
#pragma unroll
    for (int k = 0; k < NZ; k++)
#pragma unroll
      for (int j = 0; j < NY; j++)
#pragma unroll
        for (int i = 0; i < NX; i++) {
          const float a = __fmul_rn(__fmul_rn(wx[i], wy[j]), wz[k]);
          const int e = i + NX * (j + NY * k);
          // (a velocity that is not finite reaches its own eight faces alone)
          if ((unsigned)(i - lx) < 2u && (unsigned)(j - ly) < 2u && (unsigned)(k - lz) < 2u)
            v[e] = fmaf(u, a, v[e]);
          w[e] += a;
          r[e] = fmaf(mp, a, r[e]);
        }
  }
#pragma unroll
  for (int k = 0; k < NZ; k++)
#pragma unroll
    for (int j = 0; j < NY; j++)
#pragma unroll
      for (int i = 0; i < NX; i++) {
        const int o = at + (i + X0) + FACE_ROW * ((j + Y0) + FACE_ROW * (k + Z0));
        const int e = i + NX * (j + NY * k);
        if (cnt) {
          sums[0][o] += v[e];
          sums[1][o] += w[e];
          sums[2][o] += r[e];
        }
        __syncthreads();
      }
  return liquid;
}

__global__ void __launch_bounds__(SUB_T, 3) k_p2g_cells(
    const msbg_flip_particle* __restrict__ p, GridF g, int64_t n, float rhoL, float rhoG, P2GBoxes B,
    float* __restrict__ mass, int* __restrict__ liq, const int* __restrict__ perm,
    float* __restrict__ acc) {
  __shared__ float sums[3][FACES];
  __shared__ int total, fullest, first;
  const int t = threadIdx.x;
  for (int i = blockIdx.x; i < B.n[0]; i += gridDim.x) {
    int bx, by, bz, x, y, z;
    const int64_t ci = box_cell(g, B.crowded[i], t, bx, by, bz, x, y, z);
    const int all = reinterpret_cast<const int*>(mass)[ci], m = min(all, P2G_CELL_MAX);
    mass[ci] = (float)all;
    if (t == 0) {
      total = fullest = 0;
      first = B.start[ci];
    }
    __syncthreads();
    const int wm = __reduce_max_sync(0xffffffffu, m), ws = __reduce_add_sync(0xffffffffu, m);
    if ((t & 31) == 0) {
      atomicAdd(&total, ws);
      atomicMax(&fullest, wm);
    }
    __syncthreads();
    if (!box_pays(total, fullest)) {  // its particles, one after the other in perm
      for (int k = t; k < total; k += SUB_T) {
        const msbg_flip_particle& q = p[perm[first + k]];
        int box;
        if (q.phase == 0) atomicAdd(&liq[cell_of(q, g, box)], 1);
        scatter_faces(q, g, n, q.phase == 0 ? rhoL : rhoG, acc);
      }
      __syncthreads();  // total is read
      continue;
    }
    const int* list = perm + B.start[ci];
    const int at = (x - bx + 1) + FACE_ROW * ((y - by + 1) + FACE_ROW * (z - bz + 1));
    auto direction = [&](auto dd) {
      constexpr int D = decltype(dd)::value;
      for (int q = t; q < 3 * FACES; q += SUB_T) sums[q / FACES][q % FACES] = 0.f;
      __syncthreads();
      const int liquid = p2g_direction<D>(p, list, m, x, y, z, at, rhoL, rhoG, sums);
      if (D == 0 && liquid) liq[ci] += liquid;
      for (int q = t; q < FACES; q += SUB_T) {
        const float w = sums[1][q];
        const float v = sums[0][q], r = sums[2][q];
        if (w == 0.f && v == 0.f && r == 0.f) continue;
        const int64_t f = g.idx(bx + q % FACE_ROW - 1, by + q / FACE_ROW % FACE_ROW - 1,
                                bz + q / (FACE_ROW * FACE_ROW) - 1);
        if (f < 0) continue;
        atomicAdd(&acc[(size_t)D * n + f], v);
        atomicAdd(&acc[(size_t)(3 + D) * n + f], w);
        atomicAdd(&acc[(size_t)(6 + D) * n + f], r);
      }
      __syncthreads();
    };
    direction(std::integral_constant<int, 0>{});
    direction(std::integral_constant<int, 1>{});
    direction(std::integral_constant<int, 2>{});
  }
}

struct P2GConst {
  float massEps, rhoL, rhoG, betaMin, rtMin, phiDen;
};

// Phase of a cell for the interface clamp: -1 empty or outside, 0 liquid
// (more than half of its particles liquid), 1 air.
__device__ __forceinline__ int cell_phase(const GridF& g, const float* mass, const int* liq,
                                          float eps, int x, int y, int z) {
  const int64_t j = g.idx(x, y, z);
  if (j < 0 || !(mass[j] > eps)) return -1;
  return liq[j] * 2 > (int)__fadd_rn(mass[j], 0.5f) ? 0 : 1;
}

// Face velocities normalised by their weights; beta = max(1/rho, betaMin)
// from the two-phase density, clamped where both cells of a face agree; the
// blocks holding mass.
__global__ void k_p2g_finish(GridF g, int64_t n, P2GConst c, const float* __restrict__ acc,
                             const float* __restrict__ mass, const int* __restrict__ liq,
                             float* __restrict__ vel, float* __restrict__ beta,
                             int* __restrict__ active) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    int x, y, z;
    g.coords(i, x, y, z);
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const float w = acc[(size_t)(3 + d) * n + i];
      vel[3 * i + d] = w > c.massEps ? __fdiv_rn(acc[(size_t)d * n + i], w) : 0.f;
    }
    if (mass[i] > c.massEps) active[i >> (3 * g.sh)] = 1;
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const float rt = acc[(size_t)(6 + d) * n + i];
      float phi = 0.f;
      if (!(rt < c.rtMin)) phi = fminf(__fsqrt_rn(__fdiv_rn(fmaxf(__fsub_rn(rt, c.rtMin), 0.f), c.phiDen)), 1.f);
      const int pa = cell_phase(g, mass, liq, c.massEps, x - (d == 0), y - (d == 1), z - (d == 2));
      const int pb = cell_phase(g, mass, liq, c.massEps, x, y, z);
      if (pa == 0 && pb == 0)
        phi = 1.f;
      else if (pa == 1 && pb == 1)
        phi = 0.f;
      const float rho = __fadd_rn(c.rhoG, __fmul_rn(phi, __fsub_rn(c.rhoL, c.rhoG)));
      beta[3 * i + d] = fmaxf(__fdiv_rn(1.f, rho), c.betaMin);
    }
  }
}

// vel_old = vel; gravity on the v faces next to liquid; the reference's wall
// faces set to 0 (x at 0 and sx-1, y at 0, z at 0 and sz-1).
__global__ void k_gravity(GridF g, int64_t n, float* __restrict__ vel,
                          float* __restrict__ velOld, const float* __restrict__ mass, float gdt,
                          float eps) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    int x, y, z;
    g.coords(i, x, y, z);
    float v[3] = {vel[3 * i], vel[3 * i + 1], vel[3 * i + 2]};
    velOld[3 * i] = v[0];
    velOld[3 * i + 1] = v[1];
    velOld[3 * i + 2] = v[2];
    const int64_t lo = g.idx(x, y - 1, z);
    if ((lo >= 0 && mass[lo] > eps) || mass[i] > eps) v[1] = __fadd_rn(v[1], gdt);
    if (x == 0 || x == g.sx - 1) v[0] = 0.f;
    if (y == 0) v[1] = 0.f;
    if (z == 0 || z == g.sz - 1) v[2] = 0.f;
    vel[3 * i] = v[0];
    vel[3 * i + 1] = v[1];
    vel[3 * i + 2] = v[2];
  }
}

// u -= dt beta (p_b - p_a) on each lower face, pressure 0 in a cell without
// liquid; faces between two cells without liquid and the lower domain faces 0.
__global__ void k_gradient(GridF g, int64_t n, float* __restrict__ vel,
                           const float* __restrict__ mass, const float* __restrict__ beta,
                           const float* __restrict__ pres, float dt, float eps) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    int x, y, z;
    g.coords(i, x, y, z);
    const int p[3] = {x, y, z};
    const bool fb = mass[i] > eps;
#pragma unroll
    for (int d = 0; d < 3; d++) {
      if (p[d] == 0) {
        vel[3 * i + d] = 0.f;
        continue;
      }
      const int64_t j = g.idx(x - (d == 0), y - (d == 1), z - (d == 2));
      const bool fa = mass[j] > eps;
      if (!fa && !fb) {
        vel[3 * i + d] = 0.f;
        continue;
      }
      const float pa = fa ? pres[j] : 0.f, pb = fb ? pres[i] : 0.f;
      const float v =
          __fsub_rn(vel[3 * i + d], __fmul_rn(__fmul_rn(dt, beta[3 * i + d]), __fsub_rn(pb, pa)));
      vel[3 * i + d] = isfinite(v) ? v : 0.f;
    }
  }
}

// (vel, velOld) of every value side by side.
__global__ void __launch_bounds__(256) k_pair_channels(const float* __restrict__ a,
                                                       const float* __restrict__ b, int64_t n,
                                                       float2* __restrict__ out) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    out[i] = make_float2(a[i], b[i]);
}

// (vel, velOld) of component d at a position, trilinear.  The index of the block
// layout is a sum of one term per axis; a corner outside the grid counts as 0.
template <bool PAIR>
__device__ __forceinline__ void interp_comp(const GridF& g, const float* __restrict__ vel,
                                            const float* __restrict__ velOld,
                                            const float2* __restrict__ pair, const float pos[3],
                                            int d, float& pic, float& old) {
  pic = old = 0.f;
  if (!isfinite(pos[0]) || !isfinite(pos[1]) || !isfinite(pos[2])) return;  // no cell
  const float gx = __fsub_rn(pos[0], kOff[d][0]), gy = __fsub_rn(pos[1], kOff[d][1]),
              gz = __fsub_rn(pos[2], kOff[d][2]);
  const int ix0 = (int)floorf(gx), iy0 = (int)floorf(gy), iz0 = (int)floorf(gz);
  const float fx = __fsub_rn(gx, (float)ix0), fy = __fsub_rn(gy, (float)iy0),
              fz = __fsub_rn(gz, (float)iz0);
  const int m = (1 << g.sh) - 1;
  int64_t ox[2], oy[2], oz[2];
  bool vx[2], vy[2], vz[2];
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const int x = ix0 + k, y = iy0 + k, z = iz0 + k;
    vx[k] = x >= 0 && x < g.sx;
    vy[k] = y >= 0 && y < g.sy;
    vz[k] = z >= 0 && z < g.sz;
    ox[k] = ((int64_t)(x >> g.sh) << (3 * g.sh)) + (x & m);
    oy[k] = (((int64_t)(y >> g.sh) * g.nbx) << (3 * g.sh)) + ((y & m) << g.sh);
    oz[k] = (((int64_t)(z >> g.sh) * g.nbx * g.nby) << (3 * g.sh)) + ((z & m) << (2 * g.sh));
  }
  const float ex = __fsub_rn(1.f, fx), ey = __fsub_rn(1.f, fy), ez = __fsub_rn(1.f, fz);
#pragma unroll
  for (int c = 0; c < 8; c++) {
    const int dx = c & 1, dy = (c >> 1) & 1, dz = c >> 2;
    const bool in = vx[dx] && vy[dy] && vz[dz];
    float2 v = make_float2(0.f, 0.f);
    if (PAIR) {
      if (in) v = pair[3 * (ox[dx] + oy[dy] + oz[dz]) + d];
    } else {
      // no branch around the loads, so that all are in flight together (4 M particles in no order
      // on 128^3 cells: 0.69 -> 0.59 ms); pairs are faster with it
      const int64_t i = in ? 3 * (ox[dx] + oy[dy] + oz[dz]) + d : 0;
      v = make_float2(vel[i], velOld[i]);
      if (!in) v = make_float2(0.f, 0.f);
    }
    const float w = __fmul_rn(__fmul_rn(dx ? fx : ex, dy ? fy : ey), dz ? fz : ez);
    pic = __fadd_rn(pic, __fmul_rn(w, v.x));
    old = __fadd_rn(old, __fmul_rn(w, v.y));
  }
}

// 13.3 M particles in cell order, 160^3 cells (B200): 1.12 ms with the channels apart and a
// block index per corner, 0.37 ms (and 0.03 for the pairing).
template <bool PAIR>
__global__ void __launch_bounds__(256) k_g2p(msbg_flip_particle* __restrict__ p, int64_t np, GridF g,
                                             const float* __restrict__ vel,
                                             const float* __restrict__ velOld,
                                             const float2* __restrict__ pair, BinsOrder order,
                                             float alpha) {
  const int* perm = order.get();
  for (int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; n < np;
       n += (int64_t)gridDim.x * blockDim.x) {
    const int64_t k = perm ? perm[n] : n;
    msbg_flip_particle q = p[k];
#pragma unroll
    for (int d = 0; d < 3; d++) {
      float pic, old;
      interp_comp<PAIR>(g, vel, velOld, pair, q.pos, d, pic, old);
      q.vel[d] = __fadd_rn(__fmul_rn(__fsub_rn(1.f, alpha), pic),
                           __fmul_rn(alpha, __fadd_rn(q.vel[d], __fsub_rn(pic, old))));
    }
    p[k].vel[0] = q.vel[0];
    p[k].vel[1] = q.vel[1];
    p[k].vel[2] = q.vel[2];
  }
}

int grid_of(msbg_gpu_ctx* ctx, GridF& g) {
  if (!ctx->bsx0 || ctx->nLevels < 1)
    return set_error(ctx, MSBG_EINVARG, "msbg_gpu_sync_topology not called");
  for (int l : ctx->blockLevel)
    if (l != 0) return set_error(ctx, MSBG_ENOTIMPL, "the FLIP transfers need every block at level 0");
  int sh = 0;
  while ((1 << sh) < ctx->bsx0) sh++;
  g = GridF{ctx->sx, ctx->sy, ctx->sz, sh, ctx->nbx, ctx->nby};
  return MSBG_OK;
}

// The grid channels of a context for its current topology (reallocated when
// the topology changed).
int state_of(msbg_gpu_ctx* ctx, FlipState** out, GridF& g) {
  int rc = grid_of(ctx, g);
  if (rc) return rc;
  auto& sp = states()[ctx];
  if (!sp || sp->sx != ctx->sx || sp->sy != ctx->sy || sp->sz != ctx->sz || sp->bsx != ctx->bsx0) {
    sp.reset(new FlipState());
    FlipState& S = *sp;
    S.sx = ctx->sx;
    S.sy = ctx->sy;
    S.sz = ctx->sz;
    S.bsx = ctx->bsx0;
    S.n = (int64_t)S.sx * S.sy * S.sz;
    const size_t n = (size_t)S.n;
    MSBG_CUDA_TRY(ctx, S.vel.ensure(12 * n));
    MSBG_CUDA_TRY(ctx, S.velOld.ensure(12 * n));
    MSBG_CUDA_TRY(ctx, S.beta.ensure(12 * n));
    MSBG_CUDA_TRY(ctx, S.mass.ensure(4 * n));
    MSBG_CUDA_TRY(ctx, S.liq.ensure(4 * n));
    MSBG_CUDA_TRY(ctx, S.active.ensure(4 * (size_t)ctx->nb()));
    for (DeviceBuffer* b : {&S.vel, &S.velOld, &S.beta, &S.mass})
      MSBG_CUDA_TRY(ctx, cudaMemsetAsync(b->p, 0, b->bytes, ctx->stream));
  }
  *out = sp.get();
  return MSBG_OK;
}

int grid_blocks(int64_t n) { return (int)std::min<int64_t>((n + 255) / 256, 148 * 32); }

// From how many particles on P2G looks for crowded boxes: four launches more, 10 to 15 us, which
// 0.5 M particles on 64^3 to 256^3 cells give back where they lie 8 (127 against 193 us on 64^3,
// B200) or 2 to a cell (138 against 130), and 0.25 M do not.
constexpr int64_t P2G_MANY = 1 << 19;
// From how many particles on G2P looks whether it should order them (five launches, 10 us, where
// it should not), and lays the channels side by side first (48 bytes per voxel against half the
// loads), if there is at least one particle per G2P_PAIR_VOXELS voxels: 4 M particles on 128^3
// cells take 0.16 ms either way in cell order, 0.39 against 0.59 ms in none.
constexpr int64_t G2P_ORDER_MANY = 1 << 19, G2P_PAIR_MANY = 1 << 16, G2P_PAIR_VOXELS = 2;

}  // namespace

void flip_release(msbg_gpu_ctx* ctx) { states().erase(ctx); }

}  // namespace msbg

using namespace msbg;

namespace {

int flip_p2g(msbg_gpu_ctx* ctx, const msbg_flip_particle* particles, int64_t np,
             const msbg_flip_params* prm, int* activeBlocks, int64_t* nActive, bool onDevice) {
  if (!ctx || (!particles && np) || np < 0 || !prm) return MSBG_EINVARG;
  if (!(prm->rhoL > 0.f) || !(prm->rhoG > 0.f) || prm->particlesPerVoxel <= 0 ||
      !(prm->alphaPhi > 0.f))
    return set_error(ctx, MSBG_EINVARG, "FLIP parameters: densities, alphaPhi and particles "
                                        "per voxel must be positive");
  cudaSetDevice(ctx->device);
  FlipState* S = nullptr;
  GridF g;
  int rc = state_of(ctx, &S, g);
  if (rc) return rc;
  cudaStream_t st = ctx->stream;
  const int64_t n = S->n;
  MSBG_CUDA_TRY(ctx, S->acc.ensure(sizeof(float) * 9 * (size_t)n));
  MSBG_CUDA_TRY(ctx, cudaMemsetAsync(S->acc.p, 0, sizeof(float) * 9 * (size_t)n, st));
  MSBG_CUDA_TRY(ctx, cudaMemsetAsync(S->active.p, 0, S->active.bytes, st));
  const msbg_flip_particle* dp = particles;
  if (np && !onDevice) {
    MSBG_CUDA_TRY(ctx, S->parts.ensure(sizeof(msbg_flip_particle) * (size_t)np));
    MSBG_CUDA_TRY(ctx, cudaMemcpyAsync(S->parts.p, particles, sizeof(msbg_flip_particle) * np,
                                       cudaMemcpyHostToDevice, st));
    dp = S->parts.as<msbg_flip_particle>();
  }
  bool cells = np >= P2G_MANY && np <= INT_MAX && n <= INT_MAX;
  if (cells && S->lists.ensure(12 * (size_t)np) != cudaSuccess) {
    cudaGetLastError();  // no room for the lists: particle by particle
    cells = false;
  }
  MSBG_CUDA_TRY(ctx, cudaMemsetAsync(S->mass.p, 0, 4 * (size_t)n, st));
  MSBG_CUDA_TRY(ctx, cudaMemsetAsync(S->liq.p, 0, 4 * (size_t)n, st));
  if (cells) {
    // beta, which k_p2g_finish writes in full, holds the boxes and the cells' entries until then
    const int boxes = (int)(n / SUB_T);
    P2GBoxes B;
    B.cnt = S->beta.as<int>();
    B.n = B.cnt + boxes;
    B.crowded = B.n + 2;
    B.start = B.crowded + boxes;
    int2* place = S->lists.as<int2>();  // cell (-1: none) and rank in it of a particle
    int* perm = reinterpret_cast<int*>(place + np);
    MSBG_CUDA_TRY(ctx, cudaMemsetAsync(B.cnt, 0, 4 * (size_t)(boxes + 2), st));
    k_p2g_sample<<<grid_blocks(np / P2G_SAMPLE), 256, 0, st>>>(dp, np, g, B);
    k_p2g_count<<<grid_blocks(np), 256, 0, st>>>(dp, np, g, n, prm->rhoL, prm->rhoG, B,
                                                 S->mass.as<float>(), S->liq.as<int>(), place,
                                                 S->acc.as<float>());
    k_p2g_start<<<std::min(boxes, 148 * 8), SUB_T, 0, st>>>(g, B, S->mass.as<float>());
    k_p2g_place<<<grid_blocks(np), 256, 0, st>>>(np, place, B, perm);
    k_p2g_cells<<<std::min(boxes, 148 * 3), SUB_T, 0, st>>>(dp, g, n, prm->rhoL, prm->rhoG, B,
                                                            S->mass.as<float>(), S->liq.as<int>(),
                                                            perm, S->acc.as<float>());
  } else if (np) {
    k_p2g_scatter<<<grid_blocks(np), 256, 0, st>>>(dp, np, g, n, prm->rhoL, prm->rhoG,
                                                   S->acc.as<float>(), S->mass.as<float>(),
                                                   S->liq.as<int>());
  }
  P2GConst c;
  c.massEps = prm->massEps;
  c.rhoL = prm->rhoL;
  c.rhoG = prm->rhoG;
  c.betaMin = prm->betaMin;
  const float rt0 = (float)prm->particlesPerVoxel;
  c.rtMin = logf(prm->rhoL / prm->rhoG) * prm->rhoG * rt0;
  c.phiDen = prm->alphaPhi * rt0 * prm->rhoL;
  k_p2g_finish<<<grid_blocks(n), 256, 0, st>>>(g, n, c, S->acc.as<float>(), S->mass.as<float>(),
                                               S->liq.as<int>(), S->vel.as<float>(),
                                               S->beta.as<float>(), S->active.as<int>());
  MSBG_CUDA_TRY(ctx, cudaGetLastError());
  if (activeBlocks || nActive) {
    std::vector<int> flags((size_t)ctx->nb());
    MSBG_CUDA_TRY(ctx, cudaMemcpyAsync(flags.data(), S->active.p, 4 * flags.size(),
                                       cudaMemcpyDeviceToHost, st));
    MSBG_CUDA_TRY(ctx, cudaStreamSynchronize(st));
    int64_t k = 0;
    for (size_t b = 0; b < flags.size(); b++)
      if (flags[b]) {
        if (activeBlocks) activeBlocks[k] = (int)b;
        k++;
      }
    if (nActive) *nActive = k;
  }
  return msbg_gpu_sync(ctx);
}

int flip_g2p(msbg_gpu_ctx* ctx, msbg_flip_particle* particles, int64_t np, float flipAlpha,
             bool onDevice) {
  if (!ctx || (!particles && np) || np < 0) return MSBG_EINVARG;
  cudaSetDevice(ctx->device);
  FlipState* S = nullptr;
  GridF g;
  int rc = state_of(ctx, &S, g);
  if (rc) return rc;
  if (!np) return MSBG_OK;
  cudaStream_t st = ctx->stream;
  msbg_flip_particle* dp = particles;
  if (!onDevice) {
    MSBG_CUDA_TRY(ctx, S->parts.ensure(sizeof(msbg_flip_particle) * (size_t)np));
    MSBG_CUDA_TRY(ctx, cudaMemcpyAsync(S->parts.p, particles, sizeof(msbg_flip_particle) * np,
                                       cudaMemcpyHostToDevice, st));
    dp = S->parts.as<msbg_flip_particle>();
  }
  BinsOrder order;
  if (np >= G2P_ORDER_MANY)
    MSBG_CUDA_TRY(ctx, bins_build(S->lists, dp, np, BinsGrid{g.sx, g.sy, g.sz, g.sh, g.nbx, g.nby},
                                  ctx->nb(), 24.0 * (double)(S->n / ctx->nb()), st, order));
  const float* vel = S->vel.as<float>();
  const float* velOld = S->velOld.as<float>();
  float2* pair = nullptr;
  if (np >= G2P_PAIR_MANY && np * G2P_PAIR_VOXELS >= S->n) {
    if (S->acc.ensure(24 * (size_t)S->n) == cudaSuccess) {
      pair = S->acc.as<float2>();
      k_pair_channels<<<grid_blocks(3 * S->n), 256, 0, st>>>(vel, velOld, 3 * S->n, pair);
    } else {
      cudaGetLastError();
    }
  }
  if (pair)
    k_g2p<true><<<grid_blocks(np), 256, 0, st>>>(dp, np, g, vel, velOld, pair, order, flipAlpha);
  else
    k_g2p<false><<<grid_blocks(np), 256, 0, st>>>(dp, np, g, vel, velOld, pair, order, flipAlpha);
  MSBG_CUDA_TRY(ctx, cudaGetLastError());
  if (!onDevice)
    MSBG_CUDA_TRY(ctx, cudaMemcpyAsync(particles, dp, sizeof(msbg_flip_particle) * np,
                                       cudaMemcpyDeviceToHost, st));
  return msbg_gpu_sync(ctx);
}

}  // namespace

extern "C" int msbg_gpu_flip_p2g(msbg_gpu_ctx* ctx, const msbg_flip_particle* particles,
                                 int64_t np, const msbg_flip_params* prm, int* activeBlocks,
                                 int64_t* nActive) {
  return flip_p2g(ctx, particles, np, prm, activeBlocks, nActive, false);
}

extern "C" int msbg_gpu_flip_p2g_device(msbg_gpu_ctx* ctx, const msbg_flip_particle* particles,
                                        int64_t np, const msbg_flip_params* prm,
                                        int* activeBlocks, int64_t* nActive) {
  return flip_p2g(ctx, particles, np, prm, activeBlocks, nActive, true);
}

extern "C" int msbg_gpu_flip_gravity(msbg_gpu_ctx* ctx, float gravity, float dt, float massEps) {
  if (!ctx) return MSBG_EINVARG;
  cudaSetDevice(ctx->device);
  FlipState* S = nullptr;
  GridF g;
  int rc = state_of(ctx, &S, g);
  if (rc) return rc;
  k_gravity<<<grid_blocks(S->n), 256, 0, ctx->stream>>>(g, S->n, S->vel.as<float>(),
                                                         S->velOld.as<float>(),
                                                         S->mass.as<float>(), gravity * dt,
                                                         massEps);
  MSBG_CUDA_TRY(ctx, cudaGetLastError());
  return msbg_gpu_sync(ctx);
}

extern "C" int msbg_gpu_flip_pressure_gradient(msbg_gpu_ctx* ctx, const float* pressure,
                                               float dt, float massEps) {
  if (!ctx || !pressure) return MSBG_EINVARG;
  cudaSetDevice(ctx->device);
  FlipState* S = nullptr;
  GridF g;
  int rc = state_of(ctx, &S, g);
  if (rc) return rc;
  cudaStream_t st = ctx->stream;
  MSBG_CUDA_TRY(ctx, S->acc.ensure(sizeof(float) * (size_t)S->n));
  MSBG_CUDA_TRY(ctx, cudaMemcpyAsync(S->acc.p, pressure, sizeof(float) * S->n,
                                     cudaMemcpyHostToDevice, st));
  k_gradient<<<grid_blocks(S->n), 256, 0, st>>>(g, S->n, S->vel.as<float>(), S->mass.as<float>(),
                                                S->beta.as<float>(), S->acc.as<float>(), dt,
                                                massEps);
  MSBG_CUDA_TRY(ctx, cudaGetLastError());
  return msbg_gpu_sync(ctx);
}

extern "C" int msbg_gpu_flip_g2p(msbg_gpu_ctx* ctx, msbg_flip_particle* particles, int64_t np,
                                 float flipAlpha) {
  return flip_g2p(ctx, particles, np, flipAlpha, false);
}

extern "C" int msbg_gpu_flip_g2p_device(msbg_gpu_ctx* ctx, msbg_flip_particle* particles,
                                        int64_t np, float flipAlpha) {
  return flip_g2p(ctx, particles, np, flipAlpha, true);
}

namespace {
DeviceBuffer* flip_channel(FlipState* S, int which, int& comps) {
  comps = which == MSBG_FLIP_MASS ? 1 : 3;
  switch (which) {
    case MSBG_FLIP_VEL: return &S->vel;
    case MSBG_FLIP_VEL_OLD: return &S->velOld;
    case MSBG_FLIP_BETA: return &S->beta;
    case MSBG_FLIP_MASS: return &S->mass;
    default: return nullptr;
  }
}
}  // namespace

extern "C" int msbg_gpu_flip_channel(msbg_gpu_ctx* ctx, int which, float* data, int64_t n,
                                     int get) {
  if (!ctx || !data) return MSBG_EINVARG;
  cudaSetDevice(ctx->device);
  FlipState* S = nullptr;
  GridF g;
  int rc = state_of(ctx, &S, g);
  if (rc) return rc;
  int comps = 0;
  DeviceBuffer* b = flip_channel(S, which, comps);
  if (!b) return set_error(ctx, MSBG_EINVARG, "FLIP channel %d unknown", which);
  if (n != comps * S->n)
    return set_error(ctx, MSBG_EINVARG, "FLIP channel %d holds %lld floats, not %lld", which,
                     (long long)(comps * S->n), (long long)n);
  MSBG_CUDA_TRY(ctx, cudaMemcpyAsync(get ? (void*)data : b->p, get ? b->p : (const void*)data,
                                     sizeof(float) * n,
                                     get ? cudaMemcpyDeviceToHost : cudaMemcpyHostToDevice,
                                     ctx->stream));
  return msbg_gpu_sync(ctx);
}
