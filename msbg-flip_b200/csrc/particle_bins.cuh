// Order in which a gather kernel visits its particles, so that neighbouring threads read
// the same blocks of the grid (included inside namespace msbg of flip.cu and flip_mr.cu).
//
// A gather from a grid of a few hundred MB reads about 20 sectors per particle.  Particles
// that a program keeps near some order of space find them in L1 and L2; particles in no order pull
// each of them from DRAM, if the blocks that they lie in exceed L2.  The particles themselves
// are not moved: `perm` lists their indices block by block, built per call from their positions.
//   k_bins_sample  looks at up to 4096 groups of 32 consecutive particles; where the boxes around
//                  most groups, and the blocks that all of them lie in, hold more than L2 does,
//                  the particles count as scattered
//   k_bins_count, k_bins_start, k_bins_place  a counting sort by block (the bins in no
//                  order of their own); they return at once when the particles are not
//                  scattered, and the gather then takes them as they come
// No count comes back to the host.
#pragma once

// Scratch of an order: [np] rank of a particle in its block, [np] perm, [nb] particles per
// block, then their first entries in perm, [nb] blocks seen in the sample, [3] groups with large
// boxes, cursor of the bins, number of blocks seen.
inline size_t bins_bytes(int64_t np, int64_t nb) { return 4 * (size_t)(2 * np + 2 * nb + 3); }

constexpr int BINS_GROUPS = 4096;

// Blocks of the raster by the particle's clamped cell.
struct BinsGrid {
  int sx, sy, sz, sh, nbx, nby;
  // (a coordinate that is not a number ends up in cell 0 of its axis)
  __device__ __forceinline__ void cell(const float* p, int& x, int& y, int& z) const {
    x = min(max((int)floorf(p[0]), 0), sx - 1);
    y = min(max((int)floorf(p[1]), 0), sy - 1);
    z = min(max((int)floorf(p[2]), 0), sz - 1);
  }
  __device__ __forceinline__ int block(const float* p) const {
    int x, y, z;
    cell(p, x, y, z);
    return (x >> sh) + nbx * ((y >> sh) + nby * (z >> sh));
  }
};

// What the sample has to show: more than half of `groups` in boxes of `cells` cells or more, and
// so many blocks in use.
struct BinsRule {
  int groups, blocks;
  float cells;
};
__device__ __forceinline__ bool bins_scattered(const int* flag, BinsRule r) {
  return flag[0] * 2 > r.groups && flag[2] >= r.blocks;
}

__global__ void __launch_bounds__(256) k_bins_sample(const msbg_flip_particle* __restrict__ p,
                                                     int64_t np, BinsGrid g, BinsRule rule,
                                                     int* seen, int* flag) {
  const int w = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (w >= rule.groups) return;
  const msbg_flip_particle& q = p[(np / 32) * w / rule.groups * 32 + lane];
  int c[3];
  g.cell(q.pos, c[0], c[1], c[2]);
  float box = 1.f;
#pragma unroll
  for (int k = 0; k < 3; k++)
    box *= (float)(__reduce_max_sync(0xffffffffu, c[k]) - __reduce_min_sync(0xffffffffu, c[k]) + 1);
  if (lane == 0 && box >= rule.cells) atomicAdd(&flag[0], 1);
  const int b = g.block(q.pos);
  const unsigned peers = __match_any_sync(0xffffffffu, b);
  if (__ffs(peers) - 1 == lane && !seen[b] && !atomicExch(&seen[b], 1)) atomicAdd(&flag[2], 1);
}

__global__ void __launch_bounds__(256) k_bins_count(const msbg_flip_particle* __restrict__ p,
                                                    int64_t np, BinsGrid g, BinsRule rule,
                                                    const int* __restrict__ flag,
                                                    int* __restrict__ cnt, int* __restrict__ rank) {
  if (!bins_scattered(flag, rule)) return;
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < np;
       k += (int64_t)gridDim.x * blockDim.x)
    rank[k] = atomicAdd(&cnt[g.block(p[k].pos)], 1);
}

// Counts to first entries: a CTA's 1024 blocks back to back, the CTAs in any order.
__global__ void __launch_bounds__(1024) k_bins_start(int64_t nb, BinsRule rule, int* __restrict__ flag,
                                                     int* __restrict__ cnt) {
  if (!bins_scattered(flag, rule)) return;
  __shared__ int sum[32], base;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t b = blockIdx.x * (int64_t)1024 + threadIdx.x;
  const int v = b < nb ? cnt[b] : 0;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) sum[w] = x;
  __syncthreads();
  if (w == 0) {
    int s = sum[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += y;
    }
    sum[lane] = s;
    if (lane == 31) base = atomicAdd(&flag[1], s);
  }
  __syncthreads();
  if (b < nb) cnt[b] = base + (w ? sum[w - 1] : 0) + x - v;
}

__global__ void __launch_bounds__(256) k_bins_place(const msbg_flip_particle* __restrict__ p,
                                                    int64_t np, BinsGrid g, BinsRule rule,
                                                    const int* __restrict__ flag,
                                                    const int* __restrict__ start,
                                                    const int* __restrict__ rank,
                                                    int* __restrict__ perm) {
  if (!bins_scattered(flag, rule)) return;
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < np;
       k += (int64_t)gridDim.x * blockDim.x)
    perm[start[g.block(p[k].pos)] + rank[k]] = (int)k;
}

// The visiting order as a kernel argument: perm and the flag that says whether it is used.
struct BinsOrder {
  const int* perm = nullptr;
  const int* flag = nullptr;
  BinsRule rule{0, 0, 0.f};
  __device__ __forceinline__ const int* get() const {
    return perm && bins_scattered(flag, rule) ? perm : nullptr;
  }
};

// From how many bytes on an order pays: of a group's box, and of the blocks in use.  G2P (B200, 126
// MB of L2), as the particles come and ordered.  4 M in no order on 160^3 cells (98 MB; the box
// around 32 of them holds 0.83 of the grid) 0.43 and 0.76 ms, on 192^3 (170 MB) 0.56 and 0.70, on
// 208^3 (216 MB) 1.04 and 0.68, on 256^3 (403 MB) 1.46 and 0.72; in an eighth of 256^3 0.51 and
// 1.43; in order, but shuffled among 262 144 neighbours, 0.68 and 0.73, among 8192 0.57 and 0.57.
// 16 M on 512^3 with three levels, 222 to 484 MB, 2.25 to 2.35 and 2.29 to 2.31; with 630 MB 2.50
// and 2.03, shuffled among 262 144 1.80 and 2.10.
constexpr double BINS_BYTES = 160e6;

// Builds the order of np device particles on stream st, in scratch memory that the gather
// reads; blockBytes: what a gather reads of a block, on average.  Without enough device memory
// the particles are taken as they come.
inline cudaError_t bins_build(DeviceBuffer& scratch, const msbg_flip_particle* p, int64_t np,
                              const BinsGrid& g, int64_t nb, double blockBytes, cudaStream_t st,
                              BinsOrder& out) {
  out = BinsOrder();
  const int groups = (int)std::min<int64_t>(np / 32, BINS_GROUPS);
  if (groups < 1 || np > INT_MAX || nb > INT_MAX || (double)nb * blockBytes < BINS_BYTES)
    return cudaSuccess;
  // (no more blocks than the sample can see)
  const BinsRule rule{groups, (int)std::min(BINS_BYTES / blockBytes, 8.0 * groups),
                      (float)(BINS_BYTES / blockBytes * (1ll << (3 * g.sh)))};
  if (scratch.ensure(bins_bytes(np, nb)) != cudaSuccess) {
    cudaGetLastError();
    return cudaSuccess;
  }
  int* rank = scratch.as<int>();
  int* perm = rank + np;
  int* cnt = perm + np;
  int* seen = cnt + nb;
  int* flag = seen + nb;
  const cudaError_t e = cudaMemsetAsync(cnt, 0, 4 * (size_t)(2 * nb + 3), st);
  if (e != cudaSuccess) return e;
  // (few CTAs at the smaller sizes: where there is no order to make, they start to return at once)
  const int grid = (int)std::min<int64_t>((np + 2047) / 2048, 148 * 32);
  k_bins_sample<<<(groups * 32 + 255) / 256, 256, 0, st>>>(p, np, g, rule, seen, flag);
  k_bins_count<<<grid, 256, 0, st>>>(p, np, g, rule, flag, cnt, rank);
  k_bins_start<<<(unsigned)((nb + 1023) / 1024), 1024, 0, st>>>(nb, rule, flag, cnt);
  k_bins_place<<<grid, 256, 0, st>>>(p, np, g, rule, flag, cnt, rank, perm);
  out.perm = perm;
  out.flag = flag;
  out.rule = rule;
  return cudaGetLastError();
}
