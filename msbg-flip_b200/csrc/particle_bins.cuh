// Order in which a gather kernel visits its particles, so that neighbouring threads read
// the same blocks of the grid (included inside namespace msbg of flip.cu and flip_mr.cu).
//
// A gather from a grid of a few hundred MB reads about 20 sectors per particle.  Particles
// that a program keeps near block order find them in L1 and L2; particles in no order pull
// each of them from DRAM.  The particles themselves are not moved: `perm` lists their indices
// block by block, built per call from their positions.
//   k_bins_sample  looks at up to 4096 groups of 32 consecutive particles; where most groups
//                  lie in more than 8 blocks the particles count as scattered
//   k_bins_count, k_bins_start, k_bins_place  a counting sort by block (the bins in no
//                  order of their own); they return at once when the particles are not
//                  scattered, and the gather then takes them as they come
// No count comes back to the host.
#pragma once

// Scratch of an order: [np] rank of a particle in its block, [np] perm, [nb] particles per
// block, then their first entries in perm, [2] scattered groups, cursor of the bins.
inline size_t bins_bytes(int64_t np, int64_t nb) { return 4 * (size_t)(2 * np + nb + 2); }

constexpr int BINS_GROUPS = 4096;

// Blocks of the raster by the particle's clamped cell.
struct BinsGrid {
  int sx, sy, sz, sh, nbx, nby;
  __device__ __forceinline__ int block(float x, float y, float z) const {
    // (a coordinate that is not a number ends up in block 0 of its axis)
    const int cx = min(max((int)floorf(x), 0), sx - 1), cy = min(max((int)floorf(y), 0), sy - 1),
              cz = min(max((int)floorf(z), 0), sz - 1);
    return (cx >> sh) + nbx * ((cy >> sh) + nby * (cz >> sh));
  }
};

__device__ __forceinline__ bool bins_scattered(const int* flag, int groups) {
  return flag[0] * 2 > groups;
}

__global__ void __launch_bounds__(256) k_bins_sample(const msbg_flip_particle* __restrict__ p,
                                                     int64_t np, BinsGrid g, int groups,
                                                     int* __restrict__ flag) {
  const int w = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (w >= groups) return;
  const msbg_flip_particle& q = p[(np / 32) * w / groups * 32 + lane];
  const unsigned peers = __match_any_sync(0xffffffffu, g.block(q.pos[0], q.pos[1], q.pos[2]));
  const unsigned first = __ballot_sync(0xffffffffu, __ffs(peers) - 1 == lane);
  if (lane == 0 && __popc(first) > 8) atomicAdd(flag, 1);
}

__global__ void __launch_bounds__(256) k_bins_count(const msbg_flip_particle* __restrict__ p,
                                                    int64_t np, BinsGrid g, int groups,
                                                    const int* __restrict__ flag,
                                                    int* __restrict__ cnt, int* __restrict__ rank) {
  if (!bins_scattered(flag, groups)) return;
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < np;
       k += (int64_t)gridDim.x * blockDim.x)
    rank[k] = atomicAdd(&cnt[g.block(p[k].pos[0], p[k].pos[1], p[k].pos[2])], 1);
}

// Counts to first entries: a CTA's 1024 blocks back to back, the CTAs in any order.
__global__ void __launch_bounds__(1024) k_bins_start(int64_t nb, int groups, int* __restrict__ flag,
                                                     int* __restrict__ cnt) {
  if (!bins_scattered(flag, groups)) return;
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
                                                    int64_t np, BinsGrid g, int groups,
                                                    const int* __restrict__ flag,
                                                    const int* __restrict__ start,
                                                    const int* __restrict__ rank,
                                                    int* __restrict__ perm) {
  if (!bins_scattered(flag, groups)) return;
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < np;
       k += (int64_t)gridDim.x * blockDim.x)
    perm[start[g.block(p[k].pos[0], p[k].pos[1], p[k].pos[2])] + rank[k]] = (int)k;
}

// The visiting order as a kernel argument: perm and the flag that says whether it is used.
struct BinsOrder {
  const int* perm = nullptr;
  const int* flag = nullptr;
  int groups = 0;
  __device__ __forceinline__ const int* get() const {
    return perm && bins_scattered(flag, groups) ? perm : nullptr;
  }
};

// Builds the order of np device particles on stream st, in scratch memory that the gather
// reads.  Without enough device memory the particles are taken as they come.
inline cudaError_t bins_build(DeviceBuffer& scratch, const msbg_flip_particle* p, int64_t np,
                              const BinsGrid& g, int64_t nb, cudaStream_t st, BinsOrder& out) {
  out = BinsOrder();
  const int groups = (int)std::min<int64_t>(np / 32, BINS_GROUPS);
  if (groups < 1 || np > INT_MAX || nb > INT_MAX) return cudaSuccess;
  if (scratch.ensure(bins_bytes(np, nb)) != cudaSuccess) {
    cudaGetLastError();
    return cudaSuccess;
  }
  int* rank = scratch.as<int>();
  int* perm = rank + np;
  int* cnt = perm + np;
  int* flag = cnt + nb;
  const cudaError_t e = cudaMemsetAsync(cnt, 0, 4 * (size_t)(nb + 2), st);
  if (e != cudaSuccess) return e;
  const int grid = (int)std::min<int64_t>((np + 255) / 256, 148 * 32);
  k_bins_sample<<<(groups * 32 + 255) / 256, 256, 0, st>>>(p, np, g, groups, flag);
  k_bins_count<<<grid, 256, 0, st>>>(p, np, g, groups, flag, cnt, rank);
  k_bins_start<<<(unsigned)((nb + 1023) / 1024), 1024, 0, st>>>(nb, groups, flag, cnt);
  k_bins_place<<<grid, 256, 0, st>>>(p, np, g, groups, flag, cnt, rank, perm);
  out.perm = perm;
  out.flag = flag;
  out.groups = groups;
  return cudaGetLastError();
}
