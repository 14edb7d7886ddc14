// Shared definitions of the B200 sparse block-grid solver library.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <map>
#include <memory>
#include <string>
#include <utility>
#include <vector>

#include "msbg_gpu.h"

namespace msbg {

#ifdef __CUDACC__
// Programmatic dependent launch.  The kernels of a solver iteration, or the colour passes of a
// smoother, follow each other in one stream, each reading what the last one wrote, and where
// they are short a launch is mostly latency.  Launched through launch(), a kernel may start while its predecessor still
// runs (once all CTAs of that one have called pdl_go or ended): it sets itself up and reads
// what no kernel of the chain writes (an operator, block lists), then calls pdl_wait, which
// returns when the predecessor has completed and its writes are visible.  Every thread of
// such a kernel calls pdl_wait before it touches what a predecessor wrote and before it returns, so that its
// own completion says the same of all kernels before it.  Without the launch attribute both
// are no-ops.
// What a kernel of the chain writes changes while the next one is resident already.  So in a
// kernel that calls pdl_wait no pointer to it is __restrict__ and no load of it is __ldg: both
// say that nothing else writes there while the kernel runs, and let the compiler take the
// non-coherent path or move the load above the wait.  Block lists, tile offsets and the
// operator, which no kernel of a chain writes, may have either.
__device__ __forceinline__ void pdl_go() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... P, typename... A>
void launch_if(bool dependent, void (*kernel)(P...), unsigned grid, unsigned block, size_t smem,
               cudaStream_t st, A&&... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = dim3(grid);
  c.blockDim = dim3(block);
  c.dynamicSmemBytes = smem;
  c.stream = st;
  c.attrs = &at;
  c.numAttrs = dependent ? 1 : 0;
  cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
}
template <typename... P, typename... A>
void launch(void (*kernel)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t st,
            A&&... args) {
  launch_if(true, kernel, grid, block, smem, st, std::forward<A>(args)...);
}
#endif

// Neighbour / block-map codes stored in slot tables (slot >= 0 = value block).
enum : int {
  SLOT_NULL = -1,   // no block in the map: BC_NEUMANN clamp to own block
  SLOT_EMPTY = -2,  // const empty block
  SLOT_FULL = -3,   // const full block
  SLOT_OUT = -4     // outside the domain: BC_NEUMANN clamp to own block
};

// Bits of the device error flag that kernels set (msbg_gpu_sync reads it).
enum : int {
  ERR_WAIT_TIMEOUT = 1,   // a bounded wait gave up
  MCF_ERR_NOT_VALUE = 2   // a listed block is not a value block; it was skipped
};

// Device blocks on their way from one owner to the next.  While a PoolScope is open on a
// thread, buffers that it releases there go to the scope's pool, and buffers that need memory
// look there first; what is left is freed when the scope closes, or before an allocation fails.
// For work on one stream: a block may still be read by what its last owner has issued there.
// A block may be up to 1/4 larger than asked for, and its new owner keeps what is too much.  That
// comes to 1/64 of the memory that was free when the scope opened, and to nothing but the rest
// of a 2 MB page (which cudaMalloc keeps as well) where less than a quarter of the card was: what
// fits without a pool is not to be refused with one.
class DevicePool {
 public:
  DevicePool() {
    size_t free = 0, total = 0;
    if (cudaMemGetInfo(&free, &total) == cudaSuccess && free >= total / 4) allowed_ = free / 64;
  }
  ~DevicePool() { clear(); }
  DevicePool(const DevicePool&) = delete;
  DevicePool& operator=(const DevicePool&) = delete;
  void clear() {
    for (auto& b : blocks_) cudaFree(b.second);
    blocks_.clear();
  }
  void give(void* p, size_t cap) noexcept {
    try {
      blocks_.emplace(cap, p);
    } catch (...) {  // no memory for the entry
      cudaFree(p);
    }
  }
  void* take(size_t n, size_t& cap) {
    auto it = blocks_.lower_bound(n);
    if (it == blocks_.end() || it->first > n + n / 4 + 4096) return nullptr;
    const size_t more = it->first - n;
    if (n < PAGE || (n + PAGE - 1) / PAGE != (it->first + PAGE - 1) / PAGE) {
      if (more > allowed_) return nullptr;
      allowed_ -= more;
      wasted_ += more;
    }
    void* p = it->second;
    cap = it->first;
    blocks_.erase(it);
    return p;
  }
  // What the owners of this pool's blocks have too much.
  size_t wasted() const { return wasted_; }
  static DevicePool*& current() {
    static thread_local DevicePool* c = nullptr;
    return c;
  }

 private:
  static constexpr size_t PAGE = 2 << 20;
  std::multimap<size_t, void*> blocks_;
  size_t allowed_ = 0, wasted_ = 0;
};
class PoolScope {
 public:
  PoolScope() : before_(DevicePool::current()) { DevicePool::current() = &pool_; }
  ~PoolScope() { DevicePool::current() = before_; }
  PoolScope(const PoolScope&) = delete;
  PoolScope& operator=(const PoolScope&) = delete;
  size_t wasted() const { return pool_.wasted(); }

 private:
  DevicePool* before_;
  DevicePool pool_;
};

// No pool while a caller's code runs: what it releases is of another owner, stream or device.
class PoolPause {
 public:
  PoolPause() : before_(DevicePool::current()) { DevicePool::current() = nullptr; }
  ~PoolPause() { DevicePool::current() = before_; }
  PoolPause(const PoolPause&) = delete;
  PoolPause& operator=(const PoolPause&) = delete;

 private:
  DevicePool* before_;
};

struct DeviceBuffer {
  void* p = nullptr;
  size_t bytes = 0;  // asked for
  size_t cap = 0;    // of the block
  DeviceBuffer() = default;
  DeviceBuffer(const DeviceBuffer&) = delete;
  DeviceBuffer& operator=(const DeviceBuffer&) = delete;
  ~DeviceBuffer() { release(); }
  void release() {
    if (p) {
      if (DevicePool* pool = DevicePool::current())
        pool->give(p, cap);
      else
        cudaFree(p);
    }
    p = nullptr;
    bytes = cap = 0;
  }
  cudaError_t ensure(size_t n) {
    if (n <= cap && p) {
      if (n > bytes) bytes = n;
      return cudaSuccess;
    }
    release();
    const size_t want = n ? n : 16;
    DevicePool* pool = DevicePool::current();
    if (pool) p = pool->take(want, cap);
    if (!p) {
      cudaError_t e = cudaMalloc(&p, want);
      if (e != cudaSuccess && pool) {  // what the last owner left makes room
        cudaGetLastError();
        pool->clear();
        e = cudaMalloc(&p, want);
      }
      if (e != cudaSuccess) {
        p = nullptr;
        return e;
      }
      cap = want;
    }
    bytes = n;
    return cudaSuccess;
  }
  template <typename T>
  T* as() const { return reinterpret_cast<T*>(p); }
  // takes over o's allocation (o is left empty)
  void adopt(DeviceBuffer& o) {
    if (&o == this) return;
    release();
    p = o.p;
    bytes = o.bytes;
    cap = o.cap;
    o.p = nullptr;
    o.bytes = o.cap = 0;
  }
};

// One uploaded channel at one resolution level: FP32 or 16-bit render
// density (dtype MSBG_F32 / MSBG_U16).
struct Channel {
  int level = 0;
  int bsx = 0;
  int dtype = MSBG_F32;
  uint16_t emptyQ = 0, fullQ = 0;  // const values of a 16-bit channel (raw)
  int64_t nValue = 0;
  float emptyVal = 0.f, fullVal = 0.f;
  std::vector<int> slotHost;   // [nb] slot or SLOT_* code
  std::vector<int8_t> kindHost;
  DeviceBuffer pool;           // [nValue][bsx^3] float or uint16_t
  DeviceBuffer xfaces;         // [nValue][2][bsx^2]: the x = 0 and x = bsx-1 planes
  DeviceBuffer slot;           // [nb] int
  // a channel that replaces an earlier one of the same id keeps its device
  // allocations (no cudaMalloc / cudaFree per upload when the sizes fit)
  void reuse(Channel& old) {
    pool.adopt(old.pool);
    xfaces.adopt(old.xfaces);
    slot.adopt(old.slot);
  }
};

}  // namespace msbg

struct msbg_cnn;

struct msbg_gpu_ctx {
  int device = 0;
  msbg_cnn* cnn = nullptr;      // learned initial guess of the pressure solves (not owned)
  msbg_cnn* cnnCorr = nullptr;  // learned per-V-cycle correction (not owned)
  cudaStream_t stream = nullptr;
  int sx = 0, sy = 0, sz = 0, bsx0 = 0, nLevels = 1;
  int nbx = 0, nby = 0, nbz = 0;
  std::vector<int> blockLevel;
  std::map<int, std::unique_ptr<msbg::Channel>> channels;
  std::string lastError;
  // scratch for block lists (grouped by colour)
  msbg::DeviceBuffer listBuf;
  msbg::DeviceBuffer errBuf;  // int: set by kernels whose bounded wait gave up
  std::vector<int> listHost;
  void* pinned = nullptr;
  size_t pinnedBytes = 0;
  int64_t nb() const { return (int64_t)nbx * nby * nbz; }
};

namespace msbg {

int set_error(msbg_gpu_ctx* ctx, int code, const char* fmt, ...);

#define MSBG_CUDA_TRY(ctx, expr)                                                   \
  do {                                                                             \
    cudaError_t _e = (expr);                                                       \
    if (_e != cudaSuccess)                                                         \
      return ::msbg::set_error((ctx), _e == cudaErrorMemoryAllocation ? MSBG_ENOMEM \
                                                                      : MSBG_ERROR, \
                               "%s: %s (%s:%d)", #expr, cudaGetErrorString(_e),   \
                               __FILE__, __LINE__);                                \
  } while (0)

// Releases the pressure solver state of a context (pressure.cu).
void pressure_release(msbg_gpu_ctx* ctx);
// Releases the FLIP transfer channels of a context (flip.cu).
void flip_release(msbg_gpu_ctx* ctx);
// Releases the particle-splatting buffers of a context (splat.cu).
void splat_release(msbg_gpu_ctx* ctx);
// Releases the mixed-resolution G2P state of a context (flip_mr.cu).
void flip_mr_release(msbg_gpu_ctx* ctx);

// Launches of the 8-colour mean-curvature-flow passes (mcf.cu).  xfaces:
// optional face cache of nSlots value blocks (2 * bsx^2 values each, the
// pool's element type), refilled at the start of the call and kept current by
// the passes; NULL reads the neighbours' x faces from the pool.
cudaError_t launch_mcf(float* pool, const int* slotOf, const int* colourList,
                       const int* colourStart, int nbx, int nby, int nbz, int bsx,
                       float emptyVal, float fullVal, int nIter, float dt, int clamp01,
                       int* errFlag, cudaStream_t stream, void* xfaces = nullptr,
                       int64_t nSlots = 0);
// The same passes on a 16-bit render-density pool (const values raw).
cudaError_t launch_mcf_u16(uint16_t* pool, const int* slotOf, const int* colourList,
                           const int* colourStart, int nbx, int nby, int nbz, int bsx,
                           uint16_t emptyVal, uint16_t fullVal, int nIter, float dt, int clamp01,
                           int* errFlag, cudaStream_t stream, void* xfaces = nullptr,
                           int64_t nSlots = 0);

}  // namespace msbg
