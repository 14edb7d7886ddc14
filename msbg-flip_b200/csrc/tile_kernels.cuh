// Reductions, PCG vector kernels and per-tile kernels of the pressure solver
// (included inside namespace msbg::ps of pressure.cu).  Vectors are stored
// as VT (float, __half or __nv_bfloat16) and computed in FP32; inner products
// accumulate in FP64.

// ---------------------------------------------------------------------------
// reductions
// ---------------------------------------------------------------------------
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// Sum over the CTA; result valid in thread 0.
__device__ __forceinline__ double block_sum(double v) {
  __shared__ double ws[32];
  v = warp_sum(v);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) ws[w] = v;
  __syncthreads();
  const int nw = (blockDim.x + 31) >> 5;
  v = (threadIdx.x < nw) ? ws[threadIdx.x] : 0.0;
  if (w == 0) v = warp_sum(v);
  __syncthreads();
  return v;
}

struct Scalars {
  double bb, rho, rhoNew, dq, rr, alpha, beta, amax;
  double cc, cr, omega;  // energy-optimal scaling of a learned vector c
  int status;  // 0 ok, 2 breakdown, 3 non-finite
  int pad;
};

enum {
  FIN_BB = 0,
  FIN_DQ_ALPHA = 1,
  FIN_RR = 2,
  FIN_RHO = 3,
  FIN_RHONEW_BETA = 4,
  FIN_FCG_BETA = 5,      // flexible CG: beta = -(z.q)/(d.q)
  FIN_FCG_DQ_ALPHA = 6,  // flexible CG: alpha = (d.r)/(d.q), d.r of either sign
  FIN_CC = 7,            // c.Ac
  FIN_CR = 8,            // c.r
  FIN_OMEGA_CORR = 9,    // omega = (c.r)/(c.Ac): v = c.r
  FIN_OMEGA_GUESS = 10,  // omega = (g.b)/(g.b - g.r), r = b - A g: v = g.r
};

// Deterministic second stage: fixed-order sum of the CTA partials, then the
// scalar step of PCG that depends on it.
static __global__ void __launch_bounds__(1024) k_finalize(const double* partial, int n,
                                                   Scalars* s, int what) {
  pdl_go();
  pdl_wait();
  double v = 0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) v += partial[i];
  v = block_sum(v);
  if (threadIdx.x != 0) return;
  switch (what) {
    case FIN_BB: s->bb = v; break;
    case FIN_RHO: s->rho = v; break;
    case FIN_RR:
      s->rr = v;
      if (!isfinite(v)) s->status = 3;
      break;
    case FIN_DQ_ALPHA:
      s->dq = v;
      if (!isfinite(v) || !isfinite(s->rho)) s->status = 3;
      else if (!(v > 1e-300) || !(s->rho > 1e-300)) s->status = 2;
      else s->alpha = s->rho / v;
      break;
    case FIN_RHONEW_BETA:
      s->rhoNew = v;
      if (!isfinite(v)) s->status = 3;
      else if (!(v > 1e-300)) s->status = 2;
      else {
        s->beta = v / s->rho;
        s->rho = v;
      }
      break;
    case FIN_FCG_BETA:  // q = A d of the last step
      if (!isfinite(v)) s->status = 3;
      else s->beta = -v / s->dq;
      break;
    case FIN_CC: s->cc = v; break;
    case FIN_CR: s->cr = v; break;
    // The scaled vector omega*c minimises |e - omega c|_A for A e = r: it
    // never leaves a larger energy error than c = 0 does.  A degenerate c
    // gets omega = 0.
    case FIN_OMEGA_CORR:
      s->omega = (isfinite(v) && isfinite(s->cc) && s->cc > 1e-300) ? v / s->cc : 0.0;
      break;
    case FIN_OMEGA_GUESS: {
      const double gag = s->cr - v;  // g.Ag = g.b - g.(b - Ag)
      s->omega = (isfinite(v) && isfinite(s->cr) && gag > 1e-300) ? s->cr / gag : 0.0;
      break;
    }
    case FIN_FCG_DQ_ALPHA:
      // a non-linear preconditioner need not make d.r positive; the step
      // along d still minimises the energy norm as long as d.q > 0
      s->dq = v;
      if (!isfinite(v) || !isfinite(s->rho)) s->status = 3;
      else if (!(v > 1e-300)) s->status = 2;
      else s->alpha = s->rho / v;
      break;
  }
}

// ---------------------------------------------------------------------------
// level-0 vector kernels (grid-stride over groups of 4, fixed grid so the
// partial sums are deterministic)
// ---------------------------------------------------------------------------
constexpr int VEC_GRID = 148 * 4, VEC_BLOCK = 512;
// Dependent launches (common.cuh) of the vector kernels and their scalar steps: where they
// are short.  On long vectors an early start of the next kernel takes from the running one.
// Plain FP32 solves with them and without (B200, kernel by kernel; in a CUDA graph the small ones
// take the same either way): 64^3 cells 1.09 and 1.18 ms, 192^3 4.42 and 4.52, 256^3 6.58 and 6.61,
// 320^3 9.79 and 9.56, 512^3 41.6 and 40.8.
inline bool vectors_dependent(int64_t n) { return n <= (8 << 20); }

template <typename VA, typename VB>
__global__ void __launch_bounds__(VEC_BLOCK) k_dot(const VA* a,
                                                   const VB* b, int64_t n,
                                                   double* partial) {
  pdl_go();
  pdl_wait();
  double acc = 0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < (n >> 2);
       i += (int64_t)gridDim.x * blockDim.x) {
    const F4 u = load4(a + 4 * i), v = load4(b + 4 * i);
    acc += (double)u.x * v.x + (double)u.y * v.y + (double)u.z * v.z + (double)u.w * v.w;
  }
  acc = block_sum(acc);
  if (threadIdx.x == 0) partial[blockIdx.x] = acc;
}

// x += alpha d; r -= alpha q; partial |r|^2.  Skipped (norm only) after a breakdown.
template <typename VT>
__global__ void __launch_bounds__(VEC_BLOCK) k_axpy_norm(VT* x, VT* r,
                                                         const VT* d,
                                                         const VT* q, int64_t n,
                                                         const Scalars* s,
                                                         double* partial) {
  pdl_go();
  pdl_wait();
  const bool ok = s->status == 0;
  const float alpha = (float)s->alpha;
  double acc = 0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < (n >> 2);
       i += (int64_t)gridDim.x * blockDim.x) {
    F4 rv = load4(r + 4 * i);
    if (ok) {
      F4 xv = load4(x + 4 * i);
      const F4 dv = load4(d + 4 * i), qv = load4(q + 4 * i);
      xv.x = fmaf(alpha, dv.x, xv.x); xv.y = fmaf(alpha, dv.y, xv.y);
      xv.z = fmaf(alpha, dv.z, xv.z); xv.w = fmaf(alpha, dv.w, xv.w);
      rv.x = fmaf(-alpha, qv.x, rv.x); rv.y = fmaf(-alpha, qv.y, rv.y);
      rv.z = fmaf(-alpha, qv.z, rv.z); rv.w = fmaf(-alpha, qv.w, rv.w);
      store4(x + 4 * i, xv);
      store4(r + 4 * i, rv);
      rv = load4(r + 4 * i);  // the norm of what is stored
    }
    acc += (double)rv.x * rv.x + (double)rv.y * rv.y + (double)rv.z * rv.z + (double)rv.w * rv.w;
  }
  acc = block_sum(acc);
  if (threadIdx.x == 0) partial[blockIdx.x] = acc;
}

// d = z + beta d
template <typename VT>
__global__ void __launch_bounds__(VEC_BLOCK) k_update_d(VT* d,
                                                        const VT* z, int64_t n,
                                                        const Scalars* s) {
  pdl_go();
  pdl_wait();
  if (s->status) return;
  const float beta = (float)s->beta;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < (n >> 2);
       i += (int64_t)gridDim.x * blockDim.x) {
    F4 dv = load4(d + 4 * i);
    const F4 zv = load4(z + 4 * i);
    dv.x = fmaf(beta, dv.x, zv.x); dv.y = fmaf(beta, dv.y, zv.y);
    dv.z = fmaf(beta, dv.z, zv.z); dv.w = fmaf(beta, dv.w, zv.w);
    store4(d + 4 * i, dv);
  }
}

// y = scale * x (type conversion)
template <typename VS, typename VD>
__global__ void __launch_bounds__(VEC_BLOCK) k_convert(VD* __restrict__ y, const VS* __restrict__ x,
                                                       int64_t n, float scale) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < (n >> 2);
       i += (int64_t)gridDim.x * blockDim.x) {
    F4 v = load4(x + 4 * i);
    v.x *= scale; v.y *= scale; v.z *= scale; v.w *= scale;
    store4(y + 4 * i, v);
  }
}

// ---------------------------------------------------------------------------
// per-tile kernels (any tile size TS <= 16; one CTA per tile)
// ---------------------------------------------------------------------------
// The passes and groups of 8^3 tiles and smaller are short: what they cost is
// one chain of dependent global loads and a few barriers, so a thread owns one cell
// (four on 16^3 tiles, where the pipelined kernels of smooth_pipe.cuh take over): all its
// loads are in flight together, the face data come resolved from the tile's record, and
// a half sweep is one update per thread.  With a thread per z column of a tile, a
// smoothing pass of 8^3 / 4^3 tiles took 18 / 14 us and a residual 23 / 14 us (256^3 grid
// of 16^3 blocks, 3 levels, B200), and the FP16 solve 17.4 ms; with these kernels 13.1.
template <int TS>
struct TileGeo {
  static constexpr int N = TS * TS * TS;
  static constexpr int NT = TS == 16 ? 1024 : (N < 32 ? 32 : N);  // threads
  static constexpr int PER = N > NT ? N / NT : 1;                  // cells per thread
  static constexpr int P = TS + 2;                                 // padded edge
  __device__ static constexpr int pad(int i, int j, int k) {
    return (i + 1) + P * ((j + 1) + P * (k + 1));
  }
};

// Coupling times neighbour of face cell (a, b) of face (dir, side), as ghost_sum.
template <int TS, typename VT>
__device__ __forceinline__ float halo_term(const LevelView& L, const TileRec& r, int ti,
                                           const VT* x, int dir, int side, int a,
                                           int b, int zeroStart) {
  const FaceRes& F = r.f[2 * dir + side];
  const int kind = F.kind;
  if (kind == FACE_NONE || ((zeroStart >> kind) & 1)) return 0.f;
  const float* cd = dir == 0 ? L.cx : dir == 1 ? L.cy : L.cz;
  if (kind == FACE_SAME)
    return cd[(side ? F.nOff : r.off) + plane_idx(TS, dir, 0, a, b)] *
           to_f(x[F.nOff + plane_idx(TS, dir, side ? 0 : TS - 1, a, b)]);
  if (kind == FACE_COARSER)
    return L.ifc[F.ifOwn + a + TS * b] *
           to_f(x[F.nOff + plane_idx(F.nts, dir, side ? 0 : F.nts - 1, F.oa + (a >> 1),
                                     F.ob + (b >> 1))]);
  return ghost_sum(L, x, ti, TS, dir, side, a, b);
}

// A tile in shared memory: x inside a padded cube whose face halos hold the halo
// terms (coupling times neighbour), and per cell of a thread the six couplings, 1
// towards a halo: the neighbour sum is one multiply-add per face either way.
template <int TS, typename VT>
struct TileCells {
  using G = TileGeo<TS>;
  float c[G::PER][6];
  // the couplings; then, once x is there, x and the halo
  __device__ __forceinline__ void load(const LevelView& L, const TileRec& r) {
    const int t = threadIdx.x;
    const float* cx = L.cx + r.off;
    const float* cy = L.cy + r.off;
    const float* cz = L.cz + r.off;
#pragma unroll
    for (int q = 0; q < G::PER; q++) {
      const int e = t + G::NT * q;
      if (e >= G::N) continue;
      const int i = e % TS, j = (e / TS) % TS, k = e / (TS * TS);
      c[q][0] = i > 0 ? cx[e] : 1.f;
      c[q][1] = i < TS - 1 ? cx[e + 1] : 1.f;
      c[q][2] = j > 0 ? cy[e] : 1.f;
      c[q][3] = j < TS - 1 ? cy[e + TS] : 1.f;
      c[q][4] = k > 0 ? cz[e] : 1.f;
      c[q][5] = k < TS - 1 ? cz[e + TS * TS] : 1.f;
    }
  }
  __device__ __forceinline__ void load_x(const LevelView& L, const TileRec& r, int ti,
                                         const VT* x, float* xs, int zeroStart = 0) {
    const int t = threadIdx.x;
#pragma unroll
    for (int q = 0; q < G::PER; q++) {
      const int e = t + G::NT * q;
      if (e < G::N)
        xs[G::pad(e % TS, (e / TS) % TS, e / (TS * TS))] =
            zeroStart & ZERO_OWN ? 0.f : to_f(x[r.off + e]);
    }
    for (int h = t; h < 6 * TS * TS; h += G::NT) {
      const int f = h / (TS * TS), a = h % TS, b = (h / TS) % TS, dir = f >> 1, side = f & 1;
      const int p = side ? TS : -1;
      xs[dir == 0 ? G::pad(p, a, b) : dir == 1 ? G::pad(a, p, b) : G::pad(a, b, p)] =
          halo_term<TS>(L, r, ti, x, dir, side, a, b, zeroStart);
    }
  }
  // in the order x-, x+, y-, y+, z-, z+
  __device__ __forceinline__ float sum(const float* at, int q) const {
    float S = 0.f;
    S = fmaf(c[q][0], at[-1], S);
    S = fmaf(c[q][1], at[1], S);
    S = fmaf(c[q][2], at[-G::P], S);
    S = fmaf(c[q][3], at[G::P], S);
    S = fmaf(c[q][4], at[-G::P * G::P], S);
    S = fmaf(c[q][5], at[G::P * G::P], S);
    return S;
  }
};

// q = A d on tiles tileBase.., partial d.q per CTA.
template <int TS, typename VT>
__global__ void __launch_bounds__(TileGeo<TS>::NT) k_matvec_dot(LevelView L, int tileBase,
                                                                const VT* d,
                                                                VT* q,
                                                                double* partial) {
  using G = TileGeo<TS>;
  __shared__ float xs[G::P * G::P * G::P];
  const int ti = tileBase + blockIdx.x, t = threadIdx.x;
  const TileRec& r = reinterpret_cast<const TileRec*>(L.tileRec)[ti];
  pdl_go();
  TileCells<TS, VT> C;
  C.load(L, r);
  float dg[G::PER];
#pragma unroll
  for (int p = 0; p < G::PER; p++) dg[p] = t + G::NT * p < G::N ? L.diag[r.off + t + G::NT * p] : 0.f;
  pdl_wait();
  C.load_x(L, r, ti, d, xs);
  __syncthreads();
  double acc = 0;
#pragma unroll
  for (int p = 0; p < G::PER; p++) {
    const int e = t + G::NT * p;
    if (e >= G::N) continue;
    const float* at = xs + G::pad(e % TS, (e / TS) % TS, e / (TS * TS));
    float y = 0.f;
    if (dg[p] > 0.f) y = fmaf(dg[p], *at, -C.sum(at, p));
    q[r.off + e] = from_f<VT>(y);
    acc += (double)*at * (double)to_f(from_f<VT>(y));
  }
  acc = block_sum(acc);
  if (t == 0 && partial) partial[blockIdx.x] = acc;
}

// r = b - A x on tiles tileBase.., restricted (sum over the liquid children,
// P^T) into the coarse right-hand side bc (vectors VT, coarse vectors VC).
template <int TS, typename VT, typename VC>
__global__ void __launch_bounds__(TileGeo<TS>::NT)
    k_residual_restrict(LevelView L, int tileBase, const VT* x,
                        const VT* b, VC* bc,
                        const int64_t* __restrict__ coarseOff) {
  using G = TileGeo<TS>;
  __shared__ float xs[G::P * G::P * G::P];
  __shared__ float rs[G::N];
  const int ti = tileBase + blockIdx.x, t = threadIdx.x;
  const TileRec& r = reinterpret_cast<const TileRec*>(L.tileRec)[ti];
  pdl_go();
  TileCells<TS, VT> C;
  C.load(L, r);
  const int* tc = L.toCoarse + (size_t)ti * 6;
  const int ct = tc[0], ox = tc[1], oy = tc[2], oz = tc[3], agg = tc[4], cts = tc[5];
  VC* dst = ct >= 0 ? bc + coarseOff[ct] : nullptr;
  float dg[G::PER], bv[G::PER];
#pragma unroll
  for (int p = 0; p < G::PER; p++) {
    const int e = t + G::NT * p;
    dg[p] = e < G::N ? L.diag[r.off + e] : 0.f;
  }
  pdl_wait();
#pragma unroll
  for (int p = 0; p < G::PER; p++)
    bv[p] = t + G::NT * p < G::N ? to_f(b[r.off + t + G::NT * p]) : 0.f;
  C.load_x(L, r, ti, x, xs);
  __syncthreads();
  if (!dst) return;
#pragma unroll
  for (int p = 0; p < G::PER; p++) {
    const int e = t + G::NT * p;
    if (e >= G::N) continue;
    const int i = e % TS, j = (e / TS) % TS, k = e / (TS * TS);
    const float* at = xs + G::pad(i, j, k);
    float v = 0.f;
    if (dg[p] > 0.f) v = bv[p] - fmaf(dg[p], *at, -C.sum(at, p));
    if (agg)
      rs[e] = v;
    else
      dst[tidx(cts, ox + i, oy + j, oz + k)] = from_f<VC>(v);
  }
  if (!agg) return;
  __syncthreads();
  constexpr int H = TS / 2;
  for (int c = t; c < H * H * H; c += G::NT) {
    const int ci = c % H, cj = (c / H) % H, ck = c / (H * H);
    const int e = tidx(TS, 2 * ci, 2 * cj, 2 * ck);
    const float s = rs[e] + rs[e + 1] + rs[e + TS] + rs[e + TS + 1] + rs[e + TS * TS] +
                    rs[e + TS * TS + 1] + rs[e + TS * TS + TS] + rs[e + TS * TS + TS + 1];
    dst[tidx(cts, ox + ci, oy + cj, oz + ck)] = from_f<VC>(s);
  }
}

// The x = 0 plane of cx of the TS^3 tiles tileBase, tileBase+1, ... (one CTA
// per tile) into the packed layout of LevelView::cxf.
template <int TS = 16>
__global__ void __launch_bounds__(TS* TS) k_pack_cx_plane(const int64_t* __restrict__ tileOff,
                                                          int tileBase,
                                                          const float* __restrict__ cx,
                                                          float* __restrict__ cxf) {
  const int64_t off = tileOff[tileBase + blockIdx.x];
  const int c = threadIdx.x;  // y + TS z
  cxf[(off >> 4) + c] = cx[off + TS * c];
}

// x += scale * P xc (liquid cells only; vectors VT, coarse vectors VC).  On
// 16^3 tiles the packed x faces xf (if given) are written too.
template <int TS, typename VT, typename VC>
__global__ void __launch_bounds__(TS* TS) k_prolong(LevelView L, const int* __restrict__ tiles,
                                                    VT* x,
                                                    const VC* xc,
                                                    const int64_t* __restrict__ coarseOff,
                                                    float scale, VT* xf) {
  constexpr int N = TS * TS * TS, NT = TS * TS;
  pdl_go();
  const int ti = tiles[blockIdx.x];
  const int64_t off = L.tileOff[ti];
  const int* tc = L.toCoarse + (size_t)ti * 6;
  const int ct = tc[0], ox = tc[1], oy = tc[2], oz = tc[3], agg = tc[4], cts = tc[5];
  pdl_wait();
  if (ct < 0) return;
  const VC* src = xc + coarseOff[ct];
  const int sh = agg ? 1 : 0;
  if constexpr (TS >= 4) {
    // groups of 4 x-consecutive cells: every load of a thread's groups is
    // issued before any is used (non-liquid cells are written back unchanged)
    constexpr int PER = (N / 4 + NT - 1) / NT;
    F4 dv[PER], xv[PER], cv[PER];
#pragma unroll
    for (int p = 0; p < PER; p++) {
      const int e = 4 * (threadIdx.x + NT * p);
      if (e >= N) continue;
      const int i = e % TS, j = (e / TS) % TS, k = e / (TS * TS);
      dv[p] = load4(L.diag + off + e);
      xv[p] = load4(x + off + e);
      const VC* row = src + tidx(cts, 0, oy + (j >> sh), oz + (k >> sh));
      cv[p].x = to_f(row[ox + (i >> sh)]);
      cv[p].y = to_f(row[ox + ((i + 1) >> sh)]);
      cv[p].z = to_f(row[ox + ((i + 2) >> sh)]);
      cv[p].w = to_f(row[ox + ((i + 3) >> sh)]);
    }
#pragma unroll
    for (int p = 0; p < PER; p++) {
      const int e = 4 * (threadIdx.x + NT * p);
      if (e >= N) continue;
      F4 o = xv[p];
      if (dv[p].x > 0.f) o.x = to_f(from_f<VT>(xv[p].x + scale * cv[p].x));
      if (dv[p].y > 0.f) o.y = to_f(from_f<VT>(xv[p].y + scale * cv[p].y));
      if (dv[p].z > 0.f) o.z = to_f(from_f<VT>(xv[p].z + scale * cv[p].z));
      if (dv[p].w > 0.f) o.w = to_f(from_f<VT>(xv[p].w + scale * cv[p].w));
      store4(x + off + e, o);
      if (TS == 16 && xf) {
        const int i = e % TS, j = (e / TS) % TS, k = e / (TS * TS);
        if (i == 0) xf[xface_slot(off, 0, j, k)] = from_f<VT>(o.x);
        if (i == TS - 4) xf[xface_slot(off, 1, j, k)] = from_f<VT>(o.w);
      }
    }
  } else {
    for (int e = threadIdx.x; e < N; e += NT) {
      if (!(L.diag[off + e] > 0.f)) continue;
      const int i = e % TS, j = (e / TS) % TS, k = e / (TS * TS);
      const float c = to_f(src[tidx(cts, ox + (i >> sh), oy + (j >> sh), oz + (k >> sh))]);
      x[off + e] = from_f<VT>(to_f(x[off + e]) + scale * c);
    }
  }
}

// Red-black Gauss-Seidel inside tiles tileBase.., `inner` iterations, ghosts
// frozen at their values when the tile is loaded.  reverse=0: red then black;
// reverse=1: black then red (the adjoint order).  zeroStart: see pressure_kernels.cuh.
template <int TS, typename VT>
__global__ void __launch_bounds__(TileGeo<TS>::NT) k_smooth(LevelView L, int tileBase,
                                                            VT* x,
                                                            const VT* b, int inner,
                                                            int reverse, int zeroStart) {
  using G = TileGeo<TS>;
  __shared__ float xs[G::P * G::P * G::P];
  const int ti = tileBase + blockIdx.x, t = threadIdx.x;
  const TileRec& r = reinterpret_cast<const TileRec*>(L.tileRec)[ti];
  pdl_go();
  TileCells<TS, VT> C;
  C.load(L, r);
  float inv[G::PER], bb[G::PER];
  int col[G::PER], at[G::PER];
#pragma unroll
  for (int p = 0; p < G::PER; p++) {
    const int e = t + G::NT * p;
    const int i = e % TS, j = (e / TS) % TS, k = e / (TS * TS);
    inv[p] = e < G::N ? L.invdiag[r.off + e] : 0.f;
    col[p] = (i + j + k) & 1;
    at[p] = e < G::N ? G::pad(i, j, k) : G::pad(0, 0, 0);
  }
  pdl_wait();
#pragma unroll
  for (int p = 0; p < G::PER; p++)
    bb[p] = t + G::NT * p < G::N ? to_f(b[r.off + t + G::NT * p]) : 0.f;
  C.load_x(L, r, ti, x, xs, zeroStart);
  __syncthreads();
  for (int it = 0; it < inner; it++) {
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int colour = reverse ? 1 - h : h;
#pragma unroll
      for (int p = 0; p < G::PER; p++)
        if (col[p] == colour && inv[p] != 0.f)
          xs[at[p]] = (bb[p] + C.sum(xs + at[p], p)) * inv[p];
      __syncthreads();
    }
  }
#pragma unroll
  for (int p = 0; p < G::PER; p++)
    if (t + G::NT * p < G::N) x[r.off + t + G::NT * p] = from_f<VT>(xs[at[p]]);
}

// Coarsest level: x = A^-1 b with the dense FP64 inverse (symmetric).  A CTA has 16
// rows and 32 parts of the columns, summed part by part in a fixed order.  (One CTA with
// a thread per row reads up to 2 MB of the inverse alone: 45 us at 500 cells.)
constexpr int COARSE_ROWS = 16, COARSE_PARTS = 32;
template <typename VT>
__global__ void __launch_bounds__(COARSE_ROWS* COARSE_PARTS)
    k_coarse_solve(const double* __restrict__ Ainv, int n, const int64_t* __restrict__ cells,
                   const VT* b, VT* x) {
  __shared__ double bs[512];
  __shared__ double part[COARSE_PARTS][COARSE_ROWS];
  const int t = threadIdx.x, r = t % COARSE_ROWS, q = t / COARSE_ROWS;
  const int row = blockIdx.x * COARSE_ROWS + r;
  pdl_go();
  pdl_wait();
  for (int i = t; i < n; i += COARSE_ROWS * COARSE_PARTS) bs[i] = to_f(b[cells[i]]);
  __syncthreads();
  double s = 0;
  if (row < n) {
#pragma unroll 8
    for (int j = q; j < n; j += COARSE_PARTS) s += Ainv[(size_t)j * n + row] * bs[j];
  }
  part[q][r] = s;
  __syncthreads();
  if (t >= COARSE_ROWS || row >= n) return;
  s = 0;
#pragma unroll
  for (int i = 0; i < COARSE_PARTS; i++) s += part[i][t];
  x[cells[row]] = from_f<VT>((float)s);
}
