// The learned 3D CNN of the pressure solver: shapes, weight layout and the
// device kernels (forward / backward-data convolution on the tensor cores,
// weight gradients, loss, Adam).  No counterpart in the reference.
//
// Network (per 16^3 tile with a 1-cell halo, 18^3 inputs):
//   conv1 4->16, 3^3, valid on the 18^3 box (-> 16^3), ReLU
//   conv2 16->16, 3^3, zero padding, ReLU
//   conv3 16->16, 3^3, zero padding, ReLU
//   conv4 16->1,  3^3, zero padding
// No biases: the network is positively homogeneous in its value channel
// scale, which the per-tile normalisation relies on.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "msbg_cnn.h"

namespace msbg {
namespace cnn {

constexpr int TS = 16;                  // tile edge
constexpr int PD = 18;                  // padded edge
constexpr int NPAD = PD * PD * PD;      // 5832 padded cells
constexpr int NCELL = TS * TS * TS;     // 4096 cells
constexpr int NC = 16;                  // channels of the hidden layers
constexpr int NFEAT = 4;                // input channels
constexpr int NLAYER = 4;
constexpr uint32_t HALF_BYTES = NPAD * 16;  // one channel half (8 x bf16) of the padded box
constexpr int WIMG = 27 * 256;              // bf16 elements of one layer's weight image

// Master weights, FP32, PyTorch Conv3d order per layer: [cout][cin][kz][ky][kx].
__host__ __device__ constexpr int layer_cin(int l) { return l == 0 ? NFEAT : NC; }
__host__ __device__ constexpr int layer_cout(int l) { return l == NLAYER - 1 ? 1 : NC; }
__host__ __device__ constexpr int layer_off(int l) {
  return l == 0 ? 0 : l == 1 ? 27 * NFEAT * NC : l == 2 ? 27 * NFEAT * NC + 27 * NC * NC
                                                        : 27 * NFEAT * NC + 2 * 27 * NC * NC;
}
constexpr int NPARAM = 27 * NFEAT * NC + 2 * 27 * NC * NC + 27 * NC;  // 15984

// Activation tensors in global memory use the shared-memory layout of the
// convolution: per tile two channel halves, each NPAD padded cells x 16 bytes
// (8 bf16 channels), z slowest; halo cells are zero except in the first
// layer's input.  One padded z plane of one half is PLANE_BYTES contiguous.
constexpr int PLANE = PD * PD;
constexpr uint32_t PLANE_BYTES = PLANE * 16;        // 5184
constexpr size_t ACT_BYTES = 2 * (size_t)HALF_BYTES;  // per tile
__host__ __device__ constexpr int pad_index(int cell) {
  return (cell % TS + 1) + PD * ((cell / TS) % TS + 1 + PD * (cell / (TS * TS) + 1));
}

enum { EPI_RELU = 0, EPI_MASK = 1, EPI_OUT0 = 2 };

// One layer of a chain.  out: padded layout in global memory, interior written
// (null: not kept); mask (EPI_MASK): padded layout, out = acc where mask > 0.
struct ConvLayer {
  uint4* out;
  const uint4* mask;
  const __nv_bfloat16* wimg;          // [9][2][48][8] bf16 image of the layer
  int epi;
};
struct ConvChain {
  int n, nl;                          // tiles, layers
  // the first layer's input: FP32 features [n][4][NPAD] (packed into half 0 of x0
  // too, if given), or half 0 of a padded layout
  const float* feat;
  const uint4* in;
  uint4* x0;
  ConvLayer L[NLAYER];
  float* out0;                        // EPI_OUT0: channel 0
  const int64_t* outOff;              // EPI_OUT0: per-tile first cell in out0 (null: t*NCELL)
  const float* outScale;              // EPI_OUT0: per-tile factor (null: 1)
  int* err;                           // set when a bounded wait gives up
};

// 16 epilogue warps, one that issues MMAs, 4 that fill the ring.  Shared memory:
// 16 planes of activations (166 KB), two weight images (28 KB), the ring (36 KB).
constexpr int EPI_WARPS = 16;
constexpr int CONV_THREADS = (EPI_WARPS + 5) * 32;
constexpr int CONV_SLOTS = 6;
constexpr size_t CONV_SMEM = TS * 2 * (size_t)PLANE_BYTES + 2 * WIMG * 2 +
                             (CONV_SLOTS + 1) * (size_t)PLANE_BYTES +
                             (PD + TS + 2 * CONV_SLOTS + 2) * 8 + 16;
static_assert(CONV_SMEM <= 227 * 1024, "one CTA's shared memory");

// Inference of n tiles on stream st: out0[outOff[t] + cell] = outScale[t] *
// net(feat[t]) (cnn.cu).
int forward(msbg_cnn* net, const float* feat, float* out0, const int64_t* outOff,
            const float* outScale, int n, cudaStream_t st);
// Status of the network's bounded waits since the last call (0 = none gave up); clears it.
int take_error(msbg_cnn* net, cudaStream_t st);

}  // namespace cnn
}  // namespace msbg
