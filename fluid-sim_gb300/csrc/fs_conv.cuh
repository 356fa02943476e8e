// fs_conv.cuh -- the tensor-core convolution as the network calls it (fs_conv.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace fs {
namespace conv {

// what the epilogue does with a layer's output (bias added), as flags
enum {
  kOutStore = 1,      // bf16 NHWC to out
  kOutRelu = 2,       // after ReLU
  kOutPlanar = 4,     // instead: channel 0 as f32 planes to out (c_out must be 16)
  kOutMask = 8,       // 0 where mask (same shape) is not > 0
  kOutPool = 16,      // 2 x 2 sums times pool_scale to pool
  kOutPoolMask = 32,  // those 0 where pool_mask is not > 0
  kOutUp = 64,        // fine + scale * (nearest upsampling) to up (twice the size)
  kOutUpMask = 128    // those 0 where up_mask is not > 0
};

struct ConvOut {
  void* out = nullptr;
  const void* mask = nullptr;
  void* pool = nullptr;
  const void* pool_mask = nullptr;
  float pool_scale = 1.f;
  void* up = nullptr;
  const void* fine = nullptr;
  const void* up_mask = nullptr;
  float scale = 1.f;
};

// images of B x H x W pixels; the flag combinations the network uses.  dependent:
// the launch may start while the one ahead of it finishes, which has not written w
cudaError_t conv3x3(int cin, int cout, int flags, const void* in, const void* w, const float* bias, const ConvOut& o,
                    int B, int H, int W, int* err, cudaStream_t st, bool dependent = false);

}  // namespace conv
}  // namespace fs
