// Allocation-free variant of get_marked_video (stspix_get_marked_video_noalloc).
//
// Some callers cannot allocate device memory at call time, and have no engine context: a
// process that reserves all of its GPU memory up front and forbids later cudaMalloc, a
// plugin whose host application owns every device allocation, or a real-time loop where an
// allocation (and the device synchronisation cudaFree implies) is not allowed.
//
// Rules:
//  * inputs of up to kMarkedMaxPixels = 2^24 pixels (T*H*W across all frames); larger
//    inputs are rejected with STSPIX_ERR_TOO_LARGE before any work;
//  * frames have 3 channels (nftrs == 3), as for stspix_get_marked_video;
//  * `stream` must belong to the current device (checked: STSPIX_ERR_ARG otherwise);
//  * launch failures are read from the launch call itself, so an error left
//    pending by unrelated earlier work is neither reported here nor cleared.
#include <cstdint>

#include <cuda_runtime.h>

#include "engine.h"
#include "kernels.h"

namespace {
constexpr long long kMarkedMaxPixels = 1LL << 24;
}  // namespace

extern "C" int stspix_get_marked_video_noalloc(void* stream, const float* vid,
                                                const int32_t* spix, const float* color, int T,
                                                int H, int W, int nftrs, float* marked_out) {
  if (!vid || !spix || !color || !marked_out) return STSPIX_ERR_ARG;
  if (nftrs != 3 || T < 0 || H < 1 || W < 1) return STSPIX_ERR_ARG;
  const long long n = (long long)T * H * W;
  if (n > kMarkedMaxPixels) return STSPIX_ERR_TOO_LARGE;
  if (n == 0) return STSPIX_OK;
  int dev = -1, sdev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess) return STSPIX_ERR_CUDA;
  cudaStream_t st = (cudaStream_t)stream;
  if (cudaStreamGetDevice(st, &sdev) != cudaSuccess) return STSPIX_ERR_ARG;
  if (sdev != dev) return STSPIX_ERR_ARG;
  const unsigned blocks = (unsigned)((n + stspix::kMarkPix - 1) / stspix::kMarkPix);
  int h = H, w = W;
  long long nn = n;
  void* a[] = {(void*)&marked_out, (void*)&vid, (void*)&spix, (void*)&color,
               (void*)&h, (void*)&w, (void*)&nn};
  if (cudaLaunchKernel((const void*)stspix::k_marked, dim3(blocks), dim3(256), a, 0, st) !=
      cudaSuccess)
    return STSPIX_ERR_CUDA;
  return STSPIX_OK;
}
