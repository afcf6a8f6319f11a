// nn_tile.h — the tile kernels of nn_conv_tile.cu (forward and data gradient)
// as nn_conv.cu's launchers see them.  Each returns false when it does not
// take the shape or alignment (nothing was launched); otherwise *e holds the
// launch's result.
#pragma once
#include <cuda.h>

#include "nn.h"

namespace rtx {
namespace nn {

bool conv_tile_fwd(const ConvFwd& a, cudaStream_t st, cudaError_t* e);
bool conv_tile_dgrad(const ConvDgrad& a, cudaStream_t st, cudaError_t* e);

// Tensor map of an [imgs][H * step][W * step][C] BF16 tensor as (C, x, y,
// image) over every step-th pixel and row, swizzled boxes of KC channels x bw
// x bh pixels (KC * 2 bytes per pixel row; zeros outside the image).  False
// if it cannot be encoded.
bool pixel_map(CUtensorMap* m, const bf16* base, int imgs, int H, int W, int C, int step, int KC, int bw, int bh);
int tile_sm_count();

}  // namespace nn
}  // namespace rtx
