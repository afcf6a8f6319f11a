// nn_tile.h — the tile kernels of nn_conv_tile.cu (forward, data gradient)
// and nn_wgrad_tile.cu as nn_conv.cu's launchers see them.  Each returns false when it does not
// take the shape or alignment (nothing was launched); otherwise *e holds the
// launch's result.
#pragma once
#include <cuda.h>

#include "nn.h"

namespace rtx {
namespace nn {

// wide: additions in slab-major order (the rule for rows of 64 pixels or
// more), else tap-major
bool conv_tile_fwd(const ConvFwd& a, bool wide, cudaStream_t st, cudaError_t* e);
bool conv_tile_head(const ConvFwd& a, const KpHead& h, cudaStream_t st, cudaError_t* e);
bool conv_tile_dgrad(const ConvDgrad& a, bool wide, cudaStream_t st, cudaError_t* e);

bool conv_tile_wgrad(const ConvWgrad& a, cudaStream_t st, cudaError_t* e);

// Tensor map of a BF16 NHWC tensor's every step_x-th pixel of every step_y-th
// row as (C, x, y, image), H x W counted in those pixels: swizzled boxes of KC
// channels (KC * 2 bytes per pixel row) x bw x bh pixels, zeros outside.
// False if it cannot be encoded.
bool pixel_map(CUtensorMap* m, const bf16* base, int imgs, int H, int W, int C, int step_x, int step_y, int KC, int bw,
               int bh);
int tile_sm_count();

}  // namespace nn
}  // namespace rtx
