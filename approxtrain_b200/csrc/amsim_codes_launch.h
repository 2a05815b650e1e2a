// Host interface of the tensor-core table GEMM (amsim_codes.cu).
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

namespace amsim {

struct CodeParams;

// Tile shapes of code_gemm: 0 = 256 x 256, 1 = 256 x 128, 2 = 256 x 64 (rows of V x columns of U of a CTA pair).
struct CodeTile {
  int bm, bn;
  size_t slot_bytes;  // one parked tile (both CTAs' halves)
  int accumulators;   // tiles in tensor memory whose sum is a chunk's
};
CodeTile code_tile(int shape);
cudaError_t code_gemm_launch(cudaStream_t st, const CodeParams& cp, int shape, int device);

}  // namespace amsim
