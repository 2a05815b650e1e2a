// Launches of the tensor-core table GEMM (amsim_codes.cuh).  Compiled on its own by _build.py, in
// parallel with amsim.cu (-DAMSIM_SPLIT_TU), or included by amsim.cu when that is built alone.
#ifdef AMSIM_SPLIT_TU
#define AMSIM_TEMPLATES_ONLY
#include <algorithm>
#include <mutex>
#endif
#include "amsim_codes.cuh"
#include "amsim_codes_launch.h"

namespace amsim {
namespace {

template <int S, int BN>
cudaError_t code_launch_t(cudaStream_t st, const CodeParams& cp, int device) {
  using L = CodeSmem<S, BN>;
  static std::mutex mu;
  static size_t allowed[64] = {};
  const size_t smem = L::bytes(cp.rows_v, cp.rows_u);
  if (device >= 0 && device < 64) {
    std::lock_guard<std::mutex> lk(mu);
    if (allowed[device] < smem) {
      const cudaError_t e = cudaFuncSetAttribute(code_gemm<S, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return e;
      allowed[device] = smem;
    }
  }
  code_gemm<S, BN><<<2 * cp.prm.sk_grid, L::NT, smem, st>>>(cp);
  return cudaGetLastError();
}

template <int S>
cudaError_t code_launch_s(cudaStream_t st, const CodeParams& cp, int shape, int device) {
  if (shape == 0) return code_launch_t<S, 256>(st, cp, device);
  if (shape == 1) return code_launch_t<S, 128>(st, cp, device);
  return code_launch_t<S, 64>(st, cp, device);
}

}  // namespace

CodeTile code_tile(int shape) {
  if (shape == 0) return {CT_ROWS, 256, (size_t)CodeAcc<64, 256>::SLOT_FLOATS * 8, CodeSmem<64, 256>::NACC};
  if (shape == 1) return {CT_ROWS, 128, (size_t)CodeAcc<64, 128>::SLOT_FLOATS * 8, CodeSmem<64, 128>::NACC};
  return {CT_ROWS, 64, (size_t)CodeAcc<64, 64>::SLOT_FLOATS * 8, CodeSmem<64, 64>::NACC};
}

cudaError_t code_gemm_launch(cudaStream_t st, const CodeParams& cp, int shape, int device) {
  if (cp.prm.ct_slots == 32) return code_launch_s<32>(st, cp, shape, device);
  if (cp.prm.ct_slots == 64) return code_launch_s<64>(st, cp, shape, device);
  return code_launch_s<128>(st, cp, shape, device);
}

}  // namespace amsim
