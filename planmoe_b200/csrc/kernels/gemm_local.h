// Entry points of kernels/gemm_local.cu for the GEMM launcher.
#pragma once

#include "planmoe.h"

#include <cuda.h>
#include <cuda_bf16.h>

namespace planmoe {

constexpr int kLocalMaxGroups = 64;

struct LocalGemm {
  int groups, M, N, K;
  int activation, has_aux;
  const __nv_bfloat16* bias;     // [groups][N] or null
  const int* rows_used;          // [groups] token rows in use (M dim, or the contraction of a weight gradient), or null
  float* colsum;                 // see GemmArgs
  unsigned long long budget_ns;
  int* status;
};

// Whether the kernel exists for an epilogue and operand layouts.
bool local_gemm_takes(int epilogue, bool a_mn, bool b_mn);

// `ta` / `tb`: boxes of 128 (K-major) or 64 (MN-major) rows; `td`: D, `tx`: the activation derivative, 64 x 32 boxes.  `ctas`:
// even, all resident at once.
cudaError_t launch_local_gemm(int epilogue, bool a_mn, bool b_mn, const CUtensorMap& ta, const CUtensorMap& tb,
                             const CUtensorMap& td, const CUtensorMap& tx, const LocalGemm& p, int ctas, cudaStream_t stream);

}  // namespace planmoe
