// Entry points of kernels/gemm_local.cu and kernels/gemm_stream.cu for the GEMM launcher.
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
  float* q8_scales;              // kEpiStoreQ8
  unsigned long long budget_ns;
  int* status;
};

// Whether the kernel exists for an epilogue and operand layouts.
bool local_gemm_takes(int epilogue, bool a_mn, bool b_mn);

// `ta` / `tb`: boxes of 128 (K-major) or 64 (MN-major) rows; `td`: D, `tx`: the activation derivative, 64 x 32 boxes
// (kEpiStoreQ8: D as uint8 [groups * M][N], 128 x 32 boxes).  `ctas`:
// even, all resident at once.
cudaError_t launch_local_gemm(int epilogue, bool a_mn, bool b_mn, const CUtensorMap& ta, const CUtensorMap& tb,
                             const CUtensorMap& td, const CUtensorMap& tx, const LocalGemm& p, int ctas, cudaStream_t stream);

// kernels/gemm_stream.cu: at most kStreamRows rows a group, B MN-major, D = act(A . B + bias), aux (optional) = act'.
constexpr int kStreamRows = 32;
struct StreamGemm {
  int groups, M, N, K;
  int activation;
  const __nv_bfloat16* bias;     // [groups][N], on 16 bytes, or null
  __nv_bfloat16* D; long long d_row_stride, d_group_stride;
  __nv_bfloat16* aux; long long aux_row_stride, aux_group_stride;
  const int* rows_used;          // [groups] rows in use, or null; the rows of a group without any are zeros
  unsigned long long budget_ns;
  int* status;
};
bool stream_gemm_pays(int groups, int M, int N, int sms);
// `ta`: boxes of kStreamRows rows, `tb`: of 64
cudaError_t launch_stream_gemm(const CUtensorMap& ta, const CUtensorMap& tb, const StreamGemm& p, cudaStream_t stream);

}  // namespace planmoe
