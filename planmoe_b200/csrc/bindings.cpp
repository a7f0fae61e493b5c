// Python bindings of the planmoe_b200 native extension (module planmoe_b200._C).
//
// Thin adapters from torch::Tensor to the raw-pointer launchers of planmoe.h; every CUDA op
// runs on the current torch stream.  The list of exported functions covers what the
// reference binds in PlanMoE/custom/custom_kernel.cpp:292-321 (CPU sparse ops, JIT invoke,
// collective bootstrap, codec/comm pipeline), re-expressed for this design: the NCCL bootstrap
// becomes the symmetric-heap runtime, the FIFO compress/comm/decompress triple becomes explicit
// handles on the Python side.

#include <climits>
#include <torch/extension.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAStream.h>
#include <c10/cuda/CUDAGuard.h>

#include "planmoe.h"
#include "runtime/symm_heap.h"
#include "runtime/jit.h"
#include "codec/codecs.h"
#include "codec/abstract.h"
#include "comm/abstract.h"

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <atomic>

namespace py = pybind11;
using torch::Tensor;
using namespace planmoe;

namespace {

cudaStream_t cur_stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

// Kernels of this extension launched so far in this process (benchmarks report the delta).
std::atomic<long long> g_launches{0};
void count_launch(int n) { g_launches.fetch_add(n, std::memory_order_relaxed); }

void check_cuda(cudaError_t e, const char* what) {
  TORCH_CHECK(e == cudaSuccess, what, ": ", cudaGetErrorString(e));
}

#define DISPATCH_FLOAT(t, NAME, ...)                                                     \
  [&] {                                                                                  \
    switch ((t).scalar_type()) {                                                         \
      case at::kFloat: { using scalar_t = float; return __VA_ARGS__(); }                 \
      case at::kBFloat16: { using scalar_t = __nv_bfloat16; return __VA_ARGS__(); }      \
      case at::kHalf: { using scalar_t = __half; return __VA_ARGS__(); }                 \
      default: TORCH_CHECK(false, NAME, ": unsupported dtype ", (t).scalar_type());      \
    }                                                                                    \
  }()

const float* opt_f32(const c10::optional<Tensor>& t) {
  if (!t.has_value() || !t->defined()) return nullptr;
  TORCH_CHECK(t->scalar_type() == at::kFloat && t->is_contiguous(), "gates must be contiguous fp32");
  return t->data_ptr<float>();
}

// What kernels that move rows as 16-byte vectors read: a contiguous view may start anywhere in its storage, and a vector
// access off its boundary is a fault.
const void* rows16(const Tensor& t) {
  TORCH_CHECK(t.is_contiguous() && reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0, "rows must be contiguous and 16-byte aligned");
  return t.data_ptr();
}

// ---- CPU sparse ops -------------------------------------------------------------------------
template <class T>
const T* opt_ptr(const c10::optional<Tensor>& t) {
  return (t.has_value() && t->defined()) ? t->data_ptr<T>() : nullptr;
}

Tensor cpu_scatter_op(const Tensor& x, const Tensor& idx, const Tensor& loc, const c10::optional<Tensor>& gates,
                      int64_t E, int64_t C) {
  TORCH_CHECK(!x.is_cuda() && x.dim() == 2 && x.is_contiguous());
  const int K = idx.size(0), S = idx.size(1), M = x.size(1);
  Tensor out = torch::empty({E * C, M}, x.options());
  if (x.scalar_type() == at::kFloat)
    cpu_scatter<float>(x.data_ptr<float>(), idx.data_ptr<int>(), loc.data_ptr<int>(), opt_ptr<float>(gates),
                       out.data_ptr<float>(), K, S, M, E, C);
  else
    cpu_scatter<double>(x.data_ptr<double>(), idx.data_ptr<int>(), loc.data_ptr<int>(), opt_ptr<double>(gates),
                        out.data_ptr<double>(), K, S, M, E, C);
  return out;
}
Tensor cpu_gather_op(const Tensor& disp, const Tensor& idx, const Tensor& loc, const c10::optional<Tensor>& gates,
                     int64_t C) {
  TORCH_CHECK(!disp.is_cuda() && disp.dim() == 2 && disp.is_contiguous());
  const int K = idx.size(0), S = idx.size(1), M = disp.size(1);
  Tensor out = torch::empty({S, M}, disp.options());
  if (disp.scalar_type() == at::kFloat)
    cpu_gather<float>(disp.data_ptr<float>(), idx.data_ptr<int>(), loc.data_ptr<int>(), opt_ptr<float>(gates),
                      out.data_ptr<float>(), K, S, M, C);
  else
    cpu_gather<double>(disp.data_ptr<double>(), idx.data_ptr<int>(), loc.data_ptr<int>(), opt_ptr<double>(gates),
                       out.data_ptr<double>(), K, S, M, C);
  return out;
}
Tensor cpu_gate_grad_op(const Tensor& disp, const Tensor& dy, const Tensor& idx, const Tensor& loc, int64_t C) {
  TORCH_CHECK(!disp.is_cuda() && disp.is_contiguous() && dy.is_contiguous());
  const int K = idx.size(0), S = idx.size(1), M = disp.size(1);
  Tensor out = torch::empty({K, S}, disp.options());
  if (disp.scalar_type() == at::kFloat)
    cpu_gate_grad<float>(disp.data_ptr<float>(), dy.data_ptr<float>(), idx.data_ptr<int>(), loc.data_ptr<int>(),
                         out.data_ptr<float>(), K, S, M, C);
  else
    cpu_gate_grad<double>(disp.data_ptr<double>(), dy.data_ptr<double>(), idx.data_ptr<int>(), loc.data_ptr<int>(),
                          out.data_ptr<double>(), K, S, M, C);
  return out;
}

// ---- CUDA dispatch ops ----------------------------------------------------------------------
Tensor build_slot_map_op(const Tensor& idx, const Tensor& loc, int64_t E, int64_t C) {
  count_launch(1);
  TORCH_CHECK(idx.is_cuda() && idx.scalar_type() == at::kInt && idx.is_contiguous() && loc.is_contiguous());
  c10::cuda::CUDAGuard guard(idx.device());
  Tensor smap = torch::empty({E * C}, idx.options());
  launch_build_slot_map(idx.data_ptr<int>(), loc.data_ptr<int>(), smap.data_ptr<int>(), idx.size(0), idx.size(1), E, C,
                        cur_stream());
  return smap;
}

Tensor dispatch_scatter_op(const Tensor& x, const Tensor& slot_map, const c10::optional<Tensor>& gates, int64_t K,
                           int64_t n_slots, bool round_gates) {
  count_launch(1);
  TORCH_CHECK(x.is_cuda() && x.dim() == 2 && x.is_contiguous(), "x must be contiguous [S, M] on CUDA");
  const int S = x.size(0), M = x.size(1);
  TORCH_CHECK((M * x.element_size()) % 16 == 0, "row bytes must be a multiple of 16");
  c10::cuda::CUDAGuard guard(x.device());
  Tensor out = torch::empty({n_slots, M}, x.options());
  DISPATCH_FLOAT(x, "dispatch_scatter", [&] {
    launch_scatter_rows<scalar_t>(reinterpret_cast<const scalar_t*>(rows16(x)), slot_map.data_ptr<int>(),
                                  opt_f32(gates), reinterpret_cast<scalar_t*>(out.data_ptr()), K, S, M, 1, n_slots,
                                  nullptr, false, cur_stream(), round_gates);
  });
  return out;
}

Tensor dispatch_gather_op(const Tensor& disp, const Tensor& idx, const Tensor& loc, const c10::optional<Tensor>& gates,
                          int64_t C, bool round_gates) {
  count_launch(1);
  TORCH_CHECK(disp.is_cuda() && disp.dim() == 2 && disp.is_contiguous());
  const int K = idx.size(0), S = idx.size(1), M = disp.size(1);
  TORCH_CHECK(K <= 8, "top-k above 8 is not supported by the gather kernel");
  TORCH_CHECK((M * disp.element_size()) % 16 == 0, "row bytes must be a multiple of 16");
  c10::cuda::CUDAGuard guard(disp.device());
  Tensor out = torch::empty({S, M}, disp.options());
  DISPATCH_FLOAT(disp, "dispatch_gather", [&] {
    launch_gather_rows<scalar_t>(rows16(disp), nullptr, idx.data_ptr<int>(), loc.data_ptr<int>(), opt_f32(gates),
                                 reinterpret_cast<scalar_t*>(out.data_ptr()), K, S, M, C, nullptr, cur_stream(), 0, round_gates);
  });
  return out;
}

Tensor dispatch_gate_grad_op(const Tensor& disp, const Tensor& dy, const Tensor& idx, const Tensor& loc, int64_t C) {
  count_launch(1);
  TORCH_CHECK(disp.is_cuda() && disp.is_contiguous() && dy.is_contiguous() && disp.scalar_type() == dy.scalar_type());
  TORCH_CHECK((disp.size(1) * disp.element_size()) % 16 == 0, "row bytes must be a multiple of 16");
  const int K = idx.size(0), S = idx.size(1), M = disp.size(1);
  c10::cuda::CUDAGuard guard(disp.device());
  Tensor out = torch::empty({K, S}, disp.options().dtype(at::kFloat));
  DISPATCH_FLOAT(disp, "dispatch_gate_grad", [&] {
    launch_gate_grad<scalar_t>(reinterpret_cast<const scalar_t*>(rows16(disp)),
                               reinterpret_cast<const scalar_t*>(rows16(dy)), idx.data_ptr<int>(),
                               loc.data_ptr<int>(), out.data_ptr<float>(), nullptr, nullptr, K, S, M, C, cur_stream());
  });
  return out;
}

// Gate gradient plus the gate-weighted copies of dy: returns (dgates [K, S] fp32, scaled [S * K, M]) with
// scaled[t * K + k] = gates[k][t] * dy[t] for every pick that holds a slot (other rows are left unwritten).
std::vector<Tensor> dispatch_gate_grad_scaled_op(const Tensor& disp, const Tensor& dy, const Tensor& idx,
                                                 const Tensor& loc, const Tensor& gates, int64_t C) {
  count_launch(1);
  TORCH_CHECK(disp.is_cuda() && disp.is_contiguous() && dy.is_contiguous() && disp.scalar_type() == dy.scalar_type());
  TORCH_CHECK((disp.size(1) * disp.element_size()) % 16 == 0, "row bytes must be a multiple of 16");
  TORCH_CHECK(gates.is_cuda() && gates.scalar_type() == at::kFloat && gates.is_contiguous());
  const int K = idx.size(0), S = idx.size(1), M = disp.size(1);
  TORCH_CHECK(gates.numel() == (int64_t)K * S && dy.size(0) == S && dy.size(1) == M);
  c10::cuda::CUDAGuard guard(disp.device());
  Tensor out = torch::empty({K, S}, disp.options().dtype(at::kFloat));
  Tensor scaled = torch::empty({(int64_t)S * K, (int64_t)M}, dy.options());
  DISPATCH_FLOAT(disp, "dispatch_gate_grad_scaled", [&] {
    launch_gate_grad<scalar_t>(reinterpret_cast<const scalar_t*>(rows16(disp)),
                               reinterpret_cast<const scalar_t*>(rows16(dy)), idx.data_ptr<int>(),
                               loc.data_ptr<int>(), out.data_ptr<float>(), gates.data_ptr<float>(),
                               reinterpret_cast<scalar_t*>(scaled.data_ptr()), K, S, M, C, cur_stream());
  });
  return {out, scaled};
}

// The same for expert outputs that arrived as uint8 rows with a (scale, low) pair per 128 columns and row (the int8
// push epilogue's layout): `disp_ptr` uint8 [E * C, M], `scales_ptr` fp32 [M / 128][group_rows][2].  `gates` may be
// absent (then no scaled copies are produced and the second result is empty).  The scaled copies come out as int8 wire
// rows, uint8 [S * K, M + 16]: M quantised bytes + {scale, low, 0, 0}.
std::vector<Tensor> dispatch_gate_grad_q8_op(int64_t disp_ptr, int64_t scales_ptr, int64_t group_rows, const Tensor& dy,
                                             const Tensor& idx, const Tensor& loc, const c10::optional<Tensor>& gates,
                                             int64_t C, bool want_scaled) {
  count_launch(1);
  TORCH_CHECK(dy.is_cuda() && dy.is_contiguous() && dy.dim() == 2 && dy.size(1) % 128 == 0);
  const int K = idx.size(0), S = idx.size(1), M = dy.size(1);
  c10::cuda::CUDAGuard guard(dy.device());
  Tensor out = torch::empty({K, S}, dy.options().dtype(at::kFloat));
  Tensor scaled;       // int8 wire rows [S * K, M + 16] of gate * dy (rows of picks without a slot stay unwritten)
  if (want_scaled) {
    TORCH_CHECK(gates.has_value() && gates->defined(), "scaled copies need the gates");
    scaled = torch::empty({(int64_t)S * K, (int64_t)M + 16}, dy.options().dtype(at::kByte));
  }
  DISPATCH_FLOAT(dy, "dispatch_gate_grad_q8", [&] {
    launch_gate_grad<scalar_t>(reinterpret_cast<const scalar_t*>(disp_ptr), reinterpret_cast<const scalar_t*>(rows16(dy)),
                               idx.data_ptr<int>(), loc.data_ptr<int>(), out.data_ptr<float>(), opt_f32(gates),
                               nullptr, K, S, M, C, cur_stream(), reinterpret_cast<const float*>(scales_ptr), group_rows,
                               want_scaled ? scaled.data_ptr<uint8_t>() : nullptr);
  });
  return {out, want_scaled ? scaled : Tensor()};
}

// (rank [S] i32, perm [S] i32) of the batch-prioritised token order
std::vector<Tensor> importance_order_op(const Tensor& logits) {
  count_launch(2);
  TORCH_CHECK(logits.is_cuda() && logits.dim() == 2 && logits.is_contiguous());
  const int S = logits.size(0), E = logits.size(1);
  c10::cuda::CUDAGuard guard(logits.device());
  Tensor ws = torch::empty({importance_workspace(S)}, logits.options().dtype(at::kLong));
  Tensor rank = torch::empty({S}, logits.options().dtype(at::kInt)), perm = torch::empty({S}, logits.options().dtype(at::kInt));
  DISPATCH_FLOAT(logits, "importance_order", [&] {
    launch_importance_order<scalar_t>(reinterpret_cast<const scalar_t*>(logits.data_ptr()), S, E,
                                      reinterpret_cast<unsigned long long*>(ws.data_ptr()), rank.data_ptr<int>(), perm.data_ptr<int>(), cur_stream());
  });
  return {rank, perm};
}
void remap_slot_map_op(Tensor& slot_map, const Tensor& perm, int64_t K) {
  count_launch(1);
  TORCH_CHECK(slot_map.is_cuda() && slot_map.is_contiguous() && slot_map.scalar_type() == at::kInt && perm.scalar_type() == at::kInt);
  c10::cuda::CUDAGuard guard(slot_map.device());
  launch_remap_slot_map(slot_map.data_ptr<int>(), slot_map.numel(), perm.data_ptr<int>(), (int)K, cur_stream());
}

// ---- fused gate -------------------------------------------------------------------------------
// returns (idx[K,S] i32, loc[K,S] i32, gates[K,S] f32, slot_map[E*C] i32, top1_count[E] i32, l_aux[1] f32)
constexpr float kFloatEps = 1.1920929e-07f;
float gate_eps(at::ScalarType t) { return t == at::kFloat ? kFloatEps : (t == at::kHalf ? 9.765625e-04f : 7.8125e-03f); }

// {idx, loc, gates, slot_map, top1, l_aux, used}
std::vector<Tensor> gate_forward_used_op(const Tensor& logits, int64_t K, int64_t C, bool normalize) {
  count_launch(2);
  TORCH_CHECK(logits.is_cuda() && logits.dim() == 2 && logits.is_contiguous());
  const int S = logits.size(0), E = logits.size(1);
  TORCH_CHECK(E <= 64 && K <= 4 && K <= E, "fused gate supports up to 64 experts and top-4");
  c10::cuda::CUDAGuard guard(logits.device());
  auto iopt = logits.options().dtype(at::kInt);
  auto fopt = logits.options().dtype(at::kFloat);
  const int nblk = gate_workspace_blocks(S);
  Tensor idx = torch::empty({K, S}, iopt), loc = torch::empty({K, S}, iopt);
  Tensor gates = torch::empty({K, S}, fopt);
  Tensor smap = torch::empty({(int64_t)E * C}, iopt);
  Tensor top1 = torch::empty({2, E}, iopt), laux = torch::empty({1}, fopt);   // first picks, used slots of every expert
  // scratch of this call: raw gates, in-block ranks, per-block histograms and score sums
  Tensor ws = torch::empty({2 * K * S + (K + 1) * (int64_t)nblk * E}, iopt);
  int* w = ws.data_ptr<int>();
  GatePtrs gp{};
  for (int k = 0; k < K; ++k) gp.p[k] = gates.data_ptr<float>() + (int64_t)k * S;
  DISPATCH_FLOAT(logits, "gate_forward", [&] {
    launch_gate_forward<scalar_t, false>(reinterpret_cast<const scalar_t*>(logits.data_ptr()), S, E, K, C, normalize,
                                         gate_eps(logits.scalar_type()), idx.data_ptr<int>(), loc.data_ptr<int>(), gp,
                                         reinterpret_cast<float*>(w), smap.data_ptr<int>(), top1.data_ptr<int>(),
                                         top1.data_ptr<int>() + E, laux.data_ptr<float>(), w + K * S, w + 2 * K * S,
                                         reinterpret_cast<float*>(w + 2 * K * S + K * (int64_t)nblk * E), cur_stream());
  });
  return {idx, loc, gates, smap, top1[0], laux, top1[1]};
}
std::vector<Tensor> gate_forward_op(const Tensor& logits, int64_t K, int64_t C, bool normalize) {
  std::vector<Tensor> r = gate_forward_used_op(logits, K, C, normalize);
  r.pop_back();
  return r;
}

Tensor gate_backward_op(const Tensor& logits, const Tensor& idx, const c10::optional<Tensor>& dgates,
                        const c10::optional<Tensor>& dl_aux, const Tensor& top1, bool normalize) {
  count_launch(1);
  const int S = logits.size(0), E = logits.size(1), K = idx.size(0);
  c10::cuda::CUDAGuard guard(logits.device());
  Tensor out = torch::empty_like(logits);
  GatePtrs gp{};
  if (opt_f32(dgates) != nullptr)
    for (int k = 0; k < K; ++k) gp.p[k] = dgates->data_ptr<float>() + (int64_t)k * S;
  DISPATCH_FLOAT(logits, "gate_backward", [&] {
    launch_gate_backward<scalar_t, false>(reinterpret_cast<const scalar_t*>(logits.data_ptr()), S, E, K, normalize,
                                          gate_eps(logits.scalar_type()), idx.data_ptr<int>(), gp, opt_f32(dl_aux),
                                          top1.data_ptr<int>(), reinterpret_cast<scalar_t*>(out.data_ptr()), cur_stream());
  });
  return out;
}

// Routing from a [S, E] fp32 score matrix (extract_critical): {idx, loc, slot_map, top1, loss, own, gate of pick 0, 1, ...}.
// own [3, K, S]: idx, loc and gates (fp32) once more, for the gradients and the slots, which no caller gets to write to.
std::vector<Tensor> route_scores_op(const Tensor& scores, int64_t K, int64_t C, bool normalize) {
  count_launch(2);
  TORCH_CHECK(scores.is_cuda() && scores.dim() == 2 && scores.is_contiguous() && scores.scalar_type() == at::kFloat);
  const int64_t S = scores.size(0), E = scores.size(1);
  TORCH_CHECK(S > 0 && E >= 1 && E <= 64 && K >= 1 && K <= 4 && K <= E && C >= 0 && K * S <= INT_MAX,
              "route_scores supports up to 64 experts and top-4");
  c10::cuda::CUDAGuard guard(scores.device());
  auto iopt = scores.options().dtype(at::kInt);
  const int64_t nblk = gate_workspace_blocks(S);
  Tensor idx = torch::empty({K, S}, iopt), loc = torch::empty({K, S}, iopt), smap = torch::empty({E * C}, iopt);
  Tensor top1 = torch::empty({E}, iopt), loss = torch::empty({}, scores.options());
  Tensor own = torch::empty({3, K, S}, iopt);
  Tensor ws = torch::empty({2 * K * S + (K + 1) * nblk * E}, iopt);
  int* w = ws.data_ptr<int>();
  std::vector<Tensor> out{idx, loc, smap, top1, loss, own};
  GatePtrs gp{};
  for (int k = 0; k < K; ++k) {                   // tensors of their own, no views of one another
    out.push_back(torch::empty({S}, scores.options()));
    gp.p[k] = out.back().data_ptr<float>();
  }
  launch_gate_forward<float, true>(scores.data_ptr<float>(), S, E, K, C, normalize, kFloatEps, idx.data_ptr<int>(),
                                   loc.data_ptr<int>(), gp, reinterpret_cast<float*>(w), smap.data_ptr<int>(),
                                   top1.data_ptr<int>(), nullptr, loss.data_ptr<float>(), w + K * S, w + 2 * K * S,
                                   reinterpret_cast<float*>(w + 2 * K * S + K * nblk * E), cur_stream(), nullptr, nullptr,
                                   own.data_ptr<int>());
  return out;
}

// Gradient [S, E] of the scores from that of the gates (picks: own[0]) or, without picks, of the loss.
Tensor route_scores_backward_op(const c10::optional<Tensor>& scores, const c10::optional<Tensor>& picks,
                                const std::vector<c10::optional<Tensor>>& dgates, const c10::optional<Tensor>& dloss,
                                const Tensor& top1, int64_t S, bool normalize) {
  count_launch(1);
  const int64_t E = top1.numel(), K = dgates.size();
  c10::cuda::CUDAGuard guard(top1.device());
  TORCH_CHECK(K == 0 || (scores.has_value() && scores->is_contiguous() && scores->numel() == S * E &&
                         scores->scalar_type() == at::kFloat && picks.has_value() && picks->is_contiguous() &&
                         picks->numel() == K * S));
  Tensor out = torch::empty({S, E}, top1.options().dtype(at::kFloat));
  std::vector<Tensor> keep;
  GatePtrs gp{};
  for (int k = 0; k < K; ++k) {
    if (!dgates[k].has_value() || !dgates[k]->defined()) continue;
    keep.push_back(dgates[k]->to(at::kFloat).contiguous());
    TORCH_CHECK(keep.back().numel() == S);
    gp.p[k] = keep.back().data_ptr<float>();
  }
  Tensor dl;
  if (dloss.has_value() && dloss->defined()) dl = dloss->to(at::kFloat).contiguous();
  launch_gate_backward<float, true>(K > 0 ? scores->data_ptr<float>() : nullptr, S, E, K, normalize, kFloatEps,
                                    K > 0 ? picks->data_ptr<int>() : nullptr, gp,
                                    dl.defined() ? dl.data_ptr<float>() : nullptr, top1.data_ptr<int>(),
                                    out.data_ptr<float>(), cur_stream());
  return out;
}

#include "routing_nodes.h"

Tensor cumsum_sub_one_op(const Tensor& x) {
  count_launch(2);
  TORCH_CHECK(x.is_cuda() && x.dim() == 2 && x.scalar_type() == at::kInt && x.is_contiguous());
  c10::cuda::CUDAGuard guard(x.device());
  const int S = x.size(0), E = x.size(1);
  Tensor out = torch::empty_like(x);
  Tensor ws = torch::empty({cumsum_tiles(S), E}, x.options());
  launch_cumsum_sub_one(x.data_ptr<int>(), out.data_ptr<int>(), ws.data_ptr<int>(), S, E, cur_stream());
  return out;
}

// ---- int8 codec ---------------------------------------------------------------------------------
std::vector<Tensor> int8_encode_op(const Tensor& rows) {
  count_launch(1);
  TORCH_CHECK(rows.is_cuda() && rows.dim() == 2 && rows.is_contiguous());
  c10::cuda::CUDAGuard guard(rows.device());
  const int R = rows.size(0), M = rows.size(1);
  Tensor q = torch::empty({R, M}, rows.options().dtype(at::kByte));
  Tensor scale = torch::empty({R}, rows.options().dtype(at::kFloat)), bias = torch::empty_like(scale);
  DISPATCH_FLOAT(rows, "int8_encode", [&] {
    launch_int8_encode<scalar_t>(reinterpret_cast<const scalar_t*>(rows16(rows)), q.data_ptr<uint8_t>(),
                                 scale.data_ptr<float>(), bias.data_ptr<float>(), R, M, cur_stream());
  });
  return {q, scale, bias};
}
Tensor int8_decode_op(const Tensor& q, const Tensor& scale, const Tensor& bias, at::ScalarType dtype) {
  count_launch(1);
  TORCH_CHECK(q.is_cuda() && q.dim() == 2 && q.is_contiguous() && q.scalar_type() == at::kByte);
  c10::cuda::CUDAGuard guard(q.device());
  const int R = q.size(0), M = q.size(1);
  Tensor out = torch::empty({R, M}, q.options().dtype(dtype));
  DISPATCH_FLOAT(out, "int8_decode", [&] {
    launch_int8_decode<scalar_t>(static_cast<const uint8_t*>(rows16(q)), scale.data_ptr<float>(), bias.data_ptr<float>(),
                                 reinterpret_cast<scalar_t*>(out.data_ptr()), R, M, cur_stream());
  });
  return out;
}

// ---- grouped GEMM ---------------------------------------------------------------------------
// Generic entry: operands are 3-D bf16 tensors [groups, rows, cols] with contiguous last dim
// (4-D [chunks, groups, rows, cols] when `chunks` > 1); `*_mn` says the MN dim is the contiguous one.
struct GemmOpts {
  int64_t epilogue = 0, activation = 0;
  c10::optional<Tensor> bias, aux, out;
  c10::optional<Tensor> q8_out, q8_scales;      // kEpiStoreQ8: uint8 [groups * M, N], fp32 [N / 128, groups * M, 2]
  // flag gate
  int64_t gate_flags_ptr = 0, gate_rows = 0, gate_want = 0, gate_want_ptr = 0;
  int64_t gate_mode = 0, gate_nblk = 0, perm_w = 0, perm_seg_rows = 0, perm_local_first = 0;
  // push
  int64_t heap_bases_ptr = 0, push_data_off = 0, push_flag_off = 0, push_rows = 0, push_C = 0, push_c0 = 0,
          push_chunk = 0, W = 1, my_rank = 0, chunk_groups = 0, push_q8 = 0, push_scale_off = 0;
  int64_t budget_ms = 0, status_ptr = 0, max_ctas = 0, cta_group = 0;
  std::vector<int64_t> heap_bases_host;      // peers' mapped base addresses (push epilogue with bulk stores)
  // dispatch send fused into the launch (copy role)
  c10::optional<Tensor> copy_x, copy_slot_map, copy_gates;
  int64_t copy_K = 0, copy_E_local = 0, copy_C = 0, copy_chunks = 0, copy_ctas = 0, copy_data_off = 0,
          copy_flag_off = 0, copy_nblk = 0;
  // de-quantiser role (int8 wire): local landing buffer, arrival flags (set by peers), ready flags (set by the role)
  int64_t dq_ptr = 0, dq_arrival_ptr = 0, dq_ready_ptr = 0;
  int64_t trace_ptr = 0;                     // optional u64 [grid][8] role trace (see GemmArgs::trace)
  c10::optional<Tensor> rows_used;           // optional int32 [groups] (see GemmArgs::rows_used)
  c10::optional<Tensor> colsum;              // optional fp32 [groups, (M + 31) / 32, N] (see GemmArgs::colsum)
};

GemmOperand operand_of(const Tensor& t, bool mn_major) {
  TORCH_CHECK(t.is_cuda() && t.scalar_type() == at::kBFloat16, "GEMM operands must be CUDA bf16");
  TORCH_CHECK(t.dim() == 3 || t.dim() == 4, "GEMM operand must be [groups, rows, cols] or [chunks, groups, rows, cols]");
  TORCH_CHECK(t.stride(-1) == 1, "GEMM operand needs a contiguous last dim");
  GemmOperand o{};
  o.ptr = t.data_ptr();
  o.mn_major = mn_major ? 1 : 0;
  const int d = t.dim();
  o.rows = t.size(d - 2); o.cols = t.size(d - 1);
  o.row_stride = t.stride(d - 2);
  o.group_stride = t.size(d - 3) > 1 ? t.stride(d - 3) : 0;
  o.chunks = d == 4 ? t.size(0) : 1;
  o.chunk_stride = (d == 4 && t.size(0) > 1) ? t.stride(0) : 0;
  return o;
}

Tensor grouped_gemm_op(const Tensor& A, bool a_mn, const Tensor& B, bool b_mn, const GemmOpts& o) {
  count_launch(1);
  c10::cuda::CUDAGuard guard(A.device());
  GemmArgs g{};
  g.A = operand_of(A, a_mn);
  g.B = operand_of(B, b_mn);
  const int groups = A.size(A.dim() - 3);
  TORCH_CHECK(o.chunk_groups > 0 ? (groups % o.chunk_groups == 0 && B.size(B.dim() - 3) == o.chunk_groups)
                                 : B.size(B.dim() - 3) == groups, "group count mismatch");
  g.groups = groups;
  g.M = a_mn ? g.A.cols : g.A.rows;
  g.K = a_mn ? g.A.rows : g.A.cols;
  g.N = b_mn ? g.B.cols : g.B.rows;
  const int64_t kb = b_mn ? g.B.rows : g.B.cols;
  TORCH_CHECK(kb == g.K, "contraction extents differ: ", g.K, " vs ", kb);
  g.epilogue = o.epilogue; g.activation = o.activation;

  Tensor out;
  if (o.epilogue == kEpiStoreQ8) {
    out = o.q8_out.value();
    g.D = out.data_ptr(); g.d_row_stride = g.N; g.d_group_stride = (long long)g.M * g.N;
    g.q8_scales = o.q8_scales.value().data_ptr<float>();
  } else if (o.epilogue != kEpiPush) {
    if (o.out.has_value() && o.out->defined()) {
      out = *o.out;
      TORCH_CHECK(out.scalar_type() == at::kBFloat16 && out.stride(-1) == 1 && out.dim() == 3);
    } else {
      out = torch::empty({groups, g.M, g.N}, A.options());
    }
    g.D = out.data_ptr(); g.d_row_stride = out.stride(1); g.d_group_stride = out.stride(0);
  }
  if (o.aux.has_value() && o.aux->defined()) {
    const Tensor& aux = *o.aux;
    TORCH_CHECK(aux.scalar_type() == at::kBFloat16 && aux.stride(-1) == 1 && aux.dim() == 3);
    g.aux = aux.data_ptr(); g.aux_row_stride = aux.stride(1); g.aux_group_stride = aux.stride(0);
  } else {
    TORCH_CHECK(o.epilogue != kEpiDAct, "activation-backward epilogue needs aux");
  }
  if (o.bias.has_value() && o.bias->defined()) {
    const Tensor& b = *o.bias;
    TORCH_CHECK(b.scalar_type() == at::kBFloat16 && b.is_contiguous() &&
                b.numel() == (int64_t)(o.chunk_groups > 0 ? o.chunk_groups : groups) * g.N);
    g.bias = b.data_ptr(); g.bias_group_stride = g.N;
  }
  g.gate_flags = reinterpret_cast<const unsigned long long*>(o.gate_flags_ptr);
  g.gate_rows = o.gate_rows; g.gate_want = o.gate_want;
  g.gate_want_ptr = reinterpret_cast<const unsigned long long*>(o.gate_want_ptr);
  g.gate_mode = o.gate_mode; g.gate_nblk = o.gate_nblk; g.perm_w = o.perm_w; g.perm_seg_rows = o.perm_seg_rows; g.perm_local_first = (int)o.perm_local_first;
  g.heap_bases = reinterpret_cast<const unsigned long long*>(o.heap_bases_ptr);
  g.push_data_off = o.push_data_off; g.push_flag_off = o.push_flag_off; g.push_rows = o.push_rows;
  g.push_C = o.push_C; g.push_c0 = o.push_c0; g.push_chunk = o.push_chunk; g.W = o.W; g.my_rank = o.my_rank;
  g.chunk_groups = o.chunk_groups;
  g.push_q8 = o.push_q8; g.push_scale_off = o.push_scale_off;
  std::vector<unsigned long long> bases_host(o.heap_bases_host.begin(), o.heap_bases_host.end());
  if (!bases_host.empty() && (int64_t)bases_host.size() == o.W) g.heap_bases_host = bases_host.data();
  g.budget_ns = (unsigned long long)o.budget_ms * 1000000ull;
  g.status = reinterpret_cast<int*>(o.status_ptr);
  g.trace = reinterpret_cast<unsigned long long*>(o.trace_ptr);
  if (o.rows_used.has_value() && o.rows_used->defined()) {
    const Tensor& u = *o.rows_used;
    TORCH_CHECK(u.is_cuda() && u.scalar_type() == at::kInt && u.is_contiguous() && u.numel() == groups, "rows_used: int32 [groups]");
    g.rows_used = u.data_ptr<int>();
  }
  if (o.colsum.has_value() && o.colsum->defined()) {
    const Tensor& c = *o.colsum;
    TORCH_CHECK(c.is_cuda() && c.scalar_type() == at::kFloat && c.is_contiguous() &&
                c.numel() == (int64_t)groups * ((g.M + 31) / 32) * g.N, "colsum: fp32 [groups, (M + 31) / 32, N]");
    g.colsum = c.data_ptr<float>();
  }
  g.max_ctas = o.max_ctas;
  g.cta_group = o.cta_group;
  if (o.epilogue == kEpiPush) TORCH_CHECK(g.heap_bases != nullptr, "push epilogue needs heap bases");
  if (o.copy_ctas > 0) {
    TORCH_CHECK(o.copy_x.has_value() && o.copy_slot_map.has_value(), "copy role needs x and slot_map");
    const Tensor& cx = *o.copy_x;
    const Tensor& sm = *o.copy_slot_map;
    TORCH_CHECK(cx.is_cuda() && (cx.scalar_type() == at::kBFloat16 || cx.scalar_type() == at::kByte) && cx.dim() == 2 &&
                cx.is_contiguous(), "copy role: x must be contiguous rows, bf16 [S, M] or uint8 [S, M + 16]");
    TORCH_CHECK(sm.is_cuda() && sm.scalar_type() == at::kInt && sm.is_contiguous(), "copy role: slot_map must be int32");
    TORCH_CHECK(g.heap_bases != nullptr && o.copy_K > 0 && o.copy_E_local > 0 && o.copy_C > 0 && o.copy_chunks > 0,
                "copy role: incomplete geometry");
    TORCH_CHECK(sm.numel() == o.copy_E_local * o.W * o.copy_C, "copy role: slot_map size");
    g.copy.x = cx.data_ptr(); g.copy.slot_map = sm.data_ptr<int>();
    g.copy.S = cx.size(0); g.copy.M = cx.size(1);
    if (o.copy_gates.has_value() && o.copy_gates->defined()) {
      const Tensor& cg = *o.copy_gates;
      TORCH_CHECK(cg.is_cuda() && cg.scalar_type() == at::kFloat && cg.is_contiguous() &&
                  cg.numel() == o.copy_K * cx.size(0), "copy role: gates must be fp32 [K, S]");
      g.copy.gates = cg.data_ptr<float>();
    }
    g.copy.K = o.copy_K; g.copy.E_local = o.copy_E_local; g.copy.C = o.copy_C; g.copy.chunks = o.copy_chunks;
    g.copy.ctas = o.copy_ctas; g.copy.data_off = o.copy_data_off; g.copy.flag_off = o.copy_flag_off;
    g.copy.nblk = o.copy_nblk; g.copy.row_bytes = (int)(cx.size(1) * cx.element_size());
  }
  if (o.dq_ptr != 0) {
    g.dequant.q = reinterpret_cast<const void*>(o.dq_ptr);
    g.dequant.arrival = reinterpret_cast<const unsigned long long*>(o.dq_arrival_ptr);
    g.dequant.ready = reinterpret_cast<unsigned long long*>(o.dq_ready_ptr);
    g.dequant.M = g.K;
  }
  check_cuda(launch_grouped_gemm(g, cur_stream()), "grouped_gemm");
  return out;
}

// fp32 column sums [groups / fold, N] of a bf16 [groups, rows, N] tensor; with `as_bf16` the result is
// returned in bf16 (written by the same kernel).  Two launches: partial sums, then their sum.
static void colsum_check(const Tensor& x, int64_t fold) {
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == at::kBFloat16 && x.dim() == 3 && x.stride(2) == 1);
  TORCH_CHECK(fold >= 1 && x.size(0) % fold == 0, "colsum: groups must be a multiple of fold");
  TORCH_CHECK(x.size(2) % 8 == 0 && x.stride(1) % 8 == 0 && x.stride(0) % 8 == 0 &&
              reinterpret_cast<uintptr_t>(x.data_ptr()) % 16 == 0, "colsum needs 16-byte aligned rows");
}

// scratch of one job: [out][partials][counters]; fills `j`, returns the buffer
static Tensor colsum_job(const Tensor& x, int64_t fold, bool as_bf16, ColsumJob& j, Tensor& ob, const int* rows_used = nullptr) {
  const int groups = x.size(0), N = x.size(2);
  const int64_t rows = x.size(1), slabs = colsum_slabs(rows), out_groups = groups / fold;
  const int64_t counters = out_groups * colsum_colblocks(N);
  Tensor buf = torch::empty({out_groups * N + (int64_t)groups * N * slabs + counters}, x.options().dtype(at::kFloat));
  if (as_bf16) ob = torch::empty({out_groups, (int64_t)N}, x.options());
  j.x = x.data_ptr(); j.out = buf.data_ptr<float>(); j.out_bf16 = as_bf16 ? ob.data_ptr() : nullptr;
  j.partial = j.out + out_groups * N;
  j.counters = reinterpret_cast<unsigned*>(j.partial + (int64_t)groups * N * slabs);
  j.rows = rows; j.row_stride = x.stride(1); j.group_stride = x.stride(0);
  j.N = N; j.groups = groups; j.fold = (int)fold; j.rows_used = rows_used;
  return buf;
}

Tensor colsum_op(const Tensor& x, int64_t fold, bool as_bf16) {
  count_launch(2);
  colsum_check(x, fold);
  c10::cuda::CUDAGuard guard(x.device());
  ColsumJob j{};
  Tensor ob;
  Tensor buf = colsum_job(x, fold, as_bf16, j, ob);
  launch_colsum_jobs(&j, 1, cur_stream());
  if (as_bf16) return ob;
  const int64_t out_groups = x.size(0) / fold;
  return buf.narrow(0, 0, out_groups * x.size(2)).view({out_groups, x.size(2)});
}

// Column sums of two tensors in the same two launches (the two bias gradients of the expert FFN).
std::vector<Tensor> colsum2_op(const Tensor& xa, const Tensor& xb, int64_t fold, bool as_bf16) {
  count_launch(2);
  colsum_check(xa, fold);
  colsum_check(xb, fold);
  TORCH_CHECK(xa.device() == xb.device());
  c10::cuda::CUDAGuard guard(xa.device());
  ColsumJob j[2] = {};
  Tensor oa, ob;
  Tensor ba = colsum_job(xa, fold, as_bf16, j[0], oa);
  Tensor bb = colsum_job(xb, fold, as_bf16, j[1], ob);
  launch_colsum_jobs(j, 2, cur_stream());
  if (as_bf16) return {oa, ob};
  const int64_t ga = xa.size(0) / fold, gb = xb.size(0) / fold;
  return {ba.narrow(0, 0, ga * xa.size(2)).view({ga, xa.size(2)}), bb.narrow(0, 0, gb * xb.size(2)).view({gb, xb.size(2)})};
}

// ---- one rank: a pass of the layer, or of its experts, in one call --------------------------------
// A stage of the pass for the per-stage timers: `stages` is None (or null, without the interpreter), or a callable that makes a context manager of a name.
struct Stage {
  py::object cm;
  Stage(const py::object& stages, const char* name) {
    if (stages && !stages.is_none()) { cm = stages(name); cm.attr("__enter__")(); }
  }
  ~Stage() {
    if (!cm) return;
    try { cm.attr("__exit__")(py::none(), py::none(), py::none()); } catch (...) {}
  }
};

// What a pass is done with, and its routing: idx, loc int32 [K, S]; slot_map int32 [E * C]; used int32 [E]; gates fp32
// [K, S].
struct LocalRoute {
  Tensor idx, loc, slot_map, used, gates;
  int64_t C, act;
  bool postscore, int8;                           // int8: rows as int8 transfers deliver them, both ways (C % 32 == 0)
  int64_t budget_ms, status_ptr;
};

static void local_check(const Tensor& x, const LocalRoute& r, const Tensor& w1) {
  const int64_t K = r.idx.size(0), S = r.idx.size(1), E = w1.size(0);
  auto i32 = [&](const Tensor& t, int64_t n) {
    return t.is_cuda() && t.scalar_type() == at::kInt && t.is_contiguous() && t.numel() == n;
  };
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == at::kBFloat16 && x.dim() == 2 && x.size(0) == S && x.size(1) % 8 == 0);
  rows16(x);
  TORCH_CHECK(i32(r.idx, K * S) && i32(r.loc, K * S) && i32(r.slot_map, E * r.C) && i32(r.used, E) && K <= 4 && E <= 64);
  TORCH_CHECK(r.gates.is_cuda() && r.gates.scalar_type() == at::kFloat && r.gates.is_contiguous() && r.gates.numel() == K * S);
  TORCH_CHECK(!r.int8 || (r.postscore && r.C % 32 == 0 && x.size(1) % 128 == 0), "int8 rows: post-score, 128-column groups, whole slices");
}

static GemmOpts local_opts(const LocalRoute& r, int64_t epilogue) {
  GemmOpts o;
  o.epilogue = epilogue; o.activation = r.act; o.budget_ms = r.budget_ms; o.status_ptr = r.status_ptr;
  o.rows_used = r.used;
  return o;
}

// The expert GEMM whose epilogue writes int8 rows: [E * C, N] bytes and a (scale, low) pair per 128 columns and row.
struct Int8Out { Tensor rows, scales; };
static Int8Out local_gemm_int8(const Tensor& a, const Tensor& w, bool w_mn, const c10::optional<Tensor>& bias, const LocalRoute& r) {
  const int64_t E = a.size(0), N = w_mn ? w.size(2) : w.size(1);
  TORCH_CHECK(N % 128 == 0 && r.C % 32 == 0 && a.size(1) == r.C, "int8 rows: 128-column groups, slices of 32 rows");
  Int8Out out{torch::empty({E * r.C, N}, a.options().dtype(at::kByte)),
              torch::empty({N / 128, E * r.C, 2}, a.options().dtype(at::kFloat))};
  GemmOpts o = local_opts(r, kEpiStoreQ8);
  o.bias = bias;
  o.q8_out = out.rows; o.q8_scales = out.scales;
  grouped_gemm_op(a, false, w, w_mn, o);
  return out;
}

// {y [S, O], xs [E, C, M], dact [E, C, H], h [E, C, H], ys [E, C, O], scales}; without `want_grad` no derivative is saved
// (dact is empty); with int8 rows ys is [E * C, O] bytes and has scales
std::vector<Tensor> local_forward_op(const Tensor& x, const LocalRoute& r, const Tensor& w1, const Tensor& b1, const Tensor& w2,
                                     const Tensor& b2, bool want_grad, const py::object& stages) {
  local_check(x, r, w1);
  c10::cuda::CUDAGuard guard(x.device());
  const int64_t K = r.idx.size(0), S = x.size(0), M = x.size(1), E = w1.size(0), C = r.C, H = w1.size(2), O = w2.size(2);
  Tensor xs = torch::empty({E, C, M}, x.options()), dact, h, ys, y = torch::empty({S, O}, x.options());
  {
    Stage st(stages, "fwd.slots");
    count_launch(1);
    launch_slots_fill(x.data_ptr(), r.slot_map.data_ptr<int>(), r.postscore ? nullptr : r.gates.data_ptr<float>(),
                      r.used.data_ptr<int>(), xs.data_ptr(), K, S, M, E, C, r.int8, cur_stream());
  }
  Tensor scales;
  {
    Stage st(stages, "fwd.gemm1");
    GemmOpts o = local_opts(r, kEpiBiasAct);
    o.bias = b1;
    if (want_grad) o.aux = dact = torch::empty({E, C, H}, x.options());
    h = grouped_gemm_op(xs, false, w1, true, o);
  }
  {
    Stage st(stages, "fwd.gemm2");
    if (r.int8) {
      const Int8Out q = local_gemm_int8(h, w2, true, b2, r);
      ys = q.rows; scales = q.scales;
    } else {
      GemmOpts o = local_opts(r, kEpiStore);
      o.bias = b2;
      ys = grouped_gemm_op(h, false, w2, true, o);
    }
  }
  {
    Stage st(stages, "fwd.combine");
    count_launch(1);
    launch_gather_rows<__nv_bfloat16>(ys.data_ptr(), r.int8 ? scales.data_ptr<float>() : nullptr, r.idx.data_ptr<int>(),
                                      r.loc.data_ptr<int>(), r.postscore ? r.gates.data_ptr<float>() : nullptr,
                                      reinterpret_cast<__nv_bfloat16*>(y.data_ptr()), K, S, O, C, nullptr, cur_stream(),
                                      r.int8 ? E * C : 0);
  }
  return {y, xs, dact, h, ys, scales};
}

// The linear gate of a pass: logits fp32 [S, E] and what its backward needs.
struct LocalGate {
  Tensor w, logits, top1;
  bool normalize, bf16_logits;
  float eps() const { return bf16_logits ? 7.8125e-03f : kFloatEps; }
};

// `dgates` undefined: the loss alone has a gradient.
static Tensor local_gate_backward(const LocalGate& g, const LocalRoute& r, const Tensor& dgates,
                                  const c10::optional<Tensor>& dl_aux) {
  const int S = g.logits.size(0), E = g.logits.size(1), K = r.idx.size(0);
  Tensor dl = torch::empty_like(g.logits);
  GatePtrs gp{};
  if (dgates.defined())
    for (int k = 0; k < K; ++k) gp.p[k] = dgates.data_ptr<float>() + (int64_t)k * S;
  const float* f = nullptr;
  const void* h = nullptr;
  if (dl_aux.has_value() && dl_aux->defined()) {
    TORCH_CHECK(dl_aux->is_cuda() && dl_aux->numel() == 1);
    if (dl_aux->scalar_type() == at::kBFloat16) h = dl_aux->data_ptr();
    else f = dl_aux->data_ptr<float>();
  }
  count_launch(1);
  launch_gate_backward<float, false>(g.logits.data_ptr<float>(), S, E, K, g.normalize, g.eps(), r.idx.data_ptr<int>(), gp, f,
                                     g.top1.data_ptr<int>(), dl.data_ptr<float>(), cur_stream(), h);
  return dl;
}

// The gradient of the gate's weight from that of the logits, as partial sums and the job that adds them up into `dwg`;
// returns the partial sums' memory.
static Tensor gate_wgrad_job(const LocalGate& g, const Tensor& x, const Tensor& dl, ColsumJob& j, Tensor& dwg) {
  const int64_t S = x.size(0), M = x.size(1), E = g.w.size(0);
  const int chunks = gate_wgrad_chunks(S, M);
  Tensor keep = torch::empty({(int64_t)chunks + 1, E * M}, dl.options());
  const bool bf16 = g.w.scalar_type() == at::kBFloat16;
  dwg = torch::empty_like(g.w);
  float* partial = keep.data_ptr<float>();
  count_launch(1);
  launch_gate_wgrad(x.data_ptr(), dl.data_ptr<float>(), partial, S, E, M, cur_stream());
  j.partial = partial;
  j.out = bf16 ? partial + (int64_t)chunks * E * M : dwg.data_ptr<float>();
  j.out_bf16 = bf16 ? dwg.data_ptr() : nullptr;
  j.rows = (long long)chunks * 128; j.N = (int)(E * M); j.groups = j.fold = 1;
  return keep;
}

// A backward that only the balance loss takes part in: the experts have no gradient then, the tokens and the gate's weight
// theirs through the logits.
static std::vector<Tensor> local_loss_backward(const Tensor& x, const LocalRoute& r, const LocalGate& gate,
                                               const c10::optional<Tensor>& dl_aux, const std::vector<bool>& need,
                                               const py::object& stages) {
  c10::cuda::CUDAGuard guard(x.device());
  const int64_t S = x.size(0), M = x.size(1), E = gate.w.size(0);
  Tensor dx, dwg;
  Stage st(stages, "bwd.gate_grad");
  const Tensor dl = local_gate_backward(gate, r, Tensor(), dl_aux);
  if (need[0]) {
    const Tensor none = torch::full({1, S}, -1, r.idx.options());     // no pick has a slot: no row is read
    dx = torch::empty_like(x);
    count_launch(1);
    launch_gather_gate(nullptr, nullptr, none.data_ptr<int>(), none.data_ptr<int>(), nullptr, dl.data_ptr<float>(),
                       gate.w.data_ptr(), gate.w.scalar_type() == at::kBFloat16, dx.data_ptr(), 1, S, M, E, 0, cur_stream());
  }
  if (need[1]) {
    ColsumJob j{};
    const Tensor keep = gate_wgrad_job(gate, x, dl, j, dwg);
    count_launch(1);
    launch_colsum_jobs(&j, 1, cur_stream());
  }
  return {dx, dwg, {}, {}, {}, {}};
}

// {dx, dgates or dwg, dw1, db1, dw2, db2}: with `gate` the second is the gradient of the gate's weight and dx has the
// gate's part in it, without it the gradient of the gates.  `need`: which of x, (gates or wg), w1, b1, w2, b2 are asked for.
static std::vector<Tensor> local_backward(const Tensor& dy, const Tensor& x, const LocalRoute& r, const Tensor& w1,
                                          const Tensor& w2, const Tensor& xs, const Tensor& dact, const Tensor& h,
                                          const Tensor& ys, const c10::optional<Tensor>& scales,
                                          const std::vector<bool>& need, const LocalGate* gate,
                                          const c10::optional<Tensor>& dl_aux, const py::object& stages) {
  local_check(x, r, w1);
  c10::cuda::CUDAGuard guard(x.device());
  const int64_t K = r.idx.size(0), S = x.size(0), M = x.size(1), E = w1.size(0), C = r.C, O = w2.size(2);
  TORCH_CHECK(dy.is_cuda() && dy.scalar_type() == at::kBFloat16 && dy.dim() == 2 && dy.size(0) == S && dy.size(1) == O);
  const void* dyp = rows16(dy);
  const int *idx = r.idx.data_ptr<int>(), *loc = r.loc.data_ptr<int>(), *used = r.used.data_ptr<int>();
  const float* gates = r.gates.data_ptr<float>();
  Tensor dgates = torch::empty({K, S}, r.gates.options()), dys = torch::empty({E, C, O}, x.options());
  Tensor dx, dh, dxs, dx_scales, dh_sums, dl, dwg, dw1, dw2, db1, db2;
  {
    Stage st(stages, "bwd.gate_grad");
    count_launch(1);
    if (r.int8)
      launch_slots_gate_grad_q8(ys.data_ptr(), scales->data_ptr<float>(), dyp, idx, loc, gates, used, dgates.data_ptr<float>(),
                                dys.data_ptr(), K, S, O, E, C, cur_stream());
    else if (r.postscore)
      launch_slots_gate_grad(ys.data_ptr(), dyp, idx, loc, gates, used, dgates.data_ptr<float>(), dys.data_ptr(), K, S, O, E, C,
                             cur_stream());
    else
      launch_slots_fill(dyp, r.slot_map.data_ptr<int>(), nullptr, used, dys.data_ptr(), K, S, O, E, C, false, cur_stream());
    if (gate != nullptr && r.postscore) dl = local_gate_backward(*gate, r, dgates, dl_aux);
  }
  {
    Stage st(stages, "bwd.dgrad2");               // dH = (dY . W2^T) * act'
    GemmOpts o = local_opts(r, kEpiDAct);
    o.aux = dact;
    if (need[3]) o.colsum = dh_sums = torch::empty({E, (C + 31) / 32, w2.size(1)}, r.gates.options());
    dh = grouped_gemm_op(dys, false, w2, false, o);
  }
  const bool gate_from_dx = !r.postscore && (need[1] || gate != nullptr);
  if (need[0] || gate_from_dx) {
    Stage st(stages, "bwd.dgrad1");               // dX slots = dH . W1^T
    if (r.int8) {
      const Int8Out q = local_gemm_int8(dh, w1, false, c10::nullopt, r);
      dxs = q.rows; dx_scales = q.scales;
    } else {
      dxs = grouped_gemm_op(dh, false, w1, false, local_opts(r, kEpiStore));
    }
  }
  {
    Stage st(stages, "bwd.dispatch");
    if (gate_from_dx) {
      count_launch(1);
      launch_gate_grad<__nv_bfloat16>(reinterpret_cast<const __nv_bfloat16*>(dxs.data_ptr()),
                                      reinterpret_cast<const __nv_bfloat16*>(x.data_ptr()), idx, loc, dgates.data_ptr<float>(),
                                      nullptr, nullptr, K, S, M, C, cur_stream());
      if (gate != nullptr) dl = local_gate_backward(*gate, r, dgates, dl_aux);
    }
    if (need[0]) {
      dx = torch::empty_like(x);
      count_launch(1);
      if (gate != nullptr)
        launch_gather_gate(dxs.data_ptr(), r.int8 ? dx_scales.data_ptr<float>() : nullptr, idx, loc, r.postscore ? nullptr : gates, dl.data_ptr<float>(), gate->w.data_ptr(),
                           gate->w.scalar_type() == at::kBFloat16, dx.data_ptr(), K, S, M, E, C, cur_stream());
      else
        launch_gather_rows<__nv_bfloat16>(dxs.data_ptr(), r.int8 ? dx_scales.data_ptr<float>() : nullptr, idx, loc,
                                          r.postscore ? nullptr : gates, reinterpret_cast<__nv_bfloat16*>(dx.data_ptr()), K, S,
                                          M, C, nullptr, cur_stream(), r.int8 ? E * C : 0);
    }
  }
  if (need[4]) {
    Stage st(stages, "bwd.wgrad2");
    dw2 = grouped_gemm_op(h, true, dys, true, local_opts(r, kEpiStore));
  }
  if (need[2]) {
    Stage st(stages, "bwd.wgrad1");
    dw1 = grouped_gemm_op(xs, true, dh, true, local_opts(r, kEpiStore));
  }
  {
    Stage st(stages, "bwd.bias_grads");
    ColsumJob j[3] = {};
    Tensor keep[3];
    int n = 0;
    if (need[5]) { keep[n] = colsum_job(dys, 1, true, j[n], db2, used); ++n; }
    if (n > 0) count_launch(1);
    if (need[3]) {                                // the slices' sums came with dH
      const int64_t H = w2.size(1);
      db1 = torch::empty({E, H}, x.options());
      keep[n] = torch::empty({E, H}, r.gates.options());
      j[n].partial = dh_sums.data_ptr<float>(); j[n].out = keep[n].data_ptr<float>(); j[n].out_bf16 = db1.data_ptr();
      j[n].rows = C; j[n].slab_rows = 32; j[n].N = (int)H; j[n].groups = (int)E; j[n].fold = 1; j[n].rows_used = used;
      ++n;
    }
    if (gate != nullptr && need[1]) {
      keep[n] = gate_wgrad_job(*gate, x, dl, j[n], dwg);
      ++n;
    }
    if (n > 0) {
      count_launch(1);
      launch_colsum_jobs(j, n, cur_stream());
    }
  }
  return {dx, gate != nullptr ? dwg : dgates, dw1, db1, dw2, db2};
}

std::vector<Tensor> local_backward_op(const Tensor& dy, const Tensor& x, const LocalRoute& r, const Tensor& w1, const Tensor& w2,
                                      const Tensor& xs, const Tensor& dact, const Tensor& h, const Tensor& ys,
                                      const c10::optional<Tensor>& scales, const std::vector<bool>& need,
                                      const py::object& stages) {
  return local_backward(dy, x, r, w1, w2, xs, dact, h, ys, scales, need, nullptr, c10::nullopt, stages);
}

// The whole layer with a linear gate `wg` [E, M].  capacity < 0: as many slots as the busiest expert needs, rounded up by
// `round_up` (one host read).  Returns {y, l_aux, logits, top1, slot_map, used, idx, loc, gates, xs, dact, h, ys, scales, loc as
// routed} and the capacity.  int8 rows are stored in slices of 32: the experts' slots are then laid out C = capacity rounded
// up to that apart (xs.size(1)), and the first `loc` has a dropped pick behind all of them; what is dropped stays a matter of
// the capacity.
std::tuple<std::vector<Tensor>, int64_t> local_moe_forward_op(
    const Tensor& x, const Tensor& wg, const Tensor& w1, const Tensor& b1, const Tensor& w2, const Tensor& b2, int64_t K,
    int64_t capacity, const py::object& round_up, bool normalize, bool bf16_logits, bool prio, int64_t act, bool postscore, bool int8,
    int64_t budget_ms, int64_t status_ptr, bool want_grad, const py::object& stages) {
  TORCH_CHECK(x.is_cuda() && x.dim() == 2 && x.scalar_type() == at::kBFloat16);
  const int64_t S = x.size(0), M = x.size(1), E = w1.size(0);
  TORCH_CHECK(wg.is_cuda() && wg.is_contiguous() && wg.dim() == 2 && wg.size(0) == E && wg.size(1) == M && M % 32 == 0 &&
              (wg.scalar_type() == at::kFloat || wg.scalar_type() == at::kBFloat16) && E <= kProjMaxE && K >= 1 && K <= 4 &&
              K <= E && S > 0 && S * K <= INT_MAX, "linear gate outside the kernels' range");
  rows16(wg);
  c10::cuda::CUDAGuard guard(x.device());
  auto iopt = x.options().dtype(at::kInt);
  auto fopt = x.options().dtype(at::kFloat);
  const int64_t nblk = gate_workspace_blocks(S);
  LocalRoute r{torch::empty({K, S}, iopt), torch::empty({K, S}, iopt), {}, {}, torch::empty({K, S}, fopt), capacity, act,
               postscore, int8, budget_ms, status_ptr};
  const Tensor loc = r.loc;
  Tensor logits = torch::empty({S, E}, fopt), counts = torch::empty({2, E}, iopt);
  Tensor laux = torch::empty({}, fopt), laux_bf16;
  if (bf16_logits) laux_bf16 = torch::empty({}, x.options());
  Tensor ws = torch::empty({2 * K * S + (K + 1) * nblk * E}, iopt), order;
  const int* perm = nullptr;
  {
    Stage st(stages, "fwd.gate_linear");
    count_launch(1);
    launch_gate_project(rows16(x), wg.data_ptr(), wg.scalar_type() == at::kBFloat16, logits.data_ptr<float>(), S, E, M,
                        bf16_logits, cur_stream());
  }
  {
    Stage st(stages, "fwd.gate_topk_scan");
    if (prio) {
      const int64_t words = importance_workspace(S);
      order = torch::empty({words + S}, x.options().dtype(at::kLong));        // sorted tiles, ranks and permutation
      unsigned long long* const ws64 = reinterpret_cast<unsigned long long*>(order.data_ptr());
      int* const o = reinterpret_cast<int*>(ws64 + words);
      count_launch(2);
      launch_importance_order<float>(logits.data_ptr<float>(), S, E, ws64, o, o + S, cur_stream());
      perm = o + S;
    }
    const bool dynamic = capacity < 0, map_later = dynamic || (int8 && capacity % 32 != 0);
    if (!map_later) r.slot_map = torch::empty({E * capacity}, iopt);
    GatePtrs gp{};
    for (int k = 0; k < K; ++k) gp.p[k] = r.gates.data_ptr<float>() + (int64_t)k * S;
    int* w = ws.data_ptr<int>();
    count_launch(2);
    launch_gate_forward<float, false>(logits.data_ptr<float>(), S, E, K, dynamic ? INT_MAX : (int)capacity, normalize,
                                      bf16_logits ? 7.8125e-03f : kFloatEps, r.idx.data_ptr<int>(), r.loc.data_ptr<int>(), gp,
                                      reinterpret_cast<float*>(w), map_later ? nullptr : r.slot_map.data_ptr<int>(),
                                      counts.data_ptr<int>(), counts.data_ptr<int>() + E, laux.data_ptr<float>(), w + K * S,
                                      w + 2 * K * S, reinterpret_cast<float*>(w + 2 * K * S + K * nblk * E), cur_stream(), perm,
                                      bf16_logits ? laux_bf16.data_ptr() : nullptr);
    if (dynamic) {
      Tensor host;
      {
        py::gil_scoped_release others;            // the wait for the stream keeps no other Python thread waiting
        host = counts[1].cpu();
      }
      int peak = 0;
      for (int64_t e = 0; e < E; ++e) peak = std::max(peak, host.data_ptr<int>()[e]);
      capacity = round_up(peak).cast<int64_t>();
      TORCH_CHECK(capacity >= peak);
    } else if (map_later) {
      r.loc = loc.masked_fill(loc.ge(capacity), INT_MAX);
    }
    if (map_later) {
      r.C = int8 ? (capacity + 31) / 32 * 32 : capacity;
      r.slot_map = torch::empty({E * r.C}, iopt);
      count_launch(1);
      launch_build_slot_map(r.idx.data_ptr<int>(), r.loc.data_ptr<int>(), r.slot_map.data_ptr<int>(), K, S, E, r.C, cur_stream());
    }
  }
  r.used = counts[1];
  std::vector<Tensor> e = local_forward_op(x, r, w1, b1, w2, b2, want_grad, stages);
  return {{e[0], bf16_logits ? laux_bf16 : laux, logits, counts[0], r.slot_map, r.used, r.idx, r.loc, r.gates, e[1], e[2], e[3],
           e[4], e[5], loc}, capacity};
}

// `dy` undefined: see local_loss_backward
std::vector<Tensor> local_moe_backward_op(const c10::optional<Tensor>& dy, const c10::optional<Tensor>& dl_aux, const Tensor& x, const Tensor& wg,
                                          const LocalRoute& r, const Tensor& w1, const Tensor& w2, const Tensor& logits,
                                          const Tensor& top1, const Tensor& xs, const Tensor& dact, const Tensor& h,
                                          const Tensor& ys, const c10::optional<Tensor>& scales, bool normalize,
                                          bool bf16_logits, const std::vector<bool>& need, const py::object& stages) {
  const LocalGate g{wg, logits, top1, normalize, bf16_logits};
  if (!dy.has_value() || !dy->defined()) return local_loss_backward(x, r, g, dl_aux, need, stages);
  return local_backward(*dy, x, r, w1, w2, xs, dact, h, ys, scales, need, &g, dl_aux, stages);
}

#include "layer_node.h"
#include "layer32.h"

// rows [R, M] -> uint8 [R, M + 16]: M quantised bytes + {scale, low, 0, 0} (the wire rows of the fused send)
Tensor int8_rows_encode_op(const Tensor& x) {
  count_launch(1);
  TORCH_CHECK(x.is_cuda() && x.dim() == 2 && x.is_contiguous() && x.size(1) % 16 == 0,
              "int8_rows_encode: contiguous CUDA [R, M] with M % 16 == 0");
  c10::cuda::CUDAGuard guard(x.device());
  const int R = x.size(0), M = x.size(1);
  Tensor out = torch::empty({(int64_t)R, (int64_t)M + 16}, x.options().dtype(at::kByte));
  DISPATCH_FLOAT(x, "int8_rows_encode", [&] {
    launch_int8_rows_encode<scalar_t>(reinterpret_cast<const scalar_t*>(rows16(x)), out.data_ptr<uint8_t>(), R, M,
                                      cur_stream());
  });
  return out;
}

// ---- push / wait wrappers for the fused MoE path ------------------------------------------------
void scatter_push_op(const Tensor& x, const Tensor& slot_map, const c10::optional<Tensor>& gates, int64_t K, int64_t E,
                     int64_t C, int64_t heap_bases_ptr, int64_t data_off, int64_t flag_off, int64_t W, int64_t my_rank,
                     int64_t chunks, int64_t ctas, int64_t chunk_begin, int64_t chunk_count) {
  count_launch(1);
  TORCH_CHECK(x.is_cuda() && x.dim() == 2 && x.is_contiguous());
  c10::cuda::CUDAGuard guard(x.device());
  PushArgs pa{};
  pa.heap_bases = reinterpret_cast<const unsigned long long*>(heap_bases_ptr);
  pa.data_off = data_off; pa.flag_off = flag_off; pa.scale_off = 0;
  pa.W = W; pa.my_rank = my_rank; pa.chunks = chunks; pa.ctas_per_msg = ctas;
  pa.chunk_begin = chunk_begin; pa.chunk_count = chunk_count;
  TORCH_CHECK(E % W == 0 && C % chunks == 0);
  const int S = x.size(0), M = x.size(1);
  DISPATCH_FLOAT(x, "scatter_push", [&] {
    launch_scatter_rows<scalar_t>(reinterpret_cast<const scalar_t*>(rows16(x)), slot_map.data_ptr<int>(),
                                  opt_f32(gates), nullptr, K, S, M, E, C, &pa, false, cur_stream());
  });
}

Tensor gather_wait_op(int64_t disp_ptr, at::ScalarType dtype, int64_t M, const Tensor& idx, const Tensor& loc,
                      const c10::optional<Tensor>& gates, int64_t C, int64_t flags_ptr, int64_t n_flags, int64_t want,
                      int64_t budget_ms, int64_t status_ptr, int64_t want_ptr, int64_t q8_scales_ptr,
                      int64_t q8_group_rows) {
  count_launch(1);
  c10::cuda::CUDAGuard guard(idx.device());
  const int K = idx.size(0), S = idx.size(1);
  Tensor out = torch::empty({S, M}, idx.options().dtype(dtype));
  WaitArgs wa{};
  wa.flags = reinterpret_cast<const unsigned long long*>(flags_ptr);
  wa.n_flags = n_flags; wa.want = want; wa.budget_ns = (unsigned long long)budget_ms * 1000000ull;
  wa.want_ptr = reinterpret_cast<const unsigned long long*>(want_ptr);
  wa.status = reinterpret_cast<int*>(status_ptr);
  DISPATCH_FLOAT(out, "gather_wait", [&] {
    launch_gather_rows<scalar_t>(reinterpret_cast<const void*>(disp_ptr), reinterpret_cast<const float*>(q8_scales_ptr),
                                 idx.data_ptr<int>(), loc.data_ptr<int>(), opt_f32(gates),
                                 reinterpret_cast<scalar_t*>(out.data_ptr()), K, S, M, C, flags_ptr ? &wa : nullptr,
                                 cur_stream(), q8_scales_ptr ? q8_group_rows : 0);
  });
  return out;
}

// ---- ZFP / LZ codecs (CPU or CUDA by the tensor's device) ------------------------------------------
int elem_code(at::ScalarType t) {
  if (t == at::kFloat) return 0;
  if (t == at::kBFloat16) return 1;
  if (t == at::kHalf) return 2;
  TORCH_CHECK(false, "zfp codec: unsupported dtype ", t);
}

Tensor zfp_encode_op(const Tensor& x, int64_t rate) {
  TORCH_CHECK(x.dim() == 3 && x.is_contiguous(), "zfp_encode expects a contiguous [lead, rows, M] tensor");
  TORCH_CHECK(rate == 4 || rate == 8 || rate == 16, "zfp rate must be 4, 8 or 16 bits per value");
  TORCH_CHECK(x.size(2) % 4 == 0, "zfp codec needs the last dim to be a multiple of 4");
  const int64_t lead = x.size(0), rows = x.size(1), M = x.size(2);
  const int64_t bytes = (int64_t)zfp_stream_bytes(rows, M, rate);
  Tensor out = torch::empty({lead, bytes}, x.options().dtype(at::kByte));
  if (x.is_cuda()) {
    count_launch(1);
    c10::cuda::CUDAGuard guard(x.device());
    launch_zfp_encode(x.data_ptr(), elem_code(x.scalar_type()), out.data_ptr<uint8_t>(), lead, rows, M, rate, cur_stream());
  } else {
    zfp_encode_cpu(x.data_ptr(), elem_code(x.scalar_type()), out.data_ptr<uint8_t>(), lead, rows, M, rate);
  }
  return out;
}

Tensor zfp_decode_op(const Tensor& stream, int64_t lead, int64_t rows, int64_t M, int64_t rate, at::ScalarType dtype) {
  TORCH_CHECK(stream.is_contiguous() && stream.scalar_type() == at::kByte);
  TORCH_CHECK(stream.numel() == lead * (int64_t)zfp_stream_bytes(rows, M, rate), "zfp stream size mismatch");
  TORCH_CHECK(reinterpret_cast<uintptr_t>(stream.data_ptr()) % 4 == 0, "zfp stream must be 4-byte aligned");
  Tensor out = torch::empty({lead, rows, M}, stream.options().dtype(dtype));
  if (stream.is_cuda()) {
    count_launch(1);
    c10::cuda::CUDAGuard guard(stream.device());
    launch_zfp_decode(stream.data_ptr<uint8_t>(), out.data_ptr(), elem_code(dtype), lead, rows, M, rate, cur_stream());
  } else {
    zfp_decode_cpu(stream.data_ptr<uint8_t>(), out.data_ptr(), elem_code(dtype), lead, rows, M, rate);
  }
  return out;
}

std::vector<Tensor> lz_encode_op(const Tensor& raw, int64_t sym) {
  TORCH_CHECK(raw.dim() == 2 && raw.is_contiguous() && raw.scalar_type() == at::kByte);
  TORCH_CHECK((sym == 2 || sym == 4) && raw.size(1) % sym == 0 && raw.size(1) % 16 == 0,
              "lz codec: slice bytes must be a multiple of 16 and of the symbol size");
  TORCH_CHECK(reinterpret_cast<uintptr_t>(raw.data_ptr()) % sym == 0, "lz codec: symbols must be aligned");
  const int64_t slices = raw.size(0), raw_bytes = raw.size(1);
  const int64_t cap = (int64_t)lz_payload_capacity(raw_bytes);
  Tensor payload = torch::empty({slices, cap}, raw.options());
  Tensor sizes = torch::empty({slices}, raw.options().dtype(at::kInt));
  if (raw.is_cuda()) {
    count_launch(3);
    c10::cuda::CUDAGuard guard(raw.device());
    Tensor scratch = torch::empty({(int64_t)lz_scratch_bytes(slices, raw_bytes)}, raw.options());
    launch_lz_encode(raw.data_ptr<uint8_t>(), payload.data_ptr<uint8_t>(), sizes.data_ptr<int>(),
                     scratch.data_ptr<uint8_t>(), slices, raw_bytes, cap, sym, cur_stream());
  } else {
    lz_encode_cpu(raw.data_ptr<uint8_t>(), payload.data_ptr<uint8_t>(), sizes.data_ptr<int>(), slices, raw_bytes, cap, sym);
  }
  return {payload, sizes};
}

Tensor lz_decode_op(const Tensor& payload, const Tensor& sizes, int64_t raw_bytes, int64_t sym) {
  TORCH_CHECK(payload.dim() == 2 && payload.is_contiguous() && payload.scalar_type() == at::kByte);
  TORCH_CHECK((sym == 2 || sym == 4) && raw_bytes >= 0 && raw_bytes % sym == 0, "lz codec: slice bytes must be a multiple of the symbol size");
  TORCH_CHECK(payload.size(1) % 4 == 0 && reinterpret_cast<uintptr_t>(payload.data_ptr()) % 4 == 0,
              "lz codec: slices must be 4-byte aligned");
  long long len_off = 0, header = 0;
  lz_slice_layout(raw_bytes, &len_off, &header);
  TORCH_CHECK(payload.size(1) >= header, "lz codec: slices are shorter than their header");
  const int64_t slices = payload.size(0);
  Tensor raw = torch::empty({slices, raw_bytes}, payload.options());
  if (payload.is_cuda()) {
    count_launch(1);
    c10::cuda::CUDAGuard guard(payload.device());
    launch_lz_decode(payload.data_ptr<uint8_t>(), raw.data_ptr<uint8_t>(), slices, raw_bytes, payload.size(1), sym,
                     cur_stream());
  } else {
    lz_decode_cpu(payload.data_ptr<uint8_t>(), raw.data_ptr<uint8_t>(), slices, raw_bytes, payload.size(1), sym);
  }
  return raw;
}

// ---- C++ extension points: run a registered comm / codec on tensors -----------------------------
// A comm object registered in C++, kept alive across calls (it owns call counters and cached tables).
struct NativeCommHandle {
  std::unique_ptr<AbstractComm> comm;
  NativeCommHandle(const std::string& name, int64_t world_size, int64_t world_rank, int64_t local_size,
                   int64_t heap_bases_ptr, int64_t local_base, int64_t scratch_off, int64_t scratch_bytes,
                   int64_t status_ptr, int64_t budget_ms) {
    CommContext ctx;
    ctx.world_size = world_size; ctx.world_rank = world_rank; ctx.local_size = local_size > 0 ? local_size : world_size;
    ctx.local_rank = world_rank % ctx.local_size;
    ctx.heap_bases = reinterpret_cast<const unsigned long long*>(heap_bases_ptr);
    ctx.local_base = (unsigned long long)local_base;
    ctx.scratch_off = (unsigned long long)scratch_off; ctx.scratch_bytes = (unsigned long long)scratch_bytes;
    ctx.status = reinterpret_cast<int*>(status_ptr);
    if (budget_ms > 0) ctx.budget_ns = (unsigned long long)budget_ms * 1000000ull;
    comm = make_comm(name, ctx);
    TORCH_CHECK(comm != nullptr, "no native comm registered under `", name, "`");
  }
  int64_t scratch_bytes_for(int64_t payload) const { return (int64_t)comm->scratch_bytes_for((size_t)payload); }
  Tensor all_to_all(const Tensor& t) {
    Tensor in = t.contiguous();
    Tensor out = torch::empty_like(in);
    cudaStream_t s = nullptr;
    if (in.is_cuda()) { count_launch(2); s = cur_stream(); }
    c10::cuda::OptionalCUDAGuard guard;
    if (in.is_cuda()) guard.set_device(in.device());
    comm->all_to_all(in.data_ptr(), out.data_ptr(), in.numel() * in.element_size(), s);
    return out;
  }
};

Tensor native_codec_roundtrip_op(const std::string& name, const Tensor& t, int64_t parts, bool decode, int64_t out_bytes) {
  auto codec = make_compressor(name);
  TORCH_CHECK(codec != nullptr, "no native compressor registered under `", name, "`");
  Tensor in = t.contiguous();
  const size_t bytes = decode ? (size_t)out_bytes : in.numel() * in.element_size();
  cudaStream_t s = in.is_cuda() ? cur_stream() : nullptr;
  if (!decode) {
    Tensor wire = torch::empty({(int64_t)codec->wire_bytes(bytes, parts)}, in.options().dtype(at::kByte));
    codec->compress(in.data_ptr(), wire.data_ptr(), bytes, parts, in.element_size(), in.size(-1), s);
    return wire;
  }
  Tensor out = torch::empty({out_bytes}, in.options().dtype(at::kByte));
  codec->decompress(in.data_ptr(), out.data_ptr(), bytes, parts, 1, 1, s);
  return out;
}

// ---- stand-alone transfers --------------------------------------------------------------------
void xfer_op(int64_t src_ptr, const Tensor& msgs, int64_t ctas_per_msg, int64_t heap_bases_ptr, int64_t flag_off,
             int64_t wait_flags_ptr, const c10::optional<Tensor>& wait_idx, int64_t want, int64_t budget_ms,
             int64_t status_ptr, int64_t local_dst_ptr, int64_t len_off, int64_t len_base) {
  count_launch(1);
  TORCH_CHECK(msgs.is_cuda() && msgs.scalar_type() == at::kLong && msgs.is_contiguous() && msgs.dim() == 2 &&
              msgs.size(1) == 6, "msgs must be a contiguous CUDA int64 [n, 6] tensor");
  c10::cuda::CUDAGuard guard(msgs.device());
  const int n_wait = (wait_idx.has_value() && wait_idx->defined()) ? wait_idx->numel() : 0;
  launch_xfer(reinterpret_cast<const void*>(src_ptr), reinterpret_cast<const long long*>(msgs.data_ptr<int64_t>()),
              msgs.size(0), ctas_per_msg, reinterpret_cast<const unsigned long long*>(heap_bases_ptr), flag_off,
              reinterpret_cast<const unsigned long long*>(wait_flags_ptr), n_wait ? wait_idx->data_ptr<int>() : nullptr,
              n_wait, want, (unsigned long long)budget_ms * 1000000ull, reinterpret_cast<int*>(status_ptr),
              reinterpret_cast<void*>(local_dst_ptr), cur_stream(), len_off, (unsigned long long)len_base);
}

void wait_flags_op(int64_t flags_ptr, int64_t n, int64_t want, int64_t budget_ms, int64_t status_ptr) {
  count_launch(1);
  launch_wait_flags(reinterpret_cast<const unsigned long long*>(flags_ptr), n, want,
                    (unsigned long long)budget_ms * 1000000ull, reinterpret_cast<int*>(status_ptr), cur_stream());
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.doc() = "planmoe_b200 native extension (sm_100a kernels, symmetric heap, CPU reference ops)";
  m.def("cpu_scatter", &cpu_scatter_op);
  m.def("cpu_gather", &cpu_gather_op);
  m.def("cpu_gate_grad", &cpu_gate_grad_op);
  m.def("build_slot_map", &build_slot_map_op);
  m.def("dispatch_scatter", &dispatch_scatter_op, py::arg("x"), py::arg("slot_map"), py::arg("gates"), py::arg("K"),
        py::arg("n_slots"), py::arg("round_gates") = false);
  m.def("dispatch_gather", &dispatch_gather_op, py::arg("disp"), py::arg("idx"), py::arg("loc"), py::arg("gates"), py::arg("C"),
        py::arg("round_gates") = false);
  m.def("dispatch_gate_grad", &dispatch_gate_grad_op);
  m.def("dispatch_gate_grad_scaled", &dispatch_gate_grad_scaled_op);
  m.def("dispatch_gate_grad_q8", &dispatch_gate_grad_q8_op);
  m.def("gate_forward", &gate_forward_op);
  m.def("gate_forward_used", &gate_forward_used_op);
  py::class_<LocalRoute>(m, "LocalRoute")
      .def(py::init([](Tensor idx, Tensor loc, Tensor slot_map, Tensor used, Tensor gates, int64_t C, int64_t act, bool postscore,
                       bool int8, int64_t budget_ms, int64_t status_ptr) {
        return LocalRoute{idx, loc, slot_map, used, gates, C, act, postscore, int8, budget_ms, status_ptr};
      }));
  m.def("local_forward", &local_forward_op);
  m.def("local_backward", &local_backward_op);
  m.def("local_moe_forward", &local_moe_forward_op);
  m.def("local_layer_node", &local_layer_node);
  m.def("local_moe_backward", &local_moe_backward_op);
  m.attr("gate_max_experts") = kProjMaxE;
  // whether the environment leaves a single rank to the direct path (read at every call, like all of these switches)
  m.def("local_by_env", [] {
    auto is = [](const char* v, char c) { return v != nullptr && v[0] == c && v[1] == 0; };
    return !is(getenv("PLANMOE_LOCAL"), '0') && getenv("PLANMOE_FUSE_SEND") == nullptr &&
           !is(getenv("PLANMOE_DEBUG_GUARDS"), '1') && !is(getenv("PLANMOE_GEMM_TRACE"), '1');
  });
  m.def("importance_order", &importance_order_op);
  m.def("remap_slot_map", &remap_slot_map_op);
  m.def("gate_backward", &gate_backward_op);
  m.def("route_scores_node", &route_scores_node);
  m.def("scatter_node", &scatter_node);
  m.def("gather_picks_node", &gather_picks_node);
  m.def("layer32_forward", &layer32_forward_op);
  m.def("layer32_backward", &layer32_backward_op);
  m.def("route_scores", &route_scores_op);
  m.def("route_scores_backward", &route_scores_backward_op);
  m.def("cumsum_sub_one", &cumsum_sub_one_op);
  m.def("int8_encode", &int8_encode_op);
  m.def("int8_decode", &int8_decode_op);
  m.def("int8_rows_encode", &int8_rows_encode_op);
  m.def("colsum", &colsum_op, py::arg("x"), py::arg("fold") = 1, py::arg("as_bf16") = false);
  m.def("colsum2", &colsum2_op, py::arg("xa"), py::arg("xb"), py::arg("fold") = 1, py::arg("as_bf16") = false);
  m.def("scatter_push", &scatter_push_op);
  m.def("gather_wait", &gather_wait_op, py::arg("disp_ptr"), py::arg("dtype"), py::arg("M"), py::arg("idx"), py::arg("loc"),
        py::arg("gates"), py::arg("C"), py::arg("flags_ptr"), py::arg("n_flags"), py::arg("want"), py::arg("budget_ms"),
        py::arg("status_ptr"), py::arg("want_ptr") = 0, py::arg("q8_scales_ptr") = 0, py::arg("q8_group_rows") = 0);
  m.def("zfp_encode", &zfp_encode_op);
  m.def("zfp_decode", &zfp_decode_op);
  m.def("lz_encode", &lz_encode_op);
  m.def("lz_decode", &lz_decode_op);
  m.def("native_comm_names", &comm_names);
  m.def("native_compressor_names", &compressor_names);
  py::class_<NativeCommHandle>(m, "NativeCommHandle")
      .def(py::init<const std::string&, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t>(),
           py::arg("name"), py::arg("world_size") = 1, py::arg("world_rank") = 0, py::arg("local_size") = 0,
           py::arg("heap_bases_ptr") = 0, py::arg("local_base") = 0, py::arg("scratch_off") = 0,
           py::arg("scratch_bytes") = 0, py::arg("status_ptr") = 0, py::arg("budget_ms") = 0)
      .def("scratch_bytes_for", &NativeCommHandle::scratch_bytes_for)
      .def("all_to_all", &NativeCommHandle::all_to_all);
  m.def("native_codec_run", &native_codec_roundtrip_op);
  m.def("xfer", &xfer_op, py::arg("src_ptr"), py::arg("msgs"), py::arg("ctas_per_msg"), py::arg("heap_bases_ptr"),
        py::arg("flag_off"), py::arg("wait_flags_ptr"), py::arg("wait_idx"), py::arg("want"), py::arg("budget_ms"),
        py::arg("status_ptr"), py::arg("local_dst_ptr"), py::arg("len_off") = -1, py::arg("len_base") = 0);
  m.def("lz_layout", [](int64_t raw_bytes) {
    // (payload capacity per slice, byte offset of the u32 holding the code size, header bytes) of an LZ slice
    long long len_off = 0, header = 0;
    lz_slice_layout(raw_bytes, &len_off, &header);
    return std::make_tuple((int64_t)lz_payload_capacity(raw_bytes), (int64_t)len_off, (int64_t)header);
  });
  m.def("wait_flags", &wait_flags_op);
  m.def("delay", [](int64_t ns) { count_launch(1); launch_delay((unsigned long long)(ns < 0 ? 0 : ns), cur_stream()); });
  m.def("gemm_push_arrivals", &gemm_push_arrivals);
  m.def("launch_count", [] { return (long long)g_launches.load(); });

  py::class_<GemmOpts>(m, "GemmOpts")
      .def(py::init<>())
      .def_readwrite("epilogue", &GemmOpts::epilogue)
      .def_readwrite("activation", &GemmOpts::activation)
      .def_readwrite("bias", &GemmOpts::bias)
      .def_readwrite("aux", &GemmOpts::aux)
      .def_readwrite("out", &GemmOpts::out)
      .def_readwrite("gate_flags_ptr", &GemmOpts::gate_flags_ptr)
      .def_readwrite("gate_rows", &GemmOpts::gate_rows)
      .def_readwrite("gate_want", &GemmOpts::gate_want)
      .def_readwrite("gate_want_ptr", &GemmOpts::gate_want_ptr)
      .def_readwrite("gate_mode", &GemmOpts::gate_mode)
      .def_readwrite("gate_nblk", &GemmOpts::gate_nblk)
      .def_readwrite("perm_w", &GemmOpts::perm_w)
      .def_readwrite("perm_seg_rows", &GemmOpts::perm_seg_rows)
      .def_readwrite("perm_local_first", &GemmOpts::perm_local_first)
      .def_readwrite("copy_nblk", &GemmOpts::copy_nblk)
      .def_readwrite("rows_used", &GemmOpts::rows_used)
      .def_readwrite("colsum", &GemmOpts::colsum)
      .def_readwrite("trace_ptr", &GemmOpts::trace_ptr)
      .def_readwrite("dq_ptr", &GemmOpts::dq_ptr)
      .def_readwrite("dq_arrival_ptr", &GemmOpts::dq_arrival_ptr)
      .def_readwrite("dq_ready_ptr", &GemmOpts::dq_ready_ptr)
      .def_readwrite("heap_bases_ptr", &GemmOpts::heap_bases_ptr)
      .def_readwrite("push_data_off", &GemmOpts::push_data_off)
      .def_readwrite("push_flag_off", &GemmOpts::push_flag_off)
      .def_readwrite("push_rows", &GemmOpts::push_rows)
      .def_readwrite("push_C", &GemmOpts::push_C)
      .def_readwrite("push_c0", &GemmOpts::push_c0)
      .def_readwrite("push_chunk", &GemmOpts::push_chunk)
      .def_readwrite("push_q8", &GemmOpts::push_q8)
      .def_readwrite("push_scale_off", &GemmOpts::push_scale_off)
      .def_readwrite("W", &GemmOpts::W)
      .def_readwrite("my_rank", &GemmOpts::my_rank)
      .def_readwrite("chunk_groups", &GemmOpts::chunk_groups)
      .def_readwrite("budget_ms", &GemmOpts::budget_ms)
      .def_readwrite("status_ptr", &GemmOpts::status_ptr)
      .def_readwrite("max_ctas", &GemmOpts::max_ctas)
      .def_readwrite("cta_group", &GemmOpts::cta_group)
      .def_readwrite("heap_bases_host", &GemmOpts::heap_bases_host)
      .def_readwrite("copy_x", &GemmOpts::copy_x)
      .def_readwrite("copy_slot_map", &GemmOpts::copy_slot_map)
      .def_readwrite("copy_gates", &GemmOpts::copy_gates)
      .def_readwrite("copy_K", &GemmOpts::copy_K)
      .def_readwrite("copy_E_local", &GemmOpts::copy_E_local)
      .def_readwrite("copy_C", &GemmOpts::copy_C)
      .def_readwrite("copy_chunks", &GemmOpts::copy_chunks)
      .def_readwrite("copy_ctas", &GemmOpts::copy_ctas)
      .def_readwrite("copy_data_off", &GemmOpts::copy_data_off)
      .def_readwrite("copy_flag_off", &GemmOpts::copy_flag_off);
  m.def("gemm_grid_ctas", &gemm_grid_ctas, py::arg("groups"), py::arg("M"), py::arg("N"), py::arg("max_ctas") = 0,
        py::arg("cta_group") = 0);
  m.def("grouped_gemm", &grouped_gemm_op);
  m.def("tensor_from_ptr", [](int64_t ptr, int64_t nbytes, int64_t device) {
    return torch::from_blob(reinterpret_cast<void*>(ptr), {nbytes},
                            torch::TensorOptions().dtype(at::kByte).device(at::kCUDA, device));
  });

  bind_symm_heap(m);
  bind_jit(m);
}
