// A pass of the fp32 layer of one rank (ops/layer32.py) in one call each way: the routing, encode and decode kernels around
// library products.  Included by bindings.cpp behind the operations that it calls.
#pragma once

static Tensor act32(const Tensor& t, int64_t act) {
  switch (act) {
    case kActRelu: return at::relu(t);
    case kActGelu: return at::gelu(t);
    case kActSilu: return at::silu(t);
    default: return t;
  }
}
static Tensor act32_backward(const Tensor& dh, const Tensor& t, const Tensor& h, int64_t act) {
  switch (act) {
    case kActRelu: return at::threshold_backward(dh, h, 0);
    case kActGelu: return at::gelu_backward(dh, t);
    case kActSilu: return at::silu_backward(dh, t);
    default: return dh;
  }
}

// {y, loss, scores, top1, slot_map, idx, loc, gates [K, S], slots [E, C, M], t, h, outputs [E, C, O]}
std::vector<Tensor> layer32_forward_op(const Tensor& x, const Tensor& wg, const Tensor& w1, const Tensor& b1, const Tensor& w2,
                                       const Tensor& b2, int64_t K, int64_t C, bool normalize, int64_t act) {
  at::NoGradGuard none;
  c10::cuda::CUDAGuard guard(x.device());
  const int64_t E = w1.size(0), O = w2.size(2);
  const Tensor scores = at::softmax(at::linear(x, wg), 1);
  const std::vector<Tensor> r = route_scores_op(scores, K, C, normalize);      // idx, loc, slot_map, top1, loss, own, gates
  const Tensor rows = r[5].select(0, 2).view(at::kFloat);
  const Tensor xs = dispatch_scatter_op(x, r[2], c10::nullopt, K, E * C, false).view({E, C, x.size(1)});
  const Tensor t = at::bmm(xs, w1).add_(b1.unsqueeze(1)), h = act32(t, act);
  const Tensor ys = at::bmm(h, w2).add_(b2.unsqueeze(1));
  const Tensor y = dispatch_gather_op(ys.view({E * C, O}), r[0], r[1], rows, C, false);
  return {y, r[4], scores, r[3], r[2], r[0], r[1], rows, xs, t, h, ys};
}

// {dx, dwg, dw1, db1, dw2, db2}, those that `need` asks for; dy undefined: the loss alone has a gradient, the experts none
std::vector<Tensor> layer32_backward_op(const c10::optional<Tensor>& dy_, const c10::optional<Tensor>& dloss, const Tensor& x, const Tensor& wg,
                                        const Tensor& w1, const Tensor& w2, const std::vector<Tensor>& saved, bool normalize, int64_t act,
                                        const std::vector<bool>& need) {
  at::NoGradGuard none;
  c10::cuda::CUDAGuard guard(x.device());
  const Tensor &scores = saved[0], &top1 = saved[1], &slot_map = saved[2], &idx = saved[3], &loc = saved[4], &rows = saved[5],
               &xs = saved[6], &t = saved[7], &h = saved[8], &ys = saved[9];
  const int64_t K = idx.size(0), S = x.size(0), E = w1.size(0), C = xs.size(1), O = w2.size(2);
  const bool has_dy = dy_.has_value() && dy_->defined();
  Tensor dx, dwg, dw1, db1, dw2, db2, dscores;
  std::vector<c10::optional<Tensor>> dgates;
  if (has_dy) {
    const Tensor dy = vector_rows(*dy_);
    if (need[0] || need[1]) {
      const Tensor dg = dispatch_gate_grad_op(ys.view({E * C, O}), dy, idx, loc, C);
      for (int64_t k = 0; k < K; ++k) dgates.emplace_back(dg.select(0, k));
    }
    const Tensor dys = dispatch_scatter_op(dy, slot_map, rows, K, E * C, false).view({E, C, O});
    if (need[5]) db2 = dys.sum(1);
    if (need[4]) dw2 = at::bmm(h.transpose(1, 2), dys);
    if (need[0] || need[2] || need[3]) {
      const Tensor dt = act32_backward(at::bmm(dys, w2.transpose(1, 2)), t, h, act);
      if (need[3]) db1 = dt.sum(1);
      if (need[2]) dw1 = at::bmm(xs.transpose(1, 2), dt);
      if (need[0]) dx = dispatch_gather_op(at::bmm(dt, w1.transpose(1, 2)).view({E * C, x.size(1)}), idx, loc, c10::nullopt, C, false);
    }
  }
  if (need[0] || need[1]) {
    if (!dgates.empty()) dscores = route_scores_backward_op(scores, idx, dgates, dloss, top1, S, normalize);
    else                 dscores = route_scores_backward_op(c10::nullopt, c10::nullopt, {}, dloss, top1, S, normalize);
    const Tensor dl = at::_softmax_backward_data(dscores, scores, 1, at::kFloat);
    if (need[0]) dx = dx.defined() ? dx.addmm_(dl, wg) : at::mm(dl, wg);
    if (need[1]) dwg = at::mm(dl.t(), x);
  }
  return {dx, dwg, dw1, db1, dw2, db2};
}
