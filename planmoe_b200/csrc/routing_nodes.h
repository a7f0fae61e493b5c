// Autograd nodes of routing, encode and decode (impls/fast_dispatch.py, ops/dispatch.py) in C++: their backward runs on the
// engine's thread without the interpreter.  Encode and decode have Python functions that do the same, which stay for function
// transforms, forward-mode, tracing, tensor subclasses, rows that are no whole vectors, and the CPU.  Included by bindings.cpp
// behind the operations that it calls.
#pragma once

using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

// A contiguous tensor on a 16-byte boundary, which is what kernels that move rows as vectors take.
Tensor vector_rows(const Tensor& t) {
  const Tensor c = t.contiguous();
  return reinterpret_cast<uintptr_t>(c.data_ptr()) % 16 == 0 ? c : c.clone();
}

// Encode, decode and the gates' gradient as differentiable operations, for a gradient of a gradient.  Sums are fp32 and gates are
// rounded to the data's type, as in the kernels.
struct PickOps {
  const Tensor &idx, &loc;
  int64_t E, C;
  variable_list gates;                             // one a pick, or none at all

  Tensor kept(int64_t k) const { return ((loc[k] < C).logical_and_(loc[k] >= 0).logical_and_(idx[k] >= 0)).unsqueeze(1); }
  Tensor slot(int64_t k) const { return (idx[k].to(at::kLong) * C + loc[k].to(at::kLong)).clamp(0, E * C - 1); }
  Tensor weighted(const Tensor& rows, int64_t k, at::ScalarType dtype) const {
    const Tensor r = at::where(kept(k), rows.to(at::kFloat), at::zeros({}, rows.options().dtype(at::kFloat)));
    return gates.empty() ? r : r * gates[k].to(dtype).to(at::kFloat).unsqueeze(1);
  }
  Tensor scatter(const Tensor& x) const {
    Tensor out = at::zeros({E * C, x.size(1)}, x.options().dtype(at::kFloat));
    for (int64_t k = 0; k < idx.size(0); ++k) out = out.index_add(0, slot(k), weighted(x, k, x.scalar_type()));
    return out.to(x.scalar_type());
  }
  Tensor gather(const Tensor& disp) const {
    Tensor out;
    for (int64_t k = 0; k < idx.size(0); ++k) {
      const Tensor r = weighted(disp.index_select(0, slot(k)), k, disp.scalar_type());
      out = out.defined() ? out + r : r;
    }
    return out.to(disp.scalar_type());
  }
  Tensor gate_grad(const Tensor& disp, const Tensor& dy, int64_t k) const {
    return PickOps{idx, loc, E, C, {}}.weighted(disp.index_select(0, slot(k)), k, at::kFloat).mul(dy.to(at::kFloat)).sum(1);
  }
};

// Tokens [S, M] -> slots [E * C, M], without gates.
struct ScatterNode : torch::autograd::Function<ScatterNode> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& idx, const Tensor& loc, const Tensor& slot_map,
                        int64_t E, int64_t C) {
    ctx->set_materialize_grads(false);
    ctx->save_for_backward({idx, loc});
    ctx->saved_data["E"] = E;
    ctx->saved_data["C"] = C;
    return dispatch_scatter_op(vector_rows(x), slot_map, c10::nullopt, idx.size(0), E * C, false);
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    variable_list out(6);
    if (!grads[0].defined()) return out;
    const variable_list saved = ctx->get_saved_variables();
    const int64_t C = ctx->saved_data["C"].toInt();
    if (at::GradMode::is_enabled())                // create_graph
      out[0] = PickOps{saved[0], saved[1], ctx->saved_data["E"].toInt(), C, {}}.gather(grads[0]);
    else
      out[0] = dispatch_gather_op(vector_rows(grads[0]), saved[0], saved[1], c10::nullopt, C, false);
    return out;
  }
};

// In-place changes of a tensor so far; those of inference tensors are not counted.
int64_t version_of(const Tensor& t) { return t.is_inference() ? 0 : (int64_t)t._version(); }

// Slots [E * C, M] -> tokens [S, M], weighted by fp32 `rows` [K, S], which the kernels round to the data's type; the gradient
// of the gates goes to the picks' own tensors g0 .. g3, the first K of which are there.  No `slot_map`: made when the
// backward needs it.  The gates are kept beside the saved tensors: a gradient uses `rows`, whatever has become of them since, and
// only a gradient of a gradient, which runs through their history, wants them as they were.
using OptTensor = c10::optional<Tensor>;
struct GatherPicksNode : torch::autograd::Function<GatherPicksNode> {
  static constexpr int kGates = 4, kInputs = 1 + kGates + 6;
  static Tensor forward(AutogradContext* ctx, const Tensor& disp, const OptTensor& g0, const OptTensor& g1, const OptTensor& g2, const OptTensor& g3,
                        const Tensor& idx, const Tensor& loc, const Tensor& rows, const OptTensor& slot_map, int64_t E, int64_t C) {
    ctx->set_materialize_grads(false);
    ctx->save_for_backward({disp, idx, loc, rows, slot_map.value_or(Tensor())});
    ctx->saved_data["E"] = E;
    ctx->saved_data["C"] = C;
    std::vector<Tensor> gates;
    std::vector<int64_t> made;
    for (const OptTensor* g : {&g0, &g1, &g2, &g3})
      if (g->has_value()) { gates.push_back(**g); made.push_back(version_of(**g)); }
    ctx->saved_data["gates"] = std::move(gates);
    ctx->saved_data["made"] = std::move(made);
    return dispatch_gather_op(vector_rows(disp), idx, loc, rows, C, disp.scalar_type() != at::kFloat);
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    const int64_t E = ctx->saved_data["E"].toInt(), C = ctx->saved_data["C"].toInt();
    variable_list out(kInputs);
    if (!grads[0].defined()) return out;
    const variable_list saved = ctx->get_saved_variables();
    const Tensor &disp = saved[0], &idx = saved[1], &loc = saved[2], &rows = saved[3];
    const int64_t K = idx.size(0);
    if (at::GradMode::is_enabled()) {              // create_graph
      const std::vector<Tensor> gates = ctx->saved_data["gates"].toTensorVector();
      const std::vector<int64_t> made = ctx->saved_data["made"].toIntVector();
      for (int64_t k = 0; k < K; ++k)
        TORCH_CHECK(version_of(gates[k]) == made[k], "gates needed for the gradient of a gradient have been modified by an inplace operation");
      const PickOps ops{idx, loc, E, C, gates};
      out[0] = ops.scatter(grads[0]);
      for (int64_t k = 0; k < K; ++k)
        if (ctx->needs_input_grad(1 + k)) out[1 + k] = ops.gate_grad(disp, grads[0], k);
      return out;
    }
    const Tensor dy = vector_rows(grads[0]);
    const Tensor map = saved[4].defined() ? saved[4] : build_slot_map_op(idx, loc, E, C);
    out[0] = dispatch_scatter_op(dy, map, rows, K, E * C, disp.scalar_type() != at::kFloat);
    bool wanted = false;
    for (int64_t k = 0; k < K; ++k) wanted = wanted || ctx->needs_input_grad(1 + k);
    if (wanted) {
      const Tensor dg = dispatch_gate_grad_op(vector_rows(disp), dy, idx, loc, C);
      for (int64_t k = 0; k < K; ++k) out[1 + k] = dg.select(0, k);
    }
    return out;
  }
};

// Per-pick gates from the picked scores [S, K], as differentiable operations.
std::vector<Tensor> gates_of(const Tensor& picked, bool normalize) {
  std::vector<Tensor> g;
  Tensor denom;
  if (picked.size(1) > 1 && normalize) denom = picked.sum(1).clamp_min(kFloatEps);
  for (int64_t k = 0; k < picked.size(1); ++k) g.push_back(denom.defined() ? picked.select(1, k) / denom : picked.select(1, k));
  return g;
}

// Top-k, gates, locations, slot map and the value of the GShard loss of fp32 scores (route_scores_op).  Gradients and slots use
// `own`, a second copy of picks, locations and gates: the caller may change the lists of a plan in place.
struct RouteScoresNode : torch::autograd::Function<RouteScoresNode> {
  static variable_list forward(AutogradContext* ctx, const Tensor& scores, int64_t K, int64_t C, bool normalize) {
    ctx->set_materialize_grads(false);
    variable_list out = route_scores_op(scores, K, C, normalize);       // idx, loc, slot_map, top1, loss, own, gates
    ctx->save_for_backward({scores, out[5], out[3]});
    ctx->saved_data["normalize"] = normalize;
    ctx->mark_non_differentiable({out[0], out[1], out[2], out[3], out[4], out[5]});
    return out;
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    variable_list out(4);
    const int64_t K = (int64_t)grads.size() - 6;
    bool any = false;
    for (int64_t k = 0; k < K; ++k) any = any || grads[6 + k].defined();
    if (!any) return out;
    const variable_list saved = ctx->get_saved_variables();
    const Tensor &scores = saved[0], picks = saved[1].select(0, 0), &top1 = saved[2];
    const bool normalize = ctx->saved_data["normalize"].toBool();
    if (at::GradMode::is_enabled()) {              // create_graph: the same gradient as differentiable operations
      const std::vector<Tensor> all = gates_of(scores.gather(1, picks.t().to(at::kLong)), normalize);
      variable_list g, d;
      for (int64_t k = 0; k < K; ++k)
        if (grads[6 + k].defined()) { g.push_back(all[k]); d.push_back(grads[6 + k]); }
      out[0] = torch::autograd::grad(g, {scores}, d, c10::nullopt, true)[0];
      return out;
    }
    std::vector<c10::optional<Tensor>> dg;
    for (int64_t k = 0; k < K; ++k) dg.emplace_back(grads[6 + k].defined() ? c10::optional<Tensor>(grads[6 + k]) : c10::nullopt);
    out[0] = route_scores_backward_op(scores, picks, dg, c10::nullopt, top1, scores.size(0), normalize);
    return out;
  }
};

// The GShard loss that the routing kernels computed, as a node of its own: its backward can run before, after or without the
// gates'.  It is linear in the scores, sum_t sum_e scores[t, e] * top1[e] * E / S^2: their values may change before the backward.
struct RouteLossNode : torch::autograd::Function<RouteLossNode> {
  static Tensor forward(AutogradContext* ctx, const Tensor& scores, const Tensor& value, const Tensor& top1) {
    ctx->set_materialize_grads(false);
    ctx->save_for_backward({top1});
    ctx->saved_data["S"] = scores.size(0);
    return value.detach();                         // its own tensor on the value's memory
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    variable_list out(3);
    if (!grads[0].defined()) return out;
    const Tensor top1 = ctx->get_saved_variables()[0];
    const int64_t S = ctx->saved_data["S"].toInt(), E = top1.numel();
    if (at::GradMode::is_enabled())
      out[0] = (grads[0] * ((double)E / ((double)S * (double)S)) * top1.to(grads[0].scalar_type())).expand({S, E});
    else
      out[0] = route_scores_backward_op(c10::nullopt, c10::nullopt, {}, grads[0], top1, S, false);
    return out;
  }
};

Tensor scatter_node(const Tensor& x, const Tensor& idx, const Tensor& loc, const Tensor& slot_map, int64_t E, int64_t C) {
  return ScatterNode::apply(x, idx, loc, slot_map, E, C);
}
Tensor gather_picks_node(const Tensor& disp, const Tensor& idx, const Tensor& loc, const Tensor& rows, const std::vector<Tensor>& gates,
                         const c10::optional<Tensor>& slot_map, int64_t E, int64_t C) {
  TORCH_CHECK(gates.size() == (size_t)idx.size(0) && gates.size() <= GatherPicksNode::kGates);
  OptTensor g[GatherPicksNode::kGates];
  for (size_t k = 0; k < gates.size(); ++k) g[k] = gates[k];
  return GatherPicksNode::apply(disp, g[0], g[1], g[2], g[3], idx, loc, rows, slot_map, E, C);
}
// {idx, loc, slot_map, top1, loss value, own, gates ...} and the loss as a node, if asked for
std::vector<Tensor> route_scores_node(const Tensor& scores, int64_t K, int64_t C, bool normalize, bool with_loss) {
  variable_list out = RouteScoresNode::apply(scores, K, C, normalize);
  if (with_loss) out.push_back(RouteLossNode::apply(scores, out[4], out[3]));
  return out;
}
