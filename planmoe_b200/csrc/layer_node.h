// The autograd node of a layer of one rank (ops/fused_moe.py) in C++: its backward runs on the engine's thread without the
// interpreter.  It does what the Python function _LocalLayer does, which stays for the stage timers, function transforms,
// forward-mode and tracing.  Included by bindings.cpp behind local_moe_forward_op and local_moe_backward_op.
#pragma once

static const char* const kSecondOrder =
    "the gradient was computed by kernels and cannot be differentiated twice; PLANMOE_GEMM=cublas makes a layer of operations that can";

// What a pass is done with; capacity, idx and loc are set by the forward.
struct LayerArgs {
  int64_t K, capacity;
  const py::object& round_up;
  bool normalize, bf16_logits, prio;
  int64_t act;
  bool postscore, int8;
  int64_t budget_ms;
  std::shared_ptr<StatusWord> status;
  Tensor idx, loc;
};
// Keeps the status word that a backward may report to.
struct StatusHolder : torch::CustomClassHolder {
  std::shared_ptr<StatusWord> word;
  explicit StatusHolder(std::shared_ptr<StatusWord> w) : word(std::move(w)) {}
};

// Results of a backward under create_graph (ops/native.py, first_order): the same values, which raise when they are
// differentiated by what they depend on.
static variable_list once(variable_list found, const std::vector<variable_list>& depends) {
  const size_t n = found.size();
  bool any = false;
  for (Tensor& t : found) {
    any = any || t.defined();
    if (t.defined()) t = t.detach();
  }
  for (const variable_list& list : depends)
    for (const Tensor& t : list)
      if (t.defined() && t.requires_grad()) found.push_back(t);
  if (any && found.size() > n) found = torch::autograd::DelayedError(kSecondOrder, (int64_t)found.size())(std::move(found));
  found.resize(n);
  return found;
}

struct LayerNode : torch::autograd::Function<LayerNode> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& wg, const Tensor& w1, const Tensor& b1,
                               const Tensor& w2, const Tensor& b2, LayerArgs* a) {
    ctx->set_materialize_grads(false);
    const auto [t, capacity] = local_moe_forward_op(x, wg, w1, b1, w2, b2, a->K, a->capacity, a->round_up, a->normalize, a->bf16_logits,
                                                    a->prio, a->act, a->postscore, a->int8, a->budget_ms,
                                                    (int64_t)a->status->device_ptr(), true, py::none());
    a->capacity = capacity; a->idx = t[6]; a->loc = t[14];
    ctx->save_for_backward({x, wg, w1, w2, t[2], t[3], t[4], t[5], t[6], t[7], t[8], t[9], t[10], t[11], t[12], t[13]});
    ctx->saved_data["also"] = std::vector<Tensor>{b1, b2};
    ctx->saved_data["act"] = a->act;
    ctx->saved_data["flags"] = (int64_t)(a->postscore | a->int8 << 1 | a->normalize << 2 | a->bf16_logits << 3);
    ctx->saved_data["budget_ms"] = a->budget_ms;
    ctx->saved_data["status"] = c10::IValue::make_capsule(c10::make_intrusive<StatusHolder>(a->status));
    return {t[0], t[1]};
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    variable_list out(7);
    if (!grads[0].defined() && !grads[1].defined()) return out;
    const variable_list s = ctx->get_saved_variables();
    const int64_t flags = ctx->saved_data["flags"].toInt();
    const auto status = c10::static_intrusive_pointer_cast<StatusHolder>(ctx->saved_data["status"].toCapsule());
    const LocalRoute r{s[8], s[9], s[6], s[7], s[10], s[11].size(1), ctx->saved_data["act"].toInt(), (flags & 1) != 0, (flags & 2) != 0,
                       ctx->saved_data["budget_ms"].toInt(), (int64_t)status->word->device_ptr()};
    std::vector<bool> need;
    for (int i = 0; i < 6; ++i) need.push_back(ctx->needs_input_grad(i));
    auto opt = [](const Tensor& t) { return t.defined() ? c10::optional<Tensor>(t) : c10::nullopt; };
    const std::vector<Tensor> d = local_moe_backward_op(opt(grads[0].defined() ? vector_rows(grads[0]) : Tensor()), opt(grads[1]), s[0], s[1], r,
                                                        s[2], s[3], s[4], s[5], s[11], s[12], s[13], s[14], opt(s[15]),
                                                        (flags & 4) != 0, (flags & 8) != 0, need, py::object());
    for (int i = 0; i < 6; ++i) out[i] = d[i];
    return at::GradMode::is_enabled() ? once(std::move(out), {grads, s, ctx->saved_data["also"].toTensorVector()}) : out;
  }
};

// {y, l_aux, idx, loc}, capacity
std::tuple<std::vector<Tensor>, int64_t> local_layer_node(
    const Tensor& x, const Tensor& wg, const Tensor& w1, const Tensor& b1, const Tensor& w2, const Tensor& b2, int64_t K,
    int64_t capacity, const py::object& round_up, bool normalize, bool bf16_logits, bool prio, int64_t act, bool postscore, bool int8,
    int64_t budget_ms, std::shared_ptr<StatusWord> status) {
  LayerArgs a{K, capacity, round_up, normalize, bf16_logits, prio, act, postscore, int8, budget_ms, std::move(status), {}, {}};
  variable_list out = LayerNode::apply(x, wg, w1, b1, w2, b2, &a);
  return {{out[0], out[1], a.idx, a.loc}, a.capacity};
}
