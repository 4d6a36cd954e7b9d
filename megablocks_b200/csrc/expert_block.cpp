// The routed expert computation of one device - plan, permute, expert GEMMs, weighted un-permute - as one
// native call where nothing is differentiated, else as two each way (the experts, the un-permutation), each
// behind an autograd node.  The kernels are those behind the separate ops; what this saves is the
// host's time between them: some 20 us of Python per op (an autograd node, argument checks and
// conversions), which bounds small calls (a decode step of 8 tokens has 60 us of kernels, a 256-token
// training pass 110).  Two nodes and not one, because y, which only the un-permutation's backward reads,
// has to be free before the experts' backward allocates.
//
// Two layouts, as in the layers (megablocks/layers/dmoe.py:196-249, moe.py:185-245 of the reference):
//   capacity < 0   dropless: ragged row groups, weights [E, f, h], groups given by the plan's `bins`;
//   capacity > 0   token-dropping: [E, capacity, h] slots, w1 [E, h, f], groups given by `gemm_bins`.
#include "kernels.h"
#include "torch_ops.h"

namespace mb {

namespace {

struct Gemm {
  bool trans_a = false, trans_b = false;
  int64_t epilogue = gemm::kEpiNone, act = 0;
  OptTensor aux1, aux2, a2, b2, sqnorm;
  bool want_out2 = true, want_out3 = true, only_out2 = false;
  double alpha = 1.0;

  std::vector<at::Tensor> run(const at::Tensor& a, const at::Tensor& b, const at::Tensor& bins, int64_t pair) const {
    return grouped_gemm(a, b, bins, trans_a, trans_b, epilogue, act, aux1, aux2, want_out2, want_out3, bins.numel(), {},
                        true, {}, 0, 0, 0, 0, pair, {}, {}, alpha, a2, b2, sqnorm, {}, only_out2);
  }
};

at::Tensor rows_of(const at::Tensor& t) { return t.dim() == 3 ? t.view({-1, t.size(2)}) : t; }

}  // namespace

// {y, tokens_per_expert, indices, inverse, bins} and, with `save`, {x rows, z1, z2, h} (z2 undefined for the
// MLP): plan, permutation and expert GEMMs; y[rows, hidden] is in expert order.
std::vector<at::Tensor> expert_rows_forward(const at::Tensor& x, const at::Tensor& top_experts, const at::Tensor& w1,
                                            const at::Tensor& w2, const OptTensor& v1, const OptTensor& gemm_bins,
                                            int64_t num_experts, int64_t top_k, int64_t act, int64_t capacity, bool save,
                                            int64_t pair) {
  const auto plan = route_plan_rows(top_experts, num_experts, 128, capacity);
  const at::Tensor &indices = plan[0], &bin_ids = plan[1], &bins = plan[2], &inverse = plan[5];
  const bool binned = capacity > 0;
  TORCH_CHECK(!binned || (gemm_bins.has_value() && !v1.has_value()), "capacity layout: uniform bins, no gate weight");
  at::Tensor rows = binned ? rows_of(binned_gather_rows(x, indices, {}, bins, capacity, top_k))
                           : gather_rows_op(x, indices, bin_ids, {}, bins, bins, top_k, indices.numel());
  const at::Tensor& groups = binned ? *gemm_bins : bins;
  at::Tensor z1, z2, h;
  Gemm up;
  up.trans_b = !binned;
  up.act = act;
  up.only_out2 = !save;         // the pre-activations are for the backward pass
  if (v1.has_value()) {
    up.epilogue = gemm::kEpiGluDual;
    up.b2 = v1;
    auto o = up.run(rows, w1, groups, pair);
    z2 = o[0]; h = o[1]; z1 = o[2];
  } else {
    up.epilogue = gemm::kEpiAct;
    auto o = up.run(rows, w1, groups, pair);
    z1 = o[0]; h = o[1];
  }
  at::Tensor y = Gemm{}.run(h, w2, groups, pair)[0];
  if (!save) return {y, plan[4], indices, inverse, bins};
  return {y, plan[4], indices, inverse, bins, rows, z1, z2, h};
}

// {out, tokens_per_expert}: the whole block where nothing is differentiated.
std::vector<at::Tensor> expert_block_forward(const at::Tensor& x, const at::Tensor& top_experts,
                                             const at::Tensor& weights, const at::Tensor& w1, const at::Tensor& w2,
                                             const OptTensor& v1, const OptTensor& bias, const OptTensor& gemm_bins,
                                             int64_t num_experts, int64_t top_k, int64_t act, int64_t capacity,
                                             int64_t pair) {
  auto o = expert_rows_forward(x, top_experts, w1, w2, v1, gemm_bins, num_experts, top_k, act, capacity, false, pair);
  return {combine_rows_op(o[0], o[3], weights, top_k, x.size(0), bias), o[1]};
}

namespace {

// Weighted un-permutation and output bias behind a node of its own: it alone keeps y, and frees it before the
// experts' backward starts.  A C++ node, which the host passes in a few microseconds each way where a Python
// one takes some 15.
struct Combine : torch::autograd::Function<Combine> {
  static at::Tensor forward(torch::autograd::AutogradContext* ctx, const at::Tensor& y, const at::Tensor& weights,
                            const OptTensor& bias, const at::Tensor& indices, const at::Tensor& inverse,
                            const at::Tensor& bins, int64_t top_k, int64_t capacity) {
    ctx->save_for_backward({y, weights, indices, bins});
    ctx->saved_data["top_k"] = top_k;
    ctx->saved_data["capacity"] = capacity;
    ctx->saved_data["bias"] = bias.has_value();
    ctx->set_materialize_grads(false);
    return combine_rows_op(y, inverse, weights, top_k, inverse.numel() / top_k, bias);
  }

  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx,
                                                 torch::autograd::variable_list grads) {
    torch::autograd::variable_list out(8);      // undefined: no gradient
    if (!grads[0].defined()) return out;
    const auto saved = ctx->get_saved_variables();
    const at::Tensor &weights = saved[1], &indices = saved[2], &bins = saved[3];
    const int64_t top_k = ctx->saved_data["top_k"].toInt(), capacity = ctx->saved_data["capacity"].toInt();
    const at::Tensor dout = grads[0].contiguous();
    const bool binned = capacity > 0;
    const at::Tensor y = binned ? saved[0].view({bins.numel(), capacity, saved[0].size(1)}) : saved[0];
    if (ctx->saved_data["bias"].toBool() && ctx->needs_input_grad(2)) out[2] = column_sum_op(dout);
    if (ctx->needs_input_grad(0)) {
      auto un = scatter_backward_op(y, dout, indices, weights, bins, binned ? OptTensor() : OptTensor(bins), top_k);
      out[0] = rows_of(un[0]);
      if (ctx->needs_input_grad(1)) out[1] = un[1];
    } else if (ctx->needs_input_grad(1)) {
      out[1] = binned ? binned_scatter_wgrad(y, dout, indices, bins, top_k)
                      : scatter_wgrad_op(y, dout, indices, indices, bins, bins, top_k);
    }
    return out;
  }
};

}  // namespace

at::Tensor expert_combine(const at::Tensor& y, const at::Tensor& weights, const OptTensor& bias,
                          const at::Tensor& indices, const at::Tensor& inverse, const at::Tensor& bins, int64_t top_k,
                          int64_t capacity) {
  return Combine::apply(y, weights, bias, indices, inverse, bins, top_k, capacity);
}

// {dx, dw1, dw2, dv1} from the gradient of y, undefined where `needs` says so.  `slots`: per weight gradient
// (w1, w2, v1) an optional accumulator of its squared norm.
std::vector<at::Tensor> expert_rows_backward(const at::Tensor& dy, const at::Tensor& inverse, const at::Tensor& bins,
                                             const OptTensor& gemm_bins, const at::Tensor& rows, const at::Tensor& z1,
                                             const OptTensor& z2, const OptTensor& h_in, const at::Tensor& w1,
                                             const at::Tensor& w2, const OptTensor& v1, const std::vector<bool>& needs,
                                             const std::vector<OptTensor>& slots, int64_t top_k, int64_t act,
                                             double wgrad_scale, int64_t capacity, int64_t pair) {
  const bool binned = capacity > 0;
  const at::Tensor& groups = binned ? *gemm_bins : bins;
  at::Tensor dx, dw1, dw2, dv1;
  at::Tensor dz1, dz2, h = h_in.has_value() ? *h_in : at::Tensor();
  {
    Gemm down;
    down.trans_b = true;
    down.act = act;
    down.aux1 = z1;
    if (v1.has_value()) {
      down.epilogue = gemm::kEpiDGlu;
      down.aux2 = z2;
      down.want_out3 = !h.defined();
      auto o = down.run(dy, w2, groups, pair);
      dz1 = o[0]; dz2 = o[1];
      if (!h.defined()) h = o[2];
    } else {
      down.epilogue = gemm::kEpiDAct;
      down.want_out2 = !h.defined();
      auto o = down.run(dy, w2, groups, pair);
      dz1 = o[0];
      if (!h.defined()) h = o[1];
    }
  }
  auto wgrad = [&](const at::Tensor& a, const at::Tensor& b, const OptTensor& slot) {
    Gemm g;
    g.trans_a = true;
    g.alpha = wgrad_scale;
    g.sqnorm = slot;
    return g.run(a, b, groups, pair)[0];
  };
  if (needs[2]) dw2 = wgrad(h, dy, slots[1]);
  if (needs[1]) dw1 = binned ? wgrad(rows, dz1, slots[0]) : wgrad(dz1, rows, slots[0]);
  if (v1.has_value() && needs[3]) dv1 = wgrad(dz2, rows, slots[2]);
  if (needs[0]) {
    at::Tensor d;
    {
      Gemm in;
      in.trans_b = binned;
      if (v1.has_value()) {       // dx = dz1 w1 + dz2 v1 as one contraction over both pairs
        in.a2 = dz2;
        in.b2 = v1;
      }
      d = in.run(dz1, w1, groups, pair)[0];
    }
    dz1.reset();                  // free before dx is allocated
    dz2.reset();
    h.reset();
    dx = combine_rows_op(d, inverse, {}, top_k, inverse.numel() / top_k, {});
  }
  return {dx, dw1, dw2, dv1};
}

}  // namespace mb
