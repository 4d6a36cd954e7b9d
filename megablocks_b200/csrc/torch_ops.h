// Ops on tensors (torch_glue.cpp) that the expert block (expert_block.cpp) launches one after another and
// the module (bindings.cpp) also exposes one by one.
#pragma once

#include <torch/extension.h>

#include <vector>

namespace mb {

using OptTensor = c10::optional<at::Tensor>;

std::vector<at::Tensor> route_plan_rows(const at::Tensor& top_experts, int64_t num_experts, int64_t block,
                                        int64_t capacity);
at::Tensor gather_rows_op(const at::Tensor& x, const at::Tensor& indices, const at::Tensor& bin_ids,
                          const OptTensor& weights, const at::Tensor& bins, const at::Tensor& padded_bins,
                          int64_t top_k, int64_t out_rows);
at::Tensor binned_gather_rows(const at::Tensor& x, const at::Tensor& indices, const OptTensor& weights,
                              const at::Tensor& bins, int64_t capacity, int64_t top_k);
at::Tensor combine_rows_op(const at::Tensor& x, const at::Tensor& inverse, const OptTensor& weights, int64_t top_k,
                           int64_t tokens, const OptTensor& bias);
std::vector<at::Tensor> scatter_backward_op(const at::Tensor& x, const at::Tensor& grad, const at::Tensor& indices,
                                            const at::Tensor& weights, const at::Tensor& bins,
                                            const OptTensor& padded_bins, int64_t top_k);
at::Tensor scatter_wgrad_op(const at::Tensor& x, const at::Tensor& grad, const at::Tensor& indices,
                            const at::Tensor& bin_ids, const at::Tensor& bins, const at::Tensor& padded_bins,
                            int64_t top_k);
at::Tensor binned_scatter_wgrad(const at::Tensor& x, const at::Tensor& grad, const at::Tensor& indices,
                                const at::Tensor& bins, int64_t top_k);
at::Tensor column_sum_op(const at::Tensor& x);
// `only_out2`: the activation epilogues (kEpiAct, kEpiGluDual) store nothing but the activation; c and out3
// come back undefined.
std::vector<at::Tensor> grouped_gemm(const at::Tensor& a, const at::Tensor& b, const at::Tensor& bins, bool trans_a,
                                     bool trans_b, int64_t epilogue, int64_t act, const OptTensor& aux1,
                                     const OptTensor& aux2, bool want_out2, bool want_out3, int64_t num_groups,
                                     const OptTensor& c_in, bool zero_tail, const OptTensor& wait_flags,
                                     int64_t wait_count, int64_t wait_stride, int64_t wait_seq, int64_t rows_hint,
                                     int64_t pair_mode, const c10::optional<std::vector<at::Tensor>>& scatter,
                                     const std::vector<int64_t>& scatter_args, double alpha, const OptTensor& a2,
                                     const OptTensor& b2, const OptTensor& sqnorm, const OptTensor& seq_base,
                                     bool only_out2);

}  // namespace mb
