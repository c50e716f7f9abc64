// The operators of torch_ops.cpp as C++ functions, for the Python binding in torch_bind.cpp.
#pragma once

#include <ATen/ATen.h>

#include <vector>

namespace t2fw_ops {

// {outputs [B,T,D], ckpt_states [B,slots,D,K]}
std::vector<at::Tensor> lfw_forward(const at::Tensor &x, const at::Tensor &f, const at::Tensor &query,
                                    const at::Tensor &key, const at::Tensor &f_key, const at::Tensor &state);
// {d_x, d_f, d_query, d_key, d_f_key, d_state}; `outputs` is only checked for its shape
std::vector<at::Tensor> lfw_backward(const at::Tensor &grad_output, const at::Tensor &grad_state,
                                     const at::Tensor &value, const at::Tensor &forget, const at::Tensor &query,
                                     const at::Tensor &key, const at::Tensor &f_key, const at::Tensor &outputs,
                                     const at::Tensor &state, const at::Tensor &ckpt_states);
void lfw_decode_step(const at::Tensor &x, const at::Tensor &f, const at::Tensor &query, const at::Tensor &key,
                     const at::Tensor &f_key, const at::Tensor &state_in, const at::Tensor &state_out,
                     const at::Tensor &outputs);
bool lfw_decode_ring(const at::Tensor &x, const at::Tensor &f, const at::Tensor &query, const at::Tensor &key,
                     const at::Tensor &f_key, const at::Tensor &state, const at::Tensor &outputs);
std::vector<at::Tensor> lfw_fused_forward(const at::Tensor &qkvg, const at::Tensor &state, int64_t n_head);
std::vector<at::Tensor> lfw_fused_backward(const at::Tensor &grad_output, const at::Tensor &grad_state,
                                           const at::Tensor &qkvg, const at::Tensor &state,
                                           const at::Tensor &ckpt_states, int64_t n_head);
// {outputs, final_state, delta}
std::vector<at::Tensor> dfw_forward(const at::Tensor &query, const at::Tensor &key, const at::Tensor &value,
                                    const at::Tensor &state);
// {d_query, d_key, d_value, d_state}
std::vector<at::Tensor> dfw_backward(const at::Tensor &grad_output, const at::Tensor &grad_state,
                                     const at::Tensor &query, const at::Tensor &key, const at::Tensor &delta_value,
                                     const at::Tensor &final_state);

}  // namespace t2fw_ops
