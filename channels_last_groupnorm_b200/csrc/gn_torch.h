// What gnb200_torch.so offers besides its ops.
#pragma once
#include <ATen/Tensor.h>

namespace gnb200_ops {

// The module's call, if it is a plain one (see gn_torch.cpp); an undefined tensor otherwise.
__attribute__((visibility("default"))) at::Tensor group_norm_act_direct(const at::Tensor& X, const at::Tensor& weight,
                                                                        const at::Tensor& bias, int64_t G, double eps, int64_t act);

}  // namespace gnb200_ops
