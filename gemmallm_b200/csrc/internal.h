// Entry points of libmoe_b200.so that the package's own host extension (host.cpp) calls besides the
// C ABI of include/moe_b200.h. C++ linkage, same conventions and return codes.
#pragma once
#include <stddef.h>
#include <stdint.h>

namespace moe {

// moe_b200_forward with the load-balancing loss written to `aux` (nullptr: the workspace's own word).
int forward_into(const void* x, const void* Wg, const void* bg, const void* plan, const void* residual,
                 const void* norm_weight, const void* norm_bias, float norm_eps, int64_t N, int d, int f,
                 int E, int k, int dtype, int flags, void* workspace, size_t workspace_bytes, void* out,
                 float* aux, void* stream);

}  // namespace moe
