// The fixed-order sums of measurements: block sizes, and the marginals of
// mq_marginal.cu for mq_reduce.cu.
#pragma once

#include "mq_internal.cuh"

namespace mq {

constexpr uint32_t kBlock = 1024;  // entries of a block sum
constexpr uint32_t kSuper = 1024;  // partial sums of one sequential run

// Deterministic marginal over `wires` (k < n or permuted order) into device
// memory: *q = the 2^k values, somewhere in work[0 .. 2 nc + 2^k).
int marginal_device(mq_state* h, const int32_t* wires, int k, double* work, double** q);

}  // namespace mq
