// Entry points of the tensor-memory HPE kernels (hpe_tmem.cu).
#ifndef MOPS_B200_HPE_TMEM_HPP
#define MOPS_B200_HPE_TMEM_HPP

#include "runtime.hpp"

namespace mops_b200 {

// Enqueue the forward / VJP of a checked problem (K >= 1, J >= 1, I >= 1) on the call's stream
// and return true, or return false when the operand is too wide for them.
template <typename T>
bool hpe_forward_tmem(const Call& call, T* O, const T* A, const T* C, const int32_t* P, int64_t I,
                      int N, int64_t J, int K);
template <typename T>
bool hpe_backward_tmem(const Call& call, T* gA, const T* gO, const T* A, const T* C,
                       const int32_t* P, int64_t I, int N, int64_t J, int K);

} // namespace mops_b200

#endif
