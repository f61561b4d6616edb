// Outer-product scatter-add behind a sorted order of the entries (opsa_gathered.cu).
#ifndef MOPS_B200_OPSA_GATHERED_HPP
#define MOPS_B200_OPSA_GATHERED_HPP

#include "runtime.hpp"

namespace mops_b200 {

// For calls that know their index to be unsorted (device status included): sort the entries and stream them
// in that order. False when the kernels do not apply (widths, alignment) or, for gradients, are not the faster
// ones; nothing is enqueued then.
template <typename T, bool WEIGHTED>
bool opsa_forward_gathered(const Call& call, T* O, const T* A, const T* B, const T* W, const int32_t* PW,
                           const int32_t* P, int64_t J, int K, int L, int64_t nO);
template <typename T, bool WEIGHTED>
bool opsa_backward_gathered(const Call& call, T* gA, T* gB, T* gW, const T* gO, const T* A, const T* B, const T* W,
                            const int32_t* PW, const int32_t* P, int64_t J, int K, int L, int64_t nO);

} // namespace mops_b200

#endif
