// Entry points of the tensor-memory SAP kernels (sap_tmem.cu).
#ifndef MOPS_B200_SAP_TMEM_HPP
#define MOPS_B200_SAP_TMEM_HPP

#include "runtime.hpp"

namespace mops_b200 {

// One SAP problem: operand and result widths, triplets. I, K, nA, nB, nO >= 1.
template <typename T> struct SapProblem {
    const T *A, *B, *C;
    const int32_t *PA, *PB, *PO;
    int64_t I, K;
    int nA, nB, nO;
};

// Enqueue the operation on the call's stream and return true, or return false when its operands
// are too wide (or its triplets too many) for these kernels. Results that are nullptr are skipped;
// grad_grad_A / grad_grad_B may be nullptr (zero).
template <typename T> bool sap_forward_tmem(const Call& call, const SapProblem<T>& p, T* O);
template <typename T>
bool sap_backward_tmem(const Call& call, const SapProblem<T>& p, T* gA, T* gB, const T* gO);
template <typename T>
bool sap_second_tmem(const Call& call, const SapProblem<T>& p, T* ggO, T* gA2, T* gB2, const T* ggA,
                     const T* ggB, const T* gO);

} // namespace mops_b200

#endif
