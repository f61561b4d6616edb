// Entry points of the row kernels of SASAW (sasaw_rows.cu).
#ifndef MOPS_B200_SASAW_ROWS_HPP
#define MOPS_B200_SASAW_ROWS_HPP

#include "runtime.hpp"

namespace mops_b200 {

template <typename T> struct SasawProblem {
    const T *A, *B, *C, *W;
    const int32_t *M1, *J, *M2, *I, *M3;
    int64_t E, N, rows; // edges, coupling entries, output rows (= rows of W)
    int nA, nW, nO, L;
};

// Enqueue the operation on the call's stream and return true, or return false when its channel
// counts are too large for these kernels. Gradients that are nullptr are skipped.
template <typename T> bool sasaw_forward_rows(const Call& call, const SasawProblem<T>& p, T* O);
template <typename T>
bool sasaw_backward_rows(const Call& call, const SasawProblem<T>& p, T* gA, T* gB, T* gW, const T* gO);

} // namespace mops_b200

#endif
