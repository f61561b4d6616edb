// Entry points of the row kernels of SASAW (sasaw_rows.cu).
#ifndef MOPS_B200_SASAW_ROWS_HPP
#define MOPS_B200_SASAW_ROWS_HPP

#include <initializer_list>

#include "runtime.hpp"

namespace mops_b200 {

template <typename T> struct SasawProblem {
    const T *A, *B, *C, *W;
    const int32_t *M1, *J, *M2, *I, *M3;
    int64_t E, N, rows; // edges, coupling entries, output rows (= rows of W)
    int nA, nW, nO, L;
};

// Which kernels of a forward to enqueue: for a scatter index that is sorted, for one that is not (they
// stand down on the device where the index is the other), or both.
enum class ScatterPart { kBoth, kSorted, kUnsorted };
// What a forward then returns: its kernels do not apply; the result is complete; the sorted part is
// enqueued, and the one for an unsorted index is still to come.
enum : int { kNotApplicable = 0, kComplete = 1, kUnsortedLeft = 2 };

// Whether the kernels on the FP64 tensor-core instruction take this work (f64, 16-byte aligned operands), with `others`
// beside the operands of `p`: the result of a forward, gO and gB of the gradients.
enum class RowsWork { kSorted, kUnsorted, kGradients };
template <typename T>
bool sasaw_rows_by_mma(const SasawProblem<T>& p, RowsWork work, std::initializer_list<const void*> others);
// Microseconds that the row kernels take, by that instruction (mma) or by multiply-adds, as fitted to measurements; infinite
// where they do not apply.
template <typename T> double sasaw_rows_cost(const SasawProblem<T>& p, RowsWork work, bool mma);

// Enqueue the operation on the call's stream and return true, or return false when its channel
// counts are too large for these kernels (the forward: as above). Gradients that are nullptr are skipped.
template <typename T> int sasaw_forward_rows(const Call& call, const SasawProblem<T>& p, T* O, ScatterPart part);
template <typename T>
bool sasaw_backward_rows(const Call& call, const SasawProblem<T>& p, T* gA, T* gB, T* gW, const T* gO);

} // namespace mops_b200

#endif
