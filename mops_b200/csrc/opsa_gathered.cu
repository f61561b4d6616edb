// OPSA / OPSAW on an index that is known not to be sorted: the streaming kernels of opsa_pipe.cuh over a sorted
// order of the entries. A, B and W rows are gathered into the same rings by asynchronous copies, so that the
// latency of the gathers is hidden as in the sorted case; the kernels with a lane per column or entry
// (unsorted.cuh, opsa_vjp_entries), which wait for eight rows at a time, remain for widths and alignments that
// cannot be streamed, for asynchronous calls, and for gradients of short rows (least_per_row).
//
// 300 000 entries of 16 x 32 in 5003 rows, f32, weighted, without the sort: forward 140 -> 33 us, VJP 104 -> 62 us
// (60 and 245 instructions per entry became 53 and 92).
#include <algorithm>
#include <type_traits>

#include "bulk.cuh"
#include "device.cuh"
#include "opsa_gathered.hpp"
#include "unsorted.cuh"

namespace mops_b200 {
namespace {

#include "opsa_pipe.cuh"

// Sorts the entries and clears the rows that no warp stores: those without entries and those that segments
// of S positions cut.
template <typename T, typename Sync>
__device__ __forceinline__ void sort_and_clear(const EntrySort& s, const int32_t* __restrict__ P, int64_t J,
                                               int64_t n_rows, T* O, int64_t row_size, int S, const Status& st,
                                               Sync&& sync) {
    sort_entries(s, P, J, n_rows, false, st, sync);
    zero_cut_rows(O, s, row_size, n_rows, S);
}
template <typename T>
__global__ void __launch_bounds__(kSortThreads)
sort_and_clear_grid(EntrySort s, const int32_t* P, int64_t J, int64_t n_rows, T* O, int64_t row_size, int S, Status st) {
    sort_and_clear(s, P, J, n_rows, O, row_size, S, st, [] { cooperative_groups::this_grid().sync(); });
}
template <typename T>
__global__ void __launch_bounds__(kSortThreads)
sort_and_clear_block(EntrySort s, const int32_t* P, int64_t J, int64_t n_rows, T* O, int64_t row_size, int S, Status st) {
    sort_and_clear(s, P, J, n_rows, O, row_size, S, st, [] { __syncthreads(); });
}

// Chunks of 8 entries (weighted: the padded B and W rows fill the ring) or 16.
template <typename T, bool WEIGHTED> PipeLayout gathered_layout(int K, int L, bool vjp) {
    return pipe_layout(sizeof(T), K, L, WEIGHTED, vjp, WEIGHTED ? kFixedChunk<true> : 16, 2, 2, true);
}

// Gradients: entries per output row from which the streaming kernel is the faster one (0: never). It copies a
// row's grad_output to shared memory and takes its fragments before the first of the row's entries, where
// opsa_vjp_entries reads it from the caches, so short rows and few products per entry do not pay; f32 pays
// for FP64 products of operands that move half the bytes. Streaming / entries, 20 000 to 500 000 entries, at
// the line and one step (a factor of 2 to 4 in entries per row) below it:
//
//   f64, K L >= 400          0.50 - 0.95 from 1 on (weighted: 0.71 - 0.94 from 4 on, 0.91 - 1.15 at 2)
//   f64, 256 <= K L < 400    0.70 - 1.06 from 8 on, 0.85 - 1.12 at 4
//   f64, K L >= 128 or L >= 24   0.77 - 1.05 from 32 on, 0.81 - 1.11 at 16; fewer products 0.88 - 1.5 at any length
//   f32, K L >= 128 and half of the tiles' 8 or 16 by 16 or 32 in use   0.82 - 1.04 from 32 on, 0.95 - 1.14 at 16;
//                            others 1.0 - 3.2
//   f32, weighted            fixed widths 0.91 - 1.03 from 16 on, 1.03 - 1.22 at 8; others 1.01 - 3.4
template <typename T, bool WEIGHTED> int64_t least_per_row(int K, int L) {
    const int products = K * L, tiles = (K <= 8 ? 8 : 16) * (L <= 16 ? 16 : 32);
    if (sizeof(T) == 4 && WEIGHTED) return fixed_shape(K, L) ? 16 : 0;
    if (sizeof(T) == 4) return products >= 128 && 2 * products >= tiles ? 32 : 0;
    return products >= 400 ? (WEIGHTED ? 4 : 1) : products >= 256 ? 8 : products >= 128 || L >= 24 ? 32 : 0;
}

// Calls f with a kernel's widths: fixed ones, or (TILES) tiles that hold K and L.
template <bool WEIGHTED, bool TILES, typename F> void for_widths(int K, int L, F&& f) {
    using std::integral_constant;
    if constexpr (WEIGHTED) {
        if (fixed_shape(K, L)) {
            if (K == 9)
                f(integral_constant<int, 9>(), integral_constant<int, 4>(), integral_constant<int, 9>());
            else if (K == 13)
                f(integral_constant<int, 13>(), integral_constant<int, 4>(), integral_constant<int, 13>());
            else
                f(integral_constant<int, 16>(), integral_constant<int, 4>(), integral_constant<int, 16>());
            return;
        }
    }
    if constexpr (TILES) {
        auto tiles = [&](auto k) {
            if (L <= 16)
                f(k, integral_constant<int, 2>(), integral_constant<int, 0>());
            else
                f(k, integral_constant<int, 4>(), integral_constant<int, 0>());
        };
        if (K <= 8)
            tiles(integral_constant<int, 8>());
        else
            tiles(integral_constant<int, 16>());
    }
}

} // namespace

template <typename T, bool WEIGHTED>
bool opsa_forward_gathered(const Call& call, T* O, const T* A, const T* B, const T* W, const int32_t* PW,
                           const int32_t* P, int64_t J, int K, int L, int64_t nO) {
    if (!pipe_usable<T, WEIGHTED>(A, B, W, nullptr, K, L)) return false;
    const PipeLayout lay = gathered_layout<T, WEIGHTED>(K, L, false);
    const size_t smem = static_cast<size_t>(lay.warp_bytes) * kPipeWarps;
    if (smem > static_cast<size_t>(max_optin_smem(call.device))) return false;
    for_widths<WEIGHTED, true>(K, L, [&](auto k, auto nt, auto kc) {
        constexpr int MT = (decltype(k)::value + 7) / 8, NT = decltype(nt)::value, KC = decltype(kc)::value;
        auto kernel = opsa_fwd_pipe<T, MT, NT, WEIGHTED, KC, (KC > 0 ? 32 : 0), true>;
        // every warp the same number of positions
        const int64_t warps = static_cast<int64_t>(sm_count(call.device)) * kPipeWarps *
                              resident_blocks(kernel, call.device, kPipeWarps * 32, smem);
        const int64_t S = std::max<int64_t>(ceil_div(ceil_div(J, warps), 4) * 4, 16);
        const int sorters = sort_blocks(call, J, nO * K * L);
        void* scratch = scratch_alloc(call, entry_sort_bytes(J, nO, sorters));
        const EntrySort sort = entry_sort_at(scratch, nO, sorters);
        launch_sorting(call, sorters, sort_and_clear_grid<T>, sort_and_clear_block<T>, sort, P, J, nO, O,
                       static_cast<int64_t>(K) * L, static_cast<int>(S), call.status);
        note_kernel_f("opsa_fwd_pipe<%s,MT=%d,NT=%d,W=%d> gathered", scalar_name<T>(), MT, NT, WEIGHTED ? 1 : 0);
        kernel<<<static_cast<unsigned>(ceil_div(ceil_div(J, S), kPipeWarps)), kPipeWarps * 32, smem, call.stream>>>(
            O, A, B, W, PW, sort.starts, J, nO, nO, sort.perm, S, lay, call.status);
        MOPS_CUDA_OK(cudaGetLastError());
        scratch_free(call, scratch);
    });
    return true;
}

template <typename T, bool WEIGHTED>
bool opsa_backward_gathered(const Call& call, T* gA, T* gB, T* gW, const T* gO, const T* A, const T* B, const T* W,
                            const int32_t* PW, const int32_t* P, int64_t J, int K, int L, int64_t nO) {
    if (!pipe_usable<T, WEIGHTED>(A, B, W, gO, K, L)) return false;
    const int64_t least = least_per_row<T, WEIGHTED>(K, L);
    if (least == 0 || J < least * nO) return false;
    const PipeLayout lay = gathered_layout<T, WEIGHTED>(K, L, true);
    const size_t smem = static_cast<size_t>(lay.warp_bytes) * kPipeWarps;
    if (smem > static_cast<size_t>(max_optin_smem(call.device))) return false;
    const int sorters = sort_blocks(call, J, nO);
    void* scratch = scratch_alloc(call, entry_sort_bytes(J, nO, sorters));
    const EntrySort sort = entry_sort_at(scratch, nO, sorters);
    launch_sorting(call, sorters, sort_if_unsorted_grid, sort_if_unsorted_block, sort, P, J, nO,
                   static_cast<uint32_t*>(nullptr), static_cast<int64_t>(0), 0, call.status);
    for_widths<WEIGHTED, !(sizeof(T) == 4 && WEIGHTED)>(K, L, [&](auto k, auto lt, auto kc) {
        constexpr int KT = (decltype(k)::value + 3) / 4, LT = decltype(lt)::value, KC = decltype(kc)::value;
        auto kernel = opsa_vjp_pipe<T, KT, LT, WEIGHTED, KC, (KC > 0 ? 32 : 0), true>;
        const int64_t held = static_cast<int64_t>(sm_count(call.device)) *
                             resident_blocks(kernel, call.device, kPipeWarps * 32, smem);
        const int64_t blocks = std::min(ceil_div(J, static_cast<int64_t>(kPipeWarps) * lay.ch), held);
        note_kernel_f("opsa_vjp_pipe<%s,KT=%d,LT8=%d,W=%d> gathered", scalar_name<T>(), KT, LT, WEIGHTED ? 1 : 0);
        kernel<<<static_cast<unsigned>(blocks), kPipeWarps * 32, smem, call.stream>>>(
            gA, gB, gW, gO, A, B, W, PW, sort.starts, J, nO, nO, sort.perm, lay, call.status);
        MOPS_CUDA_OK(cudaGetLastError());
    });
    scratch_free(call, scratch);
    return true;
}

#define INSTANTIATE(T, W)                                                                          \
    template bool opsa_forward_gathered<T, W>(const Call&, T*, const T*, const T*, const T*,       \
                                              const int32_t*, const int32_t*, int64_t, int, int,   \
                                              int64_t);                                            \
    template bool opsa_backward_gathered<T, W>(const Call&, T*, T*, T*, const T*, const T*,        \
                                               const T*, const T*, const int32_t*, const int32_t*, \
                                               int64_t, int, int, int64_t);
INSTANTIATE(float, false)
INSTANTIATE(float, true)
INSTANTIATE(double, false)
INSTANTIATE(double, true)

} // namespace mops_b200
