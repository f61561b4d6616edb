// OPSA / OPSAW on an index that is known not to be sorted: the streaming kernels of opsa_pipe.cuh over a sorted
// order of the entries. A, B and W rows are gathered into the same rings by asynchronous copies, so that the
// latency of the gathers is hidden as in the sorted case; the kernels with a lane per column or entry
// (unsorted.cuh, opsa_vjp_entries), which wait for eight rows at a time, remain for widths and alignments that
// cannot be streamed and for asynchronous calls.
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

// Calls f with a kernel's widths: fixed ones, or tiles that hold K and L.
template <bool WEIGHTED, typename F> void for_widths(int K, int L, F&& f) {
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

} // namespace

template <typename T, bool WEIGHTED>
bool opsa_forward_gathered(const Call& call, T* O, const T* A, const T* B, const T* W, const int32_t* PW,
                           const int32_t* P, int64_t J, int K, int L, int64_t nO) {
    if (!pipe_usable<T, WEIGHTED>(A, B, W, nullptr, K, L)) return false;
    const PipeLayout lay = gathered_layout<T, WEIGHTED>(K, L, false);
    const size_t smem = static_cast<size_t>(lay.warp_bytes) * kPipeWarps;
    if (smem > static_cast<size_t>(max_optin_smem(call.device))) return false;
    for_widths<WEIGHTED>(K, L, [&](auto k, auto nt, auto kc) {
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
    const PipeLayout lay = gathered_layout<T, WEIGHTED>(K, L, true);
    const size_t smem = static_cast<size_t>(lay.warp_bytes) * kPipeWarps;
    if (smem > static_cast<size_t>(max_optin_smem(call.device))) return false;
    const int sorters = sort_blocks(call, J, nO);
    void* scratch = scratch_alloc(call, entry_sort_bytes(J, nO, sorters));
    const EntrySort sort = entry_sort_at(scratch, nO, sorters);
    launch_sorting(call, sorters, sort_if_unsorted_grid, sort_if_unsorted_block, sort, P, J, nO,
                   static_cast<uint32_t*>(nullptr), static_cast<int64_t>(0), 0, call.status);
    for_widths<WEIGHTED>(K, L, [&](auto k, auto lt, auto kc) {
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
