// Scatter operations on an index that turns out not to be sorted.
//
// Whether the index is sorted is only known on the device: the kernels here run behind the sorted
// ones and return at once when those did the work. Otherwise the entries are sorted by output row
// first (a counting sort: histogram, scan, scatter) and then processed row by row: every output
// row is written once, by one warp, and the entries that share a grad_output row are neighbours.
// 300 000 entries of 16 x 32, f32: forward 735 us with atomics -> 165 us (23 of them the sort), VJP
// 209 us in the order of the entries -> 23 + 103 us. (Calls that wait for the result stream the sorted
// entries instead where that is faster: opsa_gathered.cu.)
#ifndef MOPS_B200_UNSORTED_CUH
#define MOPS_B200_UNSORTED_CUH

#include <algorithm>

#include <cooperative_groups.h>

#include "device.cuh"

namespace mops_b200 {
namespace {

constexpr int kSortThreads = 1024;         // one block per SM, 64 registers
constexpr int64_t kOneBlockEntries = 512;  // up to here one block (and an ordinary launch) will do,
constexpr int64_t kOneBlockWrites = 8192;  // if it does not have more than this to clear

// Scratch of the sort.
struct EntrySort {
    int32_t* starts; // [n_rows + 1] first position of every row in `perm`
    int32_t* cursor; // [n_rows + 1] entries per row
    int32_t* sums;   // [blocks]
    int32_t* longest; // entries of the longest row, if more than kEvenRow, else 0
    int32_t* perm;   // [J] entries in the order of their rows
};
constexpr int kEvenRow = 32;

inline size_t entry_sort_bytes(int64_t J, int64_t n_rows, int blocks) {
    return (2 * static_cast<size_t>(n_rows + 1) + blocks + 1 + static_cast<size_t>(J)) * sizeof(int32_t);
}
inline EntrySort entry_sort_at(void* p, int64_t n_rows, int blocks) {
    EntrySort s;
    s.starts = static_cast<int32_t*>(p);
    s.cursor = s.starts + n_rows + 1;
    s.sums = s.cursor + n_rows + 1;
    s.longest = s.sums + blocks;
    s.perm = s.longest + 1;
    return s;
}

// Exclusive scan of one value per thread over the block; returns the block's total.
__device__ __forceinline__ int block_scan(int v, int& exclusive, int32_t* warp_sums) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(kFullMask, incl, o);
        if (lane >= o) incl += u;
    }
    __syncthreads();
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        const int w = lane < static_cast<int>(blockDim.x >> 5) ? warp_sums[lane] : 0;
        int wi = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(kFullMask, wi, o);
            if (lane >= o) wi += u;
        }
        warp_sums[lane] = wi - w;
        if (lane == 31) warp_sums[32] = wi;
    }
    __syncthreads();
    exclusive = warp_sums[warp] + incl - v;
    return warp_sums[32];
}

// Out-of-range rows are reported, and left out or (keep_bad) taken for row 0. `starts` and `longest` are complete
// for every thread when it returns, `perm` behind the next sync.
//
// Bounded by the latencies between the grid barriers (about 3 us each), so there are three: up to kHeldEntries
// per thread the count of a row gives every entry its place in the row (no second round of atomics), and up to
// kRowsAtOnce rows every block adds up the rows before its own by itself (300 000 entries, 5003 rows:
// 29 -> 22 us).
constexpr int kHeldEntries = 8;
constexpr int64_t kRowsAtOnce = 1 << 14;
template <typename Sync>
__device__ __forceinline__ void sort_entries(const EntrySort& s, const int32_t* __restrict__ P, int64_t J,
                                             int64_t n_rows, bool keep_bad, const Status& st, Sync&& sync,
                                             int bit = 0) {
    __shared__ int32_t warp_sums[33];
    __shared__ int32_t block_longest;
    const int64_t thread = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const int64_t threads = static_cast<int64_t>(gridDim.x) * blockDim.x;
    auto row_of = [&](int64_t j) {
        const int32_t row = __ldg(P + j);
        const bool good = static_cast<uint32_t>(row) < static_cast<uint32_t>(n_rows);
        if (!good) report_bad_index(st, bit);
        return good ? row : keep_bad ? 0 : -1;
    };
    int32_t* const counts = s.cursor;
    for (int64_t r = thread; r <= n_rows; r += threads) counts[r] = 0;
    if (thread == 0) *s.longest = 0;
    if (threadIdx.x == 0) block_longest = 0;
    const bool held = J <= kHeldEntries * threads;
    int row[kHeldEntries], rank[kHeldEntries];
#pragma unroll
    for (int q = 0; q < kHeldEntries; q++) {
        const int64_t j = thread + q * threads;
        row[q] = held && j < J ? row_of(j) : -1;
    }
    sync();
    if (held) {
#pragma unroll
        for (int q = 0; q < kHeldEntries; q++) rank[q] = row[q] >= 0 ? atomicAdd(counts + row[q], 1) : 0;
    } else {
        for (int64_t j = thread; j < J; j += threads) {
            const int r = row_of(j);
            if (r >= 0) atomicAdd(counts + r, 1);
        }
    }
    sync();
    // block b scans the rows [b per, (b + 1) per)
    const int64_t per = ceil_div(n_rows, gridDim.x);
    const int64_t lo = blockIdx.x * per < n_rows ? blockIdx.x * per : n_rows;
    const int64_t hi = lo + per < n_rows ? lo + per : n_rows;
    int unused, before = 0;
    if (n_rows <= kRowsAtOnce) {
        for (int64_t r = threadIdx.x; r < lo; r += blockDim.x) before += counts[r];
    } else {
        int mine = 0;
        for (int64_t r = lo + threadIdx.x; r < hi; r += blockDim.x) mine += counts[r];
        const int total = block_scan(mine, unused, warp_sums);
        if (threadIdx.x == 0) s.sums[blockIdx.x] = total;
        sync();
        for (int b = threadIdx.x; b < static_cast<int>(blockIdx.x); b += blockDim.x) before += s.sums[b];
    }
    int run = block_scan(before, unused, warp_sums);
    int most = 0;
    for (int64_t r0 = lo; r0 < hi; r0 += blockDim.x) {
        const int64_t r = r0 + threadIdx.x;
        const int v = r < hi ? counts[r] : 0;
        most = max(most, v);
        int exclusive;
        const int all = block_scan(v, exclusive, warp_sums);
        if (r < hi) s.starts[r] = run + exclusive;
        run += all;
    }
    most = __reduce_max_sync(kFullMask, most);
    if ((threadIdx.x & 31) == 0 && most > kEvenRow) atomicMax(&block_longest, most);
    __syncthreads();
    if (threadIdx.x == 0 && block_longest > 0) atomicMax(s.longest, block_longest);
    if (hi == n_rows && (lo < hi || blockIdx.x == 0) && threadIdx.x == 0) s.starts[n_rows] = run;
    sync();
    if (held) {
#pragma unroll
        for (int q = 0; q < kHeldEntries; q++)
            if (row[q] >= 0) s.perm[s.starts[row[q]] + rank[q]] = static_cast<int32_t>(thread + q * threads);
    } else {
        for (int64_t j = thread; j < J; j += threads) {
            const int r = row_of(j);
            if (r >= 0) s.perm[s.starts[r] + atomicSub(counts + r, 1) - 1] = static_cast<int32_t>(j);
        }
    }
}

// The sort alone, for kernels that read `perm`. Where rows are longer than `limit`, `zero` (n words, or
// nullptr) is cleared for kernels that will then add to it.
template <typename Sync>
__device__ __forceinline__ void sort_if_unsorted(const EntrySort& s, const int32_t* __restrict__ P, int64_t J,
                                                 int64_t n_rows, uint32_t* zero, int64_t n, int limit,
                                                 const Status& st, Sync&& sync) {
    if (!saw_unsorted(st)) return;
    sort_entries(s, P, J, n_rows, true, st, sync);
    if (zero != nullptr && *s.longest > limit)
        for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
             i += static_cast<int64_t>(gridDim.x) * blockDim.x)
            zero[i] = 0;
}
__global__ void __launch_bounds__(kSortThreads)
sort_if_unsorted_grid(EntrySort s, const int32_t* __restrict__ P, int64_t J, int64_t n_rows, uint32_t* zero,
                      int64_t n, int limit, Status st) {
    sort_if_unsorted(s, P, J, n_rows, zero, n, limit, st, [] { cooperative_groups::this_grid().sync(); });
}
__global__ void __launch_bounds__(kSortThreads)
sort_if_unsorted_block(EntrySort s, const int32_t* __restrict__ P, int64_t J, int64_t n_rows, uint32_t* zero,
                       int64_t n, int limit, Status st) {
    sort_if_unsorted(s, P, J, n_rows, zero, n, limit, st, [] { __syncthreads(); });
}

// `writes`: the rows, or the values of the result where the kernel clears it. (500 entries for 100 000 rows
// of 13 x 32: one block takes as long for the zeros as the whole GPU for 148 times as many.)
inline int sort_blocks(const Call& call, int64_t J, int64_t writes) {
    return J <= kOneBlockEntries && writes <= kOneBlockWrites ? 1 : sm_count(call.device);
}

// Launches `grid_kernel` cooperatively, or `block_kernel` with one block for few entries.
template <typename... Params, typename... Args>
void launch_sorting(const Call& call, int blocks, void (*grid_kernel)(Params...), void (*block_kernel)(Params...),
                    Args... args) {
    if (blocks == 1) {
        block_kernel<<<1, kSortThreads, 0, call.stream>>>(args...);
        MOPS_CUDA_OK(cudaGetLastError());
        return;
    }
    cudaLaunchConfig_t config{};
    config.gridDim = dim3(static_cast<unsigned>(blocks));
    config.blockDim = dim3(kSortThreads);
    config.stream = call.stream;
    cudaLaunchAttribute attribute{};
    attribute.id = cudaLaunchAttributeCooperative;
    attribute.val.cooperative = 1;
    config.attrs = &attribute;
    config.numAttrs = 1;
    MOPS_CUDA_OK(cudaLaunchKernelEx(&config, grid_kernel, static_cast<Params>(args)...));
}

// ---- forward of OPSA / OPSAW
constexpr int kGatherEntries = 8; // entries whose rows are in flight at a time

// Entries u0 .. u0 + U - 1 of the `count` (<= 32) that the lanes hold: (B o W)[e, lc] in `b` (0 beyond
// `count`), A[e, kb .. kb + kn) in `stage`. S: the type of products and sums.
template <typename T, int KC, bool WEIGHTED, int U, typename S>
__device__ __forceinline__ void load_entries(S (&b)[U], int my_entry, int my_w, int u0, int count,
                                             const T* __restrict__ A, const T* __restrict__ B,
                                             const T* __restrict__ W, int K, int L, int kb, int kn, int lc,
                                             T* stage, int lane) {
    T w[U];
#pragma unroll
    for (int x = lane; x < U * KC; x += 32) {
        const int u = x / KC, k = x - u * KC;
        const int64_t e = __shfl_sync(kFullMask, my_entry, u0 + u);
        stage[x] = k < kn && u0 + u < count ? __ldg(A + e * K + kb + k) : T(0);
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
        const int64_t e = __shfl_sync(kFullMask, my_entry, u0 + u);
        b[u] = __ldg(B + e * L + lc);
        if (WEIGHTED) w[u] = __ldg(W + static_cast<int64_t>(__shfl_sync(kFullMask, my_w, u0 + u)) * L + lc);
    }
    __syncwarp();
#pragma unroll
    for (int u = 0; u < U; u++) {
        if (WEIGHTED) b[u] *= static_cast<S>(w[u]);
        if (u0 + u >= count) b[u] = S(0);
    }
}

// acc[k] += a[k] b
template <typename T, int KC, typename S>
__device__ __forceinline__ void add_entry(S (&acc)[KC], const T* a_row, S b) {
    constexpr int V = 16 / sizeof(T);
#pragma unroll
    for (int k = 0; k < KC; k += V) {
        T a[V];
        load_vec<T, V>(a_row + k, a);
#pragma unroll
        for (int v = 0; v < V; v++) acc[k + v] += static_cast<S>(a[v]) * b;
    }
}

// A warp takes a segment of S consecutive positions of the sorted entries and a KC by 32 part of their
// rows, lane = column l of B. The entries' numbers and rows (of O, of W) are fetched 32 at a time, one
// per lane; B rows go to registers and A rows to shared memory eight entries at a time (`stage`: [8][KC]
// of this warp), where they are read as broadcasts. A row that lies in one segment is stored; one
// that is cut is added up with atomics (zero_cut_rows has cleared it), so that few or uneven rows
// still occupy every warp: 60 000 entries in 144 rows, f32, 8 x 17: 375 us with a warp per row, 85 with
// atomics per entry. Bounded by the latency of the gathers. (Handing A around by shuffles, one per
// product, took 430 us where this takes 175.)
template <typename T, int KC, bool WEIGHTED>
__device__ __forceinline__ void opsa_rows_gathered(T* __restrict__ O, const T* __restrict__ A,
                                                   const T* __restrict__ B, const T* __restrict__ W,
                                                   const int32_t* __restrict__ PW,
                                                   const int32_t* __restrict__ P, const EntrySort& s, int K,
                                                   int L, int64_t n_rows, int S, T* stage, const Status& st) {
    constexpr int U = kGatherEntries;
    const int lane = threadIdx.x & 31;
    const int64_t warps = static_cast<int64_t>(gridDim.x) * (blockDim.x >> 5);
    const int k_units = (K + KC - 1) / KC, units = k_units * ((L + 31) / 32);
    const int total = s.starts[n_rows]; // (bad rows are left out)
    const int64_t segments = (static_cast<int64_t>(total) + S - 1) / S;
    // consecutive warps take the parts of one segment: what they both read is in the caches
    for (int64_t unit = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
         unit < segments * units; unit += warps) {
        const int p_lo = static_cast<int>(unit / units * S), p_hi = p_lo + S < total ? p_lo + S : total;
        const int part = static_cast<int>(unit % units), lb = part / k_units * 32;
        const int kb = (part - part / k_units * k_units) * KC;
        const int l = lb + lane, lc = l < L ? l : L - 1;
        const int kn = K - kb < KC ? K - kb : KC;
        // rows that go on in the neighbouring segments
        const int before = p_lo > 0 ? __ldg(P + s.perm[p_lo - 1]) : -1;
        const int after = p_hi < total ? __ldg(P + s.perm[p_hi]) : -1;
        T acc[KC];
#pragma unroll
        for (int k = 0; k < KC; k++) acc[k] = T(0);
        int row = -1;
        auto flush = [&] {
            T* dst = O + (static_cast<int64_t>(row) * K + kb) * L + l;
            const bool cut = row == before || row == after;
#pragma unroll
            for (int k = 0; k < KC; k++) {
                if (row >= 0 && l < L && k < kn) {
                    if (cut)
                        red_add(dst + static_cast<int64_t>(k) * L, acc[k]);
                    else
                        dst[static_cast<int64_t>(k) * L] = acc[k];
                }
                acc[k] = T(0);
            }
        };
        for (int p0 = p_lo; p0 < p_hi; p0 += 32) {
            const int count = p_hi - p0 < 32 ? p_hi - p0 : 32;
            const int my_entry = s.perm[p0 + (lane < count ? lane : 0)];
            const int my_row = __ldg(P + my_entry);
            int my_w = 0;
            if (WEIGHTED) {
                my_w = __ldg(PW + my_entry);
                if (clamp_index(my_w, static_cast<int32_t>(n_rows))) report_bad_index(st, 1);
            }
            for (int u0 = 0; u0 < count; u0 += U) {
                T b[U];
                load_entries<T, KC, WEIGHTED, U, T>(b, my_entry, my_w, u0, count, A, B, W, K, L, kb, kn, lc, stage, lane);
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const int r = __shfl_sync(kFullMask, my_row, u0 + u);
                    if (u0 + u < count) {
                        if (r != row) {
                            flush();
                            row = r;
                        }
                        add_entry<T, KC, T>(acc, stage + u * KC, b[u]);
                    }
                }
                __syncwarp();
            }
        }
        flush();
    }
}

// Clears the rows that nobody stores: those without entries and those that segments of S positions cut.
template <typename T>
__device__ __forceinline__ void zero_cut_rows(T* __restrict__ O, const EntrySort& s, int64_t row_size,
                                              int64_t n_rows, int S) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = static_cast<int64_t>(gridDim.x) * (blockDim.x >> 5);
    for (int64_t r = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; r < n_rows; r += warps) {
        const int lo = s.starts[r], hi = s.starts[r + 1];
        if (lo < hi && lo / S == (hi - 1) / S) continue;
        for (int64_t x = lane; x < row_size; x += 32) O[r * row_size + x] = T(0);
    }
}

template <typename T, int KC, bool WEIGHTED>
__global__ void __launch_bounds__(kSortThreads)
opsa_fwd_unsorted_grid(T* O, const T* A, const T* B, const T* W, const int32_t* PW, const int32_t* P,
                       EntrySort s, int64_t J, int K, int L, int64_t n_rows, int S, Status st) {
    __shared__ __align__(16) T stage[kSortThreads / 32][kGatherEntries * KC];
    if (!saw_unsorted(st)) return;
    auto sync = [] { cooperative_groups::this_grid().sync(); };
    sort_entries(s, P, J, n_rows, false, st, sync);
    zero_cut_rows(O, s, static_cast<int64_t>(K) * L, n_rows, S);
    sync();
    opsa_rows_gathered<T, KC, WEIGHTED>(O, A, B, W, PW, P, s, K, L, n_rows, S, stage[threadIdx.x >> 5], st);
}
template <typename T, int KC, bool WEIGHTED>
__global__ void __launch_bounds__(kSortThreads)
opsa_fwd_unsorted_block(T* O, const T* A, const T* B, const T* W, const int32_t* PW, const int32_t* P,
                        EntrySort s, int64_t J, int K, int L, int64_t n_rows, int S, Status st) {
    __shared__ __align__(16) T stage[kSortThreads / 32][kGatherEntries * KC];
    if (!saw_unsorted(st)) return;
    auto sync = [] { __syncthreads(); };
    sort_entries(s, P, J, n_rows, false, st, sync);
    zero_cut_rows(O, s, static_cast<int64_t>(K) * L, n_rows, S);
    sync();
    opsa_rows_gathered<T, KC, WEIGHTED>(O, A, B, W, PW, P, s, K, L, n_rows, S, stage[threadIdx.x >> 5], st);
}

// Positions per segment: one segment and part per warp, within bounds (32 entries are fetched at a time;
// 512 so that the warps of a large problem end together).
inline int segment_length(int64_t J, int parts, int blocks) {
    const int64_t warps = static_cast<int64_t>(blocks) * (kSortThreads / 32);
    const int64_t S = ceil_div(ceil_div(J * parts, warps), 32) * 32;
    return static_cast<int>(std::min<int64_t>(std::max<int64_t>(S, 32), 512));
}

template <typename T, bool WEIGHTED>
void launch_fwd_unsorted(const Call& call, T* O, const T* A, const T* B, const T* W, const int32_t* PW,
                         const int32_t* P, int64_t J, int K, int L, int64_t n_rows) {
    const int blocks = sort_blocks(call, J, n_rows * K * L);
    void* scratch = scratch_alloc(call, entry_sort_bytes(J, n_rows, blocks));
    const EntrySort s = entry_sort_at(scratch, n_rows, blocks);
#define MOPS_B200_LAUNCH(KC_)                                                                      \
    launch_sorting(call, blocks, opsa_fwd_unsorted_grid<T, KC_, WEIGHTED>,                         \
                   opsa_fwd_unsorted_block<T, KC_, WEIGHTED>, O, A, B, W, PW, P, s, J, K, L,       \
                   n_rows, segment_length(J, static_cast<int>(ceil_div(K, KC_) * ceil_div(L, 32)), blocks), \
                   call.status);
    if (K <= 4) {
        MOPS_B200_LAUNCH(4)
    } else {
        MOPS_B200_LAUNCH(8)
    }
#undef MOPS_B200_LAUNCH
    scratch_free(call, scratch);
}

} // namespace
} // namespace mops_b200

#endif
