// Device-side helpers shared by the kernels: status reporting, the segment search over a
// sorted scatter index, the sortedness check, and reductions.
//
// Replaces mops/src/internal/cuda_utils.{cuh,cu} (atomic add with a pre-sm_60 fallback, the
// shared-memory bump allocator) and mops/src/internal/cuda_first_occurences.cu (a memset + a
// kernel + a device synchronisation that write a first/last-occurrence table into a cached,
// process-wide global buffer before every scatter op). Here `segment_offsets` writes the
// table of segment starts in one launch on the call's stream (no memset, no synchronisation,
// call-scoped or plan-owned memory) and checks order and range in the same pass; the
// warp-wide search (`warp_segment`) serves the kernels that work without a table.
#ifndef MOPS_B200_DEVICE_CUH
#define MOPS_B200_DEVICE_CUH

#include <algorithm>
#include <cstdint>

#include "runtime.hpp"

namespace mops_b200 {

constexpr unsigned kFullMask = 0xffffffffu;

__device__ __forceinline__ void report_unsorted(const Status& st) {
    // only the first of many reporters goes to host memory
    if (atomicExch(st.dev + kUnsortedEpoch, st.epoch) == st.epoch) return;
    st.host[kUnsortedEpoch] = st.epoch;
    __threadfence_system();
}

__device__ __forceinline__ void report_bad_index(const Status& st, int which) {
    st.dev[kBadIndex0 + which] = st.epoch;
    st.host[kBadIndex0 + which] = st.epoch;
    __threadfence_system();
}

__device__ __forceinline__ bool saw_unsorted(const Status& st) {
    return *reinterpret_cast<volatile uint32_t*>(st.dev + kUnsortedEpoch) == st.epoch;
}

// Clamp an index read from a user array into [0, n) so that a bad value can never address
// memory outside the operand; returns whether it had to.
__device__ __forceinline__ bool clamp_index(int32_t& v, int32_t n) {
    bool bad = static_cast<uint32_t>(v) >= static_cast<uint32_t>(n);
    if (bad) v = 0;
    return bad;
}

// First position in the ascending array P[lo, hi) whose value is >= r, found by the whole
// warp: every round the 32 lanes probe 32 evenly spaced positions and one ballot narrows
// the range 32-fold (five rounds for 2^24 entries, each a single coalescable load per lane).
// All lanes must call it with the same arguments; all get the result. On an unsorted array
// the result is some position in [lo, hi]; callers detect that case separately.
__device__ __forceinline__ int64_t warp_lower_bound(const int32_t* __restrict__ P, int64_t lo,
                                                    int64_t hi, int32_t r, int lane) {
    while (hi > lo) {
        int64_t n = hi - lo;
        int64_t chunk = (n + 31) / 32; // >= 1
        int64_t probe = lo + (lane + 1) * chunk - 1;
        bool below = (probe < hi) && (__ldg(P + probe) < r);
        int c = __popc(__ballot_sync(kFullMask, below));
        int64_t new_lo = lo + c * chunk;
        if (new_lo >= hi) {
            lo = hi;
            break;
        }
        // The answer is in [new_lo, new_lo + chunk - 1]: position new_lo + chunk - 1 was
        // probed and is >= r (or lies at/after hi).
        int64_t new_hi = new_lo + chunk - 1;
        if (new_hi > hi) new_hi = hi;
        lo = new_lo;
        hi = new_hi;
    }
    return lo;
}

// Number of i in [0, n) with t[i] + row_weight * i <= x, for an ascending table t, found by
// the whole warp with 32-way probes (as warp_lower_bound). All lanes call it with the same
// arguments.
template <typename Off>
__device__ __forceinline__ int64_t warp_count_weighted_le(const Off* __restrict__ t, int64_t n,
                                                          int64_t row_weight, int64_t x, int lane) {
    int64_t lo = 0, hi = n;
    while (hi > lo) {
        const int64_t len = hi - lo;
        const int64_t chunk = (len + 31) / 32; // >= 1
        const int64_t probe = lo + (lane + 1) * chunk - 1;
        const bool le = (probe < hi) && (t[probe] + row_weight * probe <= x);
        const int c = __popc(__ballot_sync(kFullMask, le));
        const int64_t new_lo = lo + c * chunk;
        if (new_lo >= hi) {
            lo = hi;
            break;
        }
        int64_t new_hi = new_lo + chunk - 1;
        if (new_hi > hi) new_hi = hi;
        lo = new_lo;
        hi = new_hi;
    }
    return lo;
}

// Splits the rows of a segment table among `parts` workers so that every worker gets whole
// rows and about the same amount of work, counted as entries + kRowWeight per row: not the
// same number of rows (the rows of a shard of a larger problem, or of an uneven graph, can be
// mostly empty), and not entries alone either (a long run of empty rows still has to be
// written). offsets[0 .. n_rows] ascending, offsets[n_rows] = number of entries. Returns the
// first row of worker `part`, who owns rows [split(part), split(part + 1)). All lanes of a
// warp call it together.
constexpr int64_t kRowWeight = 4;
template <typename Off>
__device__ __forceinline__ int64_t balanced_row_split(const Off* __restrict__ offsets,
                                                      int64_t n_rows, int64_t part, int64_t parts,
                                                      int lane) {
    if (part <= 0) return 0;
    if (part >= parts) return n_rows;
    const int64_t total = offsets[n_rows] + kRowWeight * n_rows;
    const int64_t target = total / parts * part + total % parts * part / parts;
    // the last row whose weighted start is <= target
    const int64_t r = warp_count_weighted_le(offsets, n_rows + 1, kRowWeight, target, lane) - 1;
    return r < 0 ? 0 : (r > n_rows ? n_rows : r);
}

// Bounds [begin, end) of the entries whose (sorted) index equals r.
__device__ __forceinline__ void warp_segment(const int32_t* __restrict__ P, int64_t J, int32_t r,
                                             int lane, int64_t& begin, int64_t& end) {
    begin = warp_lower_bound(P, 0, J, r, lane);
    // Segments are short in practice: look in a window after `begin` first.
    int64_t stop = begin + 1024 < J ? begin + 1024 : J;
    end = warp_lower_bound(P, begin, stop, r + 1, lane);
    if (end == stop && stop < J) end = warp_lower_bound(P, stop, J, r + 1, lane);
}

// Every warp of a grid checks one slice of the scatter index for ascending order and for
// range; together the slices cover all adjacent pairs, so "no report" proves the index is
// sorted and inside [0, n_rows). `part` in [0, n_parts).
__device__ __forceinline__ void check_sorted_slice(const int32_t* __restrict__ P, int64_t J,
                                                   int64_t n_rows, int64_t part, int64_t n_parts,
                                                   int lane, const Status& st) {
    if (J == 0) return;
    int64_t per = (J + n_parts - 1) / n_parts;
    int64_t a = part * per;
    int64_t b = a + per < J ? a + per : J;
    bool unsorted = false, bad = false;
    for (int64_t j = a + lane; j < b; j += 32) {
        int32_t v = __ldg(P + j);
        int32_t next = (j + 1 < J) ? __ldg(P + j + 1) : v;
        unsorted |= next < v;
        bad |= (v < 0) || (static_cast<int64_t>(v) >= n_rows);
    }
    if (__any_sync(kFullMask, unsorted) && lane == 0) report_unsorted(st);
    // Bit 0 is the scatter index of every scatter op.
    if (__any_sync(kFullMask, bad) && lane == 0) report_bad_index(st, 0);
}

template <typename T, int N> struct VecOf;
template <> struct VecOf<float, 1> { using type = float; };
template <> struct VecOf<float, 2> { using type = float2; };
template <> struct VecOf<float, 4> { using type = float4; };
template <> struct VecOf<double, 1> { using type = double; };
template <> struct VecOf<double, 2> { using type = double2; };

template <typename T, int N> __device__ __forceinline__ void load_vec(const T* p, T (&out)[N]) {
    using V = typename VecOf<T, N>::type;
    union {
        V v;
        T s[N];
    } u;
    u.v = *reinterpret_cast<const V*>(p);
#pragma unroll
    for (int i = 0; i < N; i++) out[i] = u.s[i];
}

template <typename T, int N> __device__ __forceinline__ void store_vec(T* p, const T (&in)[N]) {
    using V = typename VecOf<T, N>::type;
    union {
        V v;
        T s[N];
    } u;
#pragma unroll
    for (int i = 0; i < N; i++) u.s[i] = in[i];
    *reinterpret_cast<V*>(p) = u.v;
}

template <typename T> __device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFullMask, v, o);
    return v;
}

// Fire-and-forget global accumulation (compiles to RED: no value comes back).
// Reductions without a return value (atomicAdd with an unused result can still be compiled
// to the returning form, which holds a register and a scoreboard until the L2 answers).
__device__ __forceinline__ void red_add(double* addr, double v) {
    asm volatile("red.global.add.f64 [%0], %1;\n" ::"l"(addr), "d"(v) : "memory");
}
__device__ __forceinline__ void red_add(float* addr, float v) {
    asm volatile("red.global.add.f32 [%0], %1;\n" ::"l"(addr), "f"(v) : "memory");
}

// Unsorted index: runs only when the segmented kernel of the same call reported it.
template <typename T>
__global__ void zero_if_unsorted(T* __restrict__ out, int64_t n, Status st) {
    if (!saw_unsorted(st)) return;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x)
        out[i] = T(0);
}


// ---------------------------------------------------------------- FP64 tensor-core MMA
// mma.sync m8n8k4, f64. Fragment layout (lane = 4*qr + qc): A[qr][qc], B[k = qc][n = qr],
// C[qr][2*qc + {0,1}].
__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}
// c = a b (no accumulator input)
__device__ __forceinline__ void dmma0(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%4,%4};\n"
                 : "=d"(c[0]), "=d"(c[1])
                 : "d"(a), "d"(b), "d"(0.0));
}

// ---------------------------------------------------------------- asynchronous staging
// Element-wise global -> shared copies that do not pass through registers (LDGSTS): a lane
// can put a whole chunk in flight and go on; completion is tracked per committed group.
template <int BYTES>
__device__ __forceinline__ void cp_async(void* smem_dst, const void* global_src) {
    const unsigned dst = static_cast<unsigned>(__cvta_generic_to_shared(smem_dst));
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(dst), "l"(global_src),
                 "n"(BYTES)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// ---------------------------------------------------------------- segment offsets
// offsets[r] = first position of the ascending index P whose value is >= r, for r in
// [0, n_rows]; offsets[n_rows] = J. Entry j starts every row in (P[j-1], P[j]]. The same pass checks
// order and range, so the kernels that consume the table can trust it, or skip their work when the
// index was not sorted (saw_unsorted). Long runs of empty rows are filled by the whole warp, one run after
// the other; runs of a few rows by each thread (65 000 entries of 197 000 rows: 16 us less).
// Replaces the reference's first-occurrence pass (memset + kernel + device synchronisation
// into a cached global buffer, mops/src/internal/cuda_first_occurences.cu:82-117).
//
// Bounded by the 4 bytes per entry: a thread takes eight entries with two 16-byte loads, a block 2048
// entries and no more (2^24 entries: 22 us, against 60 us with one entry per thread and iteration of
// a loop, whose latencies added up). A warp that sees a descent reports it and leaves its rows
// alone: their ranges would be random (1.1 ms for 300 000 entries).
// Few entries, or many empty rows, go one entry per thread: the runs of a warp are filled one after the
// other (500 entries of 100 000 rows: 61 -> 93 us with eight).
constexpr int kOwnRows = 16;        // a thread fills by itself; the warp joins in for longer runs
constexpr int64_t kWideEntries = 1 << 18; // from here on eight entries per thread
template <int Q>
static __global__ void __launch_bounds__(256)
segment_offsets(const int32_t* __restrict__ P, int64_t J, int64_t n_rows, int64_t* __restrict__ offsets,
                Status st) {
    const int lane = threadIdx.x & 31;
    const int64_t j0 = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) * Q;
    const int32_t beyond = static_cast<int32_t>(n_rows); // (n_rows fits 31 bits)
    // v[0] = P[j0 - 1], v[1 + q] = P[j0 + q]; -1 in front of the index, n_rows behind it
    int32_t v[Q + 1];
    if (Q % 4 == 0 && (reinterpret_cast<size_t>(P) & 15) == 0 && j0 + Q <= J) {
#pragma unroll
        for (int q = 0; q < Q; q += 4) {
            const int4 u = __ldg(reinterpret_cast<const int4*>(P + j0 + q));
            v[1 + q] = u.x;
            if constexpr (Q >= 4) v[2 + q] = u.y, v[3 + q] = u.z, v[4 + q] = u.w;
        }
    } else {
#pragma unroll
        for (int q = 0; q < Q; q++) v[1 + q] = j0 + q < J ? __ldg(P + j0 + q) : beyond;
    }
    int32_t edge = -1;
    if (lane == 0 && j0 > 0) edge = j0 - 1 < J ? __ldg(P + j0 - 1) : beyond;
    v[0] = __shfl_up_sync(kFullMask, v[Q], 1);
    if (lane == 0) v[0] = edge;
    bool bad = false, descent = false;
#pragma unroll
    for (int q = 0; q < Q; q++) {
        bad |= j0 + q < J && static_cast<uint32_t>(v[1 + q]) >= static_cast<uint32_t>(beyond);
        descent |= v[1 + q] < v[q];
    }
    if (__any_sync(kFullMask, bad) && lane == 0) report_bad_index(st, 0);
    if (__any_sync(kFullMask, descent)) {
        if (lane == 0 && !saw_unsorted(st)) report_unsorted(st);
        return;
    }
#pragma unroll
    for (int q = 0; q <= Q; q++) v[q] = min(max(v[q], -1), beyond);
#pragma unroll
    for (int q = 0; q < Q; q++) {
        const int32_t prev = v[q], cur = v[1 + q];
        // rows prev + 1 .. cur start at entry j0 + q
        // (64 bits: with 2^31 - 1 rows the sums leave 32)
        if (cur > prev) offsets[int64_t(prev) + 1] = j0 + q;
        if (!__any_sync(kFullMask, cur > int64_t(prev) + 1)) continue; // (no empty rows)
        const int64_t own = min(int64_t(prev) + kOwnRows, int64_t(cur));
        for (int64_t r = int64_t(prev) + 2; r <= own; r++) offsets[r] = j0 + q;
        unsigned wide = __ballot_sync(kFullMask, cur > own);
        while (wide) {
            const int src = __ffs(wide) - 1;
            wide &= wide - 1;
            const int64_t lo = int64_t(__shfl_sync(kFullMask, prev, src)) + kOwnRows + 1;
            const int64_t hi = __shfl_sync(kFullMask, cur, src);
            const int64_t at = __shfl_sync(kFullMask, j0, src) + q;
            for (int64_t r = lo + lane; r <= hi; r += 32) offsets[r] = at;
        }
    }
}

__host__ __device__ constexpr int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

// The segment table of a scatter index for one call: taken from the calling thread's plan when
// it has one for this index (then the index is known to be sorted and nothing is launched),
// else built on the call's stream into call-scoped (or, for a plan's first use, plan-owned)
// memory. release_table(call, t.ref) when the kernels that read it are enqueued.
struct SegmentTable {
    int64_t* offsets;
    TableRef ref;
    bool known_sorted; // no need to ask the device, no fallback kernels
};

inline SegmentTable segment_table(const Call& call, const int32_t* P, int64_t J, int64_t n_rows) {
    TableKey key{};
    key.kind = kSegmentTable;
    key.ptr[0] = P;
    key.n[0] = J;
    key.n[1] = n_rows;
    SegmentTable t;
    t.ref = acquire_table(call, key, static_cast<size_t>(n_rows + 1) * sizeof(int64_t));
    t.offsets = static_cast<int64_t*>(t.ref.ptr);
    if (t.ref.fresh) {
        if (J >= kWideEntries && n_rows <= 4 * J)
            segment_offsets<8><<<static_cast<unsigned>(ceil_div(J + 1, 256 * 8)), 256, 0, call.stream>>>(
                P, J, n_rows, t.offsets, call.status);
        else
            segment_offsets<1><<<static_cast<unsigned>(ceil_div(J + 1, 256)), 256, 0, call.stream>>>(
                P, J, n_rows, t.offsets, call.status);
        MOPS_CUDA_OK(cudaGetLastError());
        commit_table(call, t.ref);
    }
    t.known_sorted = t.ref.owned_by_plan && t.ref.sorted;
    return t;
}

} // namespace mops_b200

#endif
