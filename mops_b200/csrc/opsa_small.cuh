// OPSA / OPSAW on a few thousand entries: one launch, no table.
//
// The streaming kernels need the segment table of the scatter index (a launch), and behind them, where
// nobody knows the order of the index yet, the kernels for an unsorted one (two more). For a few
// thousand entries the launches are most of the time. Here every block reads the whole index into
// shared memory and sees for itself whether it is sorted; the VJP does not care about the order.
// 420 entries, 13 x 20, f32: a forward through autograd 17 -> 8 us, the VJP kernel 10 -> 4 us.
#ifndef MOPS_B200_OPSA_SMALL_CUH
#define MOPS_B200_OPSA_SMALL_CUH

#include <type_traits>

#include "unsorted.cuh"

namespace mops_b200 {
namespace {

constexpr int kSmallEntries = 4096; // 16 KB of index per block
constexpr int kSmallWarps = 4;

// Products and sums of the weighted operation are f64 at any number of entries, as in the streaming
// kernels (opsa_pipe.cuh): the precision of a model must not depend on the size of its batch.
template <typename T, bool WEIGHTED> using SmallSum = std::conditional_t<WEIGHTED, double, T>;

// Forward: a block per output row and 8 by 32 part of it. Its warps share the row's entries (or, where the
// index is not sorted, the search for them), eight or more each, and add their sums up in shared
// memory: one row with all of 2000 entries of 8 x 20, f64, took one warp 175 us (with three
// launches 72).
template <typename T, bool WEIGHTED>
__global__ void __launch_bounds__(kSmallWarps * 32)
opsa_fwd_small(T* __restrict__ O, const T* __restrict__ A, const T* __restrict__ B, const T* __restrict__ W,
               const int32_t* __restrict__ PW, const int32_t* __restrict__ P, int J, int K, int L, int n_rows,
               Status st) {
    using S = SmallSum<T, WEIGHTED>;
    constexpr int KC = 8, U = 16; // (latency: more rows in flight than in unsorted.cuh)
    __shared__ int32_t index[kSmallEntries];
    __shared__ int32_t found[kSmallWarps][64];
    __shared__ __align__(16) T stage[kSmallWarps][U * KC];
    __shared__ S partial[kSmallWarps - 1][KC][32];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    bool bad = false, descent = false;
    for (int j = tid; j < J; j += kSmallWarps * 32) {
        const int32_t v = __ldg(P + j);
        index[j] = v;
        bad |= static_cast<uint32_t>(v) >= static_cast<uint32_t>(n_rows);
        descent |= j + 1 < J && __ldg(P + j + 1) < v;
    }
    if (bad && blockIdx.x == 0) report_bad_index(st, 0);
    const bool sorted = !__syncthreads_or(descent);
    auto lower_bound = [&](int r) { // first position whose row is >= r
        int lo = 0, hi = J;
        while (lo < hi) {
            const int mid = (lo + hi) / 2;
            if (index[mid] < r)
                lo = mid + 1;
            else
                hi = mid;
        }
        return lo;
    };
    const int k_units = (K + KC - 1) / KC, units = k_units * ((L + 31) / 32);
    const int64_t all = static_cast<int64_t>(n_rows) * units;
    for (int64_t unit = blockIdx.x; unit < all; unit += gridDim.x) {
        const int r = static_cast<int>(unit / units), part = static_cast<int>(unit - static_cast<int64_t>(r) * units);
        const int lb = part / k_units * 32, kb = part % k_units * KC;
        const int l = lb + lane, lc = l < L ? l : L - 1, kn = K - kb < KC ? K - kb : KC;
        const int row_lo = sorted ? lower_bound(r) : 0, row_hi = sorted ? lower_bound(r + 1) : J;
        const int share = ((row_hi - row_lo + kSmallWarps - 1) / kSmallWarps + 7) / 8 * 8;
        const int lo = row_lo + warp * share, hi = lo + share < row_hi ? lo + share : row_hi;
        S acc[KC];
#pragma unroll
        for (int k = 0; k < KC; k++) acc[k] = S(0);
        int held = 0; // entries of this row found and not yet added
        auto add = [&](int count) {
            const int e = found[warp][lane < count ? lane : 0];
            int w = 0;
            if (WEIGHTED) {
                w = __ldg(PW + e);
                if (clamp_index(w, n_rows)) report_bad_index(st, 1);
            }
            for (int u0 = 0; u0 < count; u0 += U) {
                S b[U];
                load_entries<T, KC, WEIGHTED, U, S>(b, e, w, u0, count, A, B, W, K, L, kb, kn, lc, stage[warp], lane);
#pragma unroll
                for (int u = 0; u < U; u++) add_entry<T, KC, S>(acc, stage[warp] + u * KC, b[u]);
                __syncwarp();
            }
        };
        for (int p0 = lo; p0 < hi; p0 += 32) {
            const int p = p0 + lane;
            const bool mine = p < hi && index[p] == r;
            const unsigned who = __ballot_sync(kFullMask, mine);
            if (mine) found[warp][held + __popc(who & ((1u << lane) - 1))] = p;
            held += __popc(who);
            __syncwarp();
            if (held >= 32) {
                add(32);
                const int rest = found[warp][32 + lane];
                __syncwarp();
                found[warp][lane] = rest;
                held -= 32;
                __syncwarp();
            }
        }
        if (held > 0) add(held);
        __syncwarp();
        if (row_hi - row_lo > share) { // (the same for the whole block)
            if (warp > 0) {
#pragma unroll
                for (int k = 0; k < KC; k++) partial[warp - 1][k][lane] = acc[k];
            }
            __syncthreads();
            if (warp == 0) {
#pragma unroll
                for (int w = 0; w < kSmallWarps - 1; w++)
#pragma unroll
                    for (int k = 0; k < KC; k++) acc[k] += partial[w][k][lane];
            }
            __syncthreads(); // (the next unit writes there again)
        }
        if (warp == 0 && l < L) {
#pragma unroll
            for (int k = 0; k < KC; k++)
                if (k < kn) O[(static_cast<int64_t>(r) * K + kb + k) * L + l] = static_cast<T>(acc[k]);
        }
    }
}

// VJP, K <= 16: a warp per entry, lane = column l. gO[row, :, l] in K loads per lane; grad_B is a sum
// in the lane, grad_A one over the lanes (16 values in 16 exchanges).
template <typename T, bool WEIGHTED>
__global__ void __launch_bounds__(kSmallWarps * 32)
opsa_vjp_small(T* __restrict__ gA, T* __restrict__ gB, T* __restrict__ gW, const T* __restrict__ gO,
               const T* __restrict__ A, const T* __restrict__ B, const T* __restrict__ W,
               const int32_t* __restrict__ PW, const int32_t* __restrict__ P, int J, int K, int L, int n_rows,
               Status st) {
    constexpr int KP = 16;
    const int lane = threadIdx.x & 31;
    const int64_t e = static_cast<int64_t>(blockIdx.x) * kSmallWarps + (threadIdx.x >> 5);
    if (e >= J) return;
    int32_t row = __ldg(P + e), w_row = 0;
    if (clamp_index(row, n_rows) && lane == 0) report_bad_index(st, 0);
    if (WEIGHTED) {
        w_row = __ldg(PW + e);
        if (clamp_index(w_row, n_rows) && lane == 0) report_bad_index(st, 1);
    }
    using S = SmallSum<T, WEIGHTED>;
    S a[KP], ga[KP];
#pragma unroll
    for (int k = 0; k < KP; k++) {
        a[k] = k < K ? __ldg(A + e * K + k) : T(0);
        ga[k] = S(0);
    }
    for (int l = lane; l < L; l += 32) {
        const T* g = gO + static_cast<int64_t>(row) * K * L + l;
        S v[KP];
#pragma unroll
        for (int k = 0; k < KP; k++) v[k] = k < K ? __ldg(g + k * L) : T(0);
        const S b = __ldg(B + e * L + l);
        const S w = WEIGHTED ? __ldg(W + static_cast<int64_t>(w_row) * L + l) : T(1);
        const S bw = WEIGHTED ? b * w : b;
        S s = S(0);
#pragma unroll
        for (int k = 0; k < KP; k++) {
            s += v[k] * a[k];
            ga[k] += v[k] * bw;
        }
        if (gB != nullptr) gB[e * L + l] = static_cast<T>(WEIGHTED ? s * w : s);
        if (WEIGHTED && gW != nullptr) red_add(gW + static_cast<int64_t>(w_row) * L + l, static_cast<T>(s * b));
    }
    if (gA == nullptr) return;
    int which = 0;
#pragma unroll
    for (int level = 0; level < 4; level++) { // hand over half of the values, keep the sums of the other half
        const int o = 16 >> level, h = KP / 2 >> level;
        const bool upper = lane & o;
#pragma unroll
        for (int i = 0; i < KP / 2; i++) {
            if (i < h) {
                const S send = upper ? ga[i] : ga[i + h], keep = upper ? ga[i + h] : ga[i];
                ga[i] = keep + __shfl_xor_sync(kFullMask, send, o);
            }
        }
        which += upper ? h : 0;
    }
    const S sum = ga[0] + __shfl_xor_sync(kFullMask, ga[0], 1);
    if ((lane & 1) == 0 && which < K) gA[e * K + which] = static_cast<T>(sum);
}

// Few enough entries that three launches cost more than one slower kernel (one block per row, one round
// trip to memory per 16 entries and warp), rows not long; with a plan there is one launch anyway.
inline bool small_forward(int64_t J, int64_t n_rows, bool weighted) {
    return J <= (weighted ? 512 : 2048) && n_rows <= 4096 && J <= 64 * n_rows && plan_bound() == nullptr;
}

} // namespace
} // namespace mops_b200

#endif
