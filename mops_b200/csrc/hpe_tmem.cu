// Homogeneous polynomial evaluation with the batch rows in tensor memory (gather_tmem.cuh): forward
// and VJP for operands of up to about 200 (f64) / 250 (f32) columns and any batch size.
//
// 2^20 rows, 100 columns, 2000 monomials of order 4, f64, against the kernels that gather from
// shared memory (hpe.cu), which its pipe bounds: forward and VJP 9.16 -> 3.95 ms together (instruction issue;
// about 20 instructions per record of the VJP and two rows). 1000 rows: forward 20 -> 12 us, VJP 115 -> 17 us.
#include "checks.hpp"
#include "gather_tmem.cuh"
#include "hpe_tmem.hpp"

namespace mops_b200 {
namespace {

__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;\n" ::: "memory");
}
__device__ __forceinline__ unsigned cluster_address(const void* p, unsigned rank) {
    unsigned a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(a) : "r"(smem_address(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ double load_cluster(unsigned a, double) {
    double v;
    asm volatile("ld.shared::cluster.f64 %0, [%1];\n" : "=d"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ float load_cluster(unsigned a, float) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];\n" : "=f"(v) : "r"(a) : "memory");
    return v;
}

// ---------------------------------------------------------------- forward
// A cluster of `parts` blocks (1, 2, 4 or 8) shares a tile: each takes a contiguous part of the
// monomials, and rank 0 adds the partial sums up through distributed shared memory. Inside a block
// the four warps of a quadrant hold the same rows and take batches in turn. The monomials are
// packed into records on the fly, stage by stage, so that no table has to be built before.
template <typename T, int K, int W>
__global__ void __launch_bounds__(kTmemThreads, 1)
hpe_fwd_tmem(T* __restrict__ O, const __grid_constant__ Operands operands, const T* __restrict__ C,
             const int32_t* __restrict__ P, int64_t I, int J, int parts, int64_t tiles, Status st) {
    const int N = operands.total;
    using G = Batch<T, K, W>;
    constexpr int B = G::B, R = G::R, RB = G::RB;
    constexpr int kStage = kStageBytes / RB < kTmemThreads ? kStageBytes / RB : kTmemThreads;
    extern __shared__ __align__(16) unsigned char smem[];
    // layout: two stages of records (the partial sums reuse them) | slabs
    T* partial = reinterpret_cast<T*>(smem); // [groups][128 R]
    __shared__ uint32_t tmem_s;
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(kFullMask, tid >> 5, 0), group = warp >> 2;
    const int part = parts > 1 ? uniform(static_cast<int>(cluster_rank())) : 0;
    const int64_t first = blockIdx.x / parts, step = gridDim.x / parts;

    Tiles<T, W> t{operands, I, operands.template slab_bytes<T>(), smem + 2 * kStageBytes};
    t.start(first, tid);
    if (warp == 0) tmem_alloc(&tmem_s, kTmemColumns);

    const int j_lo = static_cast<int>(static_cast<int64_t>(J) * part / parts);
    const int j_hi = static_cast<int>(static_cast<int64_t>(J) * (part + 1) / parts);
    const int stages = (j_hi - j_lo + kStage - 1) / kStage;
    // the raw monomial this thread packs for the next stage
    T c_raw = T(0);
    int32_t p_raw[K];
    auto load_raw = [&](int stage) {
        const int j = j_lo + stage * kStage + tid;
        if (tid < kStage && j < j_hi) {
            c_raw = __ldg(C + j);
            if constexpr (K == 4) {
                if ((reinterpret_cast<size_t>(P) & 15) == 0) {
                    const int4 v = __ldg(reinterpret_cast<const int4*>(P) + j);
                    p_raw[0] = v.x, p_raw[1] = v.y, p_raw[2] = v.z, p_raw[3] = v.w;
                    return;
                }
            }
#pragma unroll
            for (int k = 0; k < K; k++) p_raw[k] = __ldg(P + static_cast<int64_t>(j) * K + k);
        }
    };
    auto pack = [&](int stage) { // every record of the stage, padding behind the monomials
        const int j = j_lo + stage * kStage + tid;
        if (tid < kStage) {
            uint32_t w[RB / 4];
#pragma unroll
            for (int q = 0; q < RB / 4; q++) w[q] = 0;
            const bool live = j < j_hi;
            bool bad = false;
#pragma unroll
            for (int k = 0; k < K; k++) {
                if (live) bad |= clamp_index(p_raw[k], N);
                const uint32_t column = static_cast<uint32_t>((live ? p_raw[k] : N) * W);
                w[words_of(sizeof(T)) + k / 2] |= column << (k & 1 ? 16 : 0);
            }
            if (bad) report_bad_index(st, 0);
            put_coefficient<T>(w, live ? c_raw : T(0));
            uint4* dst = reinterpret_cast<uint4*>(smem + (stage & 1) * kStageBytes + tid * RB);
#pragma unroll
            for (int q = 0; q < RB / 16; q++)
                dst[q] = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
        }
    };

    tmem_fence_before_sync();
    __syncthreads();
    tmem_fence_after_sync();
    const uint32_t base = tmem_quadrant(tmem_s, warp);
    t.ones(base, warp);
    load_raw(0);

    for (int64_t tile = first; tile < tiles; tile += step) {
        t.load(tile + step < tiles ? tile + step : -1, base, tid, warp, lane);
        T acc[R];
        PieceSum<T, R> sum;
        sum.clear();
#pragma unroll
        for (int r = 0; r < R; r++) acc[r] = T(0);
        for (int s = 0; s < stages; s++) {
            pack(s);
            __syncthreads();
            load_raw(s + 1 < stages ? s + 1 : 0); // after the last stage: stage 0 of the next tile
            const int left = j_hi - j_lo - s * kStage;
            const int mc = left < kStage ? left : kStage;
            const unsigned char* recs = smem + (s & 1) * kStageBytes;
            // batch i of this group is batch 4 i + group of the stage
            constexpr int kBatches = kStage / (B * kTmemGroups); // a power of two
            const int nb = (mc + B * kTmemGroups - 1) / (B * kTmemGroups);
            auto at = [&](int i) {
                return recs + ((i & (kBatches - 1)) * kTmemGroups + group) * (B * RB);
            };
            G x, y;
            Records<T, K, W> rx, ry;
            fetch<T, K, W>(rx, at(0));
            issue<T, K, W>(x, rx, base);
            fetch<T, K, W>(ry, at(1));
            for (int i = 0; i < nb; i += 2) { // (kBatches is even: batch nb may be all padding)
                await<T, K, W>(x);
                issue<T, K, W>(y, ry, base);
                add_terms<T, K, W>(x, rx, acc);
                const unsigned char* ahead = at(i + 2); // (batch i + 3 comes next: kBatches is even)
                fetch<T, K, W>(rx, ahead);
                await<T, K, W>(y);
                issue<T, K, W>(x, rx, base);
                add_terms<T, K, W>(y, ry, acc);
                sum.template piece<B>(i, acc);
                fetch<T, K, W>(ry, ahead + kTmemGroups * (B * RB));
            }
            await<T, K, W>(x); // the loads started last are not used
        }
        sum.finish(acc);
        __syncthreads(); // the stages become the partial sums
        const int own = (warp & 3) * 32 + lane;
#pragma unroll
        for (int r = 0; r < R; r++) partial[group * (kSlabRows * R) + r * kSlabRows + own] = acc[r];
        if (parts > 1)
            cluster_sync();
        else
            __syncthreads();
        if (part == 0) {
            for (int row = tid; row < kSlabRows * R; row += kTmemThreads) {
                const int64_t i = tile * (kSlabRows * R) + row;
                T sum = T(0);
                for (int p = 0; p < parts; p++)
#pragma unroll
                    for (int g = 0; g < kTmemGroups; g++) {
                        const T* src = partial + g * (kSlabRows * R) + row;
                        sum += p == 0 ? *src : load_cluster(cluster_address(src, p), T(0));
                    }
                if (i < I) O[i] = sum;
            }
        }
        if (parts > 1)
            cluster_sync();
        else
            __syncthreads();
    }
    cp_async_wait<0>();
    tmem_fence_before_sync();
    __syncthreads();
    tmem_fence_after_sync();
    if (warp == 0) tmem_free(tmem_s, kTmemColumns);
}

// ---------------------------------------------------------------- VJP
// One record per incidence (j, k): C[j] and the other K - 1 columns of monomial j, for result
// column P[j, k].
template <typename T, int K> struct HpeIncidences {
    const T* C;
    const int32_t* P;
    int N;
    __device__ int key(int x, unsigned& bad) const {
        int32_t p = __ldg(P + x);
        if (clamp_index(p, N)) bad |= 1u;
        return p;
    }
    __device__ T coefficient(int x) const { return __ldg(C + x / K); }
    __device__ int column(int x, int q) const {
        const int j = x / K, k = x - j * K;
        int32_t p = __ldg(P + j * K + q + (q >= k ? 1 : 0));
        clamp_index(p, N);
        return p;
    }
};

// Fewer than five gathers per column of a large batch: the kernels in hpe.cu are as fast (measured
// at N = 100, K = 4: the lines cross at about 100 monomials in the forward, 120 in the VJP).
bool few_terms(const Call& call, int64_t I, int N, int64_t gathers) {
    return fills_gpu(call, I) && gathers < 5 * static_cast<int64_t>(N);
}

// Very few result columns: one warp group walks all records of a column, where the kernels in hpe.cu
// split them among the lanes of a warp (batches of up to 8192 rows) or the warps of a block. In products
// per column: 4800 monomials of order 4 in one variable, 27 rows, take 170 us there and 359 here. The
// lines cross at about 1200 (25 000 for one column and a batch that fills the GPU); from eight columns
// on, and for batches between, they do not.
bool few_columns(const Call& call, int64_t I, int N, int64_t products) {
    if (fills_gpu(call, I)) return N == 1 && products > 25000;
    return I <= 8192 && N < 8 && products > 1200 * static_cast<int64_t>(N);
}

template <typename T, int K>
bool forward_order(const Call& call, T* O, const T* A, const T* C, const int32_t* P, int64_t I, int N,
                   int64_t J) {
    if (few_terms(call, I, N, J * K)) return false;
    Operands op{};
    op.add(A, N);
    GatherShape s{};
    if (!choose_gather_shape<T>(call, I, op, static_cast<double>(J), K, 8, 8, true, 0.0, 2 * kStageBytes, s))
        return false;
    note_kernel_f("hpe_fwd_tmem<%s,K=%d,W=%d> parts=%d", scalar_name<T>(), K, s.w, s.parts);
    auto go = [&](auto kernel) {
        launch_gather(call, kernel, s, s.parts, O, op, C, P, I, static_cast<int>(J), s.parts, s.tiles,
                      call.status);
    };
    if (s.w == 8) {
        if constexpr (K * 8 <= 32) go(hpe_fwd_tmem<T, K, 8>);
    } else if (s.w == 4) {
        go(hpe_fwd_tmem<T, K, 4>);
    } else {
        go(hpe_fwd_tmem<T, K, 2>);
    }
    return true;
}

template <typename T, int K>
bool backward_order(const Call& call, T* gA, const T* gO, const T* A, const T* C, const int32_t* P,
                    int64_t I, int N, int64_t J) {
    if (few_terms(call, I, N, J * K) || few_columns(call, I, N, J * K * (K - 1))) return false;
    Operands op{};
    op.add(A, N);
    Results<T> results{};
    results.add(gA, N);
    results.scale = gO;
    TableKey key{};
    key.kind = kHpeTable;
    key.ptr[0] = C, key.ptr[1] = P;
    key.n[0] = J, key.n[1] = K, key.n[2] = N, key.n[3] = 2;
    return run_gather<T, K - 1>(call, key, HpeIncidences<T, K>{C, P, N}, J * K, op, results, I, "hpe_vjp_tmem");
}

} // namespace

template <typename T>
bool hpe_forward_tmem(const Call& call, T* O, const T* A, const T* C, const int32_t* P, int64_t I, int N,
                      int64_t J, int K) {
    switch (K) {
#define CASE(KK) case KK: return forward_order<T, KK>(call, O, A, C, P, I, N, J);
        CASE(1) CASE(2) CASE(3) CASE(4) CASE(5) CASE(6) CASE(7) CASE(8) CASE(9) CASE(10)
#undef CASE
    default: return false;
    }
}

template <typename T>
bool hpe_backward_tmem(const Call& call, T* gA, const T* gO, const T* A, const T* C, const int32_t* P,
                       int64_t I, int N, int64_t J, int K) {
    switch (K) {
#define CASE(KK) case KK: return backward_order<T, KK>(call, gA, gO, A, C, P, I, N, J);
        CASE(2) CASE(3) CASE(4) CASE(5) CASE(6) CASE(7) CASE(8) CASE(9) CASE(10)
#undef CASE
    default: return false;
    }
}

#define INSTANTIATE(T)                                                                             \
    template bool hpe_forward_tmem<T>(const Call&, T*, const T*, const T*, const int32_t*, int64_t, \
                                      int, int64_t, int);                                          \
    template bool hpe_backward_tmem<T>(const Call&, T*, const T*, const T*, const T*,             \
                                       const int32_t*, int64_t, int, int64_t, int);
INSTANTIATE(float)
INSTANTIATE(double)

} // namespace mops_b200
