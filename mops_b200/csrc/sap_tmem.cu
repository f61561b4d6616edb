// Sparse accumulation of products with the batch rows in tensor memory (gather_tmem.cuh): forward,
// VJP and second-order VJP. Every result column is a sum of records with two factors:
//
//   O[o]    : C A[PA] B[PB]                      (PO = o)
//   gA[a]   : C gO[PO] B[PB]                     (PA = a)     gB[b]  : C gO[PO] A[PA]   (PB = b)
//   ggO[o]  : C ggA[PA] B[PB] + C A[PA] ggB[PB]  (PO = o)
//   gA2[a]  : C gO[PO] ggB[PB]                   (PA = a)     gB2[b] : C gO[PO] ggA[PA] (PB = b)
//
// 2^22 rows, 20 x 6 -> 50, 1000 triplets, f64, against the kernels that gather from shared memory:
// forward 2.99 -> 1.19 ms, VJP 3.04 -> 1.68 ms (the second order by gather_sums). 1000 rows: forward 12 -> 9 us,
// VJP 39 -> 13 us, second order 109 -> 19 us.
#include "gather_tmem.cuh"
#include "sap_tmem.hpp"

namespace mops_b200 {
namespace {

enum Which { kA = 0, kB = 1, kO = 2 }; // the index arrays, in the order of the error message

// One family of records: for every triplet, result column result0 + P[key] and the operand columns
// column0[q] + P[factor[q]].
struct Family {
    int key, result0;
    int factor[2], column0[2];
};

template <typename T> struct SapSource {
    const T* C;
    const int32_t* P[3];
    int size[3];
    int K;
    Family family[4];

    __device__ int index(int which, int k, unsigned* bad) const {
        int32_t p = __ldg(P[which] + k);
        if (clamp_index(p, size[which]) && bad != nullptr) *bad |= 1u << which;
        return p;
    }
    __device__ int key(int x, unsigned& bad) const {
        const int f = x / K, k = x - f * K;
        if (f == 0) // every index array once
            for (int w = 0; w < 3; w++) index(w, k, &bad);
        return family[f].result0 + index(family[f].key, k, nullptr);
    }
    __device__ T coefficient(int x) const { return __ldg(C + x % K); }
    __device__ int column(int x, int q) const {
        const int f = x / K, k = x - f * K;
        return family[f].column0[q] + index(family[f].factor[q], k, nullptr);
    }
};

// Large batches: fewer triplets per column than this and the kernels of sap.cu are as fast. Measured over
// drawn widths, 20 000 to 4 10^6 rows, against them: forward, f64 from one triplet per column on 1.0 to 4 times
// as fast (f32 0.75 to 1.25 at one, 1.2 to 1.5 from one and a half on); VJP from three on 1.1 to 1.7 times where
// rows are whole 16-byte pieces, else 0.88 to 0.98 at three to five (their copies are 4 or 8 bytes each).
template <typename T> bool few_forward_triplets(const SapProblem<T>& p) {
    return 2 * p.K < (sizeof(T) == 8 ? 2 : 3) * static_cast<int64_t>(p.nA + p.nB + p.nO);
}
template <typename T> bool few_backward_triplets(const SapProblem<T>& p) {
    const bool pieces = (p.nA | p.nB | p.nO) * static_cast<int>(sizeof(T)) % 16 == 0;
    return p.K < (pieces ? 3 : 5) * static_cast<int64_t>(p.nA + p.nB + p.nO);
}

// And so are they for narrow operands with few triplets, whatever the triplets per column: a tile's way in and
// out costs the same then, while their tables are small. Measured on 165 shapes (widths 1 to 32 and 1 to 16, 2 to
// 100 results, 20 to 3000 triplets, 25 000 to 800 000 rows) that the lines above leave to these kernels: sap.cu's
// take 0.54 to 1.27 times as long in the forward on their side of this line (one shape 1.55), 0.47 to 1.16 for both
// gradients, 0.59 to 1.27 for one; on the other side 0.83, 0.92 and 0.78 at least, mostly more than 1. 4 x 4 -> 8,
// 40 triplets, 800 000 rows, f64, forward: 72 against 111 us; both gradients, 120 triplets: 94 against 130. With
// both operands wider than 16 columns sap.cu has no register kernels.
template <typename T> bool narrow_forward(const SapProblem<T>& p) {
    const int64_t cells = static_cast<int64_t>(p.nA) * p.nB;
    if (std::min(p.nA, p.nB) > 16) return false;
    return sizeof(T) == 8 ? 2 * p.K + cells + 16 * static_cast<int64_t>(p.nO) < 384 : p.K + cells + 8 * static_cast<int64_t>(p.nO) < 300;
}
template <typename T> bool narrow_backward(const SapProblem<T>& p, bool both) {
    const int64_t cells = static_cast<int64_t>(p.nA) * p.nB, columns = static_cast<int64_t>(p.nA) + p.nB + p.nO;
    if (std::min(p.nA, p.nB) > 16) return false;
    if (both) return sizeof(T) == 8 ? p.K + 6 * columns < 324 : p.K + 2 * cells + 6 * columns < 543;
    return sizeof(T) == 8 ? p.K + 6 * cells + 8 * columns < 454 : p.K + 8 * cells + 3 * columns < 590;
}

template <typename T, bool PRODUCTS = false>
bool run(const Call& call, const SapProblem<T>& p, const Family* families, int count, const Operands& op,
         const Results<T>& results, int level, const char* name) {
    SapSource<T> source{p.C, {p.PA, p.PB, p.PO}, {p.nA, p.nB, p.nO}, static_cast<int>(p.K), {}};
    for (int f = 0; f < count; f++) source.family[f] = families[f];
    TableKey key{};
    key.kind = kSapTable;
    key.ptr[0] = p.C, key.ptr[1] = p.PA, key.ptr[2] = p.PB, key.ptr[3] = p.PO;
    key.n[0] = p.K, key.n[1] = p.nA, key.n[2] = p.nB, key.n[3] = p.nO;
    key.n[4] = level, key.n[5] = 1;
    if (p.K * count > (1 << 20)) return false;
    return run_gather<T, 2, PRODUCTS>(call, key, source, p.K * count, op, results, p.I, name);
}

// ---------------------------------------------------------------- large batches
// Two kernels for batches that give every SM a tile. The triplets' records stay in shared memory for all
// tiles of a block, and results are collected there, to leave as one bulk copy per tile: the ring, its
// meetings and the stores of single sectors of the kernels of gather_tmem.cuh cost half of the time of
// 1000 triplets (2^22 rows, 20 x 6 -> 50, f64: 25 700 clocks per 256 rows in the forward, 11 600 of them
// whatever the number of triplets; VJP 42 600 and 24 000). Now 20 700 and 11 500, VJP 29 000 and 20 000: forward
// 1.51 -> 1.19 ms, VJP 2.48 -> 1.68 ms. What bounds them is instruction issue (63 %), then latency with four
// warps per scheduler: a record takes 7.3 instructions (9.5 clocks) for two rows, 4 clocks of them FP64.

// Records in batches of four, coefficients and 16-bit TMEM columns apart.
constexpr int kLot = 4;
template <typename T, int NF, int W> struct Lot {
    uint32_t v[kLot][NF][W];
};
template <typename T, int W> constexpr int kLaneRows = W / words_of(sizeof(T));
template <typename T, int NF> struct LotRecords {
    T c[kLot];
    uint32_t q[kLot * NF / 2];
};

template <typename T, int NF> struct ResidentRecords {
    T* c;
    uint16_t* q;
    static __host__ __device__ size_t bytes(int capacity) { return static_cast<size_t>(capacity) * (sizeof(T) + 2 * NF); }

    __device__ ResidentRecords(unsigned char* smem, int capacity)
        : c(reinterpret_cast<T*>(smem)), q(reinterpret_cast<uint16_t*>(smem + capacity * sizeof(T))) {}
    // Once per block: `count` records as the table builder wrote them; zeros (column 0) behind them, which
    // are fetched ahead but not used.
    __device__ void load(const unsigned char* records, int count, int capacity, int tid) {
        static_assert(tmem_record_bytes(sizeof(T), NF) == 16, "one 16-byte piece per record");
        for (int x = tid; x < capacity; x += kTmemThreads) {
            uint4 v = make_uint4(0u, 0u, 0u, 0u);
            if (x < count) v = __ldg(reinterpret_cast<const uint4*>(records) + x);
            uint32_t columns;
            if constexpr (sizeof(T) == 8) {
                c[x] = __hiloint2double(static_cast<int>(v.y), static_cast<int>(v.x));
                columns = v.z;
            } else {
                c[x] = __uint_as_float(v.x);
                columns = v.y;
            }
#pragma unroll
            for (int k = 0; k < NF; k++) q[x * NF + k] = static_cast<uint16_t>(columns >> (16 * k));
        }
    }
    __device__ __forceinline__ void fetch(LotRecords<T, NF>& r, int lot) const {
        constexpr int V = 16 / sizeof(T);
#pragma unroll
        for (int i = 0; i < kLot; i += V) {
            T v[V];
            load_vec<T, V>(c + lot * kLot + i, v);
#pragma unroll
            for (int j = 0; j < V; j++) r.c[i + j] = v[j];
        }
        const uint2* src = reinterpret_cast<const uint2*>(q + lot * (kLot * NF));
#pragma unroll
        for (int i = 0; i < NF; i++) {
            const uint2 u = src[i];
            r.q[2 * i] = u.x, r.q[2 * i + 1] = u.y;
        }
    }
};

template <typename T, int NF, int W>
__device__ __forceinline__ void issue(Lot<T, NF, W>& g, const LotRecords<T, NF>& r, uint32_t base) {
#pragma unroll
    for (int b = 0; b < kLot; b++)
#pragma unroll
        for (int k = 0; k < NF; k++) {
            const int i = b * NF + k;
            tmem_load(__byte_perm(r.q[i / 2], base, (i & 1) ? 0x7632 : 0x7610), g.v[b][k]);
        }
}
template <typename T, int NF, int W> __device__ __forceinline__ void await(Lot<T, NF, W>& g) {
    tmem_wait_load();
#pragma unroll
    for (int b = 0; b < kLot; b++)
#pragma unroll
        for (int k = 0; k < NF; k++) tmem_pin(g.v[b][k]);
}
// CHAINS = 2: two chains of sums, even and odd records of the batches.
template <int CHAINS, typename T, int NF, int W>
__device__ __forceinline__ void add_terms(const Lot<T, NF, W>& g, const LotRecords<T, NF>& rec,
                                          T (&acc)[2][kLaneRows<T, W>]) {
#pragma unroll
    for (int b = 0; b < kLot; b++)
#pragma unroll
        for (int r = 0; r < kLaneRows<T, W>; r++) {
            T p = rec.c[b];
#pragma unroll
            for (int k = 0; k + 1 < NF; k++) p *= tmem_value<T>(g.v[b][k], r);
            acc[b & (CHAINS - 1)][r] += p * tmem_value<T>(g.v[b][NF - 1], r);
        }
}

// The batches [first, first + count) in order, added to acc; after(i) behind batch i (from 0).
template <int CHAINS, typename T, int NF, int W, typename After>
__device__ __forceinline__ void walk_lots(const ResidentRecords<T, NF>& records, int first, int count, uint32_t base,
                                          T (&acc)[2][kLaneRows<T, W>], After&& after) {
    if (count <= 0) return;
    Lot<T, NF, W> x, y;
    LotRecords<T, NF> rx, ry;
    records.fetch(rx, first);
    issue(x, rx, base);
    records.fetch(ry, first + 1);
#pragma unroll 1
    for (int i = 0; i < count; i += 2) {
        await(x);
        issue(y, ry, base);
        add_terms<CHAINS>(x, rx, acc);
        records.fetch(rx, first + i + 2);
        after(i);
        await(y);
        issue(x, rx, base);
        add_terms<CHAINS>(y, ry, acc); // (an odd count's last batch is not the group's: everything is closed by then)
        records.fetch(ry, first + i + 3);
        after(i + 1);
    }
    await(x);
}

// Results of a tile in shared memory, rows side by side as in HBM: they leave as one bulk copy. Where the
// lanes that store a column would meet in the same banks, eight or more of them, rows are 16 bytes further
// apart and all threads copy them out (a bulk copy per row took 40 clocks each: 2 10^6 rows, 5 x 10 -> 16,
// 954 triplets, f64, forward: 610 -> 830 us).
struct ResultStage {
    int columns, stride; // bytes from row to row
    int offset;          // in shared memory
    template <typename T> __device__ __forceinline__ bool whole() const {
        return stride == columns * static_cast<int>(sizeof(T));
    }
};
template <typename T> ResultStage result_stage(int columns, int rows, size_t& smem) {
    const int bytes = columns * static_cast<int>(sizeof(T));
    const bool crowded = bytes % (sizeof(T) == 8 ? 64 : 32) == 0;
    smem = (smem + 15) / 16 * 16;
    ResultStage s{columns, bytes + (crowded ? 16 : 0), static_cast<int>(smem)};
    smem += static_cast<size_t>(rows) * s.stride;
    return s;
}
__device__ __forceinline__ void bulk_copy_out(void* global_dst, const void* smem_src, unsigned bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;\n" ::"l"(global_dst),
                 "r"(smem_address(smem_src)), "r"(bytes)
                 : "memory");
}
// All threads, when all of the tile's results are there (and fence_results has been called by who wrote
// them); a barrier has to follow before the next results.
template <typename T>
__device__ __forceinline__ void send_results(const ResultStage& s, const unsigned char* smem, T* out, int64_t row0,
                                             int rows, int tid) {
    const int bytes = s.columns * static_cast<int>(sizeof(T));
    unsigned char* dst = reinterpret_cast<unsigned char*>(out + row0 * s.columns);
    const unsigned char* src = smem + s.offset;
    if (s.whole<T>()) {
        const int all = rows * bytes, whole = all & ~15;
        if (tid == 0 && whole > 0) bulk_copy_out(dst, src, static_cast<unsigned>(whole));
        const int x = whole + tid * static_cast<int>(sizeof(T));
        if (x < all) *reinterpret_cast<T*>(dst + x) = *reinterpret_cast<const T*>(src + x);
    } else {
        const int per_row = bytes / 16, total = rows * per_row;
        const int dr = kTmemThreads / per_row, dc = kTmemThreads - dr * per_row;
        int row = tid / per_row, c = tid - row * per_row;
        for (int x = tid; x < total; x += kTmemThreads) {
            *reinterpret_cast<uint4*>(dst + static_cast<int64_t>(x) * 16) =
                *reinterpret_cast<const uint4*>(src + row * s.stride + c * 16);
            row += dr;
            c += dc;
            if (c >= per_row) {
                c -= per_row;
                row++;
            }
        }
    }
    if (tid == 0) asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
}
__device__ __forceinline__ void fence_results() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }
__device__ __forceinline__ void await_results_read() { asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory"); }
__device__ __forceinline__ void await_results_sent() { asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory"); }

// The stage may be written again when the copies of the tile before have read it: warp 0, whose first
// lane issued them, says so on a barrier, and every warp waits there before its first result of a tile.
struct StageGuard {
    uint64_t* bar;
    int tile = 0; // how many tiles this block has begun
    bool passed = false;
    __device__ void begin_tile() { passed = false; }
    __device__ __forceinline__ void pass(int warp, int lane, const Status& st) {
        if (passed) return;
        passed = true;
        if (tile == 0) return;
        if (warp == 0) {
            await_results_read();
            __syncwarp();
            if (lane == 0) mbarrier_arrive_expect(bar, 0);
        } else if (!mbarrier_wait(bar, (tile - 1) & 1) && lane == 0) {
            report_stalled(st);
        }
        __syncwarp();
    }
};

// The columns [n_lo, n_hi) of a tile by factors: the records are those of products (NF = 1), but TMEM holds the
// operands, A's columns, then B's; the coefficient comes first in the terms of rows that are not `normal`.
// (`cell / nB` by multiplication is exact up to 256 cells.) A call of its own, so that the loop over products keeps
// its registers.
template <typename T, int W>
__device__ __noinline__ void sum_by_factors(const ResidentRecords<T, 1> records, const int32_t* starts, int n_lo, int n_hi,
                                            uint32_t base, int nA, int nB, int ones, unsigned normal,
                                            unsigned char* results, int row_step) {
    constexpr int R = kLaneRows<T, W>;
    const uint32_t reciprocal = (65536u + nB - 1) / nB;
    for (int n = n_lo; n < n_hi; n++) {
        const int first = uniform(starts[n]) / kLot, end = uniform(starts[n + 1]) / kLot;
        T sum[R], part[R]; // (PieceSum: f32 in pieces of 32 records)
#pragma unroll
        for (int r = 0; r < R; r++) sum[r] = part[r] = T(0);
        for (int i = first; i < end; i++) {
            Lot<T, 2, W> g;
            LotRecords<T, 1> rec;
            records.fetch(rec, i);
#pragma unroll
            for (int b = 0; b < kLot; b++) {
                const uint32_t cell = ((b & 1) ? rec.q[b / 2] >> 16 : rec.q[b / 2] & 0xffffu) / W, a = cell * reciprocal >> 16;
                const bool padding = cell == static_cast<uint32_t>(ones);
                tmem_load(base + (padding ? cell : a) * W, g.v[b][0]);
                tmem_load(base + (padding ? cell : nA + cell - a * nB) * W, g.v[b][1]);
            }
            await(g);
#pragma unroll
            for (int b = 0; b < kLot; b++)
#pragma unroll
                for (int r = 0; r < R; r++) {
                    const T va = tmem_value<T>(g.v[b][0], r), vb = tmem_value<T>(g.v[b][1], r);
                    const bool products = normal >> r & 1;
                    part[r] = fma(products ? rec.c[b] : rec.c[b] * va, products ? va * vb : vb, part[r]);
                }
            if (sizeof(T) == 4 && ((i - first) & (kPieceRecords / kLot - 1)) == kPieceRecords / kLot - 1) {
#pragma unroll
                for (int r = 0; r < R; r++) {
                    sum[r] += part[r];
                    part[r] = T(0);
                }
            }
        }
#pragma unroll
        for (int r = 0; r < R; r++) reinterpret_cast<T*>(results + r * row_step)[n] = sizeof(T) == 8 ? part[r] : sum[r] + part[r];
    }
}

// ---- forward: by products of operand columns (NF = 1: the records' columns are the cells (a, b) of A x B,
// whose products are formed once per row on the way into TMEM), where those fit, else, f32 only, by pairs
// (NF = 2; f64 has half the rows per lane here, which gather_sums does not: 10^6 rows, 24 x 11 -> 56, 1321
// triplets: 520 -> 690 us).
//
// A tile with values out_of_band is done by factors.
// 2^20 rows, 20 x 6 -> 50, 1000 triplets, a call: looking at the values makes 317 us 328 (f64) and 210 us 216
// (f32); with such a row in every tile it takes 656 and 408 (all by gather_sums, without a look: 405, 397).
template <typename T> struct ProductSource {
    const T* C;
    const int32_t *PA, *PB, *PO;
    int nA, nB, nO;
    __device__ int key(int x, unsigned& bad) const {
        int32_t a = __ldg(PA + x), b = __ldg(PB + x), o = __ldg(PO + x);
        if (clamp_index(a, nA)) bad |= 1u << kA;
        if (clamp_index(b, nB)) bad |= 1u << kB;
        if (clamp_index(o, nO)) bad |= 1u << kO;
        return o;
    }
    __device__ T coefficient(int x) const { return __ldg(C + x); }
    __device__ int column(int x, int) const {
        int32_t a = __ldg(PA + x), b = __ldg(PB + x);
        clamp_index(a, nA);
        clamp_index(b, nB);
        return a * nB + b;
    }
};

// Behind the products (NF = 1) and, for either way of taking them, the operands.
__host__ __device__ inline int ones_column(int nf, int nA, int nB) {
    return nf == 1 && nA * nB > nA + nB ? nA * nB : nA + nB;
}

template <typename T, int NF, int W>
__global__ void __launch_bounds__(kTmemThreads, 1)
sap_fwd_resident(T* __restrict__ O, const __grid_constant__ Operands operands, const unsigned char* __restrict__ table,
                 const int32_t* __restrict__ o_start, const ResultStage stage, int capacity, int slab_offset,
                 int64_t I, int64_t tiles, Status st) {
    constexpr int R = kLaneRows<T, W>;
    const int nA = operands.cols[0], nB = operands.cols[1], nO = stage.columns;
    extern __shared__ __align__(16) unsigned char smem[];
    // layout: records | starts [nO + 1] | results | slabs
    ResidentRecords<T, NF> records(smem, capacity);
    int32_t* starts = reinterpret_cast<int32_t*>(smem + (records.bytes(capacity) + 15) / 16 * 16);
    __shared__ uint32_t tmem_s;
    __shared__ uint64_t stage_free;
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(kFullMask, tid >> 5, 0), group = warp >> 2;

    Tiles<T, W> t{operands, I, operands.template slab_bytes<T>(), smem + slab_offset};
    t.start(blockIdx.x, tid);
    if (warp == 0) tmem_alloc(&tmem_s, kTmemColumns);
    if (tid == 0) {
        mbarrier_init(&stage_free, 1);
        mbarrier_init_fence();
    }
    for (int n = tid; n <= nO; n += kTmemThreads) starts[n] = __ldg(o_start + n);
    records.load(table, __ldg(o_start + nO), capacity, tid);
    tmem_fence_before_sync();
    __syncthreads();
    tmem_fence_after_sync();
    const uint32_t base = tmem_quadrant(tmem_s, warp);
    const int ones = ones_column(NF, nA, nB);
    if (warp < 4)
        for (int r = 0; r < R; r++) tmem_store(base + ones * W + r * words_of(sizeof(T)), T(1));
    const int n_lo = uniform(group_column(starts, nO, 1, group, kTmemGroups));
    const int n_hi = uniform(group_column(starts, nO, 1, group + 1, kTmemGroups));
    const int first = uniform(starts[n_lo]) / kLot, count = uniform(starts[n_hi]) / kLot - first;
    const int own = (warp & 3) * 32 + lane;
    unsigned char* own_results = smem + stage.offset + own * stage.stride;
    StageGuard guard{&stage_free};

    int64_t before = -1;
    for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        cp_async_wait<0>();
        tmem_fence_before_sync();
        __syncthreads(); // this tile's rows are there, the results of the one before, too
        tmem_fence_after_sync();
        if (before >= 0) send_results(stage, smem, O, before, kSlabRows * R, tid);
        before = tile * (kSlabRows * R);
        const int a_stride = slab_stride(nA * static_cast<int>(sizeof(T)));
        const int b_stride = slab_stride(nB * static_cast<int>(sizeof(T)));
        unsigned bad = 0; // rows of the lane's in which this thread sees a value out_of_band
        if constexpr (NF == 1) {
            const unsigned char* a_row = t.slabs + own * a_stride;
            const unsigned char* b_row = t.slabs + kSlabRows * a_stride + own * b_stride;
            constexpr int words = words_of(sizeof(T)), kHeld = 8;
            for (int a0 = group; a0 < nA; a0 += kHeld * kTmemGroups) {
                T va[kHeld][R];
#pragma unroll
                for (int i = 0; i < kHeld; i++)
#pragma unroll
                    for (int r = 0; r < R; r++)
                        if (a0 + i * kTmemGroups < nA)
                            va[i][r] = reinterpret_cast<const T*>(a_row + r * t.slab)[a0 + i * kTmemGroups];
                for (int b = 0; b < nB; b += 2) { // (behind an odd last column a row is padded)
                    T vb[R][2];
#pragma unroll
                    for (int r = 0; r < R; r++) load_vec<T, 2>(reinterpret_cast<const T*>(b_row + r * t.slab) + b, vb[r]);
                    if ((b / 2) % kTmemGroups == group) // (every value is looked at by one thread)
#pragma unroll
                        for (int r = 0; r < R; r++)
                            bad |= (out_of_band(vb[r][0]) | (out_of_band(vb[r][1]) & static_cast<unsigned>(b + 1 < nB))) << r;
#pragma unroll
                    for (int i = 0; i < kHeld; i++) {
                        const int a = a0 + i * kTmemGroups;
                        if (a >= nA) break;
                        if (b == 0)
#pragma unroll
                            for (int r = 0; r < R; r++) bad |= out_of_band(va[i][r]) << r;
                        uint32_t w[2 * W];
#pragma unroll
                        for (int c = 0; c < 2; c++)
#pragma unroll
                            for (int r = 0; r < R; r++) put_coefficient<T>(w + c * W + r * words, va[i][r] * vb[r][c]);
                        const uint32_t at = base + (a * nB + b) * W;
                        if (b + 1 < nB) {
                            tmem_store(at, w);
                        } else {
                            uint32_t one[W];
#pragma unroll
                            for (int j = 0; j < W; j++) one[j] = w[j];
                            tmem_store(at, one);
                        }
                    }
                }
            }
#pragma unroll
            for (int r = 0; r < R; r++) // (rows behind the last one hold anything)
                if (before + r * kSlabRows + own >= I) bad &= ~(1u << r);
        } else {
            slabs_to_tmem<T, W>(t.slabs, t.slab, a_stride, nA, base, warp, lane);
            slabs_to_tmem<T, W>(t.slabs + kSlabRows * a_stride, t.slab, b_stride, nB, base + nA * W, warp, lane);
        }
        tmem_wait_store();
        tmem_fence_before_sync();
        const bool by_factors = uniform(__syncthreads_or(bad)) != 0;
        tmem_fence_after_sync();
        if (NF == 1 && by_factors) {
            slabs_to_tmem<T, W>(t.slabs, t.slab, a_stride, nA, base, warp, lane);
            slabs_to_tmem<T, W>(t.slabs + kSlabRows * a_stride, t.slab, b_stride, nB, base + nA * W, warp, lane);
            tmem_wait_store();
            tmem_fence_before_sync();
            __syncthreads();
            tmem_fence_after_sync();
        }
        if (tile + gridDim.x < tiles) t.start(tile + gridDim.x, tid);

        guard.begin_tile();
        if (count == 0) guard.pass(warp, lane, st);
        T acc[2][R];
        PieceSum<T, R> sum;
        sum.clear();
#pragma unroll
        for (int r = 0; r < R; r++) acc[0][r] = acc[1][r] = T(0);
        int n = n_lo, left = n_lo < n_hi ? uniform(starts[n_lo + 1] - starts[n_lo]) / kLot : 0;
        auto after = [&](int i) {
            if constexpr (sizeof(T) == 4) { // (PieceSum: pieces of 32 records)
                if ((i & (kPieceRecords / kLot - 1)) == kPieceRecords / kLot - 1) {
#pragma unroll
                    for (int r = 0; r < R; r++) {
                        sum.total[r] += acc[0][r] + acc[1][r];
                        acc[0][r] = acc[1][r] = T(0);
                    }
                }
            }
            if (__builtin_expect(--left == 0, 0)) { // column n is complete
                guard.pass(warp, lane, st);
#pragma unroll
                for (int r = 0; r < R; r++) {
                    T v = acc[0][r] + acc[1][r];
                    if constexpr (sizeof(T) == 4) {
                        v += sum.total[r];
                        sum.total[r] = T(0);
                    }
                    reinterpret_cast<T*>(own_results + r * kSlabRows * stage.stride)[n] = v;
                    acc[0][r] = acc[1][r] = T(0);
                }
                n++;
                left = n < n_hi ? uniform(starts[n + 1] - starts[n]) / kLot : 0;
            }
        };
        constexpr int kChains = sizeof(T) == 8 ? 1 : 2; // (f64: in the order of gather_sums)
        if constexpr (NF == 1) {
            if (by_factors) {
                guard.pass(warp, lane, st);
                sum_by_factors<T, W>(records, starts, n_lo, n_hi, base, nA, nB, ones,
                                     rows_in_band<T, W>(base, nA + nB), own_results,
                                     kSlabRows * stage.stride);
            }
        }
        walk_lots<kChains, T, NF, W>(records, first, NF == 1 && by_factors ? 0 : count, base, acc, after);
        guard.tile++;
        fence_results();
    }
    cp_async_wait<0>();
    tmem_fence_before_sync();
    __syncthreads();
    tmem_fence_after_sync();
    if (before >= 0)
        send_results(stage, smem, O, before, static_cast<int>(min(static_cast<int64_t>(kSlabRows * R), I - before)), tid);
    if (warp == 0) {
        tmem_free(tmem_s, kTmemColumns);
        await_results_sent();
    }
}

// ---- VJP by cells. With S the narrower of A, B and T the wider one, both gradients are sums over the
// cells (t, s) of
//
//   X = sum of C gO[PO] over the triplets of the cell:    gT[t] += X S[s],    gS[s] += X T[t],
//
// so a triplet costs one gather and one FMA per row instead of two records of two factors. The
// cells are sorted by t, then s; a warp group owns whole t. It keeps the X of one t in TMEM columns and takes
// them from there together, two s at a time (from a cell's end alone the gradients took 75 instructions, a
// triplet 7); gS is summed in TMEM columns that every group has for itself, which are added at the end
// of a tile.
template <typename T> struct CellSource {
    const T* C;
    const int32_t *PT, *PS, *PO;
    int nT, nS, nO, t_bit, s_bit;
    __device__ int key(int x, unsigned& bad) const {
        int32_t t = __ldg(PT + x), s = __ldg(PS + x), o = __ldg(PO + x);
        if (clamp_index(t, nT)) bad |= 1u << t_bit;
        if (clamp_index(s, nS)) bad |= 1u << s_bit;
        if (clamp_index(o, nO)) bad |= 4u;
        return t * nS + s;
    }
    __device__ T coefficient(int x) const { return __ldg(C + x); }
    __device__ int column(int x, int) const {
        int32_t o = __ldg(PO + x);
        clamp_index(o, nO);
        return o;
    }
};

// Operands: gO (nO columns), T, S; cell_start[t * nS + s] in records.
template <typename T, int W>
__global__ void __launch_bounds__(kTmemThreads, 1)
sap_vjp_resident(T* __restrict__ gT, T* __restrict__ gS, const __grid_constant__ Operands operands,
                 const unsigned char* __restrict__ table, const int32_t* __restrict__ cell_start,
                 const ResultStage t_stage, const ResultStage s_stage, int capacity, int slab_offset, int64_t I,
                 int64_t tiles, Status st) {
    constexpr int R = kLaneRows<T, W>;
    const int nO = operands.cols[0], nT = operands.cols[1], nS = operands.cols[2], cells = nT * nS;
    extern __shared__ __align__(16) unsigned char smem[];
    // layout: records | starts [cells + 1] | list [cells + 1] | results | slabs
    ResidentRecords<T, 1> records(smem, capacity);
    int32_t* starts = reinterpret_cast<int32_t*>(smem + (records.bytes(capacity) + 15) / 16 * 16);
    uint4* list = reinterpret_cast<uint4*>(starts + (cells + 4) / 4 * 4);
    __shared__ uint32_t tmem_s;
    __shared__ uint64_t stage_free;
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(kFullMask, tid >> 5, 0), group = warp >> 2;

    Tiles<T, W> tile_of{operands, I, operands.template slab_bytes<T>(), smem + slab_offset};
    tile_of.start(blockIdx.x, tid);
    if (warp == 0) tmem_alloc(&tmem_s, kTmemColumns);
    if (tid == 0) {
        mbarrier_init(&stage_free, 1);
        mbarrier_init_fence();
    }
    for (int c = tid; c <= cells; c += kTmemThreads) starts[c] = __ldg(cell_start + c);
    records.load(table, __ldg(cell_start + cells), capacity, tid);
    tmem_fence_before_sync();
    __syncthreads();
    tmem_fence_after_sync();
    const uint32_t base = tmem_quadrant(tmem_s, warp);
    tile_of.ones(base, warp);

    const int t_lo = uniform(group_column(starts, nT, nS, group, kTmemGroups));
    const int t_hi = uniform(group_column(starts, nT, nS, group + 1, kTmemGroups));
    const int c_lo = t_lo * nS, c_hi = t_hi * nS;
    const int first = uniform(starts[c_lo]) / kLot, count = uniform(starts[c_hi]) / kLot - first;
    // The group's columns behind the operands and the column of ones: X [s], sums of gS [s], for an even
    // number of s.
    const int pairs = (nS + 1) / 2, group_columns = (operands.total + 1 + group * 4 * pairs) * W;
    // Its cells that have records: batches, whether the last one of its t; column of X, t; which s t has.
    if ((warp & 3) == 0) {
        int n = 0;
        for (int c0 = c_lo; c0 < c_hi; c0 += 32) {
            const int c = c0 + lane, t = c / nS, s = c - t * nS;
            const int batches = c < c_hi ? (starts[c + 1] - starts[c]) / kLot : 0;
            const unsigned some = __ballot_sync(kFullMask, batches > 0);
            if (batches > 0) {
                uint32_t present = 0;
                for (int s2 = 0; s2 < nS; s2++)
                    present |= starts[t * nS + s2 + 1] > starts[t * nS + s2] ? 1u << s2 : 0u;
                list[c_lo + n + __popc(some & ((1u << lane) - 1))] =
                    make_uint4(static_cast<uint32_t>(batches) | (starts[c + 1] == starts[(t + 1) * nS] ? 1u << 31 : 0u),
                               static_cast<uint32_t>(group_columns + s * W) | static_cast<uint32_t>(t) << 16, present, 0u);
            }
            n += __popc(some);
        }
    }
    const int own = (warp & 3) * 32 + lane;
    unsigned char* own_t = smem + t_stage.offset + own * t_stage.stride;
    unsigned char* own_s = smem + s_stage.offset + own * s_stage.stride;
    const uint32_t X = base + group_columns, sums = X + 2 * pairs * W;
    StageGuard guard{&stage_free};

    int64_t before = -1;
    for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        cp_async_wait<0>();
        tmem_fence_before_sync();
        __syncthreads(); // this tile's rows are there, the results of the one before, too
        tmem_fence_after_sync();
        if (before >= 0) {
            send_results(t_stage, smem, gT, before, kSlabRows * R, tid);
            send_results(s_stage, smem, gS, before, kSlabRows * R, tid);
        }
        before = tile * (kSlabRows * R);
        {
            const unsigned char* src = tile_of.slabs;
            uint32_t column = base;
            for (int q = 0; q < 3; q++) {
                const int stride = slab_stride(operands.cols[q] * static_cast<int>(sizeof(T)));
                slabs_to_tmem<T, W>(src, tile_of.slab, stride, operands.cols[q], column, warp, lane);
                src += kSlabRows * stride;
                column += operands.cols[q] * W;
            }
            uint32_t zeros[2 * W];
#pragma unroll
            for (int i = 0; i < 2 * W; i++) zeros[i] = 0;
            for (int s = 0; s < nS; s += 2) tmem_store(sums + s * W, zeros);
        }
        tmem_wait_store();
        tmem_fence_before_sync();
        __syncthreads();
        tmem_fence_after_sync();
        if (tile + gridDim.x < tiles) tile_of.start(tile + gridDim.x, tid);

        guard.begin_tile();
        if (t_lo == t_hi) guard.pass(warp, lane, st);
        auto keep_t = [&](int t, const T (&v)[R]) {
            guard.pass(warp, lane, st);
#pragma unroll
            for (int r = 0; r < R; r++) reinterpret_cast<T*>(own_t + r * kSlabRows * t_stage.stride)[t] = v[r];
        };
        T acc[2][R];
#pragma unroll
        for (int r = 0; r < R; r++) acc[0][r] = acc[1][r] = T(0);
        for (int t = t_lo; t < t_hi; t++)
            if (starts[t * nS] == starts[(t + 1) * nS]) keep_t(t, acc[0]); // zeros
        // gT[t], and t's part of gS
        auto end_t = [&](int t, uint32_t present) {
            uint32_t value_t[W];
            T sum_t[R];
#pragma unroll
            for (int r = 0; r < R; r++) sum_t[r] = T(0);
            tmem_wait_store(); // (X)
            tmem_load(base + (nO + t) * W, value_t);
#pragma unroll 1
            for (int s = 0; s < nS; s += 2, present >>= 2) {
                uint32_t x[2 * W], value_s[2 * W], sum_s[2 * W];
                tmem_load(X + s * W, x);
                tmem_load(base + (nO + nT + s) * W, value_s);
                tmem_load(sums + s * W, sum_s);
                tmem_wait_load();
                tmem_pin(value_t);
                tmem_pin(x);
                tmem_pin(value_s);
                tmem_pin(sum_s);
#pragma unroll
                for (int c = 0; c < 2; c++) {
                    if (!(present >> c & 1)) continue; // (no such cell: its X is an older one)
#pragma unroll
                    for (int r = 0; r < R; r++) {
                        const int i = c * R + r;
                        const T v = tmem_value<T>(x, i);
                        sum_t[r] += v * tmem_value<T>(value_s, i);
                        put_coefficient<T>(sum_s + i * words_of(sizeof(T)),
                                           tmem_value<T>(sum_s, i) + v * tmem_value<T>(value_t, r));
                    }
                }
                tmem_store(sums + s * W, sum_s);
            }
            keep_t(t, sum_t);
        };
        const uint4* next = list + c_lo;
        uint4 cell = make_uint4(0u, 0u, 0u, 0u), ahead = count > 0 ? *next++ : cell;
        int left = 0, batches_left = count;
        auto next_cell = [&] {
            cell.x = uniform(ahead.x), cell.y = uniform(ahead.y), cell.z = uniform(ahead.z);
            left = cell.x & 0x7fffffff;
            ahead = *next++; // (behind the list: not used)
        };
        if (count > 0) next_cell();
        walk_lots<2, T, 1, W>(records, first, count, base, acc, [&](int) {
            batches_left--;
            if (--left == 0) {
                uint32_t x[W];
#pragma unroll
                for (int r = 0; r < R; r++) {
                    put_coefficient<T>(x + r * words_of(sizeof(T)), acc[0][r] + acc[1][r]);
                    acc[0][r] = acc[1][r] = T(0);
                }
                tmem_store(__byte_perm(cell.y, base, 0x7610), x);
                if (cell.x >> 31) end_t(static_cast<int>(cell.y >> 16), cell.z);
                if (batches_left > 0) next_cell();
            }
        });
        guard.tile++;
        // gS: the sums of the four groups
        tmem_wait_store();
        tmem_fence_before_sync();
        __syncthreads();
        tmem_fence_after_sync();
        for (int s2 = group; s2 < nS; s2 += kTmemGroups) {
            uint32_t part[kTmemGroups][W];
#pragma unroll
            for (int g = 0; g < kTmemGroups; g++)
                tmem_load(base + (operands.total + 1 + (4 * g + 2) * pairs + s2) * W, part[g]);
            tmem_wait_load();
#pragma unroll
            for (int g = 0; g < kTmemGroups; g++) tmem_pin(part[g]);
#pragma unroll
            for (int r = 0; r < R; r++)
                reinterpret_cast<T*>(own_s + r * kSlabRows * s_stage.stride)[s2] =
                    (tmem_value<T>(part[0], r) + tmem_value<T>(part[1], r)) +
                    (tmem_value<T>(part[2], r) + tmem_value<T>(part[3], r));
        }
        fence_results();
    }
    cp_async_wait<0>();
    tmem_fence_before_sync();
    __syncthreads();
    tmem_fence_after_sync();
    if (before >= 0) {
        const int rows = static_cast<int>(min(static_cast<int64_t>(kSlabRows * R), I - before));
        send_results(t_stage, smem, gT, before, rows, tid);
        send_results(s_stage, smem, gS, before, rows, tid);
    }
    if (warp == 0) {
        tmem_free(tmem_s, kTmemColumns);
        await_results_sent();
    }
}

// The same with the records streamed, gT stored as it comes and gS summed in shared memory: for records, results or
// addresses that sap_vjp_resident does not take. A cell's end is dearer here (75 instructions), so gather_sums is
// faster up to about ten triplets per cell. 800 000 rows, f64: 32 x 8 -> 60, 8000 triplets, 5.4 ms by gather_sums,
// 3.2 here; 25 x 25 -> 30 with 1500 (2.4 per cell), 100 000 rows, 164 us there, 335 here.
template <typename T, int W>
__global__ void __launch_bounds__(kTmemThreads, 1)
sap_vjp_cells(T* __restrict__ gT, T* __restrict__ gS, const __grid_constant__ Operands operands,
              const unsigned char* __restrict__ records, const int32_t* __restrict__ cell_start, int64_t I,
              int64_t tiles, Status st) {
    using G = Batch<T, 1, W>;
    constexpr int B = G::B, R = G::R, RB = G::RB;
    using Ring = RecordRing<1024>;
    constexpr int kPerStage = 1024 / (B * RB);
    static_assert(kPerStage % 2 == 0, "pairs of batches do not straddle stages");
    const int nO = operands.cols[0], nT = operands.cols[1], nS = operands.cols[2], cells = nT * nS;
    extern __shared__ __align__(16) unsigned char smem[];
    // layout: ring | starts [cells + 1], padded | gS sums [group][nS][128 R] | slabs
    int32_t* starts = reinterpret_cast<int32_t*>(smem + kStageBytes);
    T* sums = reinterpret_cast<T*>(smem + kStageBytes + (static_cast<size_t>(cells + 1) * 4 + 15) / 16 * 16);
    unsigned char* slabs = reinterpret_cast<unsigned char*>(sums + kTmemGroups * nS * kSlabRows * R);
    __shared__ uint32_t tmem_s;
    __shared__ uint64_t full[kTmemGroups][2];
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(kFullMask, tid >> 5, 0), group = warp >> 2;

    Tiles<T, W> tile_of{operands, I, operands.template slab_bytes<T>(), slabs};
    tile_of.start(blockIdx.x, tid);
    if (warp == 0) tmem_alloc(&tmem_s, kTmemColumns);
    Ring::prepare(smem, full, tid);
    for (int c = tid; c <= cells; c += kTmemThreads) starts[c] = __ldg(cell_start + c);
    tmem_fence_before_sync();
    __syncthreads();
    tmem_fence_after_sync();
    const uint32_t base = tmem_quadrant(tmem_s, warp);
    tile_of.ones(base, warp);

    const int t_lo = uniform(group_column(starts, nT, nS, group, kTmemGroups));
    const int t_hi = uniform(group_column(starts, nT, nS, group + 1, kTmemGroups));
    const int c_hi = t_hi * nS;
    const int x_lo = uniform(starts[t_lo * nS]), batches = uniform(starts[c_hi] - starts[t_lo * nS]) / B;
    Ring ring(smem + group * 2048, full[group], group, (warp & 3) == 0 && lane == 0,
              records + static_cast<size_t>(x_lo) * RB, batches * B * RB);
    const int own = (warp & 3) * 32 + lane;
    T* mine = sums + static_cast<size_t>(group) * nS * kSlabRows * R + own; // [s][slot][128]

    for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        tile_of.load(tile + gridDim.x < tiles ? tile + gridDim.x : -1, base, tid, warp, lane);
        const int64_t row0 = tile * (kSlabRows * R) + own;
        bool live[R];
        T acc[R], sum_t[R];
#pragma unroll
        for (int r = 0; r < R; r++) {
            live[r] = row0 + r * kSlabRows < I;
            acc[r] = sum_t[r] = T(0);
        }
        for (int s = 0; s < nS * R; s++) mine[s * kSlabRows] = T(0);
        SectorWriter<T, R> writer{};
        int t = t_lo, s = 0, c = t_lo * nS;
        uint32_t value_t[1][W];
        auto load_t = [&] { // T[t] of the lane's rows
            tmem_load(base + (nO + t) * W, value_t[0]);
            tmem_wait_load();
            tmem_pin(value_t[0]);
        };
        // Moves on to the next cell that has records (or to the end), storing gT[t] on the way.
        // Returns its number of batches.
        auto next_cell = [&](bool moved) {
            for (; c < c_hi; moved = true) {
                if (moved) {
                    c++;
                    if (++s == nS) {
                        writer.put(t, gT + row0 * nT + t, kSlabRows * static_cast<int64_t>(nT), t - t_lo, t + 1 == t_hi,
                                   sum_t, live);
#pragma unroll
                        for (int r = 0; r < R; r++) sum_t[r] = T(0);
                        s = 0;
                        t++;
                        if (t < t_hi) load_t();
                    }
                    if (c == c_hi) break;
                }
                const int n = uniform(starts[c + 1] - starts[c]) / B;
                if (n > 0) return n;
            }
            return -1;
        };
        auto end_cell = [&] {
            uint32_t value_s[W];
            tmem_load(base + (nO + nT + s) * W, value_s);
            tmem_wait_load();
            tmem_pin(value_s);
#pragma unroll
            for (int r = 0; r < R; r++) {
                sum_t[r] += acc[r] * tmem_value<T>(value_s, r);
                mine[(s * R + r) * kSlabRows] += acc[r] * tmem_value<T>(value_t[0], r);
                acc[r] = T(0);
            }
        };
        if (t < t_hi) load_t();
        ring.start_tile();
        int left = next_cell(false);
        if (batches > 0) {
            G x, y;
            Records<T, 1, W> rx, ry;
            auto add = [&](const G& g, const Records<T, 1, W>& rec) {
                add_terms<T, 1, W>(g, rec, acc);
                if (--left == 0) {
                    end_cell();
                    left = next_cell(true);
                }
            };
            ring.enter_stage(0, lane, st);
            fetch<T, 1, W>(rx, ring.template at<B * RB>(0));
            issue<T, 1, W>(x, rx, base);
            fetch<T, 1, W>(ry, ring.template at<B * RB>(1));
            for (int i = 0; i < batches; i += 2) {
                await<T, 1, W>(x);
                issue<T, 1, W>(y, ry, base);
                add(x, rx);
                if ((i & (kPerStage - 1)) == kPerStage - 2 && i + 2 < batches)
                    ring.enter_stage((i + 2) / kPerStage, lane, st);
                fetch<T, 1, W>(rx, ring.template at<B * RB>(i + 2));
                await<T, 1, W>(y);
                issue<T, 1, W>(x, rx, base);
                add(y, ry); // (behind the last batch: all cells are done, nothing is kept)
                fetch<T, 1, W>(ry, ring.template at<B * RB>(i + 3));
            }
            await<T, 1, W>(x);
        }
        tmem_fence_before_sync();
        __syncthreads(); // all sums are complete; before the next tile overwrites TMEM
        tmem_fence_after_sync();
        // gS: the tile's rows are contiguous in memory
        const int64_t first_row = tile * (kSlabRows * R);
        const int64_t have = I - first_row < kSlabRows * R ? I - first_row : kSlabRows * R;
        for (int y = tid; y < have * nS; y += kTmemThreads) {
            const int row = y / nS, s2 = y - row * nS;
            T v = T(0);
#pragma unroll
            for (int g = 0; g < kTmemGroups; g++)
                v += sums[(static_cast<size_t>(g) * nS + s2) * kSlabRows * R + row];
            gS[first_row * nS + y] = v;
        }
        // (the barriers of the next tile's load come before the sums are cleared)
    }
    cp_async_wait<0>();
    __syncthreads();
    if (warp == 0) tmem_free(tmem_s, kTmemColumns);
}

inline bool at_16_bytes(const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }

// Builds (or takes from the plan) the table of records over `columns` result columns, each a whole number
// of batches, and calls go(records, starts).
template <typename T, int NF, typename Source, typename Go>
void with_lots(const Call& call, TableKey key, const Source& source, int64_t K, int columns, int w, int least,
               int ones, Go&& go) {
    const size_t b_rec = (static_cast<size_t>(K) + static_cast<size_t>(columns) * kLot) * tmem_record_bytes(sizeof(T), NF);
    key.scalar_bytes = static_cast<int>(sizeof(T));
    key.n[8] = w;
    TableRef ref = acquire_table(call, key, b_rec + (static_cast<size_t>(columns) + 1) * sizeof(int32_t));
    unsigned char* records = static_cast<unsigned char*>(ref.ptr);
    int32_t* starts = reinterpret_cast<int32_t*>(records + b_rec);
    if (ref.fresh) {
        auto build = gather_table<T, NF, Source>;
        const size_t builder = table_smem(K, columns);
        allow_dynamic_smem(build, call.device, builder);
        build<<<1, kTableThreads, builder, call.stream>>>(records, starts, source, static_cast<int>(K), columns, w,
                                                          kLot, least, ones, call.status);
        MOPS_CUDA_OK(cudaGetLastError());
        commit_table(call, ref);
    }
    go(static_cast<const unsigned char*>(records), static_cast<const int32_t*>(starts));
    release_table(call, ref);
}

template <typename T> TableKey triplet_key(const SapProblem<T>& p, int64_t level) {
    TableKey key{};
    key.kind = kSapTable;
    key.ptr[0] = p.C, key.ptr[1] = p.PA, key.ptr[2] = p.PB, key.ptr[3] = p.PO;
    key.n[0] = p.K, key.n[1] = p.nA, key.n[2] = p.nB, key.n[3] = p.nO, key.n[4] = level;
    return key;
}

// Where a block's shared memory goes; `capacity` records (with the batches fetched ahead).
inline size_t resident_smem(size_t record_bytes, int capacity, int columns) {
    return (record_bytes * capacity + 15) / 16 * 16 + (static_cast<size_t>(columns + 1) * 4 + 15) / 16 * 16;
}

template <typename T, int NF, int W>
bool forward_resident(const Call& call, const SapProblem<T>& p, T* O) {
    constexpr int rows = kSlabRows * kLaneRows<T, W>;
    const int columns = ones_column(NF, p.nA, p.nB) + 1;
    const size_t limit = static_cast<size_t>(max_optin_smem(call.device)) - 1024;
    const int64_t tiles = ceil_div(p.I, static_cast<int64_t>(rows));
    if (table_smem(p.K, p.nO) > limit || !at_16_bytes(O) || p.K > (1 << 14)) return false;
    if (columns > kTmemColumns / W || tiles < sm_count(call.device)) return false;
    Operands op{};
    op.add(p.A, p.nA);
    op.add(p.B, p.nB);
    const int capacity = static_cast<int>(ceil_div(p.K + static_cast<int64_t>(p.nO) * kLot, kLot) + 3) * kLot;
    size_t smem = resident_smem(sizeof(T) + 2 * NF, capacity, p.nO);
    const ResultStage stage = result_stage<T>(p.nO, rows, smem);
    smem = (smem + 15) / 16 * 16;
    const int slabs = static_cast<int>(smem);
    smem += static_cast<size_t>(kLaneRows<T, W>) * op.template slab_bytes<T>();
    if (smem > limit) return false;
    note_kernel_f("sap_fwd_resident<%s,NF=%d,W=%d>", scalar_name<T>(), NF, W);
    auto run = [&](const unsigned char* records, const int32_t* starts) {
        launch_gather(call, sap_fwd_resident<T, NF, W>, GatherShape{W, 1, tiles, smem}, 1, O, op, records, starts, stage,
                      capacity, slabs, p.I, tiles, call.status);
    };
    if constexpr (NF == 1) {
        with_lots<T, 1>(call, triplet_key(p, -2), ProductSource<T>{p.C, p.PA, p.PB, p.PO, p.nA, p.nB, p.nO}, p.K, p.nO,
                        W, 1, columns - 1, run);
    } else {
        SapSource<T> source{p.C, {p.PA, p.PB, p.PO}, {p.nA, p.nB, p.nO}, static_cast<int>(p.K), {}};
        source.family[0] = {kO, 0, {kA, kB}, {0, p.nA}};
        with_lots<T, 2>(call, triplet_key(p, -3), source, p.K, p.nO, W, 1, columns - 1, run);
    }
    return true;
}

// The VJP's operands, in the kernels' order, and the source of its records.
template <typename T> struct CellProblem {
    bool b_narrow;
    int nS, nT, cells;
    Operands op{};
    CellSource<T> source;
    CellProblem(const SapProblem<T>& p, const T* gO)
        : b_narrow(p.nB <= p.nA), nS(b_narrow ? p.nB : p.nA), nT(b_narrow ? p.nA : p.nB), cells(nS * nT),
          source{p.C, b_narrow ? p.PA : p.PB, b_narrow ? p.PB : p.PA, p.PO, nT, nS, p.nO, b_narrow ? 0 : 1, b_narrow ? 1 : 0} {
        op.add(gO, p.nO);
        op.add(b_narrow ? p.A : p.B, nT);
        op.add(b_narrow ? p.B : p.A, nS);
    }
};

// Rows per lane: W / words(T). Both kernels read the same table.
template <typename T, int W>
bool backward_resident(const Call& call, const SapProblem<T>& p, const CellProblem<T>& c, T* gA, T* gB) {
    constexpr int rows = kSlabRows * kLaneRows<T, W>;
    const size_t limit = static_cast<size_t>(max_optin_smem(call.device)) - 1024;
    const int64_t tiles = ceil_div(p.I, static_cast<int64_t>(rows));
    if (table_smem(p.K, c.cells) > limit || !at_16_bytes(gA) || !at_16_bytes(gB) || p.K > (1 << 14)) return false;
    if (c.op.total + 1 + kTmemGroups * ((c.nS + 1) / 2 * 4) > kTmemColumns / W || c.nS > 32 || tiles < sm_count(call.device))
        return false;
    const int64_t padded = p.K + 3 * std::min<int64_t>(p.K, c.cells);
    const int capacity = static_cast<int>(ceil_div(padded, kLot) + 3) * kLot;
    size_t smem = resident_smem(sizeof(T) + 2, capacity, 5 * c.cells + 8); // (bounds and list)
    const ResultStage t_stage = result_stage<T>(c.nT, rows, smem);
    const ResultStage s_stage = result_stage<T>(c.nS, rows, smem);
    smem = (smem + 15) / 16 * 16;
    const int slabs = static_cast<int>(smem);
    smem += static_cast<size_t>(kLaneRows<T, W>) * c.op.template slab_bytes<T>();
    if (smem > limit) return false;
    note_kernel_f("sap_vjp_resident<%s,W=%d>", scalar_name<T>(), W);
    with_lots<T, 1>(call, triplet_key(p, -1), c.source, p.K, c.cells, W, 0, c.op.total,
                    [&](const unsigned char* records, const int32_t* starts) {
                        launch_gather(call, sap_vjp_resident<T, W>, GatherShape{W, 1, tiles, smem}, 1, c.b_narrow ? gA : gB,
                                      c.b_narrow ? gB : gA, c.op, records, starts, t_stage, s_stage, capacity, slabs,
                                      p.I, tiles, call.status);
                    });
    return true;
}

template <typename T, int W>
bool backward_cells(const Call& call, const SapProblem<T>& p, const CellProblem<T>& c, T* gA, T* gB) {
    constexpr int rows = kSlabRows * kLaneRows<T, W>;
    static_assert(batch_of(1, W) == kLot, "the table's batches");
    const size_t limit = static_cast<size_t>(max_optin_smem(call.device)) - 1024;
    const int64_t tiles = ceil_div(p.I, static_cast<int64_t>(rows));
    const size_t smem = kStageBytes + (static_cast<size_t>(c.cells + 1) * 4 + 15) / 16 * 16 +
                        static_cast<size_t>(kTmemGroups) * c.nS * rows * sizeof(T) +
                        static_cast<size_t>(kLaneRows<T, W>) * c.op.template slab_bytes<T>();
    if (table_smem(p.K, c.cells) > limit || c.op.total + 1 > kTmemColumns / W || smem > limit || tiles < sm_count(call.device))
        return false;
    // cells / gather_sums, 140 drawn shapes: 0.60 - 1.18 from 12 triplets per cell on (longer: down to 0.25),
    // 0.69 - 1.26 at 8 to 12, 0.85 - 1.37 at 4 to 6, 0.94 - 3.8 below 2
    if (p.K < 12 * static_cast<int64_t>(c.cells)) return false;
    note_kernel_f("sap_vjp_cells<%s,W=%d>", scalar_name<T>(), W);
    with_lots<T, 1>(call, triplet_key(p, -1), c.source, p.K, c.cells, W, 0, c.op.total,
                    [&](const unsigned char* records, const int32_t* starts) {
                        launch_gather(call, sap_vjp_cells<T, W>, GatherShape{W, 1, tiles, smem}, 1, c.b_narrow ? gA : gB,
                                      c.b_narrow ? gB : gA, c.op, records, starts, p.I, tiles, call.status);
                    });
    return true;
}

} // namespace

template <typename T> bool sap_forward_tmem(const Call& call, const SapProblem<T>& p, T* O) {
    if (fills_gpu(call, p.I) && (few_forward_triplets(p) || narrow_forward(p))) return false;
    // Most products have to be used (3.5 10^6 rows, 25 x 5 -> 5, 141 triplets, f64: 410 -> 440 us). Kernels with
    // fewer rows per lane, where shared memory or the batch leave no more, come after those by pairs, and behind
    // gather_sums for many triplets, which it has more rows for: f64 by products with one row 0.87 to 1.06 times
    // as long as gather_sums up to 1000 triplets, 1.02 to 1.27 mostly beyond; f32 by pairs with two rows 0.58 to
    // 0.68 up to 268 triplets, 1.14 to 1.42 with 8000 (32 x 8 -> 60, which fits four rows in gather_sums alone).
    const bool products = 2 * p.K >= 3 * static_cast<int64_t>(p.nA) * p.nB;
    if (products && forward_resident<T, 1, 4>(call, p, O)) return true;
    if constexpr (sizeof(T) == 4) {
        if (forward_resident<T, 2, 4>(call, p, O) || (products && forward_resident<T, 1, 2>(call, p, O)) ||
            (p.K <= 4000 && forward_resident<T, 2, 2>(call, p, O)))
            return true;
    } else {
        // (more products than fit two rows: 130 000 rows, 14 x 10 -> 8, 254 triplets: 34 -> 38 us)
        const bool fit_two = ones_column(1, p.nA, p.nB) < kTmemColumns / 4;
        if (products && fit_two && p.K <= 1000 && forward_resident<T, 1, 2>(call, p, O)) return true;
    }
    Operands op{};
    op.add(p.A, p.nA);
    op.add(p.B, p.nB);
    Results<T> results{};
    results.add(O, p.nO);
    const Family f[] = {{kO, 0, {kA, kB}, {0, p.nA}}};
    return run<T, sizeof(T) == 8>(call, p, f, 1, op, results, 0, "sap_fwd_tmem");
}

template <typename T>
bool sap_backward_tmem(const Call& call, const SapProblem<T>& p, T* gA, T* gB, const T* gO) {
    const bool both = gA != nullptr && gB != nullptr;
    if (fills_gpu(call, p.I) && (few_backward_triplets(p) || narrow_backward(p, both))) return false;
    // Both gradients of a batch with a tile for every SM: by cells.
    if (both) {
        const CellProblem<T> cells(p, gO);
        if (backward_resident<T, 4>(call, p, cells, gA, gB) || backward_resident<T, 2>(call, p, cells, gA, gB) ||
            backward_cells<T, 4>(call, p, cells, gA, gB) || backward_cells<T, 2>(call, p, cells, gA, gB))
            return true;
    }
    Operands op{};
    Results<T> results{};
    Family f[2];
    int count = 0;
    op.add(gO, p.nO);
    if (gA != nullptr) {
        f[count++] = {kA, results.total, {kO, kB}, {0, op.total}};
        op.add(p.B, p.nB);
        results.add(gA, p.nA);
    }
    if (gB != nullptr) {
        f[count++] = {kB, results.total, {kO, kA}, {0, op.total}};
        op.add(p.A, p.nA);
        results.add(gB, p.nB);
    }
    return run(call, p, f, count, op, results, 1 + (gA ? 2 : 0) + (gB ? 4 : 0), "sap_vjp_tmem");
}

template <typename T>
bool sap_second_tmem(const Call& call, const SapProblem<T>& p, T* ggO, T* gA2, T* gB2, const T* ggA,
                     const T* ggB, const T* gO) {
    Operands op{};
    Results<T> results{};
    Family f[4];
    int count = 0;
    [[maybe_unused]] const int at_gO = 0;
    op.add(gO, p.nO);
    [[maybe_unused]] const int at_ggA = op.total;
    if (ggA != nullptr) op.add(ggA, p.nA);
    [[maybe_unused]] const int at_ggB = op.total;
    if (ggB != nullptr) op.add(ggB, p.nB);
    if (ggO != nullptr) {
        if (ggA != nullptr) {
            f[count++] = {kO, results.total, {kA, kB}, {at_ggA, op.total}};
            op.add(p.B, p.nB);
        }
        if (ggB != nullptr) {
            f[count++] = {kO, results.total, {kA, kB}, {op.total, at_ggB}};
            op.add(p.A, p.nA);
        }
        results.add(ggO, p.nO);
    }
    if (gA2 != nullptr) {
        if (ggB != nullptr) f[count++] = {kA, results.total, {kO, kB}, {at_gO, at_ggB}};
        results.add(gA2, p.nA);
    }
    if (gB2 != nullptr) {
        if (ggA != nullptr) f[count++] = {kB, results.total, {kO, kA}, {at_gO, at_ggA}};
        results.add(gB2, p.nB);
    }
    if (count == 0) return false; // nothing but zeros
    return run(call, p, f, count, op, results,
               8 + (ggO ? 16 : 0) + (gA2 ? 32 : 0) + (gB2 ? 64 : 0) + (ggA ? 128 : 0) + (ggB ? 256 : 0),
               "sap_vjp_vjp_tmem");
}

#define INSTANTIATE(T)                                                                             \
    template bool sap_forward_tmem<T>(const Call&, const SapProblem<T>&, T*);                      \
    template bool sap_backward_tmem<T>(const Call&, const SapProblem<T>&, T*, T*, const T*);       \
    template bool sap_second_tmem<T>(const Call&, const SapProblem<T>&, T*, T*, T*, const T*,      \
                                     const T*, const T*);
INSTANTIATE(float)
INSTANTIATE(double)

} // namespace mops_b200
