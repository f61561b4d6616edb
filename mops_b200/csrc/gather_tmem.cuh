// Sparse sums of products over batch rows held in tensor memory (tmem.cuh):
//
//   out[i, n] = scale[i] * sum over the records of n of c * V[i, q_1] * ... * V[i, q_NF]
//
// for every batch row i, where V is the row's operands side by side and the records (a coefficient
// and NF columns) are the same for all rows. The VJP of HPE and all of SAP have this form; the
// forward of HPE is the case of a single n (hpe_tmem.cu).
//
// A gathered column of 32 rows is one `tcgen05.ld` at a column number taken from the record, for R
// rows per lane at once (W = R words(T) columns), so that the kernels are bounded by instruction
// issue and the FP64 pipe and no longer by shared memory, through which every gather went before.
//
// The loads of a warp are asynchronous and there is one wait for all of them, so the loops are
// software-pipelined by hand: wait for batch b, start the loads of batch b + 1, multiply batch b,
// fetch the records of batch b + 2 from shared memory. (Issued and waited for batch by batch, the
// same loop took 1.4 to 1.6 times as long.)
#ifndef MOPS_B200_GATHER_TMEM_CUH
#define MOPS_B200_GATHER_TMEM_CUH

#include <algorithm>
#include <cmath>

#include "tmem_tile.cuh"

namespace mops_b200 {
namespace { // (instantiated by hpe_tmem.cu and sap_tmem.cu, each for itself)

__device__ __forceinline__ int uniform(int v) { return __shfl_sync(kFullMask, v, 0); }

constexpr int kStageBytes = 8192;

// The operands of a tile, side by side: operand q has cols[q] columns.
constexpr int kMaxOperands = 5;
struct Operands {
    const void* data[kMaxOperands];
    int cols[kMaxOperands];
    int unit[kMaxOperands]; // copy_unit_of
    int count;
    int total; // columns of all of them; column `total` of a tile holds ones

    template <typename T> void add(const T* p, int columns) {
        data[count] = p;
        cols[count] = columns;
        unit[count] = copy_unit_of(p, static_cast<size_t>(columns) * sizeof(T));
        total += columns;
        count++;
    }
    // Shared memory of one slab.
    template <typename T> __host__ __device__ int slab_bytes() const {
        int bytes = 0;
        for (int q = 0; q < count; q++) bytes += kSlabRows * slab_stride(cols[q] * static_cast<int>(sizeof(T)));
        return bytes;
    }
};

// The results, side by side in the same way.
constexpr int kMaxResults = 3;
template <typename T> struct Results {
    T* data[kMaxResults];
    int cols[kMaxResults];
    int count;
    int total;
    const T* scale; // per batch row; nullptr: 1

    void add(T* p, int columns) {
        data[count] = p;
        cols[count] = columns;
        total += columns;
        count++;
    }
};

// A record: the coefficient, then NF 16-bit TMEM column numbers, 16 or 32 bytes. Padding records
// have coefficient 0 and point at a column of ones behind the operand's N columns: they add exactly
// zero whatever A holds, and the loops below have no remainders.
__host__ __device__ constexpr int tmem_record_bytes(int scalar_bytes, int nf) {
    return scalar_bytes + 2 * nf <= 16 ? 16 : 32;
}

// Monomials per batch: enough loads in flight per wait, few enough registers for two batches.
__host__ __device__ constexpr int batch_of(int nf, int w) {
    return nf * w <= 8 ? 4 : nf * w <= 16 ? 2 : 1;
}

template <typename T, int NF, int W> struct Batch {
    static constexpr int B = batch_of(NF, W), R = W / words_of(sizeof(T));
    static constexpr int RB = tmem_record_bytes(sizeof(T), NF);
    uint32_t v[B][NF][W];
};

template <typename T, int NF, int W> struct Records {
    uint32_t w[Batch<T, NF, W>::B][Batch<T, NF, W>::RB / 4];
};

template <typename T, int NF, int W>
__device__ __forceinline__ void fetch(Records<T, NF, W>& r, const unsigned char* recs) {
    using G = Batch<T, NF, W>;
#pragma unroll
    for (int b = 0; b < G::B; b++)
#pragma unroll
        for (int q = 0; q < G::RB / 16; q++) {
            const uint4 v = *reinterpret_cast<const uint4*>(recs + b * G::RB + 16 * q);
            r.w[b][4 * q] = v.x, r.w[b][4 * q + 1] = v.y;
            r.w[b][4 * q + 2] = v.z, r.w[b][4 * q + 3] = v.w;
        }
}

// Starts the loads of a batch. A block owns all of its SM's TMEM, so that its columns start at 0
// and an address is the record's 16 bits under the upper half of `base` (the warp's quadrant): one
// byte permutation each.
template <typename T, int NF, int W>
__device__ __forceinline__ void issue(Batch<T, NF, W>& g, const Records<T, NF, W>& r, uint32_t base) {
#pragma unroll
    for (int b = 0; b < Batch<T, NF, W>::B; b++)
#pragma unroll
        for (int k = 0; k < NF; k++)
            tmem_load(__byte_perm(r.w[b][words_of(sizeof(T)) + k / 2], base, (k & 1) ? 0x7632 : 0x7610),
                      g.v[b][k]);
}

template <typename T> __device__ __forceinline__ void put_coefficient(uint32_t* w, T c) {
    if constexpr (sizeof(T) == 8) {
        w[0] = static_cast<uint32_t>(__double2loint(c));
        w[1] = static_cast<uint32_t>(__double2hiint(c));
    } else {
        w[0] = __float_as_uint(c);
    }
}

template <typename T, int NF, int W> __device__ __forceinline__ void await(Batch<T, NF, W>& g) {
    tmem_wait_load();
#pragma unroll
    for (int b = 0; b < Batch<T, NF, W>::B; b++)
#pragma unroll
        for (int k = 0; k < NF; k++) tmem_pin(g.v[b][k]);
}

// acc[r] += the coefficient times the NF factors of row r, for every record of the batch. PRODUCTS: c (a b).
template <typename T, int NF, int W, bool PRODUCTS = false>
__device__ __forceinline__ void add_terms(const Batch<T, NF, W>& g, const Records<T, NF, W>& rec,
                                          T (&acc)[Batch<T, NF, W>::R]) {
#pragma unroll
    for (int b = 0; b < Batch<T, NF, W>::B; b++) {
        T c;
        if constexpr (sizeof(T) == 8)
            c = __hiloint2double(static_cast<int>(rec.w[b][1]), static_cast<int>(rec.w[b][0]));
        else
            c = __uint_as_float(rec.w[b][0]);
#pragma unroll
        for (int r = 0; r < Batch<T, NF, W>::R; r++) {
            if constexpr (PRODUCTS) {
                acc[r] += c * (tmem_value<T>(g.v[b][0], r) * tmem_value<T>(g.v[b][1], r));
            } else {
                T p = c;
#pragma unroll
                for (int k = 0; k + 1 < NF; k++) p *= tmem_value<T>(g.v[b][k], r);
                acc[r] += p * tmem_value<T>(g.v[b][NF - 1], r);
            }
        }
    }
}

// ---------------------------------------------------------------- products of operands
// A product a b may overflow or lose bits to underflow where the term c a b does neither (f32: c = 1e-30,
// a = b = 1e25), so terms are (c a) b. The f64 forward of SAP takes c (a b) all the same, because large batches
// form the products once per row (sap_tmem.cu) and a row's sums are to be the same bits in any batch; rows whose
// products might be out of range (out_of_band) are found first, and their terms are (c a) b there, too.

// Which of the lane's rows of `columns` values in TMEM have none out_of_band, a bit each.
template <typename T, int W> __device__ __forceinline__ unsigned rows_in_band(uint32_t base, int columns) {
    unsigned rows = ~0u;
    for (int n = 0; n < columns; n++) {
        uint32_t v[W];
        tmem_load(base + n * W, v);
        tmem_wait_load();
        tmem_pin(v);
#pragma unroll
        for (int r = 0; r < W / words_of(sizeof(T)); r++)
            rows &= ~(out_of_band(tmem_value<T>(v, r)) << r);
    }
    return rows;
}

// f32 sums are taken in pieces of 32 records, which are then added up: one chain over a column's records
// (thousands) lost up to four bits against the kernels that split them among 32 lanes (201 monomials of
// order 5 in one variable: relative error 3.8e-6 against 2.1e-7). f64 keeps one chain.
constexpr int kPieceRecords = 32;
template <typename T, int R> struct PieceSum {
    static constexpr bool kPieces = sizeof(T) == 4;
    T total[kPieces ? R : 1];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int r = 0; r < (kPieces ? R : 1); r++) total[r] = T(0);
    }
    // Behind batch pair i of B records per batch.
    template <int B> __device__ __forceinline__ void piece(int i, T (&acc)[R]) {
        if constexpr (kPieces) {
            constexpr int kBatches = kPieceRecords / B;
            if ((i & (kBatches - 1)) == kBatches - 2) take(acc);
        }
    }
    __device__ __forceinline__ void take(T (&acc)[R]) {
        if constexpr (kPieces) {
#pragma unroll
            for (int r = 0; r < R; r++) {
                total[r] += acc[r];
                acc[r] = T(0);
            }
        }
    }
    // The whole sum, in acc.
    __device__ __forceinline__ void finish(T (&acc)[R]) {
        if constexpr (kPieces) {
#pragma unroll
            for (int r = 0; r < R; r++) {
                acc[r] += total[r];
                total[r] = T(0);
            }
        }
    }
};

// The slabs of the tiles one block works on.
template <typename T, int W> struct Tiles {
    static constexpr int R = W / words_of(sizeof(T));
    const Operands& op;
    int64_t I;
    int slab; // bytes of one slot's rows
    unsigned char* slabs;

    __device__ void start(int64_t tile, int tid) const {
        for (int s = 0; s < R; s++) {
            const int64_t row = (tile * R + s) * kSlabRows;
            const int64_t left = I - row;
            const int have = left < kSlabRows ? static_cast<int>(left) : kSlabRows;
            unsigned char* dst = slabs + s * slab;
            for (int q = 0; q < op.count && left > 0; q++) {
                const int bytes = op.cols[q] * static_cast<int>(sizeof(T)), stride = slab_stride(bytes);
                start_slab(dst, static_cast<const T*>(op.data[q]) + row * op.cols[q], have, bytes, stride,
                           op.unit[q], tid);
                dst += kSlabRows * stride;
            }
        }
        cp_async_commit();
    }
    // The column of ones.
    __device__ void ones(uint32_t base, int warp) const {
        if (warp < 4)
            for (int r = 0; r < R; r++) tmem_store(base + op.total * W + r * words_of(sizeof(T)), T(1));
        tmem_wait_store();
    }
    // Brings the tile started before into TMEM and starts tile `next` (if >= 0). Ends with the block
    // synchronised. CHECK: whether no value of the block's rows of the batch (`live`: the lane's, a bit each) is
    // out_of_band.
    template <bool CHECK = false>
    __device__ bool load(int64_t next, uint32_t base, int tid, int warp, int lane, unsigned live = 0) const {
        unsigned bad = 0;
        cp_async_wait<0>();
        tmem_fence_before_sync();
        __syncthreads();
        tmem_fence_after_sync();
        const unsigned char* src = slabs;
        uint32_t column = base;
        for (int q = 0; q < op.count; q++) {
            const int stride = slab_stride(op.cols[q] * static_cast<int>(sizeof(T)));
            bad |= slabs_to_tmem<T, W, CHECK>(src, slab, stride, op.cols[q], column, warp, lane);
            src += kSlabRows * stride;
            column += op.cols[q] * W;
        }
        tmem_wait_store();
        tmem_fence_before_sync();
        bool good = true;
        if constexpr (CHECK)
            good = uniform(__syncthreads_or(bad & live)) == 0;
        else
            __syncthreads();
        tmem_fence_after_sync();
        if (next >= 0) start(next, tid);
        return good;
    }
};

// ---------------------------------------------------------------- table of records
// The records grouped by result column, by a stable counting sort in one block. Every column has a
// whole number of batches, at least `least` of them (padding records). Every warp owns a contiguous chunk of
// the records; their columns are read once and kept in shared memory (16 bits each), and the ranks
// of equal columns inside a warp's 32 come from one match. (HPE, J = 2000, K = 4, N = 100: 15 us
// against 67 us in an earlier 256-thread form that read the index arrays again and again.)
//
// `Source` describes the records x = 0 .. M - 1 before the sort: int key(x, bad) (result column),
// T coefficient(x), int column(x, q) (operand column of factor q); `bad` collects which index
// arrays held values out of range.
constexpr int kTableThreads = 1024;
constexpr int kTableWarps = kTableThreads / 32;

inline size_t table_smem(int64_t M, int N) {
    return (static_cast<size_t>(kTableWarps) * N + 2 * N + 2) * sizeof(int32_t) + static_cast<size_t>(M) * 2;
}

template <typename T, int NF, typename Source>
__global__ void __launch_bounds__(kTableThreads, 1)
gather_table(unsigned char* __restrict__ records, int32_t* __restrict__ n_start, Source source, int M,
             int N, int W, int batch, int least, int ones_column, Status st) {
    constexpr int RB = tmem_record_bytes(sizeof(T), NF);
    extern __shared__ __align__(16) int32_t counts[]; // [warps][N] | starts [N + 1] | totals [N] | keys
    int32_t* starts = counts + kTableWarps * N;
    int32_t* totals = starts + N + 1;
    uint16_t* keys = reinterpret_cast<uint16_t*>(totals + N + 1);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int chunk = ((M + kTableWarps - 1) / kTableWarps + 31) / 32 * 32;
    const int x_lo = min(warp * chunk, M), x_hi = min(x_lo + chunk, M);

    for (int i = tid; i < kTableWarps * N; i += kTableThreads) counts[i] = 0;
    unsigned bad = 0;
    for (int x = tid; x < M; x += kTableThreads) keys[x] = static_cast<uint16_t>(source.key(x, bad));
    for (int b = 0; b < kMaxIndexArrays; b++)
        if (bad >> b & 1) report_bad_index(st, b);
    __syncthreads();
    int32_t* mine = counts + warp * N;
    for (int x = x_lo + lane; x < x_hi; x += 32) atomicAdd(mine + keys[x], 1);
    __syncthreads();
    // counts -> offsets of every warp inside a column (lane = warp)
    for (int n = warp; n < N; n += kTableWarps) {
        const int v = counts[lane * N + n];
        int incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(kFullMask, incl, o);
            if (lane >= o) incl += u;
        }
        counts[lane * N + n] = incl - v;
        if (lane == 31) totals[n] = incl;
    }
    __syncthreads();
    if (warp == 0) { // where every column starts, in records
        int run = 0;
        for (int b0 = 0; b0 <= N; b0 += 32) {
            const int b = b0 + lane;
            const int v = b < N ? max(least, (totals[b] + batch - 1) / batch) * batch : 0;
            int incl = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(kFullMask, incl, o);
                if (lane >= o) incl += u;
            }
            if (b <= N) starts[b] = run + incl - v;
            run += __shfl_sync(kFullMask, incl, 31);
        }
    }
    __syncthreads();
    for (int n = tid; n <= N; n += kTableThreads) n_start[n] = starts[n];
    auto put = [&](int pos, const uint32_t (&w)[RB / 4]) {
        uint4* dst = reinterpret_cast<uint4*>(records + static_cast<size_t>(pos) * RB);
#pragma unroll
        for (int q = 0; q < RB / 16; q++)
            dst[q] = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
    };
    for (int n = tid; n < N; n += kTableThreads) {
        for (int pos = starts[n] + totals[n]; pos < starts[n + 1]; pos++) {
            uint32_t w[RB / 4];
#pragma unroll
            for (int q = 0; q < RB / 4; q++) w[q] = 0;
#pragma unroll
            for (int q = 0; q < NF; q++)
                w[words_of(sizeof(T)) + q / 2] |= static_cast<uint32_t>(ones_column * W) << (q & 1 ? 16 : 0);
            put(pos, w);
        }
    }
    for (int x0 = x_lo; x0 < x_hi; x0 += 32) {
        const int x = x0 + lane;
        const bool live = x < x_hi;
        const int key = live ? keys[x] : -1 - lane;
        const unsigned same = __match_any_sync(kFullMask, key);
        const int rank = __popc(same & ((1u << lane) - 1));
        int pos = 0;
        if (live) pos = starts[key] + mine[key] + rank;
        __syncwarp();
        if (live && rank == 0) mine[key] += __popc(same);
        __syncwarp();
        if (live) {
            uint32_t w[RB / 4];
#pragma unroll
            for (int q = 0; q < RB / 4; q++) w[q] = 0;
            put_coefficient<T>(w, source.coefficient(x));
#pragma unroll
            for (int q = 0; q < NF; q++)
                w[words_of(sizeof(T)) + q / 2] |= static_cast<uint32_t>(source.column(x, q) * W)
                                                  << (q & 1 ? 16 : 0);
            put(pos, w);
        }
    }
}

// ---------------------------------------------------------------- the sums
// A whole 32-byte sector, from a 32-byte boundary on, in one store.
__device__ __forceinline__ void store_sector(double* from, const double (&v)[4]) {
    asm volatile("st.global.v4.f64 [%0], {%1,%2,%3,%4};\n" ::"l"(from), "d"(v[0]), "d"(v[1]), "d"(v[2]), "d"(v[3])
                 : "memory");
}
__device__ __forceinline__ void store_sector(float* from, const float (&v)[8]) {
    asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n" ::"l"(from), "f"(v[0]), "f"(v[1]),
                 "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
                 : "memory");
}

// Writes results to rows, one column after the other, in whole 32-byte sectors (partial ones cost
// L2 five times as much: measured 1.1 against 5 TB/s). A lane keeps its row's last E values, column n
// in held[n mod E] (the switch makes that a constant: shifting the values along took 300
// instructions per column of four rows), and stores them when they end a sector, which depends on the
// row where the row size is no multiple of 32 bytes; what lies before the first or behind the last
// whole sector goes out alone.
template <typename T, int R> struct SectorWriter {
    static constexpr int E = 32 / sizeof(T);
    T held[E][R];

    // The value at `at` (and at + r row_step for the other rows, if live), column J of E, the `run`-th
    // (from 0) that this lane writes in a row; `last`: the run ends here.
    template <int J>
    __device__ __forceinline__ void put(T* at, int64_t row_step, int run, bool last, const T (&now)[R],
                                        const bool (&live)[R]) {
#pragma unroll
        for (int r = 0; r < R; r++) held[J][r] = now[r];
        const int phase = static_cast<int>(reinterpret_cast<size_t>(at) / sizeof(T)) & (E - 1);
        if (phase == E - 1 && run >= E - 1) {
#pragma unroll
            for (int r = 0; r < R; r++) {
                T v[E];
#pragma unroll
                for (int e = 0; e < E; e++) v[e] = held[(J + 1 + e) & (E - 1)][r];
                if (live[r]) store_sector(at + r * row_step - (E - 1), v);
            }
        } else if (phase == E - 1 || last) { // at an end of the run
            const int k = min(phase, run);
#pragma unroll
            for (int e = 0; e < E - 1; e++)
                if (e <= k) {
#pragma unroll
                    for (int r = 0; r < R; r++)
                        if (live[r]) at[r * row_step - e] = held[(J - e) & (E - 1)][r];
                }
            // (a whole sector is complete only with phase == E - 1)
        }
        __syncwarp();
    }
    __device__ __forceinline__ void put(int column, T* at, int64_t row_step, int run, bool last, const T (&now)[R],
                                        const bool (&live)[R]) {
        switch (column & (E - 1)) {
        case 0: put<0>(at, row_step, run, last, now, live); break;
        case 1: put<1>(at, row_step, run, last, now, live); break;
        case 2: put<2>(at, row_step, run, last, now, live); break;
        case 3: put<3>(at, row_step, run, last, now, live); break;
        default:
            if constexpr (E > 4) {
                switch (column & (E - 1)) {
                case 4: put<4>(at, row_step, run, last, now, live); break;
                case 5: put<5>(at, row_step, run, last, now, live); break;
                case 6: put<6>(at, row_step, run, last, now, live); break;
                default: put<7>(at, row_step, run, last, now, live); break;
                }
            }
        }
    }
};

// The records of one warp group, streamed from HBM / L2 through two shared-memory stages filled by
// bulk copies. Batches are fetched into registers ahead of their use, so that the stream does not
// drain between stages. Fetches behind a group's last batch read whatever their place in the ring
// holds, zeros or older records: every column number they find lies inside the tile.
template <int STAGE> struct RecordRing {
    const unsigned char* source;
    int bytes, stages; // of the whole stream
    unsigned char* ring;
    uint64_t* full; // [2]
    int group;
    bool leader;          // the thread that issues the copies
    bool alive = true;    // no copy has failed to arrive
    unsigned filled = 0;  // stages waited for so far (all tiles)
    unsigned before = 0;  // slot of the current tile's first stage

    __device__ RecordRing(unsigned char* ring_, uint64_t* full_, int group_, bool leader_,
                          const unsigned char* source_, int bytes_)
        : source(source_), bytes(bytes_), stages((bytes_ + STAGE - 1) / STAGE), ring(ring_), full(full_),
          group(group_), leader(leader_) {}

    // Once per block, before the first __syncthreads(): zeros the rings of all groups, readies the barriers.
    static __device__ void prepare(unsigned char* rings, uint64_t (*barriers)[2], int tid) {
        if (tid < kTmemGroups * 2) {
            mbarrier_init(&barriers[tid >> 1][tid & 1], 1);
            mbarrier_init_fence();
        }
        for (int x = tid * 16; x < kTmemGroups * 2 * STAGE; x += kTmemThreads * 16)
            *reinterpret_cast<uint4*>(rings + x) = make_uint4(0u, 0u, 0u, 0u);
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    }
    __device__ void fill(int s, unsigned slot) {
        const int left = bytes - s * STAGE;
        const unsigned n = static_cast<unsigned>(left < STAGE ? left : STAGE);
        mbarrier_arrive_expect(full + slot, n);
        bulk_copy_in(ring + slot * STAGE, source + static_cast<size_t>(s) * STAGE, n, full + slot);
    }
    __device__ void start_tile() {
        before = filled & 1;
        if (alive && leader && stages > 0) {
            fill(0, before);
            if (stages > 1) fill(1, before ^ 1);
        }
    }
    // The four warps of the group meet: all of them have fetched the stage before, so its slot is
    // free again. A warp whose copy did not arrive reports it and stops waiting; the others learn
    // of it when they meet next.
    __device__ void enter_stage(int stage, int lane, const Status& st) {
        int all_alive;
        asm volatile("{\n .reg .pred p, q;\n setp.ne.s32 p, %1, 0;\n"
                     " barrier.cta.red.and.pred q, %2, 128, p;\n selp.s32 %0, 1, 0, q;\n}\n"
                     : "=r"(all_alive)
                     : "r"(alive ? 1 : 0), "r"(1 + group)
                     : "memory");
        alive = __all_sync(kFullMask, all_alive != 0) != 0;
        if (alive) {
            if (stage > 0 && stage + 1 < stages && leader) fill(stage + 1, (filled + 1) & 1);
            alive = __all_sync(kFullMask, mbarrier_wait(full + (filled & 1), (filled >> 1) & 1));
            if (!alive && lane == 0) report_stalled(st);
            filled++;
        }
        __syncwarp();
    }
    template <int PIECE> __device__ __forceinline__ const unsigned char* at(int piece) const {
        constexpr int per_stage = STAGE / PIECE; // a power of two
        return ring + ((before * per_stage + piece) & (2 * per_stage - 1)) * PIECE;
    }
};

// The first of `columns` columns that group `which` of `all` works on: the groups split `starts`
// (ascending, starts[c * stride] = first record of column c) evenly.
__device__ __forceinline__ int group_column(const int32_t* starts, int columns, int stride, int which, int all) {
    if (which <= 0) return 0;
    if (which >= all) return columns;
    const int target = static_cast<int>(static_cast<int64_t>(starts[columns * stride]) * which / all);
    int lo = 0, hi = columns;
    while (lo < hi) {
        const int mid = (lo + hi) / 2;
        if (starts[mid * stride] < target)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

// PRODUCTS: the columns [n_lo, n_hi) of a tile with values out_of_band (`normal`: the lane's rows without),
// straight from the table and to the one result.
template <typename T, int W>
__device__ __noinline__ void gather_by_factors(const unsigned char* __restrict__ records, const int32_t* starts, int n_lo,
                                            int n_hi, uint32_t base, unsigned normal, T* out, int columns,
                                            int64_t row0, int64_t I) {
    constexpr int R = W / words_of(sizeof(T)), RB = tmem_record_bytes(sizeof(T), 2);
    for (int n = n_lo; n < n_hi; n++) {
        T sum[R];
#pragma unroll
        for (int r = 0; r < R; r++) sum[r] = T(0);
        const int end = uniform(starts[n + 1]);
        for (int x = uniform(starts[n]); x < end; x++) {
            const uint4 w = __ldg(reinterpret_cast<const uint4*>(records + static_cast<size_t>(x) * RB));
            const T c = __hiloint2double(static_cast<int>(w.y), static_cast<int>(w.x));
            uint32_t a[W], b[W];
            tmem_load(__byte_perm(w.z, base, 0x7610), a);
            tmem_load(__byte_perm(w.z, base, 0x7632), b);
            tmem_wait_load();
            tmem_pin(a);
            tmem_pin(b);
#pragma unroll
            for (int r = 0; r < R; r++) {
                const T va = tmem_value<T>(a, r), vb = tmem_value<T>(b, r);
                const bool products = normal >> r & 1;
                sum[r] = fma(products ? c : c * va, products ? va * vb : vb, sum[r]);
            }
        }
#pragma unroll
        for (int r = 0; r < R; r++)
            if (row0 + r * kSlabRows < I) out[(row0 + r * kSlabRows) * columns + n] = sum[r];
    }
}

// The result columns are split among parts * 4 warp groups by number of records; a group's four
// warps (one per quadrant) walk the same records for their own rows, add them up in registers, and
// store a result when a column ends. `parts` blocks share a tile (they need no reduction).
template <typename T, int NF, int W, bool PRODUCTS = false>
__global__ void __launch_bounds__(kTmemThreads, 1)
gather_sums(const __grid_constant__ Results<T> results, const __grid_constant__ Operands operands,
            const unsigned char* __restrict__ records, const int32_t* __restrict__ n_start, int64_t I,
            int parts, int64_t tiles, Status st) {
    const int N = results.total;
    using G = Batch<T, NF, W>;
    constexpr int B = G::B, R = G::R, RB = G::RB;
    using Ring = RecordRing<2048>; // two stages and four groups: 16 KB
    constexpr int kPerStage = 2048 / (B * RB); // batches
    static_assert(kPerStage % 2 == 0, "pairs of batches do not straddle stages");
    extern __shared__ __align__(16) unsigned char smem[];
    // layout: stages [group][2][2048] | n_start [N + 1], padded | slabs
    int32_t* starts = reinterpret_cast<int32_t*>(smem + 2 * kStageBytes);
    unsigned char* slabs = smem + 2 * kStageBytes + (static_cast<size_t>(N + 1) * 4 + 15) / 16 * 16;
    __shared__ uint32_t tmem_s;
    __shared__ uint64_t full[kTmemGroups][2];
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(kFullMask, tid >> 5, 0), group = warp >> 2;
    const int part = blockIdx.x % parts;
    const int64_t first = blockIdx.x / parts, step = gridDim.x / parts;

    Tiles<T, W> t{operands, I, operands.template slab_bytes<T>(), slabs};
    t.start(first, tid);
    if (warp == 0) tmem_alloc(&tmem_s, kTmemColumns);
    Ring::prepare(smem, full, tid);
    for (int n = tid; n <= N; n += kTmemThreads) starts[n] = __ldg(n_start + n);
    tmem_fence_before_sync();
    __syncthreads();
    tmem_fence_after_sync();
    const uint32_t base = tmem_quadrant(tmem_s, warp);
    t.ones(base, warp);

    // this group's columns [n_lo, n_hi) and records [x_lo, x_hi)
    // (through a shuffle: the compiler then knows that the loops below are warp-uniform)
    const int which = part * kTmemGroups + group, all = parts * kTmemGroups;
    const int n_lo = uniform(group_column(starts, N, 1, which, all));
    const int n_hi = uniform(group_column(starts, N, 1, which + 1, all));
    const int x_lo = uniform(starts[n_lo]), batches = uniform(starts[n_hi] - starts[n_lo]) / B;
    Ring ring(smem + group * 4096, full[group], group, (warp & 3) == 0 && lane == 0,
              records + static_cast<size_t>(x_lo) * RB, batches * B * RB);
    for (int64_t tile = first; tile < tiles; tile += step) {
        const int64_t row0 = tile * (kSlabRows * R) + (warp & 3) * 32 + lane, next = tile + step < tiles ? tile + step : -1;
        bool by_factors = false;
        if constexpr (PRODUCTS) {
            unsigned in_batch = 0; // (rows behind the last one hold anything)
#pragma unroll
            for (int r = 0; r < R; r++) in_batch |= row0 + r * kSlabRows < I ? 1u << r : 0u;
            by_factors = !t.template load<true>(next, base, tid, warp, lane, in_batch);
            if (by_factors)
                gather_by_factors<T, W>(records, starts, n_lo, n_hi, base,
                                        rows_in_band<T, W>(base, operands.total), results.data[0],
                                        results.cols[0], row0, I);
        } else {
            t.load(next, base, tid, warp, lane);
        }
        T acc[R];
        PieceSum<T, R> sum;
        sum.clear();
        bool live[R];
#pragma unroll
        for (int r = 0; r < R; r++) {
            live[r] = row0 + r * kSlabRows < I;
            acc[r] = T(0);
        }
        int n = n_lo, which_result = 0, local = n_lo; // column n = column `local` of that result
        while (which_result + 1 < results.count && local >= results.cols[which_result])
            local -= results.cols[which_result++];
        int lo = local; // first column of this result that is the group's
        SectorWriter<T, R> writer{};
        int cols = results.cols[which_result];
        T* at = results.data[which_result] + row0 * cols + local;
        auto close = [&] { // column n is complete
            sum.finish(acc);
#pragma unroll
            for (int r = 0; r < R; r++)
                if (results.scale && live[r]) acc[r] *= __ldg(results.scale + row0 + r * kSlabRows);
            writer.put(local, at, kSlabRows * static_cast<int64_t>(cols), local - lo,
                       n + 1 == n_hi || local + 1 == cols, acc, live);
#pragma unroll
            for (int r = 0; r < R; r++) acc[r] = T(0);
            n++;
            at++;
            if (++local == cols && n < n_hi) {
                local = lo = 0;
                which_result++;
                cols = results.cols[which_result];
                at = results.data[which_result] + row0 * cols;
            }
        };
        if (batches > 0 && !by_factors) {
            ring.start_tile();
            G x, y;
            Records<T, NF, W> rx, ry;
            // (a column has an even number of batches: it can only end behind a y, and the code that
            // closes it is there once)
            int left = uniform(starts[n_lo + 1] - starts[n_lo]) / (2 * B); // pairs of column n
            constexpr int kPairs = kPerStage / 2;                          // of a stage
            // Pairs are counted down to the end of a stage, or looked at by their number: which is shorter depends on
            // what else the compiler keeps in registers. One gradient, 300 000 rows, 20 x 6 -> 50, 12 000 triplets,
            // f64, four rows' columns: 1157 us counted, 934 not; two more columns per load 234 and 250, f32 598 and
            // 643, products first 686 and 780; hpe_large (3 factors) 3950 and 4320.
            constexpr bool kCounted = PRODUCTS || sizeof(T) == 4 || NF != 2 || W != 4;
            int stage = 0, in_stage = kPairs; // pairs until the batches fetched ahead are the next stage's
            ring.enter_stage(0, lane, st);
            const unsigned char* ahead = ring.template at<B * RB>(0);
            fetch<T, NF, W>(rx, ahead);
            issue<T, NF, W>(x, rx, base);
            fetch<T, NF, W>(ry, ahead + B * RB);
            for (int i = 0; kCounted || i < batches; i += 2) {
                await<T, NF, W>(x);
                issue<T, NF, W>(y, ry, base);
                add_terms<T, NF, W, PRODUCTS>(x, rx, acc);
                if constexpr (kCounted) {
                    ahead += 2 * B * RB;
                    if (__builtin_expect(--in_stage == 0, 0)) {
                        if (i + 2 < batches) ring.enter_stage(++stage, lane, st);
                        ahead = ring.template at<B * RB>(i + 2);
                        in_stage = kPairs;
                    }
                } else {
                    if ((i & (kPerStage - 1)) == kPerStage - 2 && i + 2 < batches)
                        ring.enter_stage((i + 2) / kPerStage, lane, st);
                    ahead = ring.template at<B * RB>(i + 2);
                }
                fetch<T, NF, W>(rx, ahead);
                await<T, NF, W>(y);
                issue<T, NF, W>(x, rx, base);
                add_terms<T, NF, W, PRODUCTS>(y, ry, acc);
                sum.template piece<B>(i, acc);
                if (__builtin_expect(--left == 0, 0)) {
                    close();
                    if (kCounted && n == n_hi) break; // (the last column ends with the last batch)
                    left = kCounted || n < n_hi ? uniform(starts[n + 1] - starts[n]) / (2 * B) : 0;
                }
                fetch<T, NF, W>(ry, ahead + B * RB);
            }
            await<T, NF, W>(x);
        }
        tmem_fence_before_sync();
        __syncthreads(); // before the next tile overwrites TMEM
        tmem_fence_after_sync();
    }
    cp_async_wait<0>();
    __syncthreads();
    if (warp == 0) tmem_free(tmem_s, kTmemColumns);
}

// ---------------------------------------------------------------- dispatch
// A batch that gives every SM a tile of 128 rows. There a tile's way through shared memory into TMEM
// and back (about 25 us for 512 rows of 76 columns, hardly overlapped with the sums: one block per
// SM) has to be earned back by its gathers; smaller batches gain from the split of the records.
inline bool fills_gpu(const Call& call, int64_t I) {
    return I >= static_cast<int64_t>(sm_count(call.device)) * kSlabRows;
}

struct GatherShape {
    int w, parts;
    int64_t tiles;
    size_t smem;
};

// Rows per lane and blocks per tile for a problem, by estimated clocks: a record costs a
// sub-partition about 4 + 3 NF issue slots and NF operations per row (two slots each in f64, whose
// pipe takes a warp in two clocks); a tile costs its way into TMEM; whole waves count. Wide lanes
// (more rows per record read) win for large batches, narrow ones and several blocks per tile for
// batches that cannot fill the GPU. `column` is the granularity of a part (records of one result
// column), 0 where the records can be cut anywhere.
template <typename T>
bool choose_gather_shape(const Call& call, int64_t I, const Operands& op, double records, int nf,
                         int max_w, int max_parts, bool power_of_two_parts, double column, size_t fixed_smem,
                         GatherShape& best) {
    const int sms = sm_count(call.device);
    const size_t limit = static_cast<size_t>(max_optin_smem(call.device)) - 1024;
    const size_t slab = static_cast<size_t>(op.template slab_bytes<T>());
    double best_cost = -1;
    for (int w : {8, 4, 2}) {
        if (w > max_w || (op.total + 1) * w > kTmemColumns || nf * w > 32) continue;
        const int r = w / words_of(sizeof(T));
        if (fixed_smem + r * slab > limit) continue;
        const int64_t tiles = ceil_div(I, static_cast<int64_t>(kSlabRows) * r);
        const double record = 4 + 3 * nf + nf * r * (sizeof(T) == 8 ? 2 : 1);
        for (int parts = 1; parts <= max_parts; parts = power_of_two_parts ? parts * 2 : parts + 1) {
            const double waves = static_cast<double>(ceil_div(tiles * parts, sms));
            double share = records / parts;
            if (column > 0) share = std::max(share, std::ceil(records / column / (4 * parts)) * 4 * column);
            // (blocks of a cluster wait for one another at both ends of every tile)
            const double together = power_of_two_parts && parts > 1 && waves > 1 ? 2500 : 0;
            const double cost = waves * (share * record + 1500 + together + 4.0 * op.total * r);
            if (best_cost < 0 || cost < best_cost) {
                best_cost = cost;
                best = {w, parts, tiles, fixed_smem + r * slab};
            }
        }
    }
    return best_cost >= 0;
}

template <typename Kernel, typename... Args>
void launch_gather(const Call& call, Kernel kernel, const GatherShape& s, int cluster, Args... args) {
    // More than half of an SM's shared memory: one block per SM, which owns all of its TMEM.
    const size_t smem = std::max<size_t>(s.smem, 117 * 1024);
    allow_dynamic_smem(kernel, call.device, smem);
    const int64_t at_once = std::max<int64_t>(1, sm_count(call.device) / s.parts);
    cudaLaunchConfig_t config{};
    config.gridDim = dim3(static_cast<unsigned>(std::min(s.tiles, at_once) * s.parts));
    config.blockDim = dim3(kTmemThreads);
    config.dynamicSmemBytes = smem;
    config.stream = call.stream;
    cudaLaunchAttribute attribute{};
    attribute.id = cudaLaunchAttributeClusterDimension;
    attribute.val.clusterDim.x = static_cast<unsigned>(cluster);
    attribute.val.clusterDim.y = attribute.val.clusterDim.z = 1;
    config.attrs = &attribute;
    config.numAttrs = cluster > 1 ? 1 : 0;
    MOPS_CUDA_OK(cudaLaunchKernelEx(&config, kernel, args...));
}

// Builds (or takes from the plan) the table of M records over results.total columns and runs the
// sums. `key` names the table: kind, arrays and sizes; n[8], n[9] are filled in here. Returns
// false when the problem does not fit (operands too wide for TMEM, too many records to sort).
template <typename T, int NF, bool PRODUCTS = false, typename Source>
bool run_gather(const Call& call, TableKey key, const Source& source, int64_t M, const Operands& op,
                const Results<T>& results, int64_t I, const char* name) {
    constexpr int RB = tmem_record_bytes(sizeof(T), NF);
    const int N = results.total;
    const size_t builder = table_smem(M, N);
    if (N == 0 || builder > static_cast<size_t>(max_optin_smem(call.device)) - 1024) return false;
    GatherShape s{};
    const size_t fixed = 2 * kStageBytes + (static_cast<size_t>(N + 1) * 4 + 15) / 16 * 16;
    if (!choose_gather_shape<T>(call, I, op, static_cast<double>(M), NF, sizeof(T) == 8 ? 8 : 4, std::max(1, std::min(32, N / 4)),
                                false, static_cast<double>(M) / N, fixed, s))
        return false;
    const int batch = 2 * batch_of(NF, s.w); // columns end behind a pair of batches
    const size_t b_rec = (static_cast<size_t>(M) + static_cast<size_t>(N) * batch) * RB;
    const size_t b_n = (static_cast<size_t>(N) + 1) * sizeof(int32_t);
    key.scalar_bytes = static_cast<int>(sizeof(T));
    key.n[8] = s.w, key.n[9] = NF;
    TableRef ref = acquire_table(call, key, b_rec + b_n);
    unsigned char* records = static_cast<unsigned char*>(ref.ptr);
    int32_t* n_start = reinterpret_cast<int32_t*>(records + b_rec);
    if (ref.fresh) {
        auto build = gather_table<T, NF, Source>;
        allow_dynamic_smem(build, call.device, builder);
        build<<<1, kTableThreads, builder, call.stream>>>(records, n_start, source, static_cast<int>(M), N,
                                                          s.w, batch, 1, op.total, call.status);
        MOPS_CUDA_OK(cudaGetLastError());
        commit_table(call, ref);
    }
    note_kernel_f("%s<%s,NF=%d,W=%d> parts=%d", name, scalar_name<T>(), NF, s.w, s.parts);
    auto go = [&](auto kernel) {
        launch_gather(call, kernel, s, 1, results, op, static_cast<const unsigned char*>(records),
                      static_cast<const int32_t*>(n_start), I, s.parts, s.tiles, call.status);
    };
    if (s.w == 8) {
        if constexpr (NF * 8 <= 32 && sizeof(T) == 8) go(gather_sums<T, NF, 8, PRODUCTS>);
    } else if (s.w == 4) {
        go(gather_sums<T, NF, 4, PRODUCTS>);
    } else {
        go(gather_sums<T, NF, 2, PRODUCTS>);
    }
    release_table(call, ref);
    return true;
}

} // namespace
} // namespace mops_b200

#endif
