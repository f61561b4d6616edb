// Sparse accumulation of products with the batch rows in tensor memory (gather_tmem.cuh): forward,
// VJP and second-order VJP. Every result column is a sum of records with two factors:
//
//   O[o]    : C A[PA] B[PB]                      (PO = o)
//   gA[a]   : C gO[PO] B[PB]                     (PA = a)     gB[b]  : C gO[PO] A[PA]   (PB = b)
//   ggO[o]  : C ggA[PA] B[PB] + C A[PA] ggB[PB]  (PO = o)
//   gA2[a]  : C gO[PO] ggB[PB]                   (PA = a)     gB2[b] : C gO[PO] ggA[PA] (PB = b)
//
// 2^22 rows, 20 x 6 -> 50, 1000 triplets, f64, against the kernels that gather from shared memory:
// forward 2.99 -> 1.6 ms, VJP 3.04 -> 2.6 ms (a tile's way in and out takes nearly half of that: the
// time per triplet is 3 times less). 1000 rows: forward 12 -> 9 us, VJP 39 -> 13 us, second order
// 109 -> 19 us.
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

// Fewer triplets per column of a large batch than this and the kernels of sap.cu are as fast
// (measured at 76 columns, f64: the lines cross at about 260 triplets in the forward, 770 in the VJP).
constexpr int kForwardTriplets = 4, kBackwardTriplets = 10; // per column

template <typename T>
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
    return run_gather<T, 2>(call, key, source, p.K * count, op, results, p.I, name);
}

// ---------------------------------------------------------------- VJP by cells
// With S the narrower of A, B and T the wider one, both gradients are sums over the cells (t, s) of
//
//   X = sum of C gO[PO] over the triplets of the cell:    gT[t] += X S[s],    gS[s] += X T[t],
//
// so a triplet costs one gather and one FMA per row instead of two records of two factors. The
// cells are sorted by t, then s; a warp group owns whole t: gT[t] is summed in registers, gS in
// shared memory, by every group for itself, and the groups' sums are added at the end of a tile.
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

// Operands: gO (nO columns), T, S; starts[t * nS + s] in records.
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

template <typename T>
bool backward_cells(const Call& call, const SapProblem<T>& p, T* gA, T* gB, const T* gO) {
    const bool b_narrow = p.nB <= p.nA;
    const int nS = b_narrow ? p.nB : p.nA, nT = b_narrow ? p.nA : p.nB, cells = nS * nT;
    const size_t builder = table_smem(p.K, cells);
    if (builder > static_cast<size_t>(max_optin_smem(call.device)) - 1024) return false;
    Operands op{};
    op.add(gO, p.nO);
    op.add(b_narrow ? p.A : p.B, nT);
    op.add(b_narrow ? p.B : p.A, nS);
    // rows per lane: as many as fit and still give every SM a tile
    int w = 0;
    int64_t tiles = 0;
    size_t smem = 0;
    for (int candidate : {4, 2}) {
        const int r = candidate / words_of(sizeof(T));
        tiles = ceil_div(p.I, static_cast<int64_t>(kSlabRows) * r);
        smem = kStageBytes + (static_cast<size_t>(cells + 1) * 4 + 15) / 16 * 16 +
               static_cast<size_t>(kTmemGroups) * nS * kSlabRows * r * sizeof(T) +
               static_cast<size_t>(r) * op.template slab_bytes<T>();
        if ((op.total + 1) * candidate <= kTmemColumns &&
            smem <= static_cast<size_t>(max_optin_smem(call.device)) - 1024 &&
            tiles >= sm_count(call.device)) {
            w = candidate;
            break;
        }
    }
    if (w == 0) return false;
    const int batch = batch_of(1, w);
    constexpr int RB = tmem_record_bytes(sizeof(T), 1);
    const size_t b_rec = (static_cast<size_t>(p.K) + static_cast<size_t>(cells) * batch) * RB;
    TableKey key{};
    key.kind = kSapTable;
    key.scalar_bytes = static_cast<int>(sizeof(T));
    key.ptr[0] = p.C, key.ptr[1] = p.PA, key.ptr[2] = p.PB, key.ptr[3] = p.PO;
    key.n[0] = p.K, key.n[1] = p.nA, key.n[2] = p.nB, key.n[3] = p.nO, key.n[4] = -1, key.n[8] = w;
    TableRef ref = acquire_table(call, key, b_rec + (static_cast<size_t>(cells) + 1) * sizeof(int32_t));
    unsigned char* records = static_cast<unsigned char*>(ref.ptr);
    int32_t* starts = reinterpret_cast<int32_t*>(records + b_rec);
    if (ref.fresh) {
        auto build = gather_table<T, 1, CellSource<T>>;
        allow_dynamic_smem(build, call.device, builder);
        const CellSource<T> source{p.C, b_narrow ? p.PA : p.PB, b_narrow ? p.PB : p.PA, p.PO, nT, nS, p.nO,
                                   b_narrow ? 0 : 1, b_narrow ? 1 : 0};
        build<<<1, kTableThreads, builder, call.stream>>>(records, starts, source, static_cast<int>(p.K),
                                                          cells, w, batch, 0, op.total, call.status);
        MOPS_CUDA_OK(cudaGetLastError());
        commit_table(call, ref);
    }
    note_kernel_f("sap_vjp_cells<%s,W=%d>", scalar_name<T>(), w);
    const GatherShape shape{w, 1, tiles, smem};
    auto go = [&](auto kernel) {
        launch_gather(call, kernel, shape, 1, b_narrow ? gA : gB, b_narrow ? gB : gA, op,
                      static_cast<const unsigned char*>(records), static_cast<const int32_t*>(starts), p.I,
                      tiles, call.status);
    };
    if (w == 4)
        go(sap_vjp_cells<T, 4>);
    else
        go(sap_vjp_cells<T, 2>);
    release_table(call, ref);
    return true;
}

} // namespace

template <typename T> bool sap_forward_tmem(const Call& call, const SapProblem<T>& p, T* O) {
    if (fills_gpu(call, p.I) && p.K < kForwardTriplets * static_cast<int64_t>(p.nA + p.nB + p.nO)) return false;
    Operands op{};
    op.add(p.A, p.nA);
    op.add(p.B, p.nB);
    Results<T> results{};
    results.add(O, p.nO);
    const Family f[] = {{kO, 0, {kA, kB}, {0, p.nA}}};
    return run(call, p, f, 1, op, results, 0, "sap_fwd_tmem");
}

template <typename T>
bool sap_backward_tmem(const Call& call, const SapProblem<T>& p, T* gA, T* gB, const T* gO) {
    if (fills_gpu(call, p.I) && p.K < kBackwardTriplets * static_cast<int64_t>(p.nA + p.nB + p.nO)) return false;
    // Both gradients of a batch with a tile for every SM: by cells.
    if (gA != nullptr && gB != nullptr && backward_cells(call, p, gA, gB, gO)) return true;
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
