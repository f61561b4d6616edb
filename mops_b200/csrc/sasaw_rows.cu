// Sparse accumulation scatter-add with weights, row by row with the coupling applied per row and
// not per edge. With D[m3,m2,m1] the coupling as a dense table and lane = column b:
//
//   forward      G_i[m1,m2,b] = sum over the edges e of row i of A[e,m1] B[e,b] W[J_e,m2,b]
//                O[i,m3,b]    = sum_{m1,m2} D[m3,m2,m1] G_i[m1,m2,b]
//   gradients, with the edges in the order of J (row j of W):
//                F_j[m1,m3,b] = sum over the edges e with J_e = j of A[e,m1] B[e,b] gO[I_e,m3,b]
//                gW[j,m2,b]   = sum_{m1,m3} D[m3,m2,m1] F_j[m1,m3,b]
//                E_j[m1,m3,b] = sum_m2 D[m3,m2,m1] W[j,m2,b]
//                Z[m1,b]      = sum_m3 E_j[m1,m3,b] gO[I_e,m3,b]
//                gB[e,b]      = sum_m1 A[e,m1] Z[m1,b],      gA[e,m1] = sum_b B[e,b] Z[m1,b]
//
// G, F and E stay in registers while a warp walks the edges of a row, so that an edge costs
// nA x nW (forward) or 2 nA x nO (gradients) multiply-adds per column and nothing else: no coupling
// matrix per edge, no reduction over lanes but the nA sums of gA, no atomics (gW is a sum over a row)
// and hence no dependence on the order of I. The coupling costs nA x nW x nO per row and column,
// shared by the row's edges. The gathered rows (of W, of gO) come through a ring of asynchronous
// copies in shared memory, eight edges deep, into which every lane copies what it will read itself.
//
// What bounds them: latency at two warps per scheduler (the sums take 162 registers per lane), the FP64
// pipe then 39 % (sums) and 25 % (edge gradients) busy, issue slots 44 %; L2 or DRAM where the
// gathered table is large. Against the kernels of sasaw.cu, sums and gradients, 9 x 9 x 9 channels:
// f32 250 000 edges, 64 columns 0.44 + 1.13 -> 0.14 + 0.36 ms; f64 60 000 edges, 32 columns 70 + 148
// -> 45 + 120 us. Half the products per warp and three warps per scheduler were slower (62 -> 111 us):
// what an edge costs beside its products then counts twice.
#include <algorithm>
#include <cmath>
#include <initializer_list>
#include <type_traits>

#include "checks.hpp"
#include "sasaw_rows.hpp"
#include "unsorted.cuh"

namespace mops_b200 {
namespace {

enum { kBitI = 0, kBitM1 = 1, kBitJ = 2, kBitM2 = 3, kBitM3 = 4 };
constexpr int kWidest = 16;
constexpr int kDepth = 8; // steps in the ring
constexpr int kRowWarps = 8;
constexpr int kTableOut = 3; // outputs contracted together

// One 64-bit (or 32-bit) element per lane: a double, two floats, or a float.
template <typename T, int VEC> struct Pack;
template <typename T> struct Pack<T, 1> {
    using V = T;
    static __device__ __forceinline__ V dup(T x) { return x; }
    static __device__ __forceinline__ V fma(V a, V b, V c) { return a * b + c; }
    static __device__ __forceinline__ V mul(V a, V b) { return a * b; }
    static __device__ __forceinline__ V add(V a, V b) { return a + b; }
    static __device__ __forceinline__ T sum(V a) { return a; }
    static __device__ __forceinline__ V shift(V a, int o) { return __shfl_xor_sync(kFullMask, a, o); }
    static __device__ __forceinline__ void add_at(T* p, V a) { red_add(p, a); }
};
template <> struct Pack<float, 2> { // FFMA2: two multiply-adds per instruction
    using V = unsigned long long;
    static __device__ __forceinline__ V dup(float x) {
        V v;
        asm("mov.b64 %0, {%1, %1};" : "=l"(v) : "f"(x));
        return v;
    }
    static __device__ __forceinline__ V fma(V a, V b, V c) {
        V d;
        asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
        return d;
    }
    static __device__ __forceinline__ V mul(V a, V b) {
        V d;
        asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
        return d;
    }
    static __device__ __forceinline__ V add(V a, V b) {
        V d;
        asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
        return d;
    }
    static __device__ __forceinline__ float sum(V a) {
        float x, y;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a));
        return x + y;
    }
    static __device__ __forceinline__ V shift(V a, int o) { return __shfl_xor_sync(kFullMask, a, o); }
    static __device__ __forceinline__ void add_at(float* p, V a) {
        float x, y;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a));
        red_add(p, x);
        red_add(p + 1, y);
    }
};

// ---- the dense coupling table D[out][a][c], padded with zeros: `out` is m3 (forward) or m2
// (gradients), c the other one. A warp per entry of the table, lanes over the coupling entries in a
// fixed order, so the sums are reproducible. A block turns the coupling's indices into places in the table
// once, in shared memory (each warp by itself, from global memory: 9.6 us for 729 places and 500 entries).
template <typename T>
__global__ void __launch_bounds__(256)
sasaw_dense_table(T* __restrict__ D, const T* __restrict__ C, const int32_t* __restrict__ M1,
                  const int32_t* __restrict__ M2, const int32_t* __restrict__ M3, int64_t N, int nA, int nW,
                  int nO, bool out_is_m2, int pad_out, int pad_a, int pad_c, Status st) {
    constexpr int kAtOnce = 1024;
    __shared__ int32_t places[kAtOnce];
    const int lane = threadIdx.x & 31;
    const int slot = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    T sum = T(0);
    for (int64_t n0 = 0; n0 < N; n0 += kAtOnce) {
        const int count = N - n0 < kAtOnce ? static_cast<int>(N - n0) : kAtOnce;
        for (int x = threadIdx.x; x < count; x += blockDim.x) {
            int32_t m1 = __ldg(M1 + n0 + x), m2 = __ldg(M2 + n0 + x), m3 = __ldg(M3 + n0 + x);
            const bool b1 = clamp_index(m1, nA), b2 = clamp_index(m2, nW), b3 = clamp_index(m3, nO);
            if (blockIdx.x == 0) {
                if (b1) report_bad_index(st, kBitM1);
                if (b2) report_bad_index(st, kBitM2);
                if (b3) report_bad_index(st, kBitM3);
            }
            places[x] = ((out_is_m2 ? m2 : m3) * pad_a + m1) * pad_c + (out_is_m2 ? m3 : m2);
        }
        __syncthreads();
#pragma unroll 4
        for (int x = lane; x < count; x += 32)
            if (places[x] == slot) sum += __ldg(C + n0 + x);
        __syncthreads();
    }
    sum = warp_sum(sum);
    if (lane == 0 && slot < pad_out * pad_a * pad_c) D[slot] = sum;
}

// ---- walking the edges of a range of rows
template <typename T> struct RowsArgs {
    const T *A, *B, *G;          // [E][nA], [E][L], gathered rows [rows][nC][L]
    const int32_t* gather;       // [E] row of G
    const int32_t* perm;         // order of the edges; nullptr: as they are
    const T* D;                  // table [pad_out][NA][pad_c]
    int64_t rows;
    int nA, nC, nOut, L;
    int pad_out, pad_a, pad_c;
    int lanes;                   // lanes per edge (a power of two); 32 / lanes edges side by side
    int bit;                     // status bit of `gather`
    const int32_t* longest;      // with a permutation: where its rows are longer than `limit`, they are
    int limit, chunk;            // taken in chunks of this many edges, whatever rows these belong to
    int piece_at, piece_room;    // shared memory for the sums of so many pieces (Pieces)
};

// Some rows. kCut: and of their edges those at positions [p_lo, p_hi); other warps have others, so that sums
// are added to what is there. kPiece: the same, of a block's own rows; the sums of a first row that another warp
// has begun (`head`) go to shared memory, where the block adds them up. (Instantiated for each: with the choice at run time the even
// case took 3 % longer, f32, 250 000 edges.)
enum Cut { kWhole = 0, kCut = 1, kPiece = 2 };
template <Cut CUT> struct Part {
    int64_t row_lo, row_hi;
    int p_lo, p_hi;
    unsigned char* head;
};
template <> struct Part<kWhole> {
    int64_t row_lo, row_hi;
};

// One slot of a warp's ring: NC rows of 32 lanes, B, the A rows of the edges side by side, their numbers.
template <typename T, int VEC, int NA, int NC> struct Slot {
    using V = typename Pack<T, VEC>::V;
    static constexpr int kB = NC * 32 * sizeof(V);
    static constexpr int kA = kB + 32 * sizeof(V);
    static constexpr int kRow = (NA * sizeof(T) + 15) / 16 * 16; // bytes of an A row
    // (rounded up so that A rows start at a multiple of 128 bytes: kB and kA are multiples, too)
    static __host__ __device__ constexpr int bytes(int side_by_side) {
        return (kA + side_by_side * kRow + (side_by_side * 4 + 15) / 16 * 16 + 127) / 128 * 128;
    }
};

template <int BYTES, int OFFSET> __device__ __forceinline__ void cp_async_at(unsigned dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0 + %1], [%2], %3;\n" ::"r"(dst), "n"(OFFSET), "l"(src), "n"(BYTES)
                 : "memory");
}
__device__ __forceinline__ void cp_async16(unsigned dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
}
template <int BYTES, int STEP, int C, int N>
__device__ __forceinline__ void cp_async_rows(unsigned dst, const unsigned char* src, int64_t row_bytes) {
    if constexpr (C < N) {
        cp_async_at<BYTES, C * STEP>(dst, src + C * row_bytes);
        cp_async_rows<BYTES, STEP, C + 1, N>(dst, src, row_bytes);
    }
}

// How a warp takes the edges: several side by side (L <= 16 columns and f64 or f32 of one column per lane),
// one at a time, or one at a time with L = 32 VEC columns and operands at 16-byte boundaries (then
// every offset is a constant and the copies are whole 16-byte pieces).
enum Mode { kSideBySide = 0, kOneEdge = 1, kExact = 2 };

// Walks a part for columns [b0, ...) and c in [c0, c0 + nc): begin(row), step(w[NC] and B
// of this lane, A row, edge, live), end(row) in order. All lanes together.
//
// One edge at a time the copies do not care about rows: they run along the positions, and a step is
// straight-line code (wait, start the copies of the step seven ahead, read, multiply), which the
// compiler can interleave: at 9 x 9 channels, f64, 337 -> 210 instructions per edge of the sums,
// 640 -> 450 us at 10^6 edges.
template <typename T, int VEC, int NA, int NC, Mode MODE, typename Off, Cut CUT, typename Begin, typename Step,
          typename End>
__device__ __forceinline__ void walk_rows(const RowsArgs<T>& g, const Off* __restrict__ offsets,
                                          const Part<CUT>& part, int b0, int c0, unsigned char* ring, int lane,
                                          const Status& st, Begin&& begin, Step&& step, End&& end) {
    using P = Pack<T, VEC>;
    using V = typename P::V;
    using Sl = Slot<T, VEC, NA, NC>;
    constexpr bool kSide = MODE == kSideBySide;
    const int LP = kSide ? g.lanes : 32, S = kSide ? 32 / LP : 1;
    const int sub = kSide ? lane / LP : 0, lb = kSide ? lane & (LP - 1) : lane;
    const int L = MODE == kExact ? 32 * VEC : g.L;
    const int nc = g.nC - c0 < NC ? g.nC - c0 : NC;
    const int b = MODE == kExact ? lane * VEC : b0 + lb * VEC;
    const bool valid = MODE == kExact || b < L;
    const int bc = valid ? b : L - VEC; // lanes beyond the last column read it again, with B = 0
    const int slot_bytes = kSide ? Sl::bytes(S) : Sl::bytes(1);
    const unsigned ring32 = static_cast<unsigned>(__cvta_generic_to_shared(ring));
    const unsigned lane_off = lane * static_cast<unsigned>(sizeof(V));
    // what no copy writes: channels beyond nc and nA, B of the lanes beyond the last column
    for (int x = lane * 4; x < kDepth * slot_bytes; x += 128) *reinterpret_cast<int*>(ring + x) = 0;
    __syncwarp();

    const int64_t row_lo = part.row_lo, row_hi = part.row_hi;
    int p_lo = static_cast<int>(offsets[row_lo]), p_hi = static_cast<int>(offsets[row_hi]);
    if constexpr (CUT != kWhole) p_lo = max(p_lo, part.p_lo), p_hi = min(p_hi, part.p_hi);
    auto row_end = [&](int64_t row) {
        const int end = static_cast<int>(offsets[row + 1]);
        return CUT != kWhole ? min(end, p_hi) : end;
    };
    // Edge numbers and gathered rows, 32 positions per register: the block that the copies have
    // reached (0), the next (1), and of the one after that the edge numbers only (2).
    auto load_edge = [&](int base) {
        int e = min(base + lane, p_hi - 1);
        if (g.perm != nullptr) e = __ldg(g.perm + e);
        return e;
    };
    auto load_row = [&](int e) {
        int32_t r = __ldg(g.gather + e);
        if (clamp_index(r, static_cast<int32_t>(g.rows))) report_bad_index(st, g.bit);
        return r;
    };
    int block = p_lo;
    int e0 = 0, e1 = 0, e2 = 0, g0 = 0, g1 = 0;
    if (p_lo < p_hi) {
        e0 = load_edge(block), e1 = load_edge(block + 32), e2 = load_edge(block + 64);
        g0 = load_row(e0), g1 = load_row(e1);
    }
    auto next_block = [&] {
        block += 32;
        e0 = e1, g0 = g1, e1 = e2;
        g1 = load_row(e1);
        e2 = load_edge(block + 64);
    };
    constexpr int64_t kScalar = sizeof(T);
    const unsigned char* g_base = reinterpret_cast<const unsigned char*>(g.G + static_cast<int64_t>(c0) * L + bc);
    // (row sizes fit 32 bits, rows_apply: an address is one multiply-add)
    const int g_row = g.nC * L * static_cast<int>(kScalar), l_row = L * static_cast<int>(kScalar);
    const int a_size = g.nA * static_cast<int>(kScalar);
    const unsigned char* b_base = reinterpret_cast<const unsigned char*>(g.B + bc);
    const unsigned char* a_base = reinterpret_cast<const unsigned char*>(g.A + lb);
    const unsigned char* g_piece = reinterpret_cast<const unsigned char*>(g.G + static_cast<int64_t>(c0) * L) + lane * 16;
    const unsigned char* b_piece = reinterpret_cast<const unsigned char*>(g.B) + lane * 16;
    constexpr int kStep = 32 * sizeof(V);
    auto copy_edge = [&](int slot, int e, int r) { // W (or gO) row and B
        if constexpr (MODE == kExact) {
            // Both are contiguous, and so are their places in the slot: 16-byte pieces, spread over
            // the lanes (gradients of 4.2 10^6 edges, f64: 3.05 -> 2.91 ms).
            constexpr int kPieces = Sl::kB / 16, kAll = Sl::kA / 16; // with B
            const unsigned to = ring32 + slot + lane * 16;
            const unsigned char* g_src = g_piece + static_cast<int64_t>(r) * g_row;
            const unsigned char* b_src = b_piece + static_cast<int64_t>(e) * l_row;
            if (nc == NC) {
#pragma unroll
                for (int i = 0; i < kAll; i += 32) {
                    const bool in_row = i + 32 <= kPieces || i + lane < kPieces;
                    const unsigned char* src = in_row ? g_src + i * 16 : b_src + (i - kPieces) * 16;
                    if (i + 32 <= kAll || i + lane < kAll) cp_async16(to + i * 16, src);
                }
            } else {
                for (int i = lane; i < nc * (kStep / 16); i += 32)
                    cp_async16(ring32 + slot + i * 16, g_src + (i - lane) * 16);
                if (lane < kStep / 16) cp_async16(to + Sl::kB, b_src);
            }
            return;
        }
        const unsigned dst = ring32 + slot + lane_off;
        const unsigned char* src = g_base + static_cast<int64_t>(r) * g_row;
        if (nc == NC) {
            cp_async_rows<sizeof(V), kStep, 0, NC>(dst, src, l_row);
        } else {
            for (int c = 0; c < nc; c++) cp_async_at<sizeof(V), 0>(dst + c * kStep, src + c * l_row);
        }
        if (valid) cp_async_at<sizeof(V), Sl::kB>(dst, b_base + static_cast<int64_t>(e) * l_row);
    };

    // the copies: the next step to start
    int64_t f_row = row_lo;
    int f_p = p_lo, f_end = row_lo < row_hi ? row_end(row_lo) : p_lo;
    auto start = [&](int slot) { // slot: byte offset in the ring
        if constexpr (!kSide) { // (behind the last edge it is copied again: nobody reads it)
            const int at = f_p - block;
            const int e = __shfl_sync(kFullMask, e0, at), r = __shfl_sync(kFullMask, g0, at);
            copy_edge(slot, e, r);
            if (lb < g.nA)
                cp_async<sizeof(T)>(ring + slot + Sl::kA + lb * sizeof(T), a_base + static_cast<int64_t>(e) * a_size);
            if (lane == 0) *reinterpret_cast<int*>(ring + slot + Sl::kA + Sl::kRow) = e;
            f_p++;
        } else {
            while (f_p >= f_end && f_row + 1 < row_hi) {
                f_row++;
                f_end = row_end(f_row);
            }
            if (f_p < f_end) {
                if (f_p >= block + 32) next_block();
                const bool live = f_p + sub < f_end; // (a repeated edge counts as A = 0)
                const int at = (live ? f_p + sub : f_end - 1) - block;
                const int ea = __shfl_sync(kFullMask, e0, at & 31), eb = __shfl_sync(kFullMask, e1, at & 31);
                const int ra = __shfl_sync(kFullMask, g0, at & 31), rb = __shfl_sync(kFullMask, g1, at & 31);
                const int e = at < 32 ? ea : eb, r = at < 32 ? ra : rb;
                copy_edge(slot, e, r);
                unsigned char* a = ring + slot + Sl::kA + sub * Sl::kRow;
                const unsigned char* a_src = a_base + static_cast<int64_t>(e) * a_size;
                for (int x = lb; x < g.nA; x += LP) {
                    if (live)
                        cp_async<sizeof(T)>(a + x * sizeof(T), a_src + (x - lb) * kScalar);
                    else
                        *reinterpret_cast<T*>(a + x * sizeof(T)) = T(0);
                }
                if (lb == 0) *reinterpret_cast<int*>(ring + slot + Sl::kA + S * Sl::kRow + sub * 4) = e;
                f_p = min(f_p + S, f_end);
            }
        }
        cp_async_commit();
    };
    if (p_lo < p_hi) {
#pragma unroll 1
        for (int s = 0; s < kDepth - 1; s++) start(s * slot_bytes);
    }

    int slot = 0, before = (kDepth - 1) * slot_bytes; // byte offsets of this step's slot and the last one's
    int lo = p_lo;
    for (int64_t row = row_lo; row < row_hi; row++) {
        const int hi = row_end(row);
        const bool any = lo < hi;
        begin(row, any);
#pragma unroll 1
        for (int p = lo; p < hi; p += S) {
            cp_async_wait<kDepth - 2>();
            __syncwarp();
            start(before);
            V w[NC];
            const unsigned char* from = ring + slot;
#pragma unroll
            for (int c = 0; c < NC; c++)
                w[c] = *reinterpret_cast<const V*>(from + lane_off + c * (32 * sizeof(V)));
            const V bv = *reinterpret_cast<const V*>(from + lane_off + Sl::kB);
            const T* a = reinterpret_cast<const T*>(from + Sl::kA + sub * Sl::kRow);
            const int* e = reinterpret_cast<const int*>(from + Sl::kA + S * Sl::kRow) + sub;
            step(w, bv, a, e, !kSide || p + sub < hi);
            before = slot;
            slot += slot_bytes;
            if (slot == kDepth * slot_bytes) slot = 0;
            if (!kSide && f_p == block + 32) next_block();
        }
        end(row, any);
        lo = hi;
    }
    cp_async_wait<0>();
    __syncwarp();
}

// The A row of an edge in registers (16-byte loads).
template <typename T, int NA> __device__ __forceinline__ void load_a(const T* a, T (&out)[NA]) {
    constexpr int N = 16 / sizeof(T);
#pragma unroll
    for (int x = 0; x < NA; x += N) {
        T v[N];
        load_vec<T, N>(a + x, v);
#pragma unroll
        for (int i = 0; i < N; i++)
            if (x + i < NA) out[x + i] = v[i];
    }
}

// out[o] (+)= sum_{a,c} D[o][a][c0 + c] acc[a][c] for the lane's column, o = 0 .. nOut - 1. ADD: by atomics.
template <typename T, int VEC, int NA, int NC, bool ADD>
__device__ __forceinline__ void contract_row(const RowsArgs<T>& g, const T* D, T* out,
                                             typename Pack<T, VEC>::V (&acc)[NA][NC], int c0, bool store,
                                             bool add_to) {
    using P = Pack<T, VEC>;
    using V = typename P::V;
    for (int o = 0; o < g.nOut; o += kTableOut) {
        V v[kTableOut];
#pragma unroll
        for (int u = 0; u < kTableOut; u++) v[u] = V(0);
        const T* d = D + static_cast<size_t>(o) * NA * g.pad_c + c0;
#pragma unroll
        for (int a = 0; a < NA; a++)
#pragma unroll
            for (int c = 0; c < NC; c++)
#pragma unroll
                for (int u = 0; u < kTableOut; u++)
                    v[u] = P::fma(P::dup(d[(u * NA + a) * g.pad_c + c]), acc[a][c], v[u]);
#pragma unroll
        for (int u = 0; u < kTableOut; u++) {
            for (int x = g.lanes; x < 32; x <<= 1) v[u] = P::add(v[u], P::shift(v[u], x));
            if (store && o + u < g.nOut) {
                T* at = out + static_cast<int64_t>(o + u) * g.L;
                V* dst = reinterpret_cast<V*>(at);
                if constexpr (ADD)
                    P::add_at(at, v[u]);
                else
                    *dst = add_to ? P::add(*dst, v[u]) : v[u];
            }
        }
    }
}

// Forward, and the gW part of the gradients: `out` is [rows][nOut][L].
template <typename T, int VEC, int NA, int NC, Mode MODE, typename Off, Cut CUT>
__device__ __forceinline__ void outer_rows(const RowsArgs<T>& g, const Off* __restrict__ offsets,
                                           T* __restrict__ out, const Part<CUT>& part, const T* D,
                                           unsigned char* ring, int lane, const Status& st) {
    using P = Pack<T, VEC>;
    using V = typename P::V;
    const int lb = lane & (g.lanes - 1);
    for (int b0 = 0; b0 < g.L; b0 += 32 * VEC) {
        const int b = b0 + lb * VEC;
        const bool store = lane < g.lanes && b < g.L;
        for (int c0 = 0; c0 < g.nC; c0 += NC) {
            V acc[NA][NC];
            walk_rows<T, VEC, NA, NC, MODE, Off, CUT>(
                g, offsets, part, b0, c0, ring, lane, st,
                [&](int64_t, bool) {
#pragma unroll
                    for (int a = 0; a < NA; a++)
#pragma unroll
                        for (int c = 0; c < NC; c++) acc[a][c] = V(0);
                },
                [&](V(&w)[NC], V bv, const T* a_row, const int*, bool) {
                    T A[NA];
                    load_a<T, NA>(a_row, A);
#pragma unroll
                    for (int c = 0; c < NC; c++) w[c] = P::mul(w[c], bv);
#pragma unroll
                    for (int a = 0; a < NA; a++) {
                        const V av = P::dup(A[a]);
#pragma unroll
                        for (int c = 0; c < NC; c++) acc[a][c] = P::fma(av, w[c], acc[a][c]);
                    }
                },
                [&](int64_t row, bool any) {
                    T* at = out + row * g.nOut * g.L + b;
                    if (CUT != kCut || any) contract_row<T, VEC, NA, NC, CUT == kCut>(g, D, at, acc, c0, store, c0 > 0);
                });
        }
    }
}

// Adds NP values over the LP lanes of an edge and stores them, dst[0 .. n). While a lane holds several
// values it hands half of them to its partner and takes the partner's share of the other half, so
// that NP values cost about NP shuffles and not NP log LP.
template <int O, typename T, int NP, int LP>
__device__ __forceinline__ void sum_level(T (&v)[NP], int lb, int& which) {
    constexpr int kHeld = NP * O * 2 / LP; // values a lane holds at this level, if more than one
    if constexpr (kHeld > 1) {
        const bool upper = lb & O;
#pragma unroll
        for (int i = 0; i < kHeld / 2; i++) {
            const T send = upper ? v[i] : v[i + kHeld / 2];
            const T mine = upper ? v[i + kHeld / 2] : v[i];
            v[i] = mine + __shfl_xor_sync(kFullMask, send, O);
        }
        which += upper ? kHeld / 2 : 0;
    } else {
        v[0] += __shfl_xor_sync(kFullMask, v[0], O);
    }
    if constexpr (O > 1) sum_level<O / 2, T, NP, LP>(v, lb, which);
}
template <typename T, int NP, int LP>
__device__ __forceinline__ void sum_lanes(T (&v)[NP], int lb, T* dst, int n, bool live, bool first) {
    int which = 0;
    sum_level<LP / 2, T, NP, LP>(v, lb, which);
    constexpr int kLeft = NP > LP ? NP / LP : 1, kCopies = LP > NP ? LP / NP : 1;
    if (live && (lb & (kCopies - 1)) == 0) {
#pragma unroll
        for (int i = 0; i < kLeft; i++)
            if (which + i < n) dst[which + i] = first ? v[i] : dst[which + i] + v[i];
    }
}

// The same without selecting, for one edge per warp: lane `lb` holds its values in the order i ^ mask,
// with the mask below, so that what it hands over is always the upper half. M of the NA values (a
// power of two) go this way, the ninth of nine by itself.
__device__ __forceinline__ int sum_mask(int lane, int m) {
    int mask = 0;
    for (int o = 16, h = m / 2; h >= 1; o /= 2, h /= 2)
        if (lane & o) mask |= h;
    return mask;
}
template <int O, int HELD, typename T, int NA> __device__ __forceinline__ void sum_ordered(T (&v)[NA]) {
    if constexpr (HELD > 1) {
#pragma unroll
        for (int i = 0; i < HELD / 2; i++) v[i] += __shfl_xor_sync(kFullMask, v[i + HELD / 2], O);
    } else {
        v[0] += __shfl_xor_sync(kFullMask, v[0], O);
    }
    if constexpr (O > 1) sum_ordered<O / 2, (HELD > 1 ? HELD / 2 : 1), T, NA>(v);
}

// gA and gB. `own` is the matrix of the rows themselves, [rows][nOut][L] (W, where the rows are
// those of W and g.G is gO).
template <typename T, int VEC, int NA, int NC, Mode MODE, typename Off, Cut CUT>
__device__ __forceinline__ void edge_gradients(const RowsArgs<T>& g, const Off* __restrict__ offsets,
                                               T* __restrict__ gA, T* __restrict__ gB,
                                               const T* __restrict__ own, const Part<CUT>& part, const T* D,
                                               unsigned char* ring, int lane, const Status& st) {
    using P = Pack<T, VEC>;
    using V = typename P::V;
    constexpr int NP = NA <= 4 ? 4 : 16;              // values in the sums over lanes, padded
    constexpr int M = NA <= 4 ? 4 : NA <= 9 ? 8 : 16; // ... that are taken in the lane's own order
    constexpr bool kOrdered = MODE != kSideBySide;
    const int LP = g.lanes, lb = lane & (LP - 1);
    const int mask = kOrdered ? sum_mask(lane, M) : 0;
    for (int b0 = 0; b0 < g.L; b0 += 32 * VEC) {
        const int b = b0 + lb * VEC, bc = b < g.L ? b : g.L - VEC;
        for (int c0 = 0; c0 < g.nC; c0 += NC) {
            const bool first = b0 == 0 && c0 == 0;
            V E[NA][NC];
            walk_rows<T, VEC, NA, NC, MODE, Off, CUT>(
                g, offsets, part, b0, c0, ring, lane, st,
                [&](int64_t row, bool any) {
                    if (!any) return;
#pragma unroll
                    for (int a = 0; a < NA; a++)
#pragma unroll
                        for (int c = 0; c < NC; c++) E[a][c] = V(0);
                    const T* src = own + row * g.nOut * g.L + bc;
                    V next = *reinterpret_cast<const V*>(src);
                    for (int o = 0; o < g.nOut; o++) {
                        const V v = next;
                        if (o + 1 < g.nOut) next = *reinterpret_cast<const V*>(src + static_cast<int64_t>(o + 1) * g.L);
                        const T* d = D + static_cast<size_t>(o) * NA * g.pad_c + c0;
#pragma unroll
                        for (int a = 0; a < NA; a++)
#pragma unroll
                            for (int c = 0; c < NC; c++)
                                E[a][c] = P::fma(P::dup(d[(a < M ? a ^ mask : a) * g.pad_c + c]), v, E[a][c]);
                    }
                },
                [&](V(&w)[NC], V bv, const T* a_row, const int* edge, bool live) {
                    const int64_t e = *edge;
                    V z[NA];
#pragma unroll
                    for (int a = 0; a < NA; a++) {
                        z[a] = P::mul(E[a][0], w[0]);
#pragma unroll
                        for (int c = 1; c < NC; c++) z[a] = P::fma(E[a][c], w[c], z[a]);
                    }
                    if (gB != nullptr) {
                        T A[NA];
                        if constexpr (kOrdered) {
#pragma unroll
                            for (int a = 0; a < NA; a++) A[a] = a_row[a < M ? a ^ mask : a];
                        } else {
                            load_a<T, NA>(a_row, A);
                        }
                        V s0 = P::mul(P::dup(A[0]), z[0]), s1 = V(0);
#pragma unroll
                        for (int a = 1; a < NA; a++)
                            (a & 1 ? s1 : s0) = P::fma(P::dup(A[a]), z[a], a & 1 ? s1 : s0);
                        s0 = P::add(s0, s1);
                        if (live && b < g.L) {
                            V* dst = reinterpret_cast<V*>(gB + e * g.L + b);
                            *dst = c0 > 0 ? P::add(*dst, s0) : s0;
                        }
                    }
                    if (gA != nullptr) {
                        T* dst = gA + e * g.nA;
                        if constexpr (kOrdered) {
                            T v[NA];
#pragma unroll
                            for (int a = 0; a < NA; a++) v[a] = P::sum(P::mul(z[a], bv));
                            T last = T(0);
                            if constexpr (NA > M) last = warp_sum(v[M]);
                            sum_ordered<16, M, T, NA>(v);
                            if ((lane & (32 / M - 1)) == 0 && mask < g.nA)
                                dst[mask] = first ? v[0] : dst[mask] + v[0];
                            if (NA > M && lane == 1 && M < g.nA) dst[M] = first ? last : dst[M] + last;
                        } else {
                            T v[NP];
#pragma unroll
                            for (int a = 0; a < NP; a++)
                                v[a] = a < NA ? P::sum(P::mul(z[a < NA ? a : 0], bv)) : T(0);
                            switch (LP) { // (uniform)
                            case 16: sum_lanes<T, NP, 16>(v, lb, dst, g.nA, live, first); break;
                            case 8: sum_lanes<T, NP, 8>(v, lb, dst, g.nA, live, first); break;
                            default: sum_lanes<T, NP, 4>(v, lb, dst, g.nA, live, first); break;
                            }
                        }
                    }
                },
                [&](int64_t, bool) {});
        }
    }
}

// ---- kernels
// Blocks per SM: two for f32 with one column per lane, whose sums take 81 registers and not 162. That
// pays for the edge gradients (200 000 edges, 32 columns, 16 x 9 -> 16 channels: 0.67 -> 0.54 ms) and
// for short rows (10 edges: sums 0.15 -> 0.12, gradients 0.26 -> 0.19 ms); the sums of 16 channels
// stay with one block (0.31 against 0.34 ms).
template <typename T, int VEC> constexpr int kEdgeBlocks = sizeof(T) == 4 && VEC == 1 ? 2 : 1;
template <typename T, int VEC, int NA> constexpr int kSumBlocks = NA <= 9 ? kEdgeBlocks<T, VEC> : 1;

// A block owns a range of rows (the blocks share the edges evenly); its warps take them a few at a
// time, about kChunkEdges edges, so that none waits for another's long rows
// (60 000 edges, 1000 rows: 63 -> 45 us against rows dealt out beforehand).
constexpr int kChunkEdges = 256;
constexpr int kLeastChunk = 32;
template <typename Off> __device__ __forceinline__ int chunk_rows(const Off* offsets, int64_t lo, int64_t hi, int warps = kRowWarps) {
    const int64_t edges = offsets[hi] - offsets[lo], rows = hi - lo;
    if (edges <= 0) return 256;
    const int64_t n = kChunkEdges * rows / edges, fair = rows / (2 * warps);
    return static_cast<int>(n < 1 || fair < 1 ? 1 : n < fair ? n : fair);
}
//
// Rows longer than the limit (or few of them) would leave warps waiting for one another: then the blocks
// share out chunks of edges instead, and rows are cut where a chunk ends (sums of 60 000 edges, half of
// them in one of 1000 rows, f32, 9 x 9 x 9 channels: 9.3 ms without).
template <typename Off, typename F>
__device__ __forceinline__ void for_rows(const Off* offsets, int64_t lo, int64_t hi, int* counter, int lane, F&& f) {
    const int n = chunk_rows(offsets, lo, hi);
    while (true) {
        int at = 0;
        if (lane == 0) at = atomicAdd(counter, n);
        const int64_t r = lo + __shfl_sync(kFullMask, at, 0);
        if (r >= hi) break;
        f(Part<kWhole>{r, r + n < hi ? r + n : hi});
    }
}
template <typename Off, typename F>
__device__ __forceinline__ void for_cuts(const Off* offsets, int64_t rows, int chunk, int* counter, int lane, F&& f) {
    const int edges = static_cast<int>(offsets[rows]);
    while (true) {
        int at = 0;
        if (lane == 0) at = atomicAdd(counter, 1);
        const int64_t p = (blockIdx.x + static_cast<int64_t>(__shfl_sync(kFullMask, at, 0)) * gridDim.x) * chunk;
        if (p >= edges) break;
        const int end = p + chunk < edges ? static_cast<int>(p) + chunk : edges;
        // the rows of the first and of the last edge
        f(Part<kCut>{warp_count_weighted_le(offsets, rows + 1, 0, p, lane) - 1,
                     warp_count_weighted_le(offsets, rows + 1, 0, end - 1, lane), static_cast<int>(p), end, nullptr});
    }
}

// Few rows for a block's warps: dealt out whole, the last ones leave most warps waiting (60 000 edges, 1000 rows: 13.5
// tasks of a row and sixteen columns for twelve warps). Then the block's edges are cut into equal pieces, as many as
// warps, whatever rows they belong to. A row belongs to the piece that it begins in; what other pieces add to it, at
// most one row each, goes to shared memory and is added in their order when all are done: the same bits every time.
// 60 000 edges, 1000 rows, f64 sums 37 -> 33 us; 250 000 edges, 4099 rows, 64 columns, f32, gradients of A and B, which add
// up nothing over a row: 195 -> 178 us. (The sums by multiply-adds gain 2 % there, 129 -> 126 us, and lose as much on many
// rows, 2.07 -> 2.12 ms, to the third way through their loop in the kernel.) From six rows a warp on the last ones matter less than the additional coupling of the cut ones.
// (Rows are dealt out whole all the same where the sums have no room for what the pieces hand on: with nine components of A
// 9 x 9 -> 9 channels have room for twelve pieces, 10 gathered channels and 9 outputs for none; and for 5, 7 and 9 to 11 slices of
// columns, for which two pieces a warp, rounded up, are more than there is ever room for.)
constexpr int kMostPieces = 64; // of all slices of the columns
constexpr int kFewRowsPerWarp = 6;
struct Pieces {
    int64_t lo, hi; // the block's rows
    int first, edges, count;
    int64_t* heads; // [slice][piece] (shared memory): the row that the piece goes on with, -1: none
    unsigned char* sums;
    int sums_bytes; // of a piece
};
// Pieces per slice, 0: the rows are not few, or there is no room.
template <typename Off>
__device__ __forceinline__ int piece_count(const Off* offsets, int64_t lo, int64_t hi, int warps, int slices, int room) {
    if ((hi - lo) * slices >= kFewRowsPerWarp * warps) return 0;
    if (offsets[hi] - offsets[lo] < 8 * warps) return 0;
    const int n = slices <= warps && warps % slices == 0 ? warps / slices : (2 * warps + slices - 1) / slices;
    return n > 1 && n * slices <= room ? n : 0;
}
template <typename Off, typename F>
__device__ __forceinline__ void for_pieces(const Off* offsets, const Pieces& z, int slices, int* counter, int lane, F&& f) {
    auto at = [&](int t) { return z.first + static_cast<int>(static_cast<int64_t>(z.edges) * t / z.count); };
    auto row_at = [&](int t) { // the first row that begins at piece t's first edge or behind it
        if (t <= 0) return z.lo;
        if (t >= z.count) return z.hi;
        return z.lo + warp_count_weighted_le(offsets + z.lo, z.hi - z.lo + 1, 0, at(t) - 1, lane);
    };
    while (true) {
        int task = 0;
        if (lane == 0) task = atomicAdd(counter, 1);
        task = __shfl_sync(kFullMask, task, 0);
        if (task >= z.count * slices) break;
        const int t = task % z.count;
        const int64_t lo = row_at(t), hi = row_at(t + 1);
        const bool head = static_cast<int>(offsets[lo]) > at(t);
        if (lane == 0) z.heads[task] = head ? lo - 1 : -1;
        f(Part<kPiece>{head ? lo - 1 : lo, hi, at(t), at(t + 1), head ? z.sums + task * z.sums_bytes : nullptr},
          task / z.count);
    }
}
// Adds the sums of the pieces' heads to their rows, columns [b0, b0 + columns) of slice b0 / columns. All threads of
// the block, a warp per row.
template <typename T>
__device__ __forceinline__ void add_heads(const Pieces& z, int slices, int columns, int n_out, int L, T* out, int warps) {
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int task = warp; task < z.count * slices; task += warps) {
        const int t = task % z.count, b0 = task / z.count * columns;
        const int64_t row = z.heads[task];
        if (row < 0 || (t > 0 && z.heads[task - 1] == row)) continue;
        const int wide = L - b0 < columns ? L - b0 : columns;
        for (int x = lane; x < n_out * wide; x += 32) {
            const int o = x / wide, b = x - o * wide;
            T* at = out + (row * n_out + o) * L + b0 + b;
            T sum = *at;
            for (int i = task; i < task - t + z.count && z.heads[i] == row; i++)
                sum += reinterpret_cast<const T*>(z.sums + i * z.sums_bytes)[o * columns + b];
            *at = sum;
        }
    }
}
// A block's rows: f(part, slice) for pieces of them where they are few, whole(lo, hi) otherwise. `out`: what f adds
// up, nullptr where nothing is.
template <typename T, typename Off, typename F, typename Whole>
__device__ __forceinline__ void for_few_rows(const RowsArgs<T>& g, const Off* offsets, int warps, int slices, int columns,
                                             T* out, int64_t* heads, unsigned char* smem, int* counter, int lane, F&& f,
                                             Whole&& whole) {
    const int64_t lo = balanced_row_split(offsets, g.rows, blockIdx.x, gridDim.x, lane);
    const int64_t hi = balanced_row_split(offsets, g.rows, blockIdx.x + 1, gridDim.x, lane);
    const int count = piece_count(offsets, lo, hi, warps, slices, out != nullptr ? g.piece_room : kMostPieces);
    if (count == 0) {
        whole(lo, hi);
        return;
    }
    const int first = static_cast<int>(offsets[lo]);
    const Pieces z{lo, hi, first, static_cast<int>(offsets[hi]) - first, count, heads, smem + g.piece_at,
                   (g.nOut * columns * static_cast<int>(sizeof(T)) + 15) / 16 * 16};
    for_pieces(offsets, z, slices, counter, lane, f);
    if (out != nullptr) add_heads(z, slices, columns, g.nOut, g.L, out, warps);
}

// Shared memory of the kernels: the table, the rings, and a counter of rows taken.
template <typename T, int VEC, int NA, int NC> struct RowsShared {
    T* D;
    unsigned char* ring;
    int* counter;
    __device__ RowsShared(const RowsArgs<T>& g, unsigned char* smem, int* c, int warp) : counter(c) {
        D = reinterpret_cast<T*>(smem);
        const int size = g.pad_out * NA * g.pad_c;
        if (threadIdx.x == 0) *counter = 0;
        for (int x = threadIdx.x; x < size; x += kRowWarps * 32) D[x] = g.D[x];
        ring = smem + static_cast<int>(size * sizeof(T) + 127) / 128 * 128 +
               warp * kDepth * Slot<T, VEC, NA, NC>::bytes(32 / g.lanes);
        __syncthreads();
    }
};

// Forward (rows of the scatter index, `offsets`, or `starts` with a permutation when that turned out not
// to be sorted) and gW (rows of W, `starts`).
enum RowsRun { kSorted = 0, kIfUnsorted = 1, kAlways = 2 };

template <typename T, int VEC, int NA, int NC, Mode MODE>
__global__ void __launch_bounds__(kRowWarps * 32, (kSumBlocks<T, VEC, NA>))
sasaw_sum_rows(const __grid_constant__ RowsArgs<T> g, const int64_t* __restrict__ offsets,
               const int32_t* __restrict__ starts, T* __restrict__ out, RowsRun run, Status st) {
    if (run != kAlways && saw_unsorted(st) != (run == kIfUnsorted)) return;
    __shared__ int counter;
    extern __shared__ __align__(128) unsigned char smem[];
    const int warp = __shfl_sync(kFullMask, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const RowsShared<T, VEC, NA, NC> sh(g, smem, &counter, warp);
    auto sum = [&](const auto* at, const auto& part) {
        outer_rows<T, VEC, NA, NC, MODE>(g, at, out, part, sh.D, sh.ring, lane, st);
    };
    auto rows = [&](const auto* at) {
        for_rows(at, balanced_row_split(at, g.rows, blockIdx.x, gridDim.x, lane),
                 balanced_row_split(at, g.rows, blockIdx.x + 1, gridDim.x, lane), sh.counter, lane,
                 [&](const auto& part) { sum(at, part); });
    };
    if (run == kSorted)
        rows(offsets);
    else if (*g.longest <= g.limit)
        rows(starts);
    else // (`out` has been cleared by a kernel before)
        for_cuts(starts, g.rows, g.chunk, sh.counter, lane, [&](const auto& part) { sum(starts, part); });
}

#include "sasaw_rows_mma.cuh"

// gW, to which the sums that come next will add.
template <typename T> __device__ __forceinline__ void clear_for_sums(const RowsArgs<T>& g, T* gW) {
    if (gW == nullptr) return;
    const int64_t n = g.rows * g.nOut * g.L;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x)
        gW[i] = T(0);
}

#include "sasaw_edges_mma.cuh"

// gA and gB. (A kernel of its own: gathering for gW at the same time in half of the warps saves DRAM
// traffic, but with both loops in one kernel the registers do not suffice.)
template <typename T, int VEC, int NA, int NC, Mode MODE>
__global__ void __launch_bounds__(kRowWarps * 32, (kEdgeBlocks<T, VEC>))
sasaw_edge_gradients(const __grid_constant__ RowsArgs<T> g, const int32_t* __restrict__ starts, T* __restrict__ gA,
                     T* __restrict__ gB, T* __restrict__ gW, const T* __restrict__ W, Status st) {
    __shared__ int counter;
    extern __shared__ __align__(128) unsigned char smem[];
    const int warp = __shfl_sync(kFullMask, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const RowsShared<T, VEC, NA, NC> sh(g, smem, &counter, warp);
    auto gradients = [&](const auto& part) {
        edge_gradients<T, VEC, NA, NC, MODE>(g, starts, gA, gB, W, part, sh.D, sh.ring, lane, st);
    };
    if (*g.longest <= g.limit) {
        __shared__ int64_t heads[kMostPieces];
        for_few_rows<T>(g, starts, kRowWarps, 1, g.L, nullptr, heads, smem, sh.counter, lane,
                        [&](const auto& part, int) { gradients(part); },
                        [&](int64_t lo, int64_t hi) { for_rows(starts, lo, hi, sh.counter, lane, gradients); });
        return;
    }
    clear_for_sums(g, gW);
    for_cuts(starts, g.rows, g.chunk, sh.counter, lane, gradients);
}

// ---- the order of the edges by a row index: row starts and permutation (a counting sort)
__global__ void __launch_bounds__(kSortThreads)
order_edges_grid(EntrySort s, const int32_t* __restrict__ P, int64_t E, int64_t rows, int bit, Status st) {
    sort_entries(s, P, E, rows, true, st, [] { cooperative_groups::this_grid().sync(); }, bit);
}
__global__ void __launch_bounds__(kSortThreads)
order_edges_block(EntrySort s, const int32_t* __restrict__ P, int64_t E, int64_t rows, int bit, Status st) {
    sort_entries(s, P, E, rows, true, st, [] { __syncthreads(); }, bit);
}

// ---- dispatch
// Channel counts are padded to the next instantiation: A to 4, 9, 16 (spherical harmonics up to
// l = 1, 2, 3), the other one to at most 81 products, several passes where it is wider.
inline int pad_a(int n) { return n <= 4 ? 4 : n <= 9 ? 9 : 16; }
inline int chunk_c(int na, int n) { return n <= 4 ? 4 : na <= 9 ? 9 : n <= 5 || n > 8 ? 5 : 4; }

template <typename T> struct RowsShape {
    RowsArgs<T> g;
    int na, nc, vec;
    bool aligned; // G and B at 16-byte boundaries
    size_t smem;
    size_t table_bytes;
};

template <typename T>
RowsShape<T> rows_shape(const Call& call, const SasawProblem<T>& p, const T* gathered, bool out_is_m2, int vec) {
    RowsShape<T> s{};
    s.na = s.g.pad_a = pad_a(p.nA);
    s.g.nC = out_is_m2 ? p.nO : p.nW;
    s.g.nOut = out_is_m2 ? p.nW : p.nO;
    s.nc = chunk_c(s.na, s.g.nC);
    s.vec = vec;
    s.g.A = p.A, s.g.B = p.B, s.g.G = gathered;
    s.g.rows = p.rows, s.g.nA = p.nA, s.g.L = p.L;
    s.aligned = (reinterpret_cast<uintptr_t>(gathered) | reinterpret_cast<uintptr_t>(p.B)) % 16 == 0;
    s.g.pad_c = static_cast<int>(ceil_div(s.g.nC, s.nc)) * s.nc;
    s.g.pad_out = static_cast<int>(ceil_div(s.g.nOut, kTableOut)) * kTableOut;
    int lanes = 4;
    while (lanes < 32 && lanes * vec < p.L) lanes *= 2;
    s.g.lanes = lanes;
    s.table_bytes = static_cast<size_t>(s.g.pad_out) * s.na * s.g.pad_c * sizeof(T);
    // (Slot::bytes)
    size_t slot = static_cast<size_t>(s.nc + 1) * 32 * vec * sizeof(T) +
                        (32 / lanes) * ((s.na * sizeof(T) + 15) / 16 * 16) + (32 / lanes * 4 + 15) / 16 * 16;
    slot = (slot + 127) / 128 * 128;
    s.smem = (s.table_bytes + 127) / 128 * 128 + slot * kDepth * kRowWarps;
    return s;
}

template <typename T, typename F> void for_shape(const RowsShape<T>& s, F&& f) {
    auto with = [&](auto vec, auto na, auto nc) {
        constexpr int VEC = decltype(vec)::value, NA = decltype(na)::value, NC = decltype(nc)::value;
        using I = std::integral_constant<int, VEC>;
        using A = std::integral_constant<int, NA>;
        using X = std::integral_constant<int, NC>;
        if (s.g.L == 32 * VEC && s.aligned)
            f(I(), A(), X(), std::integral_constant<Mode, kExact>());
        else if (VEC == 2 || s.g.lanes == 32)
            f(I(), A(), X(), std::integral_constant<Mode, kOneEdge>());
        else if constexpr (VEC == 1)
            f(I(), A(), X(), std::integral_constant<Mode, kSideBySide>());
    };
    auto widths = [&](auto vec) {
        using I4 = std::integral_constant<int, 4>;
        using I5 = std::integral_constant<int, 5>;
        using I9 = std::integral_constant<int, 9>;
        using I16 = std::integral_constant<int, 16>;
        if (s.na == 4)
            s.nc == 4 ? with(vec, I4(), I4()) : with(vec, I4(), I9());
        else if (s.na == 9)
            s.nc == 4 ? with(vec, I9(), I4()) : with(vec, I9(), I9());
        else
            s.nc == 4 ? with(vec, I16(), I4()) : with(vec, I16(), I5());
    };
    if constexpr (sizeof(T) == 4) {
        if (s.vec == 2) {
            widths(std::integral_constant<int, 2>());
            return;
        }
    }
    widths(std::integral_constant<int, 1>());
}

template <typename T> bool rows_apply(const SasawProblem<T>& p) {
    return p.nA >= 1 && p.nA <= kWidest && p.nW >= 1 && p.nW <= kWidest && p.nO >= 1 && p.nO <= kWidest &&
           p.L >= 1 && p.L <= (1 << 20) && p.E >= 1 && positions_fit_int(p.E) && p.rows >= 1 && p.N <= (1 << 20);
}

// Shared memory for the table and the rings, beside what the kernels declare themselves (the counter, the pieces' heads).
// At most 16 channels each, all but these fit: f64, up to 4 columns, 5 to 9 components of A, 10 or more gathered
// channels and 13 or more outputs, whose table and rings alone take the whole of it.
constexpr size_t kStaticShared = 1024;
template <typename T> bool rows_fit(const Call& call, const RowsShape<T>& s) {
    return s.smem + kStaticShared <= static_cast<size_t>(max_optin_smem(call.device));
}

// Two columns per lane (f32) from 33 columns on, where every operand allows 8-byte accesses.
template <typename T> int vector_width(int L, std::initializer_list<const void*> operands) {
    if (sizeof(T) == 8 || L % 2 != 0 || L <= 32) return 1;
    for (const void* p : operands)
        if (reinterpret_cast<uintptr_t>(p) % 8 != 0) return 1;
    return 2;
}

template <typename T>
TableRef dense_table(const Call& call, const SasawProblem<T>& p, const RowsShape<T>& s, bool out_is_m2) {
    TableKey key{};
    key.kind = kSasawDenseTable;
    key.scalar_bytes = static_cast<int>(sizeof(T));
    key.ptr[0] = p.C, key.ptr[1] = p.M1, key.ptr[2] = p.M2, key.ptr[3] = p.M3;
    key.n[0] = p.N, key.n[1] = p.nA, key.n[2] = p.nW, key.n[3] = p.nO, key.n[4] = out_is_m2 ? 1 : 0;
    TableRef ref = acquire_table(call, key, s.table_bytes);
    if (ref.fresh) {
        const int64_t warps = static_cast<int64_t>(s.g.pad_out) * s.na * s.g.pad_c;
        sasaw_dense_table<T><<<static_cast<unsigned>(ceil_div(warps, 8)), 256, 0, call.stream>>>(
            static_cast<T*>(ref.ptr), p.C, p.M1, p.M2, p.M3, p.N, p.nA, p.nW, p.nO, out_is_m2, s.g.pad_out, s.na,
            s.g.pad_c, call.status);
        MOPS_CUDA_OK(cudaGetLastError());
        commit_table(call, ref);
    }
    return ref;
}

// As many blocks as the SMs hold, fewer for few rows (more blocks than rows for their warps: 23 -> 29 us).
// With a permutation rows may be cut, so that it is the edges that count.
template <typename Kernel, typename T>
unsigned rows_blocks(const Call& call, Kernel kernel, const RowsShape<T>& s, int64_t edges) {
    const int64_t sms = sm_count(call.device);
    int64_t blocks = sms * resident_blocks(kernel, call.device, kRowWarps * 32, s.smem);
    if (s.g.rows < blocks * kRowWarps) blocks = sms;
    const int64_t most = s.g.perm == nullptr ? s.g.rows : std::max(s.g.rows, ceil_div(edges, kLeastChunk));
    return static_cast<unsigned>(std::min(most, blocks));
}

// Rows longer than twice the average are cut in chunks, two or more for every warp; where there are few
// rows for the warps, those longer than kFewRowsLimit.
constexpr int kFewRowsLimit = 96;
template <typename T> void set_chunks(const Call& call, RowsShape<T>& s, const EntrySort& sort, int64_t edges) {
    const int64_t warps = static_cast<int64_t>(sm_count(call.device)) * kRowWarps;
    const int64_t average = edges / s.g.rows;
    s.g.longest = sort.longest;
    s.g.limit = s.g.rows < 2 * warps ? kFewRowsLimit : static_cast<int>(std::max<int64_t>(128, 2 * average));
    s.g.chunk = static_cast<int>(std::min<int64_t>(
        std::max<int64_t>(ceil_div(edges, 2 * warps * kLeastChunk) * kLeastChunk, kLeastChunk), kChunkEdges));
}

// The sums on the FP64 tensor-core instruction: 16-byte pieces of every operand, and columns that fill at least
// half of a warp's sixteen; at half only from ten components of A on, whose sums fill the instruction (8 columns:
// 9 x 16 -> 9 channels 66 -> 82 us, 4 x 9 -> 4 94 -> 103, but 16 x 9 -> 9 435 -> 245).
inline bool sums_shape_by_mma(int nA, int L) { return L % 2 == 0 && L >= (pad_a(nA) == 16 ? 8 : 10); }
template <typename T> bool sums_by_mma(const RowsShape<T>& s, const T* out) {
    return sizeof(T) == 8 && sums_shape_by_mma(s.g.nA, s.g.L) && s.aligned && reinterpret_cast<uintptr_t>(out) % 16 == 0;
}
// The gradients of A and B on the same instruction: up to nine channels, 16-byte pieces of every operand, and a
// gathered table that stays in L2 beside what streams through it. (A row's columns are taken eight at a time, 64 bytes: 4.2 10^6
// edges, tables of 19, 38, 75 and 151 MB: 2.33, 2.39, 2.59 to 2.81, 3.10 ms against 2.53, 2.55, 2.65, 2.82.)
inline bool gradients_shape_by_mma(int nA, int nO, int L, int64_t rows) {
    constexpr double kCacheBytes = 60e6; // of the 126 MB
    return nA <= 9 && nO <= 9 && L % 2 == 0 && L >= 8 && static_cast<double>(rows) * nO * L * 8 <= kCacheBytes;
}
template <typename T> bool gradients_by_mma(const RowsShape<T>& s, const T* W, const T* gB) {
    return sizeof(T) == 8 && gradients_shape_by_mma(s.g.nA, s.g.nC, s.g.L, s.g.rows) && s.aligned &&
           (reinterpret_cast<uintptr_t>(W) | reinterpret_cast<uintptr_t>(gB)) % 16 == 0;
}
template <typename F> void for_mma_shape(const RowsShape<double>& s, F&& f) {
    auto with = [&](auto ma, auto ninth, auto nc) {
        using Any = std::integral_constant<int, 0>;
        if (s.g.nC % decltype(nc)::value != 0)
            f(ma, ninth, nc, std::false_type(), Any());
        else if (s.g.L != 32)
            f(ma, ninth, nc, std::true_type(), Any());
        else
            f(ma, ninth, nc, std::true_type(), std::integral_constant<int, 32>());
    };
    using I1 = std::integral_constant<int, 1>;
    using I2 = std::integral_constant<int, 2>;
    using I4 = std::integral_constant<int, 4>;
    using I5 = std::integral_constant<int, 5>;
    using I9 = std::integral_constant<int, 9>;
    if (s.na == 16)
        s.nc == 4 ? with(I2(), std::false_type(), I4()) : with(I2(), std::false_type(), I5());
    else if (s.g.nA == 9)
        s.nc == 4 ? with(I1(), std::true_type(), I4()) : with(I1(), std::true_type(), I9());
    else
        s.nc == 4 ? with(I1(), std::false_type(), I4()) : with(I1(), std::false_type(), I9());
}

template <typename T>
void launch_sums(const Call& call, const RowsShape<T>& s, const int64_t* offsets, const int32_t* starts,
                 T* out, RowsRun when, int64_t edges) {
    if constexpr (sizeof(T) == 8) {
        if (sums_by_mma(s, out)) {
            for_mma_shape(s, [&](auto ma, auto ninth, auto nc, auto full, auto ll) {
                constexpr int MA = decltype(ma)::value, NC = decltype(nc)::value, LL = decltype(ll)::value;
                constexpr bool NINTH = decltype(ninth)::value, FULL = decltype(full)::value;
                auto kernel = sasaw_sum_rows_mma<MA, NINTH, NC, FULL, LL>;
                const size_t table = MmaTable<MA, NINTH>::scalars(s.g.nOut, s.g.pad_c) * sizeof(double);
                constexpr size_t rings = kMmaWarps * kMmaRing<MA, NC>;
                // (fits with the most channels there are, of every instantiation, on any GPU with 227 KB a block)
                static_assert(MmaTable<MA, NINTH>::scalars(kWidest, (kWidest + NC - 1) / NC * NC) * sizeof(double) + kMmaWarps * kMmaRing<MA, NC> <=
                              227 * 1024 - 2048);
                // (behind the rings: what pieces of rows hand on)
                const size_t head = static_cast<size_t>(s.g.nOut) * kMmaColumns * sizeof(double);
                const size_t room = (static_cast<size_t>(max_optin_smem(call.device)) - 2048 - table - rings) / head;
                RowsArgs<T> g = s.g;
                g.piece_at = static_cast<int>(table + rings);
                g.piece_room = static_cast<int>(std::min<size_t>(room, 2 * kMmaWarps));
                const size_t smem = table + rings + g.piece_room * head;
                allow_dynamic_smem(kernel, call.device, smem);
                const int64_t most = s.g.perm == nullptr ? s.g.rows : std::max(s.g.rows, ceil_div(edges, kLeastChunk));
                const int64_t blocks = std::min<int64_t>(most, sm_count(call.device));
                note_kernel_f("sasaw_sum_rows_mma<MA=%d,NINTH=%d,NC=%d,L=%d>,PIECES=%d", MA, NINTH, NC, LL, g.piece_room);
                kernel<<<static_cast<unsigned>(blocks), kMmaWarps * 32, smem, call.stream>>>(g, offsets, starts, out,
                                                                                            when, call.status);
            });
            MOPS_CUDA_OK(cudaGetLastError());
            return;
        }
    }
    note_kernel_f("sasaw_sum_rows<%s,VEC=%d,NA=%d,NC=%d>", scalar_name<T>(), s.vec, s.na, s.nc);
    for_shape(s, [&](auto vec, auto na, auto nc, auto mode) {
        auto kernel = sasaw_sum_rows<T, decltype(vec)::value, decltype(na)::value, decltype(nc)::value,
                                     decltype(mode)::value>;
        const unsigned blocks = rows_blocks(call, kernel, s, edges);
        kernel<<<blocks, kRowWarps * 32, s.smem, call.stream>>>(s.g, offsets, starts, out, when, call.status);
    });
    MOPS_CUDA_OK(cudaGetLastError());
}

template <typename T>
void launch_edges_mma(const Call& call, const RowsShape<T>& s, const int32_t* starts, T* gA, T* gB, T* gW, const T* W,
                      int64_t edges) {
    if constexpr (sizeof(T) == 8) {
        auto go = [&](auto ks, auto c9, auto a9, auto ll) {
            constexpr int KS = decltype(ks)::value, LL = decltype(ll)::value;
            constexpr bool C9 = decltype(c9)::value, A9 = decltype(a9)::value;
            auto kernel = sasaw_edge_gradients_mma<KS, C9, A9, LL>;
            const size_t table = (GradTable<KS>::scalars(s.g.nOut) * sizeof(double) + 127) / 128 * 128;
            const size_t smem = table + kGradWarps * grad_ring_bytes<KS, C9>();
            allow_dynamic_smem(kernel, call.device, smem);
            const int64_t most = std::max(s.g.rows, ceil_div(edges, kLeastChunk));
            const int64_t blocks = std::min<int64_t>(most, sm_count(call.device));
            note_kernel_f("sasaw_edge_gradients_mma<KS=%d,C9=%d,A9=%d,L=%d>", KS, C9, A9, LL);
            kernel<<<static_cast<unsigned>(blocks), kGradWarps * 32, smem, call.stream>>>(s.g, starts, gA, gB, gW, W,
                                                                                         call.status);
        };
        auto with = [&](auto ks, auto c9) {
            using Any = std::integral_constant<int, 0>;
            if (s.g.nA == 9 && s.g.L == 32)
                go(ks, c9, std::true_type(), std::integral_constant<int, 32>());
            else if (s.g.nA == 9)
                go(ks, c9, std::true_type(), Any());
            else
                go(ks, c9, std::false_type(), Any());
        };
        using I1 = std::integral_constant<int, 1>;
        using I2 = std::integral_constant<int, 2>;
        if (s.g.nC == 9)
            with(I2(), std::true_type());
        else
            s.g.nC <= 4 ? with(I1(), std::false_type()) : with(I2(), std::false_type());
        MOPS_CUDA_OK(cudaGetLastError());
    }
}

} // namespace

template <typename T>
bool sasaw_rows_by_mma(const SasawProblem<T>& p, RowsWork work, std::initializer_list<const void*> others) {
    uintptr_t all = reinterpret_cast<uintptr_t>(p.B) | reinterpret_cast<uintptr_t>(p.W);
    for (const void* x : others) all |= reinterpret_cast<uintptr_t>(x);
    if (sizeof(T) != 8 || !rows_apply(p) || all % 16 != 0) return false;
    return work == RowsWork::kGradients ? gradients_shape_by_mma(p.nA, p.nO, p.L, p.rows) : sums_shape_by_mma(p.nA, p.L);
}

// The sums on the FP64 tensor-core instruction: microseconds, fitted to 1400 shapes with a sorted index (and where they
// were off to 2281 others) and to 929 without, 1 to 200 edges per row, up to 2 10^6 edges and 1000 coupling entries. Operations of the steps (one
// more for rows whose ends cut one; those of channels that the last pass does not have apart) and of the coupling, each by whether A
// has one tile, one and a ninth component, or two; what a step and a result cost beside; what the coupling costs more where the
// last pass has fewer channels; the coupling's table; results read again by later passes; the sort; a row's steps one after the
// other where rows are few.
inline double sums_mma_cost(bool sorted, int64_t edges, int64_t rows, int nA, int nW, int nO, int L, int64_t N) {
    struct Cost {
        double call, operation[3], missing, step, couple[3], part, result, table, again, edge, few; // in 10^-6 but the first one
    };
    constexpr Cost with_order{37.6, {1.32, 1.32, 1.12}, 1.2, 84, {0.596, 0.596, 0.507}, 0.28, 117, 4.4, 1.42, 0, 13900};
    constexpr Cost without{60.2, {1.82, 2.23, 1.4}, 1.1, 39, {0.53, 0.52, 0.46}, 0.29, 152, 4.86, 2.6, 21.5, 1100};
    const Cost& c = sorted ? with_order : without;
    const int na = pad_a(nA), nc = chunk_c(na, nW), ma = na == 16 ? 2 : 1, ninth = nA == 9 ? 1 : 0, kind = ma == 2 ? 2 : ninth;
    const double E = static_cast<double>(edges), n = static_cast<double>(rows);
    const double passes = static_cast<double>(ceil_div(nW, nc)), columns = static_cast<double>(ceil_div(L, 16));
    const double steps = (E / 4 + 0.75 * n * (1 - std::exp(-E / n))) * columns * passes, results = n * columns * passes;
    const double channel = 2 * (ma * 16 + 2 * ninth + 2), channels = nW / passes;
    const double couple = (2 * ma + ninth) * nc * 32 * static_cast<double>(ceil_div(nO, 8));
    const double table = static_cast<double>(ceil_div(nO, kTableOut)) * kTableOut * na * passes * nc * static_cast<double>(N);
    const double few = std::max(0.0, 1 - n * columns / 1776) * E / n * passes * nc * ma;
    return c.call + 1e-6 * (steps * (channel * (c.operation[kind] * channels + c.missing * (nc - channels)) + c.step) +
                            results * (couple * (c.couple[kind] + (nW % nc != 0 ? c.part : 0)) + c.result) +
                            c.table * table + c.again * n * nO * L * (passes - 1) + c.edge * E + c.few * few);
}

// The gradients on the FP64 tensor-core instruction, all three of them: microseconds, fitted to 148 shapes up to
// 2 10^6 edges; eight in ten estimates are within a sixth. Clocks of the instructions of a step, of a row's E, of the sums'
// steps and coupling, and what the coupling's table takes.
inline double gradients_mma_cost(int64_t edges, int64_t rows, int nA, int nW, int nO, int L, int64_t N) {
    const int ks = nO <= 4 ? 1 : 2, c9 = nO == 9 ? 1 : 0, a9 = nA == 9 ? 1 : 0;
    const int na = pad_a(nA), nc = chunk_c(na, nO);
    const double E = static_cast<double>(edges), n = static_cast<double>(rows);
    const double slices = static_cast<double>(ceil_div(L, 8)), columns = static_cast<double>(ceil_div(L, 16));
    const double step = 8 * (ks * 16 + 4 * c9 + 8 + a9 * (2 * ks + 2 * c9 + 4)), sum_step = nc * 2 * (18 + 2 * a9);
    const double outs = static_cast<double>(ceil_div(nW, 8)), passes = static_cast<double>(ceil_div(nO, nc));
    const double table = static_cast<double>(ceil_div(nW, 3)) * 3 * na * passes * nc * static_cast<double>(N);
    const double few = std::max(0.0, 1 - n / 1184) * E / n; // a row's steps one after the other
    return 60.2 + 1e-6 * (0.647 * E / 8 * slices * step + 2.59 * n * slices * nW * (ks * 16 + 10) +
                          1.39 * E / 4 * columns * passes * sum_step + 8.31 * E / 4 * columns * passes * 100 +
                          3.58 * n * columns * passes * (2 + a9) * nc * 32 * outs + 10.2 * table) +
           1.64 * few * slices * step / 8e3;
}

// By multiply-adds: microseconds, fitted to 750 shapes up to 2 10^6 edges with 1 to 16 channels, 1 to 100 columns and rows of
// a fraction of an edge to thousands; nine in ten estimates are within a third where a call takes more
// than 80 us. A step is an edge (or the edges side by side) in one pass over columns and channels.
template <typename T> double sasaw_rows_cost(const SasawProblem<T>& p, RowsWork work, bool mma) {
    if (!rows_apply(p)) return INFINITY;
    if (mma && work == RowsWork::kGradients) return gradients_mma_cost(p.E, p.rows, p.nA, p.nW, p.nO, p.L, p.N);
    if (mma) return sums_mma_cost(work == RowsWork::kSorted, p.E, p.rows, p.nA, p.nW, p.nO, p.L, p.N);
    struct Cost {
        double call, product, step, exact_product, exact_step; // products and steps in 10^-6
        double contract, contract_once, table, pass, edge, row; // 10^-6, 10^-3, 10^-5, 1, 10^-6, 10^-3
        double few_step, few_product; // a row's steps one after the other: 10^-2, 10^-4
    };
    constexpr bool f32 = sizeof(T) == 4;
    constexpr Cost sorted = f32 ? Cost{22.3, 1.92, 247, 3.51, 79.4, 4.61, 0, 0.369, 1.27, 10.3, 0, 16.8, 18.3}
                                : Cost{20.8, 4.46, 145, 3, 163, 4.81, 0, 0.739, 1.14, 51.1, 1.02, 16, 21.7};
    constexpr Cost unsorted = f32 ? Cost{33.9, 4.21, 210, 2.79, 152, 4.3, 4.59, 1.7, 3.19, 32.5, 0, 0, 0}
                                  : Cost{30.3, 4.66, 139, 2.38, 109, 4.41, 3.32, 0.0769, 8.66, 178, 0.922, 0, 0};
    constexpr Cost gradients = f32 ? Cost{31.4, 6.26, 741, 8.67, 352, 5.62, 6.84, 1.01, 23.3, 0, 0.113, 0, 0}
                                   : Cost{38.3, 14.2, 743, 10.5, 539, 9.55, 2.48, 0.897, 15.7, 29.7, 0, 0, 0};
    const Cost& c = work == RowsWork::kSorted ? sorted : work == RowsWork::kUnsorted ? unsorted : gradients;
    const bool forward = work != RowsWork::kGradients;
    const int nC = forward ? p.nW : p.nO, nOut = forward ? p.nO : p.nW;
    const int na = pad_a(p.nA), nc = chunk_c(na, nC), vec = vector_width<T>(p.L, {});
    int lanes = 4;
    while (lanes < 32 && lanes * vec < p.L) lanes *= 2;
    const double E = static_cast<double>(p.E), rows = static_cast<double>(p.rows), side = 32 / lanes;
    const double passes = static_cast<double>(ceil_div(nC, nc) * ceil_div(p.L, lanes * vec));
    const double products = na * nc, contract = products * (ceil_div(nOut, kTableOut) * kTableOut);
    // (a row's last step is half empty)
    const double steps = E / side + std::min(E, rows) * (1 - 1 / side);
    const bool exact = p.L == 32 * vec;
    const double busy = std::max(rows, 1184.0); // (a row for each of the warps)
    double us = c.call + passes * c.pass + E * c.edge * 1e-6 + contract * static_cast<double>(p.N) * c.table * 1e-5 +
                passes * contract * (busy * c.contract * 1e-6 + c.contract_once * 1e-3) + passes * busy * c.row * 1e-3;
    us += passes * steps * 1e-6 * (exact ? products * c.exact_product + c.exact_step : products * c.product + c.step);
    const double few = std::max(0.0, 1 - rows / 2368); // (two rows for each of the warps)
    if (exact && na == 16 && (vec == 2 || !f32)) us *= 1.25; // (what the fit leaves over)
    us += few * passes * (E / rows / side) * (c.few_step * 1e-2 + products * c.few_product * 1e-4);
    return us;
}

template <typename T> int sasaw_forward_rows(const Call& call, const SasawProblem<T>& p, T* O, ScatterPart part) {
    if (!rows_apply(p)) return kNotApplicable;
    RowsShape<T> s = rows_shape(call, p, p.W, false, vector_width<T>(p.L, {p.B, p.W, O}));
    if (!rows_fit(call, s)) return kNotApplicable;
    TableRef table = dense_table(call, p, s, false);
    s.g.gather = p.J, s.g.perm = nullptr, s.g.D = static_cast<const T*>(table.ptr), s.g.bit = kBitJ;
    bool unsorted = true;
    if (part != ScatterPart::kUnsorted) {
        SegmentTable seg = segment_table(call, p.I, p.E, p.rows);
        launch_sums<T>(call, s, seg.offsets, nullptr, O, kSorted, p.E);
        unsorted = !seg.known_sorted; // asynchronous calls cannot look: always enqueue
        release_table(call, seg.ref);
        if (unsorted && call.wait) {
            wait_stream(call);
            unsorted = host_saw_unsorted(call);
        }
    }
    if (unsorted && part != ScatterPart::kSorted) {
        const int sorters = sort_blocks(call, p.E, p.rows);
        void* scratch = scratch_alloc(call, entry_sort_bytes(p.E, p.rows, sorters));
        const EntrySort sort = entry_sort_at(scratch, p.rows, sorters);
        s.g.perm = sort.perm;
        set_chunks(call, s, sort, p.E);
        launch_sorting(call, sorters, sort_if_unsorted_grid, sort_if_unsorted_block, sort, p.I, p.E, p.rows,
                       reinterpret_cast<uint32_t*>(O), p.rows * p.nO * p.L * static_cast<int64_t>(sizeof(T) / 4),
                       s.g.limit, call.status);
        launch_sums<T>(call, s, nullptr, sort.starts, O, kIfUnsorted, p.E);
        scratch_free(call, scratch);
        unsorted = false;
    }
    release_table(call, table);
    return unsorted ? kUnsortedLeft : kComplete;
}

template <typename T>
bool sasaw_backward_rows(const Call& call, const SasawProblem<T>& p, T* gA, T* gB, T* gW, const T* gO) {
    if (!rows_apply(p)) return false;
    RowsShape<T> s = rows_shape(call, p, gO, true, vector_width<T>(p.L, {p.B, p.W, gO, gB, gW}));
    if (!rows_fit(call, s)) return false;
    TableRef table = dense_table(call, p, s, true);
    // the edges in the order of J
    const int sorters = sort_blocks(call, p.E, p.rows);
    TableKey key{};
    key.kind = kEdgeOrder;
    key.ptr[0] = p.J;
    key.n[0] = p.E, key.n[1] = p.rows;
    TableRef order = acquire_table(call, key, entry_sort_bytes(p.E, p.rows, sorters));
    const EntrySort sort = entry_sort_at(order.ptr, p.rows, sorters);
    if (order.fresh) {
        launch_sorting(call, sorters, order_edges_grid, order_edges_block, sort, p.J, p.E, p.rows,
                       static_cast<int>(kBitJ), call.status);
        commit_table(call, order);
    }
    s.g.gather = p.I, s.g.perm = sort.perm, s.g.D = static_cast<const T*>(table.ptr), s.g.bit = kBitI;
    set_chunks(call, s, sort, p.E);
    if ((gA != nullptr || gB != nullptr) && gradients_by_mma(s, p.W, gB)) {
        launch_edges_mma(call, s, sort.starts, gA, gB, gW, p.W, p.E);
    } else if (gA != nullptr || gB != nullptr) {
        note_kernel_f("sasaw_edge_gradients<%s,VEC=%d,NA=%d,NC=%d>", scalar_name<T>(), s.vec, s.na, s.nc);
        for_shape(s, [&](auto vec, auto na, auto nc, auto mode) {
            auto kernel = sasaw_edge_gradients<T, decltype(vec)::value, decltype(na)::value, decltype(nc)::value,
                                               decltype(mode)::value>;
            const unsigned blocks = rows_blocks(call, kernel, s, p.E);
            kernel<<<blocks, kRowWarps * 32, s.smem, call.stream>>>(s.g, sort.starts, gA, gB, gW, p.W, call.status);
        });
        MOPS_CUDA_OK(cudaGetLastError());
    } else if (gW != nullptr) {
        MOPS_CUDA_OK(cudaMemsetAsync(gW, 0, p.rows * p.nW * p.L * sizeof(T), call.stream));
    }
    if (gW != nullptr) {
        launch_sums<T>(call, s, nullptr, sort.starts, gW, kAlways, p.E);
    }
    release_table(call, order);
    release_table(call, table);
    return true;
}

#define INSTANTIATE(T)                                                                             \
    template bool sasaw_rows_by_mma<T>(const SasawProblem<T>&, RowsWork, std::initializer_list<const void*>); \
    template double sasaw_rows_cost<T>(const SasawProblem<T>&, RowsWork, bool);                    \
    template int sasaw_forward_rows<T>(const Call&, const SasawProblem<T>&, T*, ScatterPart);      \
    template bool sasaw_backward_rows<T>(const Call&, const SasawProblem<T>&, T*, T*, T*, const T*);
INSTANTIATE(float)
INSTANTIATE(double)

} // namespace mops_b200
