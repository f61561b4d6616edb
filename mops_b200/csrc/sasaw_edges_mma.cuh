// The gradients of A and B of sasaw_rows.cu on the FP64 tensor-core instruction, f64, up to nine channels of A and of O.
//
//   Z[e,m1,b] = sum_m3 gO[I_e,m3,b] E_b[m3,m1],     E_b[m3,m1] = sum_m2 D[m3,m2,m1] W[j,m2,b]
//   gA[e,m1] = sum_b B[e,b] Z[e,m1,b],     gB[e,b] = sum_m1 A[e,m1] Z[e,m1,b]
//
// For one column b the Z of eight edges of a row j is a product of two matrices: edges by m3, m3 by m1, four m3
// to a DMMA. Lane = 4 u + q holds gO of edge u and of m3 = q (and q + 4) as the first operand, E_b[q][u] as
// the second (in registers for as long as the row lasts), and is given Z of edge u and of m1 = 2q and 2q + 1. So the sum over b of
// gA stays in the lane, and gB is a sum over the four lanes of an edge. The ninth m3 and the ninth m1 go by
// multiply-adds, the latter as partial sums of the four lanes.
//
// A warp takes the columns of its rows eight at a time: 32 registers of E and 80 of the ninths' coefficients. gA is added up
// in shared memory, by the same lanes for every eight columns. Rows of gO and B come through a ring of asynchronous
// copies, three steps of eight edges deep: the 64 bytes of a row and two edges make a line of 128, in which the four pieces of
// 16 bytes are permuted by m3, so that loads meet no bank twice. (Lines padded instead: the copies take
// twice the time, 14.7 against 7.9 clocks for 512 bytes.) Steps run along the positions: one that a row's end cuts is
// done once for each of its rows, and every edge's results are stored by its own. Windows of 96 edges bound the
// shared memory of gA; the columns of a window come one slice after the other without a gap in the copies.
//
// What bounds it: latency at two warps per scheduler (255 registers; 228 instructions per edge, issue slots 33 %, FP64 pipes 33 %). 9 x 9 x 9
// channels, 32 columns, against the multiply-adds of sasaw_rows.cu: 60 000 edges 66 -> 52 us, 4.2 10^6 edges with
// tables of 19 MB 2.53 -> 2.33 ms; gathered tables beyond L2 stay there (gradients_shape_by_mma). gA added up in
// global memory instead: 3.0 ms; with the hint to bring 256 bytes into L2: slower from 38 MB on.
#ifndef MOPS_B200_SASAW_EDGES_MMA_CUH
#define MOPS_B200_SASAW_EDGES_MMA_CUH

constexpr int kGradWarps = 8;
constexpr int kGradColumns = 8;
constexpr int kGradStep = 8; // edges
constexpr int kGradDepth = 3;
constexpr int kGradWindow = 96; // edges whose gA is added up in shared memory, eight columns after the other

// KS: m3 = 0 .. 4 KS - 1 by DMMA; C9, A9: there is a ninth m3, a ninth m1.
template <int KS, bool C9> struct GradSlot {
    static constexpr int kRows = C9 ? 9 : 4 * KS;          // of gO; B's is behind them
    static constexpr int kPair = (kRows + 1) * 128;        // two edges
    static constexpr int kA = kGradStep / 2 * kPair;       // A[u][0 .. 7], 64 bytes an edge
    static constexpr int kA9 = kA + kGradStep * 64;        // A[u][8]
    static constexpr int kBytes = (kA9 + kGradStep * 8 + 127) / 128 * 128;
};

// The coupling in shared memory: [m2][k][lane] D[4 k + q][m2][u], and [m2][i][q] the coefficients of the ninths:
// D[8][m2][2 q], D[8][m2][2 q + 1], D[q][m2][8], D[q + 4][m2][8], D[8][m2][8] (of q = 0 only).
template <int KS> struct GradTable {
    static __host__ __device__ size_t scalars(int nW) { return static_cast<size_t>(nW) * (KS * 32 + 20); }
    static __device__ void fill(double* table, const RowsArgs<double>& g) {
        const int nW = g.nOut;
        auto d = [&](int m3, int m2, int m1) {
            return m3 < g.nC && m1 < g.nA ? __ldg(g.D + (static_cast<size_t>(m2) * g.pad_a + m1) * g.pad_c + m3) : 0.0;
        };
        for (int x = threadIdx.x; x < nW * KS * 32; x += blockDim.x)
            table[x] = d((x >> 5) % KS * 4 + (x & 3), (x >> 5) / KS, x >> 2 & 7);
        for (int x = threadIdx.x; x < nW * 20; x += blockDim.x) {
            const int q = x & 3, i = (x >> 2) % 5, m2 = (x >> 2) / 5;
            const int m3 = i < 2 || i == 4 ? 8 : i == 2 ? q : q + 4, m1 = i < 2 ? 2 * q + i : 8;
            table[nW * KS * 32 + x] = i == 4 && q != 0 ? 0.0 : d(m3, m2, m1);
        }
    }
};

// The edges at positions [p_lo, p_hi), at most kGradWindow of them, of the rows [row_lo, row_hi).
template <int KS, bool C9, bool A9, int LL, typename Off>
__device__ __forceinline__ void mma_edge_window(const RowsArgs<double>& g, const Off* __restrict__ offsets,
                                                double* __restrict__ gA, double* __restrict__ gB,
                                                const double* __restrict__ W, int64_t row_lo, int64_t row_hi,
                                                int p_lo, int p_hi, const double* table, unsigned char* ring,
                                                int lane, const Status& st) {
    using Slot = GradSlot<KS, C9>;
    constexpr int kColumns = kGradColumns, kStep = kGradStep, kDepth = kGradDepth;
    const int q = lane & 3, u = lane >> 2; // of the copies, too: edge u of a step, piece q of every row
    const int L = LL > 0 ? LL : g.L, nW = g.nOut;
    const int last = p_hi - 1, steps = (p_hi - p_lo + kStep - 1) / kStep;
    const int slices = (L + kColumns - 1) / kColumns, all_steps = steps * slices;

    const int l_row = L * 8, g_row = g.nC * l_row, a_row = g.nA * 8;
    const unsigned ring32 = static_cast<unsigned>(__cvta_generic_to_shared(ring));
    const unsigned to = ring32 + (u >> 1) * Slot::kPair + (u & 1) * 64;
    unsigned char* const mine = ring + (u >> 1) * Slot::kPair + (u & 1) * 64;
    double* const w_rows = reinterpret_cast<double*>(ring + kDepth * Slot::kBytes); // [2][nW][8]
    const unsigned w_rows32 = ring32 + kDepth * Slot::kBytes;
    // gA so far, [position][0 .. 7] and [position][8]
    double* const sums = reinterpret_cast<double*>(ring + kDepth * Slot::kBytes + 2 * kWidest * 64) + u * 8 + 2 * q;
    double* const sums9 = reinterpret_cast<double*>(ring + kDepth * Slot::kBytes + 2 * kWidest * 64 + kGradWindow * 64) + u;

    // Edge numbers and gathered rows of 32 positions (four steps): of the block that the copies have reached (0), of
    // the next (1), the edge numbers of the one behind that (2). Behind the last block comes the first one again, for
    // the next columns.
    auto load_edge = [&](int base) {
        const int e = min(base + lane, last);
        return g.perm != nullptr ? __ldg(g.perm + e) : e;
    };
    auto behind = [&](int base) { return base + 32 < p_hi ? base + 32 : p_lo; };
    auto checked = [&](int32_t r) {
        if (clamp_index(r, static_cast<int32_t>(g.rows))) report_bad_index(st, g.bit);
        return r;
    };
    int block2 = behind(behind(p_lo));
    int e0 = load_edge(p_lo), e1 = load_edge(behind(p_lo)), e2 = load_edge(block2);
    int r0 = __ldg(g.gather + e0), r1 = __ldg(g.gather + e1);
    r0 = checked(r0);

    auto copy16 = [&](unsigned dst, const void* src, bool in) { // columns beyond the last one are zeros
        if (in)
            cp_async16(dst, src);
        else
            asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};\n" ::"r"(dst), "r"(0) : "memory");
    };
    int ahead = 0, ahead_step = 0, ahead_slice = 0; // the next step to copy: of all, of its slice
    int edge[kDepth - 1] = {};                      // the lane's edge of the steps under way, the oldest first
    auto start = [&](int slot) {
        if (ahead < all_steps) {
            if ((ahead_step & 3) == 0 && ahead > 0) {
                e0 = e1, r0 = checked(r1);
                e1 = e2;
                r1 = __ldg(g.gather + e1);
                block2 = behind(block2);
                e2 = load_edge(block2);
            }
            const int at = (ahead_step & 3) * kStep + u;
            const int e = __shfl_sync(kFullMask, e0, at), r = __shfl_sync(kFullMask, r0, at);
            const int b = ahead_slice * kColumns + 2 * q;
            const bool in = LL % kColumns == 0 && LL > 0 ? true : b < L;
            const unsigned char* src = reinterpret_cast<const unsigned char*>(g.G + b) + static_cast<int64_t>(r) * g_row;
            const unsigned dst = to + slot;
#pragma unroll
            for (int c = 0; c < Slot::kRows; c++)
                if (C9 || c < g.nC) copy16(dst + c * 128 + ((q ^ (c & 3)) * 16), src + c * l_row, in);
            copy16(dst + Slot::kRows * 128 + q * 16, reinterpret_cast<const unsigned char*>(g.B + b) +
                       static_cast<int64_t>(e) * l_row, in);
            const unsigned char* a = reinterpret_cast<const unsigned char*>(g.A + q) + static_cast<int64_t>(e) * a_row;
            const unsigned to_a = ring32 + slot + Slot::kA + u * 64 + q * 8;
            if (q < g.nA) cp_async_at<8, 0>(to_a, a);
            if (q + 4 < g.nA) cp_async_at<8, 32>(to_a, a + 32);
            if (A9 && q == 0) cp_async_at<8, 0>(ring32 + slot + Slot::kA9 + u * 8, a + 64);
            edge[kDepth - 2] = e;
            if (++ahead_step == steps) ahead_step = 0, ahead_slice++;
        }
        ahead++;
        cp_async_commit();
    };
    // The columns [8 slice, 8 slice + 8) of row j of W into buffer `half`, as part of the next group of copies.
    int64_t w_row = -1; // row under way or there, its slice, and the steps started since
    int w_slice = 0, w_age = 0, w_half = 0;
    auto fetch_w = [&](int64_t row, int slice, int half) {
        for (int x = lane; x < nW * 4; x += 32) {
            const int b = slice * kColumns + 2 * (x & 3);
            copy16(w_rows32 + half * (kWidest * 64) + x * 16, W + (row * nW + (x >> 2)) * L + b, b < L);
        }
        w_row = row, w_slice = slice, w_age = 0;
    };

    __syncwarp(); // (the ring's last readers)
#pragma unroll
    for (int i = 0; i < kDepth - 1; i++) {
        if (i > 0) {
#pragma unroll
            for (int d = 0; d + 1 < kDepth - 1; d++) edge[d] = edge[d + 1];
        }
        start(i * Slot::kBytes);
    }
    int slot = (kDepth - 1) * Slot::kBytes, e_now = 0; // of the step that is there; before the first one the last slot
    auto advance = [&] {
        cp_async_wait<kDepth - 2>();
        __syncwarp();
        e_now = edge[0];
#pragma unroll
        for (int d = 0; d + 1 < kDepth - 1; d++) edge[d] = edge[d + 1];
        start(slot);
        slot += Slot::kBytes;
        if (slot == kDepth * Slot::kBytes) slot = 0;
        w_age++;
    };

    for (int slice = 0; slice < slices; slice++) {
        const int b0 = slice * kColumns;
        int lo = p_lo, now = -1; // `now`: the step that is there
        for (int64_t row = row_lo; row < row_hi; row++) {
            const int hi = min(static_cast<int>(offsets[row + 1]), p_hi);
            if (lo >= hi) continue;
            // E and the ninths' coefficients
            if (w_row != row || w_slice != slice) { // (another row's may be on its way to the same place)
                cp_async_commit();
                cp_async_wait<0>();
                __syncwarp();
                fetch_w(row, slice, w_half);
            }
            if (w_age < kDepth) {
                cp_async_commit();
                cp_async_wait<0>();
            }
            __syncwarp();
            double E[KS][kColumns], ninth[5], c[5][kColumns];
#pragma unroll
            for (int b = 0; b < kColumns; b++)
#pragma unroll
                for (int k = 0; k < KS; k++) E[k][b] = 0;
#pragma unroll
            for (int i = 0; i < 5; i++) ninth[i] = 0;
            {
                const double* w = w_rows + w_half * (kWidest * 8);
                const double* d = table + lane;
                const double* d9 = table + nW * KS * 32 + q;
#pragma unroll 3
                for (int m2 = 0; m2 < nW; m2++, w += 8, d += KS * 32, d9 += 20) {
                    double x[kColumns];
#pragma unroll
                    for (int b = 0; b < kColumns; b += 2) {
                        const double2 v = *reinterpret_cast<const double2*>(w + b);
                        x[b] = v.x, x[b + 1] = v.y;
                    }
#pragma unroll
                    for (int k = 0; k < KS; k++) {
                        const double f = d[k * 32];
#pragma unroll
                        for (int b = 0; b < kColumns; b++) E[k][b] = fma(f, x[b], E[k][b]);
                    }
                    const double wu = w[u]; // (the ninths' coefficients: lane (u, q) has those of column u)
                    if constexpr (C9) ninth[0] = fma(d9[0], wu, ninth[0]), ninth[1] = fma(d9[4], wu, ninth[1]);
                    if constexpr (A9) ninth[2] = fma(d9[8], wu, ninth[2]);
                    if constexpr (A9 && KS > 1) ninth[3] = fma(d9[12], wu, ninth[3]);
                    if constexpr (A9 && C9) ninth[4] = fma(d9[16], wu, ninth[4]);
                }
            }
#pragma unroll
            for (int i = 0; i < 5; i++)
#pragma unroll
                for (int b = 0; b < kColumns; b++) {
                    const bool used = i < 2 ? C9 : i == 2 ? A9 : i == 3 ? A9 && KS > 1 : A9 && C9;
                    c[i][b] = used ? __shfl_sync(kFullMask, ninth[i], 4 * b + q) : 0.0;
                }
            __syncwarp();
            w_half ^= 1;
            if (row + 1 < row_hi)
                fetch_w(row + 1, slice, w_half);
            else if (slice + 1 < slices)
                fetch_w(row_lo, slice + 1, w_half);

#pragma unroll 1
            for (int t = (lo - p_lo) / kStep; t * kStep + p_lo < hi; t++) {
                if (t > now) {
                    advance();
                    now = t;
                }
                const int p = p_lo + t * kStep + u;
                const bool live = p >= lo && p < hi;
                const double2 a = *reinterpret_cast<const double2*>(ring + slot + Slot::kA + u * 64 + q * 16);
                const double a9 = A9 ? *reinterpret_cast<const double*>(ring + slot + Slot::kA9 + u * 8) : 0.0;
                double s[2] = {0, 0}, s9 = 0, gb[kColumns];
                const unsigned char* from = mine + slot + q * 128;
#pragma unroll
                for (int half = 0; half < kColumns; half += 4) { // (four products side by side)
                    double v[KS][4], v8[4], bv[4], z[4][2], z9[4];
                    auto load4 = [&](double(&x)[4], const unsigned char* from, int swap) {
#pragma unroll
                        for (int i = 0; i < 2; i++) {
                            const double2 y = *reinterpret_cast<const double2*>(from + ((half / 2 + i) ^ swap) * 16);
                            x[2 * i] = y.x, x[2 * i + 1] = y.y;
                        }
                    };
#pragma unroll
                    for (int k = 0; k < KS; k++) load4(v[k], from + k * 512, q);
                    if constexpr (C9) load4(v8, mine + slot + 8 * 128, 0);
                    load4(bv, mine + slot + Slot::kRows * 128, 0);
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        z[i][0] = C9 ? v8[i] * c[0][half + i] : 0;
                        z[i][1] = C9 ? v8[i] * c[1][half + i] : 0;
                    }
#pragma unroll
                    for (int k = 0; k < KS; k++)
#pragma unroll
                        for (int i = 0; i < 4; i++) dmma(z[i], v[k][i], E[k][half + i]);
                    if constexpr (A9) {
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            z9[i] = v[0][i] * c[2][half + i];
                            if constexpr (KS > 1) z9[i] = fma(v[KS - 1][i], c[3][half + i], z9[i]);
                            if constexpr (C9) z9[i] = fma(v8[i], c[4][half + i], z9[i]);
                        }
                    }
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        double sum = A9 ? a9 * z9[i] : 0;
                        sum = fma(a.x, z[i][0], sum);
                        gb[half + i] = fma(a.y, z[i][1], sum);
                        s[0] = fma(bv[i], z[i][0], s[0]);
                        s[1] = fma(bv[i], z[i][1], s[1]);
                        if constexpr (A9) s9 = fma(bv[i], z9[i], s9);
                    }
                }
                // gB: the sums over the edge's four lanes, columns 2q and 2q + 1 for lane q
                if (gB != nullptr) {
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const double send = q & 2 ? gb[i] : gb[i + 4], keep = q & 2 ? gb[i + 4] : gb[i];
                        gb[i] = keep + __shfl_xor_sync(kFullMask, send, 2);
                    }
#pragma unroll
                    for (int i = 0; i < 2; i++) {
                        const double send = q & 1 ? gb[i] : gb[i + 2], keep = q & 1 ? gb[i + 2] : gb[i];
                        gb[i] = keep + __shfl_xor_sync(kFullMask, send, 1);
                    }
                    if (live && b0 + 2 * q < L)
                        *reinterpret_cast<double2*>(gB + static_cast<int64_t>(e_now) * L + b0 + 2 * q) =
                            make_double2(gb[0], gb[1]);
                }
                if (gA != nullptr) {
                    if constexpr (A9) {
                        s9 += __shfl_xor_sync(kFullMask, s9, 1);
                        s9 += __shfl_xor_sync(kFullMask, s9, 2);
                    }
                    double2* before = reinterpret_cast<double2*>(sums + t * (kStep * 8));
                    double* before9 = sums9 + t * kStep;
                    if (slice > 0) {
                        s[0] += before->x, s[1] += before->y;
                        if constexpr (A9) s9 += *before9;
                    }
                    if (live) {
                        if (slice + 1 < slices) {
                            *before = make_double2(s[0], s[1]);
                            if (A9 && q == 0) *before9 = s9;
                        } else {
                            double* to_a = gA + static_cast<int64_t>(e_now) * g.nA + 2 * q;
                            if (2 * q < g.nA) to_a[0] = s[0];
                            if (2 * q + 1 < g.nA) to_a[1] = s[1];
                            if (A9 && q == 0) to_a[8] = s9;
                        }
                    }
                }
            }
            lo = hi;
        }
    }
    cp_async_wait<0>();
    __syncwarp();
}

// A part, window by window: whole rows where they fit one.
template <int KS, bool C9, bool A9, int LL, typename Off, Cut CUT>
__device__ __forceinline__ void mma_edge_gradients(const RowsArgs<double>& g, const Off* __restrict__ offsets,
                                                   double* __restrict__ gA, double* __restrict__ gB,
                                                   const double* __restrict__ W, const Part<CUT>& part,
                                                   const double* table, unsigned char* ring, int lane,
                                                   const Status& st) {
    int p = static_cast<int>(offsets[part.row_lo]), p_hi = static_cast<int>(offsets[part.row_hi]);
    if constexpr (CUT != kWhole) p = max(p, part.p_lo), p_hi = min(p_hi, part.p_hi);
    int64_t row = part.row_lo;
    while (p < p_hi) {
        const int64_t mine = row + 1 + lane;
        const int end = static_cast<int>(offsets[mine < part.row_hi ? mine : part.row_hi]);
        const int limit = min(p + kGradWindow, p_hi);
        const int whole = __popc(__ballot_sync(kFullMask, mine <= part.row_hi && end <= limit)); // rows that end inside
        const int to = whole > 0 ? __shfl_sync(kFullMask, end, whole - 1) : limit;
        if (to > p)
            mma_edge_window<KS, C9, A9, LL>(g, offsets, gA, gB, W, row, row + max(whole, 1), p, to, table, ring, lane, st);
        row += whole;
        p = to;
    }
}

// Shared memory: the coupling, then the warps' rings, rows of W and sums of gA.
template <int KS, bool C9> constexpr size_t grad_ring_bytes() {
    return kGradDepth * GradSlot<KS, C9>::kBytes + (2 * kWidest * kGradColumns + kGradWindow * 9) * sizeof(double);
}
template <int KS, bool C9, bool A9, int LL>
__global__ void __launch_bounds__(kGradWarps * 32, 1)
sasaw_edge_gradients_mma(const __grid_constant__ RowsArgs<double> g, const int32_t* __restrict__ starts,
                         double* __restrict__ gA, double* __restrict__ gB, double* __restrict__ gW,
                         const double* __restrict__ W, Status st) {
    __shared__ int counter;
    extern __shared__ __align__(128) unsigned char smem[];
    const int warp = __shfl_sync(kFullMask, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    double* table = reinterpret_cast<double*>(smem);
    constexpr int kRing = static_cast<int>(grad_ring_bytes<KS, C9>());
    unsigned char* ring = smem + (GradTable<KS>::scalars(g.nOut) * sizeof(double) + 127) / 128 * 128 + warp * kRing;
    if (threadIdx.x == 0) counter = 0;
    GradTable<KS>::fill(table, g);
    for (int x = lane * 16; x < kRing; x += 512) // (rows of gO and components of A that there are not stay zero)
        *reinterpret_cast<uint4*>(ring + x) = make_uint4(0, 0, 0, 0);
    __syncthreads();
    auto gradients = [&](const auto& part) {
        mma_edge_gradients<KS, C9, A9, LL>(g, starts, gA, gB, W, part, table, ring, lane, st);
    };
    if (*g.longest <= g.limit) {
        // (whole rows also where they are few: cut ones have their E made twice, 52 -> 58 us at 1000 rows)
        for_rows(starts, balanced_row_split(starts, g.rows, blockIdx.x, gridDim.x, lane),
                 balanced_row_split(starts, g.rows, blockIdx.x + 1, gridDim.x, lane), &counter, lane, gradients);
        return;
    }
    clear_for_sums(g, gW);
    for_cuts(starts, g.rows, g.chunk, &counter, lane, gradients);
}

#endif
