// The row sums of sasaw_rows.cu (forward and gW) on the FP64 tensor-core instruction, f64.
//
//   G_i[m1,c,b] = sum over the edges e of row i of A[e,m1] V[e,c,b],    V[e,c,b] = B[e,b] G[r_e,c,b]
//
// is a product of matrices with the edges as the contracted index: for a channel c and eight columns b a
// step of four edges is one DMMA with b as its rows and eight m1 as its columns. Lane = 4 n + q holds V of
// edge q and of columns 2n, 2n + 1 (one 16-byte load; two DMMA take the even and the odd columns of sixteen),
// which is what the instruction wants as its first operand, and A[q][n] as the second. The ninth of nine
// components of A goes by ordinary multiply-adds from the same registers. Results need no exchange before
// the coupling is applied: out^T[b,o] = sum_{m1} G^T[b,m1] D[m1,o] takes them as the first operand of another
// DMMA, with m1 = 2q and m1 = 2q + 1 as two contracted groups of four.
//
// A warp has sixteen columns of a row: 108 registers of sums for 9 x 9 channels, so that twelve warps
// fit an SM (168 registers, of which 9 x 9 channels spill 36 to 140 bytes and no other channels any). Its operands come through a ring of asynchronous copies, three steps deep, laid out without bank
// conflicts. (Loaded straight into registers, which needs no ring, the same loads touch four lines per eight
// lanes, and the L1 pipe was 83 % busy: 1.60 against 1.04 ms in the same run.) The steps run along the positions whatever rows they belong to: one that a row's end cuts is
// multiplied once for each of its rows, the other edges as zeros.
//
// What bounds it: the FP64 pipe (36 DMMA, 36 DFMA and 36 DMUL for four edges and 32 columns, 64 % busy), latency
// at three warps per scheduler; 107 instructions per edge. 9 x 9 x 9 channels, 32 columns, against the multiply-adds of
// sasaw_rows.cu: 4.2 10^6 edges forward 1.65 -> 1.16 to 1.27 ms (tables that fit L2: 1.47 -> 0.99), 1.2 10^6, 60 per row,
// 609 -> 377 us; 16 x 9 -> 9 channels, 16 columns, 3.9 10^5 edges 320 -> 144 to 160 us.
#ifndef MOPS_B200_SASAW_ROWS_MMA_CUH
#define MOPS_B200_SASAW_ROWS_MMA_CUH

constexpr int kMmaWarps = 12;
constexpr int kMmaColumns = 16; // of a warp
constexpr int kMmaStep = 4;     // edges
constexpr int kMmaDepth = 3;    // steps of a warp's ring

// One step's operands: for every edge NC rows of sixteen columns and B's (an odd multiple of 32 bytes apart, so that
// the 16-byte loads of eight lanes, two pieces of four edges, meet no bank twice), then the A rows.
template <int MA, int NC> struct MmaSlot {
    static constexpr int kRow = kMmaColumns * 8;
    static constexpr int kEdge = (NC + 1) * kRow + 32;
    static constexpr int kA = kMmaStep * kEdge;
    static constexpr int kARow = MA == 1 ? 96 : 160; // (four lanes' edges at 8-byte loads: other banks)
    static constexpr int kBytes = kA + kMmaStep * kARow;
};
template <int MA, int NC> constexpr int kMmaRing = kMmaDepth * MmaSlot<MA, NC>::kBytes;

// Fragments of the coupling: [tile of eight outputs][c][s][lane], s = 2 m + j the components 8 m + 2 q + j of A and
// behind them the ninth. A last tile of one output holds it for all n.
template <int MA, bool NINTH> struct MmaTable {
    static constexpr int S = 2 * MA + (NINTH ? 1 : 0);
    static constexpr __host__ __device__ size_t scalars(int n_out, int pad_c) {
        return static_cast<size_t>((n_out + 7) / 8) * pad_c * S * 32;
    }
    static __device__ void fill(double* table, const double* __restrict__ D, int n_out, int pad_c, int na) {
        const int size = static_cast<int>(scalars(n_out, pad_c));
        for (int x = threadIdx.x; x < size; x += blockDim.x) {
            const int q = x & 3, n = x >> 2 & 7, s = (x >> 5) % S, c = (x >> 5) / S % pad_c;
            const int o0 = (x >> 5) / S / pad_c * 8;
            const int o = n_out - o0 == 1 ? o0 : o0 + n;
            const int m1 = s < 2 * MA ? 8 * (s >> 1) + 2 * q + (s & 1) : 8;
            table[x] = o < n_out && m1 < na ? __ldg(D + (static_cast<size_t>(o) * na + m1) * pad_c + c) : 0.0;
        }
    }
};

// The columns [b0, b0 + 16) of a part. FULL: the channels fill every pass. LL: L where it is known (0 otherwise).
template <int MA, bool NINTH, int NC, bool FULL, int LL, typename Off, Cut CUT>
__device__ __forceinline__ void mma_sum_rows(const RowsArgs<double>& g, const Off* __restrict__ offsets,
                                             double* __restrict__ out, const Part<CUT>& part, int b0,
                                             const double* table, unsigned char* ring, int lane,
                                             const Status& st) {
    constexpr int S = MmaTable<MA, NINTH>::S;
    using Slot = MmaSlot<MA, NC>;
    const int q = lane & 3, n = lane >> 2;
    const int L = LL > 0 ? LL : g.L;
    const int64_t row_lo = part.row_lo, row_hi = part.row_hi;
    int p_lo = static_cast<int>(offsets[row_lo]), p_hi = static_cast<int>(offsets[row_hi]);
    if constexpr (CUT != kWhole) p_lo = max(p_lo, part.p_lo), p_hi = min(p_hi, part.p_hi);
    const int last = p_hi - 1, steps = (p_hi - p_lo + kMmaStep - 1) / kMmaStep;

    const bool store = b0 + 2 * n < L;
    const int b = b0 + 2 * n;
    const int l_row = L * 8, g_row = g.nC * l_row, a_row = g.nA * 8;
    // The copies: lanes 8 u ... 8 u + 7 bring edge u of a step, 16 bytes of every row each.
    const int u = lane >> 3, piece = lane & 7;
    const int from = min(b0 + 2 * piece, L - 2); // (behind the last column: read again, and not used)
    const unsigned to = static_cast<unsigned>(__cvta_generic_to_shared(ring)) + u * Slot::kEdge + piece * 16;
    const unsigned to_a = static_cast<unsigned>(__cvta_generic_to_shared(ring)) + Slot::kA + u * Slot::kARow + piece * 8;
    const unsigned char* b_base = reinterpret_cast<const unsigned char*>(g.B + from);
    const unsigned char* a_base = reinterpret_cast<const unsigned char*>(g.A + piece);
    const unsigned char* mine = ring + q * Slot::kEdge + n * 16; // this lane's operands
    const unsigned char* mine_a = ring + Slot::kA + q * Slot::kARow + n * 8;

    auto load_edge = [&](int p) {
        const int e = min(p + lane, last);
        return g.perm != nullptr ? __ldg(g.perm + e) : e;
    };
    auto checked = [&](int32_t r) {
        if (clamp_index(r, static_cast<int32_t>(g.rows))) report_bad_index(st, g.bit);
        return r;
    };

    for (int c0 = 0; c0 < g.nC; c0 += NC) {
        const int nc = g.nC - c0 < NC ? g.nC - c0 : NC;
        const unsigned char* g_base = reinterpret_cast<const unsigned char*>(g.G + static_cast<int64_t>(c0) * L + from);
        // Edge numbers and gathered rows of 32 positions: of the block that the copies have reached (0), of the
        // next (1), and the edge numbers of the one behind that (2).
        int block = p_lo, e0 = 0, r0 = 0, e1 = 0, r1 = 0, e2 = 0;
        if (steps > 0) {
            e0 = load_edge(block), e1 = load_edge(block + 32), e2 = load_edge(block + 64);
            r0 = __ldg(g.gather + e0), r1 = __ldg(g.gather + e1);
            r0 = checked(r0);
        }
        int ahead = 0; // the next step to copy
        auto start = [&](int slot) { // (behind the last edge it is copied again: nobody reads it)
            if (ahead * kMmaStep + p_lo == block + 32) {
                block += 32;
                e0 = e1, r0 = checked(r1);
                e1 = e2;
                r1 = __ldg(g.gather + e1);
                e2 = load_edge(block + 64);
            }
            const int at = (ahead & 7) * kMmaStep + u;
            const int64_t e = __shfl_sync(kFullMask, e0, at), r = __shfl_sync(kFullMask, r0, at);
            const unsigned char* src = g_base + r * g_row;
            const unsigned dst = to + slot;
#pragma unroll
            for (int c = 0; c < NC; c++)
                if (FULL || c < nc) cp_async16(dst + c * Slot::kRow, src + c * l_row);
            cp_async16(dst + NC * Slot::kRow, b_base + e * l_row);
            const unsigned char* a = a_base + e * a_row;
            if (piece < g.nA) cp_async_at<8, 0>(to_a + slot, a);
            if ((MA == 2 || NINTH) && piece + 8 < g.nA) cp_async_at<8, 64>(to_a + slot, a + 64);
            cp_async_commit();
            ahead++;
        };
        if (steps > 0) {
            __syncwarp(); // (the ring's last readers)
#pragma unroll 1
            for (int i = 0; i < kMmaDepth - 1; i++) start(i * Slot::kBytes);
        }
        // `slot`: of step `now`, whose copies have arrived; before the first one the last of the ring
        int now = -1, slot = (kMmaDepth - 1) * Slot::kBytes;

        int lo = p_lo;
        for (int64_t row = row_lo; row < row_hi; row++) {
            int hi = static_cast<int>(offsets[row + 1]);
            if constexpr (CUT != kWhole) hi = min(hi, p_hi);
            double* at = out + row * g.nOut * L + b;
            int stride = L; // from one output to the next
            if constexpr (CUT == kPiece) {
                if (row == row_lo && part.head != nullptr) {
                    at = reinterpret_cast<double*>(part.head) + 2 * n;
                    stride = kMmaColumns;
                }
            }
            if (lo >= hi) {
                if (CUT != kCut && c0 == 0 && store)
                    for (int o = q; o < g.nOut; o += 4)
                        *reinterpret_cast<double2*>(at + static_cast<int64_t>(o) * stride) = make_double2(0, 0);
                continue;
            }
            double acc[NC][2][MA][2], acc9[NC][2];
#pragma unroll
            for (int c = 0; c < NC; c++)
#pragma unroll
                for (int t = 0; t < 2; t++) {
#pragma unroll
                    for (int m = 0; m < MA; m++) acc[c][t][m][0] = acc[c][t][m][1] = 0;
                    acc9[c][t] = 0;
                }
            auto advance = [&] {
                cp_async_wait<kMmaDepth - 2>();
                __syncwarp();
                start(slot);
                slot += Slot::kBytes;
                if (slot == kMmaRing<MA, NC>) slot = 0;
                now++;
            };
            // The row's edges of step `now`: all four, or (SOME) those for which `live`.
            auto multiply = [&](auto some, bool live) {
                constexpr bool SOME = decltype(some)::value;
                double a[MA], a9 = 0;
#pragma unroll
                for (int m = 0; m < MA; m++) a[m] = *reinterpret_cast<const double*>(mine_a + slot + m * 64);
                if constexpr (NINTH) a9 = *reinterpret_cast<const double*>(ring + Slot::kA + 64 + q * Slot::kARow + slot);
                if (SOME && !live) {
#pragma unroll
                    for (int m = 0; m < MA; m++) a[m] = 0;
                    a9 = 0;
                }
                const double2 bv = *reinterpret_cast<const double2*>(mine + slot + NC * Slot::kRow);
#pragma unroll
                for (int c = 0; c < NC; c++) {
                    if (!FULL && c >= nc) break;
                    const double2 w = *reinterpret_cast<const double2*>(mine + slot + c * Slot::kRow);
                    double v[2] = {w.x * bv.x, w.y * bv.y};
                    if (SOME && !live) v[0] = v[1] = 0;
#pragma unroll
                    for (int t = 0; t < 2; t++) {
#pragma unroll
                        for (int m = 0; m < MA; m++) dmma(acc[c][t][m], v[t], a[m]);
                        if constexpr (NINTH) acc9[c][t] = fma(a9, v[t], acc9[c][t]);
                    }
                }
            };
            // (steps count from the part's first position)
            int first = lo - p_lo;
            const int end = hi - p_lo;
            if (first % kMmaStep != 0) { // the step that the last row ended in
                const int at_q = first / kMmaStep * kMmaStep + q;
                multiply(std::true_type(), at_q >= first && at_q < end);
                first = (first / kMmaStep + 1) * kMmaStep;
            }
#pragma unroll 1
            for (; first + kMmaStep <= end; first += kMmaStep) {
                advance();
                multiply(std::false_type(), true);
            }
            if (first < end) {
                advance();
                multiply(std::true_type(), first + q < end);
            }
            lo = hi;

            const double* d = table + static_cast<size_t>(c0) * S * 32 + lane;
#pragma unroll 1
            for (int o0 = 0; o0 < g.nOut; o0 += 8, d += static_cast<size_t>(g.pad_c) * S * 32) {
                double sum[2][2] = {}; // [t][j]: output o0 + 2 q + j of column b + t
                int first = o0 + 2 * q, count = g.nOut - first;
                if (g.nOut - o0 > 1) {
                    double odd[2][2] = {}; // (two chains per tile)
#pragma unroll
                    for (int c = 0; c < NC; c++)
#pragma unroll
                        for (int s = 0; s < S; s++) {
                            const double f = d[(c * S + s) * 32];
#pragma unroll
                            for (int t = 0; t < 2; t++) {
                                const double v = s < 2 * MA ? acc[c][t][s / 2 % MA][s & 1] : acc9[c][t];
                                dmma((c * S + s) & 1 ? odd[t] : sum[t], v, f);
                            }
                        }
#pragma unroll
                    for (int t = 0; t < 2; t++) sum[t][0] += odd[t][0], sum[t][1] += odd[t][1];
                } else { // one output: multiply-adds, and the sum over the lanes that share a column
#pragma unroll
                    for (int c = 0; c < NC; c++)
#pragma unroll
                        for (int s = 0; s < S; s++) {
                            const double f = d[(c * S + s) * 32];
#pragma unroll
                            for (int t = 0; t < 2; t++) {
                                const double v = s < 2 * MA ? acc[c][t][s / 2 % MA][s & 1] : acc9[c][t];
                                sum[t][(c * S + s) & 1] = fma(v, f, sum[t][(c * S + s) & 1]);
                            }
                        }
#pragma unroll
                    for (int t = 0; t < 2; t++) {
                        double v = sum[t][0] + sum[t][1];
                        v += __shfl_xor_sync(kFullMask, v, 1);
                        sum[t][0] = v + __shfl_xor_sync(kFullMask, v, 2);
                    }
                    first = o0, count = q == 0 ? 1 : 0;
                }
                if (store) {
#pragma unroll
                    for (int j = 0; j < 2; j++) {
                        if (j >= count) break;
                        double* to = at + static_cast<int64_t>(first + j) * stride;
                        if constexpr (CUT == kCut) {
                            red_add(to, sum[0][j]);
                            red_add(to + 1, sum[1][j]);
                        } else {
                            double2 v = make_double2(sum[0][j], sum[1][j]);
                            if (c0 > 0) {
                                const double2 u = *reinterpret_cast<const double2*>(to);
                                v.x += u.x, v.y += u.y;
                            }
                            *reinterpret_cast<double2*>(to) = v;
                        }
                    }
                }
            }
        }
        cp_async_wait<0>();
        __syncwarp();
    }
}

// As for_rows and for_cuts: every part once for each slice of sixteen columns, one slice of all parts after the
// other (so that what they gather is a slice of the table at a time: less to keep in L2).
template <typename F>
__device__ __forceinline__ void for_slices(int parts, int slices, int* counter, int lane, F&& f) {
    int slice = 0, before = 0; // parts of the slices before
    while (true) {
        int at = 0;
        if (lane == 0) at = atomicAdd(counter, 1);
        at = __shfl_sync(kFullMask, at, 0);
        while (at - before >= parts && slice < slices) slice++, before += parts;
        if (slice >= slices) break;
        f(at - before, slice);
    }
}

// Shared memory: fragments of the coupling, then the warps' rings.
template <int MA, bool NINTH, int NC, bool FULL, int LL>
__global__ void __launch_bounds__(kMmaWarps * 32, 1)
sasaw_sum_rows_mma(const __grid_constant__ RowsArgs<double> g, const int64_t* __restrict__ offsets,
                   const int32_t* __restrict__ starts, double* __restrict__ out, RowsRun run, Status st) {
    if (run != kAlways && saw_unsorted(st) != (run == kIfUnsorted)) return;
    __shared__ int counter;
    extern __shared__ __align__(128) unsigned char smem[];
    const int warp = __shfl_sync(kFullMask, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    double* table = reinterpret_cast<double*>(smem);
    constexpr int kRing = kMmaRing<MA, NC>;
    unsigned char* ring = smem + MmaTable<MA, NINTH>::scalars(g.nOut, g.pad_c) * sizeof(double) + warp * kRing;
    if (threadIdx.x == 0) counter = 0;
    MmaTable<MA, NINTH>::fill(table, g.D, g.nOut, g.pad_c, g.pad_a);
    for (int x = lane * 16; x < kRing; x += 512) // (components of A beyond nA stay zero)
        *reinterpret_cast<uint4*>(ring + x) = make_uint4(0, 0, 0, 0);
    __syncthreads();
    const int slices = (g.L + kMmaColumns - 1) / kMmaColumns;
    auto sum = [&](const auto* at, const auto& part, int slice) {
        mma_sum_rows<MA, NINTH, NC, FULL, LL>(g, at, out, part, slice * kMmaColumns, table, ring, lane, st);
    };
    __shared__ int64_t heads[kMostPieces];
    auto rows = [&](const auto* at) {
        for_few_rows(g, at, kMmaWarps, slices, kMmaColumns, out, heads, smem, &counter, lane,
                     [&](const auto& part, int slice) { sum(at, part, slice); }, [&](int64_t lo, int64_t hi) {
                         const int n = chunk_rows(at, lo, hi, kMmaWarps);
                         for_slices(static_cast<int>((hi - lo + n - 1) / n), slices, &counter, lane, [&](int i, int slice) {
                             const int64_t r = lo + static_cast<int64_t>(i) * n;
                             sum(at, Part<kWhole>{r, r + n < hi ? r + n : hi}, slice);
                         });
                     });
    };
    if (run == kSorted) {
        rows(offsets);
    } else if (*g.longest <= g.limit) {
        rows(starts);
    } else { // (`out` has been cleared by a kernel before)
        const int edges = starts[g.rows], chunks = (edges + g.chunk - 1) / g.chunk;
        const int mine = static_cast<int>(blockIdx.x), blocks = static_cast<int>(gridDim.x);
        for_slices(chunks > mine ? (chunks - mine + blocks - 1) / blocks : 0, slices, &counter, lane, [&](int i, int slice) {
            const int p = (mine + i * blocks) * g.chunk, end = edges - p > g.chunk ? p + g.chunk : edges;
            // the rows of the first and of the last edge
            sum(starts, Part<kCut>{warp_count_weighted_le(starts, g.rows + 1, 0, p, lane) - 1,
                                   warp_count_weighted_le(starts, g.rows + 1, 0, end - 1, lane), p, end, nullptr}, slice);
        });
    }
}

#endif
