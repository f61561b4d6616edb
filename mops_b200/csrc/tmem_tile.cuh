// Tiles of a row-major operand in tensor memory: how rows travel from HBM to TMEM lanes.
//
// A block works on 128 R batch rows at a time: row 128 r + l of the tile is TMEM lane l, slot r.
// Column n of the operand occupies W = R words(T) TMEM columns starting at n W, so that one load
// of W columns gives a lane its R values of column n. Rows arrive in slabs of 128 (one per slot):
// contiguous in HBM, copied asynchronously into shared memory with a padded row stride (an odd
// multiple of 16 bytes: no bank conflicts when every lane reads 16 bytes of its own row), from
// there to TMEM. The next tile's slabs are under way while the current tile is worked on.
#ifndef MOPS_B200_TMEM_TILE_CUH
#define MOPS_B200_TMEM_TILE_CUH

#include "tmem.cuh"

namespace mops_b200 {

constexpr int kTmemThreads = 512; // sixteen warps: four per quadrant
constexpr int kTmemGroups = kTmemThreads / 128;
constexpr int kSlabRows = 128;
constexpr int kTmemColumns = 512;

__host__ __device__ constexpr int words_of(int scalar_bytes) { return scalar_bytes / 4; }

// Shared-memory row stride of a slab: an odd number of 16-byte units.
__host__ __device__ inline int slab_stride(int row_bytes) {
    const int units = (row_bytes + 15) / 16;
    return (units | 1) * 16;
}

template <int UNIT> __device__ __forceinline__ void copy_unit(void* dst, const void* src) {
    if constexpr (UNIT == 16)
        lane_copy16(dst, src);
    else
        cp_async<UNIT>(dst, src);
}

// Starts the copy of `rows` (<= 128) rows of `row_bytes` bytes each, contiguous at `src`.
template <int UNIT>
__device__ __forceinline__ void start_slab_units(unsigned char* slab, const unsigned char* src,
                                                 int rows, int row_bytes, int stride, int tid) {
    const int per_row = row_bytes / UNIT; // >= 1
    const int total = rows * per_row;
    const int dr = kTmemThreads / per_row, dc = kTmemThreads - dr * per_row;
    int row = tid / per_row, c = tid - row * per_row;
    for (int x = tid; x < total; x += kTmemThreads) {
        copy_unit<UNIT>(slab + row * stride + c * UNIT, src + static_cast<size_t>(x) * UNIT);
        row += dr;
        c += dc;
        if (c >= per_row) {
            c -= per_row;
            row++;
        }
    }
}

// `unit`: largest of 16, 8, 4 that divides the row size and the operand's address.
__device__ __forceinline__ void start_slab(unsigned char* slab, const void* src, int rows,
                                           int row_bytes, int stride, int unit, int tid) {
    const unsigned char* s = static_cast<const unsigned char*>(src);
    if (unit == 16)
        start_slab_units<16>(slab, s, rows, row_bytes, stride, tid);
    else if (unit == 8)
        start_slab_units<8>(slab, s, rows, row_bytes, stride, tid);
    else
        start_slab_units<4>(slab, s, rows, row_bytes, stride, tid);
}

inline int copy_unit_of(const void* base, size_t row_bytes) {
    const size_t both = reinterpret_cast<size_t>(base) | row_bytes;
    return both % 16 == 0 ? 16 : both % 8 == 0 ? 8 : 4;
}

// 0 if |v| is 0 or in [2^-511, 2^512) (f32: [2^-63, 2^64)), else 1: the product of two such values is 0 or a normal
// number. (No branches: the loops that look at values also move them.)
__device__ __forceinline__ unsigned out_of_band(double v) {
    const uint32_t word = (static_cast<uint32_t>(__double2hiint(v)) & 0x7fffffffu) | min(static_cast<uint32_t>(__double2loint(v)), 1u);
    return static_cast<unsigned>(word - (512u << 20) >= (1023u << 20)) & static_cast<unsigned>(word != 0);
}
__device__ __forceinline__ unsigned out_of_band(float v) {
    const uint32_t word = __float_as_uint(v) & 0x7fffffffu;
    return static_cast<unsigned>(word - (64u << 23) >= (127u << 23)) & static_cast<unsigned>(word != 0);
}

// Moves all R slabs of a tile from shared memory to the TMEM columns of one operand. `column0`: TMEM
// address of the operand's first column in the warp's quadrant; `slab`: bytes from one slot's rows
// to the next. The sixteen warps share the columns: warp group g takes 16-byte pieces g, g + 4, ...
// of the rows; the columns of a piece, with their R slots each, are consecutive in TMEM and go
// there in one store (one store per scalar took four to eight times as many, and most of the time
// of a tile with few records). CHECK: a bit for every slot of which the thread moved a
// value out_of_band.
template <typename T, int W, bool CHECK = false>
__device__ __forceinline__ unsigned slabs_to_tmem(const unsigned char* rows, int slab, int stride, int N,
                                              uint32_t column0, int warp, int lane) {
    constexpr int per16 = 16 / sizeof(T), words = words_of(sizeof(T)), R = W / words;
    const unsigned char* row = rows + ((warp & 3) * 32 + lane) * stride;
    unsigned bad = 0;
    for (int p = warp >> 2; p * per16 < N; p += kTmemGroups) {
        uint32_t r[per16 * W];
#pragma unroll
        for (int s = 0; s < R; s++) {
            const uint4 v = *reinterpret_cast<const uint4*>(row + s * slab + p * 16);
            const uint32_t word[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int i = 0; i < 4; i++) r[i / words * W + s * words + i % words] = word[i];
        }
        if constexpr (CHECK) {
#pragma unroll
            for (int n = 0; n < per16; n++)
#pragma unroll
                for (int s = 0; s < R; s++) {
                    T v;
                    if constexpr (sizeof(T) == 8)
                        v = __hiloint2double(static_cast<int>(r[n * W + 2 * s + 1]), static_cast<int>(r[n * W + 2 * s]));
                    else
                        v = __uint_as_float(r[n * W + s]);
                    bad |= (out_of_band(v) & static_cast<unsigned>(p * per16 + n < N)) << s;
                }
        }
        const uint32_t at = column0 + p * per16 * W;
        if ((p + 1) * per16 <= N) {
            tmem_store(at, r);
        } else { // the last columns of an operand whose rows are no multiple of 16 bytes
#pragma unroll
            for (int n = 0; n + 1 < per16; n++)
                if (p * per16 + n < N)
#pragma unroll
                    for (int i = 0; i < W; i++)
                        tmem_store(at + n * W + i, __uint_as_float(r[n * W + i]));
        }
    }
    return bad;
}

} // namespace mops_b200

#endif
