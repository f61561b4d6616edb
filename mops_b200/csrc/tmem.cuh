// Tensor memory (TMEM) as a gather buffer.
//
// HPE and SAP read operands at run-time indices that are the same for every batch row: "column
// P[j,k] of my row". TMEM has exactly that shape: 128 lanes by 512 32-bit columns, and a
// `tcgen05.ld.32x32b.xW` hands every lane of a warp W consecutive columns of its own TMEM lane,
// at a column number that is warp-uniform and may come from a register. With lane = batch row
// a gather of one operand for 32 rows is one instruction, and it does not touch the
// shared-memory pipe, which moves 128 bytes per clock per SM (one f64 operand for 32 rows = 2
// clocks) and bounded both operations before. Measured on B200, loads at run-time columns:
// x2 2.0 clocks and x4 2.6 clocks per warp load and sub-partition, i.e. 510 / 790 bytes per
// clock per SM.
//
// A warp can only reach the 32 lanes of its own quadrant (warp number modulo 4).
#ifndef MOPS_B200_TMEM_CUH
#define MOPS_B200_TMEM_CUH

#include <cstdint>

#include "bulk.cuh"

namespace mops_b200 {

// Allocation by one converged warp; the address is written to shared memory. `columns` is a
// power of two, 32 to 512.
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_address_out, unsigned columns) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(
                     smem_address(smem_address_out)),
                 "r"(columns)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void tmem_free(uint32_t address, unsigned columns) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(address),
                 "r"(columns)
                 : "memory");
}

// Around a __syncthreads() that orders TMEM accesses of different warps.
__device__ __forceinline__ void tmem_fence_before_sync() {
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
}
__device__ __forceinline__ void tmem_fence_after_sync() {
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
}

// The address of column 0 of the calling warp's quadrant.
__device__ __forceinline__ uint32_t tmem_quadrant(uint32_t address, int warp) {
    return address + (static_cast<uint32_t>(warp & 3) << 21);
}

// W consecutive columns of the lane, asynchronously: the registers are valid after tmem_wait_load.
__device__ __forceinline__ void tmem_load(uint32_t a, uint32_t (&r)[1]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];\n" : "=r"(r[0]) : "r"(a));
}
__device__ __forceinline__ void tmem_load(uint32_t a, uint32_t (&r)[2]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0,%1}, [%2];\n"
                 : "=r"(r[0]), "=r"(r[1])
                 : "r"(a));
}
__device__ __forceinline__ void tmem_load(uint32_t a, uint32_t (&r)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(a));
}
__device__ __forceinline__ void tmem_load(uint32_t a, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
                   "=r"(r[6]), "=r"(r[7])
                 : "r"(a));
}
// Waits for all of the warp's loads in flight.
__device__ __forceinline__ void tmem_wait_load() {
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
}
// Keeps the uses of a loaded register behind the wait (the load is asynchronous, so the compiler
// must not move them up on the strength of the load instruction alone).
template <int N> __device__ __forceinline__ void tmem_pin(uint32_t (&r)[N]) {
#pragma unroll
    for (int i = 0; i < N; i++) asm volatile("" : "+r"(r[i]));
}

__device__ __forceinline__ void tmem_store(uint32_t a, float v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};\n" ::"r"(a),
                 "r"(__float_as_uint(v))
                 : "memory");
}
__device__ __forceinline__ void tmem_store(uint32_t a, double v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1,%2};\n" ::"r"(a),
                 "r"(__double2loint(v)), "r"(__double2hiint(v))
                 : "memory");
}
// N consecutive columns.
__device__ __forceinline__ void tmem_store(uint32_t a, const uint32_t (&r)[2]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1,%2};\n" ::"r"(a), "r"(r[0]), "r"(r[1]) : "memory");
}
__device__ __forceinline__ void tmem_store(uint32_t a, const uint32_t (&r)[4]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};\n" ::"r"(a),
                 "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3])
                 : "memory");
}
__device__ __forceinline__ void tmem_store(uint32_t a, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n" ::"r"(a),
                 "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
__device__ __forceinline__ void tmem_store(uint32_t a, const uint32_t (&r)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n" ::"r"(a),
                 "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
                 : "memory");
}
__device__ __forceinline__ void tmem_store(uint32_t a, const uint32_t (&r)[32]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};\n" ::"r"(a),
                 "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
                 : "memory");
}
__device__ __forceinline__ void tmem_wait_store() {
    asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
}

// Scalar r of a group of columns that holds W / words(T) rows.
template <typename T, int W> __device__ __forceinline__ T tmem_value(const uint32_t (&w)[W], int r) {
    if constexpr (sizeof(T) == 8)
        return __hiloint2double(static_cast<int>(w[2 * r + 1]), static_cast<int>(w[2 * r]));
    else
        return __uint_as_float(w[r]);
}

} // namespace mops_b200

#endif
