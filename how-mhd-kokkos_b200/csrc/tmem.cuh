// tmem.cuh -- tensor memory (256 KB per SM, 128 lanes x 512 columns of 32 bits)
// as a per-lane store beside the registers: allocation, and the moves between
// a warp's registers and its 32 lanes (tcgen05.alloc / st / ld / wait, PTX ISA).
// Warp w of a block of four reaches lanes 32 w .. 32 w + 31.
#pragma once

#include <cstdint>

#include "tma.cuh"

namespace how {

// One whole warp: `columns` (a power of two >= 32) of tensor memory; the
// address lands in shared memory.
template <int COLUMNS> __device__ __forceinline__ void tmem_alloc(uint32_t* where) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(where)), "n"(COLUMNS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
template <int COLUMNS> __device__ __forceinline__ void tmem_free(uint32_t address) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(address), "n"(COLUMNS));
}
__device__ __forceinline__ void tmem_wait_stores() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// N values per lane at consecutive columns
template <int N> __device__ __forceinline__ void tmem_store(uint32_t at, const uint32_t* v);
template <int N> __device__ __forceinline__ void tmem_load(uint32_t at, uint32_t* v);

template <> __device__ __forceinline__ void tmem_store<2>(uint32_t at, const uint32_t* v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1, %2};"
                 ::"r"(at), "r"(v[0]), "r"(v[1]) : "memory");
}
template <> __device__ __forceinline__ void tmem_load<2>(uint32_t at, uint32_t* v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0, %1}, [%2];"
                 : "=r"(v[0]), "=r"(v[1]) : "r"(at) : "memory");
}
template <> __device__ __forceinline__ void tmem_load<4>(uint32_t at, uint32_t* v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(at) : "memory");
}
template <> __device__ __forceinline__ void tmem_store<8>(uint32_t at, const uint32_t* v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"r"(at), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}
// The registers of the loads before are defined from here on: the values pass
// through, so that no use moves ahead of the wait.
template <int N> __device__ __forceinline__ void tmem_wait_loads(uint32_t* v) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < N; ++i) asm volatile("" : "+r"(v[i]));
}

}  // namespace how
