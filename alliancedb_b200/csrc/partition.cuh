// partition.cuh -- digit functions shared by the
// partitioned joins (paged.cuh does the partitioning itself).
// The digit is (key >> shift) & (F - 1): the low-bit radix of PRO
// (HASH_BIT_MODULO, hashing/joins/parallel_radix_join.cpp:68), shift = the bits
// an earlier pass consumed.  NPO's partitioned form and the sort-merge names take
// it from the top bits of key * kHashMul (equal keys still meet in one partition;
// the reference's range split of the high bits, sorting/joins/
// sortmergejoin_multiway.cpp:475-487, is not needed for that).
#pragma once

#include "adb_common.cuh"

namespace adb {

__device__ __forceinline__ uint64_t ld_stream(const uint64_t *p) {
    return __ldcs(reinterpret_cast<const unsigned long long *>(p));
}

// Bulk prefetch of [p, p + bytes) into L2 (p 16-byte aligned, bytes a multiple of 16).
__device__ __forceinline__ void prefetch_l2(const void *p, uint32_t bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

struct DigitFn {
    uint32_t shift;
    uint32_t mask;      // F - 1
    bool hashed = false;   // the pass applies it to key * kHashMul
    __host__ __device__ __forceinline__ uint32_t operator()(uint32_t key) const { return (key >> shift) & mask; }
};

__host__ __device__ __forceinline__ uint64_t chunk_of(uint64_t n, int G) {
    uint64_t c = (n + G - 1) / G;
    return (c + 1) & ~1ULL;                     // even -> 16-byte aligned chunk starts
}

}  // namespace adb
