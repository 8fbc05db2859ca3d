// npo_join.cuh -- no-partitioning hash join (NPO, NPO_st) on one global table.
//
// Replaces hashing/joins/no_partitioning_join.cpp:112-476 (NPO_st, npo_thread,
// np_distribute, NPO) and its table code in hashing/joins/common_functions.cpp
// (allocate_hashtable :75-102, build_hashtable_mt :350-400, probe_hashtable
// :221-280).  The reference chains 32-byte buckets of two tuples behind
// per-bucket latches; on the GPU a slot is 8 bytes, the tuple word itself,
// claimed with one 64-bit atomicCAS.  Two forms: buckets of four slots, three slots
// per build tuple (npo_build, npo_probe: NPO by default while the table stays in
// the 126 MB L2, and adb_npo_join_noalloc), and an open-addressing array of 2^l2
// slots, load <= 0.5, probed linearly from a four-slot window (by table region,
// npo.cu, where the caller asks for regions).
//
// The empty marker is the all-ones word.  A build tuple equal to it (key and
// payload both 0xFFFFFFFF) is counted on the side instead of stored, and
// probes with key 0xFFFFFFFF add those matches, so no key value is reserved.
#pragma once

#include "adb_common.cuh"
#include "partition.cuh"

namespace adb {

constexpr uint64_t kEmpty = ~0ULL;

__host__ __device__ __forceinline__ uint32_t npo_hash(uint32_t key, uint32_t log2n) {
    return log2n ? (uint32_t)((key * kHashMul) >> (32 - log2n)) : 0u;
}

// Inserts tuple word w (not the empty marker) by linear probing from `slot`.
__device__ __forceinline__ void npo_insert_from(uint64_t *table, uint64_t mask, uint64_t slot, uint64_t w,
                                                int *err) {
    for (uint64_t tries = 0;;) {
        const unsigned long long prev = atomicCAS(reinterpret_cast<unsigned long long *>(table + slot),
                                                  (unsigned long long)kEmpty, (unsigned long long)w);
        if (prev == kEmpty) return;
        slot = (slot + 1) & mask;
        if (++tries > mask) { atomicExch(err, kErrTableFull); return; }   // table full: cannot happen at load <= 0.5
    }
}

// Count, checksum and optional materialisation of a probe's matches.
template <bool kMaterialize>
struct NpoSink {
    Acc a;
    uint64_t *mat;
    unsigned long long *mat_n;
    uint64_t mat_cap;
    __device__ __forceinline__ void match(uint64_t s, uint32_t key, uint32_t rpay, uint64_t sh) {
        a.count++;
        a.sum += pair_hash_pre(key, rpay, sh);
        if (kMaterialize) {
            const unsigned long long k = atomicAdd(mat_n, 1ull);
            if (k < mat_cap) mat[k] = s;
        }
    }
};

// The matches of S tuple s (key 0xFFFFFFFF) with the nsent build tuples that
// equal the empty marker.
template <bool kMaterialize>
__device__ __forceinline__ void npo_add_sentinels(NpoSink<kMaterialize> &sink, uint64_t s, uint64_t nsent) {
    sink.a.count += nsent;
    sink.a.sum += nsent * pair_hash(0xFFFFFFFFu, 0xFFFFFFFFu, tpay(s));
    if (kMaterialize)
        for (uint64_t t = 0; t < nsent; t++) {
            const unsigned long long k = atomicAdd(sink.mat_n, 1ull);
            if (k < sink.mat_cap) sink.mat[k] = s;
        }
}

// A probe's first read: the four slots b .. b + 3 from b = slot & ~1, the
// 16-byte pair holding the start slot and the pair after it (wrapping at the
// table's end), two 16-byte loads.  Starting the window at the start slot's
// pair instead of its aligned 32-byte sector leaves one or two slots after
// the start slot in every window (the sector leaves none for a start slot in
// its last place): at load 0.5 a probe then has to read on past the window
// about 19 % of the time instead of about 47 %.
__device__ __forceinline__ void npo_window(const uint64_t *table, uint64_t mask, uint64_t slot, ulonglong2 &lo,
                                           ulonglong2 &hi) {
    const uint64_t b = slot & ~1ULL;
    lo = __ldg(reinterpret_cast<const ulonglong2 *>(table + b));
    hi = __ldg(reinterpret_cast<const ulonglong2 *>(table + ((b + 2) & mask)));
}

// The slots after a probe's window: linear probing from slot
// (slot & ~1) + 4 until the first empty slot, for a probe whose run of
// occupied slots reached the window's end.
template <bool kMaterialize>
__device__ __forceinline__ void npo_probe_rest(NpoSink<kMaterialize> &sink, const uint64_t *table, uint64_t mask,
                                               uint64_t s, uint64_t slot, uint64_t sh) {
    const uint32_t key = tkey(s);
    uint64_t sl = ((slot & ~1ULL) + 4) & mask;
    for (uint64_t tries = 0; tries <= mask; tries++) {
        const uint64_t v = table[sl];
        if (v == kEmpty) break;
        if (tkey(v) == key) sink.match(s, key, tpay(v), sh);
        sl = (sl + 1) & mask;
    }
}

// One probe's window: S tuple s with start slot `slot`, given its window
// (lo, hi, read by npo_window), scanned from the start slot; the matches of
// build tuples equal to the empty marker (nsent of them, key 0xFFFFFFFF) are
// added here too.  Returns true when the run of occupied slots reaches the
// window's end, so that npo_probe_rest must go on.
template <bool kMaterialize>
__device__ __forceinline__ bool npo_probe_window(NpoSink<kMaterialize> &sink, uint64_t s, uint64_t slot,
                                                 ulonglong2 lo, ulonglong2 hi, uint64_t nsent, uint64_t &sh) {
    const uint32_t key = tkey(s);
    sh = s_half(key, tpay(s));
    const uint64_t w4[4] = {lo.x, lo.y, hi.x, hi.y};
    bool open = true;   // no empty slot met yet
    uint32_t hits = 0;  // matching slots of the window
#pragma unroll
    for (int j = 0; j < 4; j++) {
        if (open && (uint64_t)j >= (slot & 1)) {
            if (w4[j] == kEmpty) open = false;
            else if (tkey(w4[j]) == key) hits |= 1u << j;
        }
    }
    while (hits) {       // one call site for the checksum (usually one match)
        const int j = __ffs(hits) - 1;
        hits &= hits - 1;
        const ulonglong2 h2 = j & 2 ? hi : lo;
        sink.match(s, key, tpay(j & 1 ? h2.y : h2.x), sh);
    }
    if (key == 0xFFFFFFFFu && nsent) npo_add_sentinels(sink, s, nsent);
    return open;
}

// One whole probe: the window, then the slots after it where needed.
template <bool kMaterialize>
__device__ __forceinline__ void npo_probe_one(NpoSink<kMaterialize> &sink, const uint64_t *table, uint64_t mask,
                                              uint64_t s, uint64_t slot, ulonglong2 lo, ulonglong2 hi,
                                              uint64_t nsent) {
    uint64_t sh;
    if (npo_probe_window(sink, s, slot, lo, hi, nsent, sh)) npo_probe_rest(sink, table, mask, s, slot, sh);
}

// ---------------------------------------------------------------------------
// The bucket table: nb buckets of four slots (one 32-byte sector), bucket =
// the high word of hash x nb, so any nb will do.  A tuple claims the slot its
// hash picks in its bucket with one compare-and-swap; where that is taken it
// reads the bucket for a free slot and goes on to the next bucket when there is
// none.  A probe reads its bucket with one 32-byte load and goes on only past a
// full one: rare for a lane, but some lane of a warp nearly always does, so the
// table has three slots per build tuple (24 bytes): at two, 14 % of the buckets
// are full and the probe's instructions double; at four the table outgrows the
// L2 sooner.  3,000,017 x 5,000,011 tuples, keys over 32 bits (build with the
// table's clearing / probe, us): linear probing in 2^ceil(log2 2|R|) slots with a
// four-slot window 62 / 115; buckets at two slots per tuple 77 / 96, at three
// 68 / 70, at four 90 / 64.
// ---------------------------------------------------------------------------
__host__ __device__ __forceinline__ uint64_t npo_buckets(uint64_t nR) { return nR > 2 ? (3 * nR + 3) / 4 : 1; }

__device__ __forceinline__ void npo_ld_bucket(const uint64_t *p, uint64_t (&v)[4]) {
    asm volatile("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];"
                 : "=l"(v[0]), "=l"(v[1]), "=l"(v[2]), "=l"(v[3])
                 : "l"(p));
}

static __global__ void __launch_bounds__(256)
npo_build(const uint64_t *__restrict__ R, uint64_t nR, uint64_t *__restrict__ table, uint32_t nb,
          unsigned long long *sentinel_cnt, int *err) {
    const uint64_t T = (uint64_t)gridDim.x * blockDim.x;
    auto cas = [&](uint64_t slot, uint64_t w) {
        return atomicCAS(reinterpret_cast<unsigned long long *>(table) + slot, (unsigned long long)kEmpty,
                         (unsigned long long)w) == kEmpty;
    };
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nR; i += T) {
        const uint64_t w = ld_stream(R + i);
        if (w == kEmpty) { atomicAdd(sentinel_cnt, 1ull); continue; }
        // the bucket, and the quarter of its hash range that h lies in: evenly spread hashes
        // (dense keys) then claim their slots without meeting (adb_npo_join_noalloc, 2^21 x
        // 300,000 dense: 83 -> 79 us; bits of h below the bucket's would do for others)
        const uint32_t h = tkey(w) * kHashMul, st = h * nb >> 30;
        uint32_t b = __umulhi(h, nb);
        if (cas(4ull * b + st, w)) continue;
        // the slot was taken: read the bucket for a free one, the next where there is none
        for (uint64_t tries = 0;; tries++) {
            uint64_t v[4];
            asm volatile("ld.relaxed.gpu.global.v4.b64 {%0, %1, %2, %3}, [%4];"
                         : "=l"(v[0]), "=l"(v[1]), "=l"(v[2]), "=l"(v[3])
                         : "l"(table + 4ull * b)
                         : "memory");
            uint32_t empty = 0;
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (v[j] == kEmpty) empty |= 1u << j;
            if (empty) {
                const uint32_t k = (st + __ffs((empty | empty << 4) >> st) - 1) & 3;
                if (cas(4ull * b + k, w)) break;
            } else {
                b = b + 1 == nb ? 0 : b + 1;
            }
            // cannot happen: a third of the slots is used, of the fixed table's at most half
            if (tries > 8ull * nb) { atomicExch(err, kErrTableFull); break; }
        }
    }
}

// One bucket against S tuple s: its first match into (found, pay), further ones
// (repeated build keys) to the sink.  Returns whether the bucket is full, so
// that the next one must be read too.
template <bool kMaterialize>
__device__ __forceinline__ bool npo_scan(NpoSink<kMaterialize> &sink, uint64_t s, uint64_t sh, const uint64_t (&v)[4],
                                         bool &found, uint32_t &pay) {
    const uint32_t key = tkey(s);
    uint32_t hits = 0;
    bool full = true;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const bool empty = v[j] == kEmpty;
        full = full && !empty;
        if (tkey(v[j]) == key && !empty) hits |= 1u << j;
    }
    while (hits) {
        const int j = __ffs(hits) - 1;
        hits &= hits - 1;
        const uint32_t lo = j & 1 ? tpay(v[1]) : tpay(v[0]), hi = j & 1 ? tpay(v[3]) : tpay(v[2]);
        if (found) sink.match(s, key, pay, sh);
        pay = j & 2 ? hi : lo;
        found = true;
    }
    return full;
}

template <bool kMaterialize>
__global__ void __launch_bounds__(256)
npo_probe(const uint64_t *__restrict__ S, uint64_t nS, const uint64_t *__restrict__ table, uint32_t nb,
          const unsigned long long *sentinel_cnt, unsigned long long *acc, uint64_t *mat, unsigned long long *mat_n,
          uint64_t mat_cap, unsigned long long *out) {
    __shared__ uint64_t red[64];
    const uint64_t T = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t nsent = *sentinel_cnt;
    NpoSink<kMaterialize> sink{Acc(), mat, mat_n, mat_cap};
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    uint64_t n = i < nS ? ld_stream(S + i) : 0ULL;
    for (; i < nS; i += T) {
        const uint64_t s = n;
        uint32_t b = __umulhi(tkey(s) * kHashMul, nb);
        uint64_t v[4];
        npo_ld_bucket(table + 4ull * b, v);
        n = i + T < nS ? ld_stream(S + i + T) : 0ULL;   // in flight with the bucket
        const uint64_t sh = s_half(tkey(s), tpay(s));
        bool found = false;
        uint32_t pay = 0;
        bool more = npo_scan(sink, s, sh, v, found, pay);
        for (uint32_t t = 1; more && t < nb; t++) {
            b = b + 1 == nb ? 0 : b + 1;
            uint64_t x[4];
            npo_ld_bucket(table + 4ull * b, x);
            more = npo_scan(sink, s, sh, x, found, pay);
        }
        if (tkey(s) == 0xFFFFFFFFu && nsent) npo_add_sentinels(sink, s, nsent);
        // the lanes of a warp find their matches in different buckets; the
        // checksum then runs once for all of them
        if (found) sink.match(s, tkey(s), pay, sh);
    }
    block_flush(sink.a, acc, red);
    if (out && threadIdx.x == 0) finish_call(acc, out);
}

}  // namespace adb
