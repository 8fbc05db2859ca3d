// smj_sort.cuh -- sorting building blocks of the progressive merge join:
//   chunk_sort        sort up to 8192 tuples by key inside one CTA's shared memory
//   block_sort_kernel sort consecutive blocks of a global array (one CTA per block)
//   merge_kernel      merge-path merge of two sorted global arrays
//   merge_join_kernel merge-path join of two sorted global arrays
// They restate avxsort_tuples (sorting/joins/avxsort.cpp:209-223), the merges of
// avx_merge_tuples / avx_multiway_merge (sorting/joins/merge.cpp:105-171,
// avx_multiway_merge.cpp:200-340) and merge_join (sorting/joins/
// common_functions.cpp:298-372) for the device.
#pragma once

#include "adb_common.cuh"

namespace adb {

constexpr uint32_t kSmjBucketBits = 12;

// Bitonic sort of dst[0..n) on the whole 64-bit word, padded to a power of
// two with all-ones words (which sort last); dst must hold that many words.
__device__ __forceinline__ void bitonic_words(uint64_t *dst, uint32_t n) {
    uint32_t m = 1;
    while (m < n) m <<= 1;
    for (uint32_t i = n + threadIdx.x; i < m; i += blockDim.x) dst[i] = ~0ULL;
    __syncthreads();
    for (uint32_t k = 2; k <= m; k <<= 1) {
        for (uint32_t jj = k >> 1; jj > 0; jj >>= 1) {
            for (uint32_t i = threadIdx.x; i < m; i += blockDim.x) {
                const uint32_t l = i ^ jj;
                if (l > i) {
                    const uint64_t x = dst[i], y = dst[l];
                    const bool up = (i & k) == 0;
                    if ((x > y) == up) { dst[i] = y; dst[l] = x; }
                }
            }
            __syncthreads();
        }
    }
}

// Sorts src[0..n) into dst (both shared memory, dst with room for n rounded
// up to a power of two) by key; tuples with key 0xFFFFFFFF are also ordered
// by payload, so all-ones words come last.  cnt holds 2^12 + 2 counters; red
// holds 64 scratch words.  All threads call it.
//
// MSD counting sort on the (at most) 12 highest key bits that differ within
// the chunk, all-ones words in a bucket of their own behind the rest (out of the
// bit analysis: as a bitonic sort's padding they must come last); then an
// insertion sort inside each bucket when the buckets are wider than one key.
// A bucket of more than 128 tuples that needs sorting makes the whole chunk
// take the bitonic path instead.
__device__ __forceinline__ void chunk_sort(const uint64_t *src, uint32_t n, uint64_t *dst, uint32_t *cnt, uint32_t *red) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    // key bits that differ within the chunk (all-ones words left out)
    uint32_t a = 0xFFFFFFFFu, o = 0;
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
        const uint64_t v = src[i];
        if (v != ~0ULL) {
            a &= tkey(v);
            o |= tkey(v);
        }
    }
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
        a &= __shfl_xor_sync(0xffffffffu, a, s);
        o |= __shfl_xor_sync(0xffffffffu, o, s);
    }
    if (lane == 0) { red[wid] = a; red[32 + wid] = o; }
    __syncthreads();
    a = 0xFFFFFFFFu;
    o = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) { a &= red[w]; o |= red[32 + w]; }
    __syncthreads();
    const uint32_t vary = (a & ~o) ? 0u : a ^ o;   // a & ~o != 0: no word counted (a stays all ones)
    const uint32_t hi = vary ? 31 - __clz(vary) : 0u;
    const uint32_t nbits = vary == 0 ? 0u : (hi + 1 < kSmjBucketBits ? hi + 1 : kSmjBucketBits);
    const uint32_t shift = vary == 0 ? 0u : hi + 1 - nbits;
    const uint32_t nb = 1u << nbits, bmask = nb - 1;   // bucket nb: all-ones words
    auto bucket = [&](uint64_t v) { return v == ~0ULL ? nb : (tkey(v) >> shift) & bmask; };
    for (uint32_t d = threadIdx.x; d <= nb; d += blockDim.x) cnt[d] = 0;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) atomicAdd(&cnt[bucket(src[i])], 1u);
    __syncthreads();
    {   // exclusive scan of the bucket counts, contiguous buckets per thread
        const uint32_t per = (nb + 1 + blockDim.x - 1) / blockDim.x;
        const uint32_t d0 = threadIdx.x * per, d1 = min(nb + 1, d0 + per);
        uint32_t loc = 0;
        for (uint32_t d = d0; d < d1; d++) loc += cnt[d];
        uint32_t tot;
        uint32_t ex = block_exclusive_scan(loc, red, &tot);
        for (uint32_t d = d0; d < d1; d++) {
            const uint32_t c = cnt[d];
            cnt[d] = ex;
            ex += c;
        }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
        const uint64_t v = src[i];
        dst[atomicAdd(&cnt[bucket(v)], 1u)] = v;
    }
    __syncthreads();
    // cnt[d] is now the end of bucket d.  With shift == 0 a bucket is one key
    // value: only the bucket of key 0xFFFFFFFF (the last one, if the chunk's
    // common bits are all ones) needs its payloads ordered.  With shift > 0
    // every bucket is insertion-sorted by whole word.  The all-ones bucket is
    // one word value.
    const uint32_t d_first = shift == 0 ? ((a | bmask) == 0xFFFFFFFFu ? bmask : nb) : 0u;
    int big = 0;
    for (uint32_t d = d_first + threadIdx.x; d < nb; d += blockDim.x)
        if (cnt[d] - (d ? cnt[d - 1] : 0u) > 128) big = 1;
    if (__syncthreads_or(big)) {
        bitonic_words(dst, n);
        return;
    }
    for (uint32_t d = d_first + threadIdx.x; d < nb; d += blockDim.x) {
        const uint32_t b = d ? cnt[d - 1] : 0u, e = cnt[d];
        for (uint32_t i = b + 1; i < e; i++) {
            const uint64_t v = dst[i];
            uint32_t j = i;
            while (j > b && dst[j - 1] > v) {
                dst[j] = dst[j - 1];
                j--;
            }
            dst[j] = v;
        }
    }
    __syncthreads();
}


constexpr uint32_t kSortBlock = 8192;                 // tuples a CTA sorts in shared memory
constexpr size_t kBlockSortSmem = (size_t)kSortBlock * 8 * 2 + ((size_t)(1u << kSmjBucketBits) + 4) * 4 + 1024;

// Sorts each kSortBlock-tuple block of in[0..n) into out (same positions).
static __global__ void __launch_bounds__(1024, 1) block_sort_kernel(const uint64_t *in, uint64_t n, uint64_t *out) {
    extern __shared__ __align__(16) unsigned char smem[];
    uint64_t *X = reinterpret_cast<uint64_t *>(smem);
    uint64_t *Y = X + kSortBlock;
    uint32_t *cnt = reinterpret_cast<uint32_t *>(Y + kSortBlock);
    uint32_t *red = cnt + (1u << kSmjBucketBits) + 4;
    const uint64_t b = (uint64_t)blockIdx.x * kSortBlock;
    if (b >= n) return;
    const uint32_t m = (uint32_t)min((uint64_t)kSortBlock, n - b);
    for (uint32_t i = threadIdx.x; i < m; i += blockDim.x) X[i] = in[b + i];
    __syncthreads();
    chunk_sort(X, m, Y, cnt, red);
    for (uint32_t i = threadIdx.x; i < m; i += blockDim.x) out[b + i] = Y[i];
}

// ---------------------------------------------------------------------------
// Merges, merge-path tiled: a CTA produces kMergeTile merged elements.  Two warps
// find where the tile begins and ends in A and in B, the CTA copies both parts to
// shared memory, and each thread merges kMergePer elements there, from where its
// own diagonal cuts the tile.  Bound by latency: the searches, the loads and the
// local merges of one wave of CTAs follow one another.  Runs of 1.6M tuples, us:
// a merge pass 28 with one thread per 64 elements, which read and wrote global
// memory element by element, 12 in this form; the join of two runs 82 / 40.  Tiles
// of 1024 to 2048 tuples by 128 to 512 threads: 12 to 13.6.
// ---------------------------------------------------------------------------
constexpr int kMergeThreads = 256;
constexpr uint32_t kMergePer = 8;
constexpr uint32_t kMergeTile = kMergeThreads * kMergePer;
static_assert(2 * kSortBlock % kMergeTile == 0, "a tile lies within one pair of runs");

struct MergeTile {
    uint64_t v[kMergeTile];                        // A's part, then B's
    uint64_t cut[2];                               // A elements before the tile, and before its end
};

// Number of A elements among the first k elements of merge(A, B), A first on
// equal keys; by one warp, 32 probes a round.
__device__ __forceinline__ uint64_t warp_merge_path(const uint64_t *A, uint64_t na, const uint64_t *B, uint64_t nb,
                                                    uint64_t k, int lane) {
    uint64_t lo = k > nb ? k - nb : 0, hi = k < na ? k : na;
    while (lo < hi) {
        const uint64_t step = (hi - lo + 31) / 32, mid = lo + lane * step;
        const bool before = mid < hi && tkey(A[mid]) <= tkey(B[k - mid - 1]);   // true up to the answer
        const uint32_t c = __popc(__ballot_sync(0xffffffffu, before));
        if (c == 0) break;
        hi = min(hi, lo + c * step);
        lo += (c - 1) * step + 1;
    }
    return lo;
}

// Elements k0 .. k0 + kMergeTile - 1 of merge(A, B): f(o, i, v, from_b) for each of
// the calling thread's, in order, o its place in the tile and i the number of A
// elements of the tile before it.  Every thread of the CTA calls it.
template <class F>
__device__ __forceinline__ void merge_tile(MergeTile &t, const uint64_t *A, uint64_t na, const uint64_t *B, uint64_t nb,
                                           uint64_t k0, F f) {
    const uint64_t k1 = min(na + nb, k0 + kMergeTile);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp < 2) {
        const uint64_t c = warp_merge_path(A, na, B, nb, warp ? k1 : k0, lane);
        if (lane == 0) t.cut[warp] = c;
    }
    __syncthreads();
    const uint64_t i0 = t.cut[0], j0 = k0 - i0;
    const uint32_t n = (uint32_t)(k1 - k0), ta = (uint32_t)(t.cut[1] - i0), tb = n - ta;
    for (uint32_t x = threadIdx.x; x < n; x += kMergeThreads) t.v[x] = x < ta ? A[i0 + x] : B[j0 + (x - ta)];
    __syncthreads();
    const uint64_t *a = t.v, *b = t.v + ta;
    const uint32_t d = min(n, threadIdx.x * kMergePer), e = min(n, d + kMergePer);
    uint32_t lo = d > tb ? d - tb : 0, hi = d < ta ? d : ta;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (tkey(a[mid]) <= tkey(b[d - mid - 1])) lo = mid + 1; else hi = mid;
    }
    uint32_t i = lo, j = d - lo;
    for (uint32_t o = d; o < e; o++) {
        const bool from_b = i >= ta || (j < tb && tkey(b[j]) < tkey(a[i]));
        const uint64_t v = from_b ? b[j] : a[i];
        f(o, i, v, from_b);
        if (from_b) j++; else i++;
    }
}

// The tile's elements k0 .. of merge(A, B) to out[0 ..), through shared memory
// (a pad word per thread: no bank conflicts), so that the stores are coalesced.
__device__ __forceinline__ void merge_tile_out(MergeTile &t, uint64_t *stage, const uint64_t *A, uint64_t na,
                                               const uint64_t *B, uint64_t nb, uint64_t k0, uint64_t *out) {
    merge_tile(t, A, na, B, nb, k0, [&](uint32_t o, uint32_t, uint64_t v, bool) { stage[o + o / kMergePer] = v; });
    __syncthreads();
    const uint32_t n = (uint32_t)(min(na + nb, k0 + kMergeTile) - k0);
    for (uint32_t x = threadIdx.x; x < n; x += kMergeThreads) out[x] = stage[x + x / kMergePer];
}

// Merges sorted pairs of runs: run pair q covers in[q * 2 * run .. ) as
// A = [q*2*run, q*2*run + run) and B = the next run (shorter at the end).
static __global__ void __launch_bounds__(kMergeThreads)
merge_pass_kernel(const uint64_t *in, uint64_t n, uint64_t run, uint64_t *out) {
    __shared__ MergeTile t;
    __shared__ uint64_t stage[kMergeTile + kMergeThreads];
    const uint64_t k0 = (uint64_t)blockIdx.x * kMergeTile;
    const uint64_t base = k0 / (2 * run) * (2 * run);
    const uint64_t na = min(run, n - base), nb = min(run, n - base - na);
    merge_tile_out(t, stage, in + base, na, in + base + na, nb, k0 - base, out + k0);
}

// Merges two sorted arrays into out.
static __global__ void __launch_bounds__(kMergeThreads)
merge_kernel(const uint64_t *A, uint64_t na, const uint64_t *B, uint64_t nb, uint64_t *out) {
    __shared__ MergeTile t;
    __shared__ uint64_t stage[kMergeTile + kMergeThreads];
    const uint64_t k0 = (uint64_t)blockIdx.x * kMergeTile;
    merge_tile_out(t, stage, A, na, B, nb, k0, out + k0);
}

// Joins sorted R (A) with sorted S (B): every S tuple meets the run of equal
// R keys just before its merge position (in the tile, and before it where the
// run began earlier).  r_is_a selects which side A is, for the checksum's
// (r_payload, s_payload) order.
static __global__ void __launch_bounds__(kMergeThreads)
merge_join_kernel(const uint64_t *A, uint64_t na, const uint64_t *B, uint64_t nb, int a_is_r, unsigned long long *acc) {
    __shared__ MergeTile t;
    __shared__ uint64_t red[64];
    Acc ac;
    merge_tile(t, A, na, B, nb, (uint64_t)blockIdx.x * kMergeTile, [&](uint32_t, uint32_t i, uint64_t b, bool from_b) {
        if (!from_b) return;
        const uint32_t key = tkey(b);
        auto add = [&](uint64_t x) {
            ac.count++;
            ac.sum += a_is_r ? pair_hash(key, tpay(x), tpay(b)) : pair_hash(key, tpay(b), tpay(x));
        };
        int64_t q = (int64_t)i - 1;
        for (; q >= 0 && tkey(t.v[q]) == key; q--) add(t.v[q]);
        if (q < 0)
            for (q = (int64_t)t.cut[0] - 1; q >= 0 && tkey(A[q]) == key; q--) add(A[q]);
    });
    block_flush(ac, acc, red);
}

}  // namespace adb
