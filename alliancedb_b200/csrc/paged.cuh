// paged.cuh -- radix/range partitioning of R and S into pages, one or two passes.
//
// Replaces the reference's partitioning passes
//   parallel_radix_partition (+ _optimized, software write-combining)
//                         hashing/joins/parallel_radix_join.cpp:739-806, 877-970
//   serial_radix_partition / radix_cluster          :688-729, :573-614
//   partition_relation_optimized / radix_cluster_optimized
//                         sorting/joins/partition.cpp:152-218, 327-350
// Like the reference, large fan-outs take two passes (its NUM_PASSES = 2,
// prj_params.h:19-21); unlike it, no pass needs a histogram pass first:
//   * output goes to 512-byte pages (64 tuples) taken from a per-CTA pool, a
//     partition's pages chained through the CTA's page log, so partitions
//     need not be contiguous and their sizes need not be known in advance;
//   * each tile of 6144 or 8192 tuples is counting-sorted by digit in shared memory
//     (the role of the reference's software write-combining buffers, its
//     _optimized partitioner), then copied out so that each partition's
//     tuples form one contiguous stream through its pages: warps store
//     contiguous runs, and the partial sectors at the ends of a tile's run are
//     completed in L2 by the stream's next tile, so DRAM sees whole lines;
//   * pass 2 reads the pages of pass 1 in work units of up to unit_pages pages
//     that never cross a pass-1 partition, so skewed partitions are split
//     over many CTAs;
//   * page_place turns the per-CTA page logs into one page list per partition.
// Traffic per pass: 8 bytes read + 8 bytes written per tuple, plus about 5
// bytes of page-list and count metadata per 64 tuples.
#pragma once

#include <type_traits>

#include "adb_common.cuh"
#include "partition.cuh"

namespace adb {

constexpr int kPageTuples = 64;                 // 512-byte pages
constexpr int kPassThreads = 512;               // threads per CTA of a pass, two CTAs per SM
constexpr int kPassMinBlocks = 2;
constexpr int kFlatTile = 6144;                 // tuples per tile: flat input with a second pass to follow,
constexpr int kPagedTile = 8192;                //   paged input,
constexpr int kSegTile = 8192;                  //   segmented input,
constexpr int kWideThreads = 1024;              //   flat input in a single pass (one CTA per SM)
constexpr int kWideTile = 8192;
constexpr uint32_t kMaxPassBits = 9;            // <= 512 partitions per pass
constexpr uint32_t kMaxUnitPages = 2048;        // pass-2 work unit: <= 128K tuples
constexpr uint32_t kMinUnitPages = kPagedTile / 64;  // one tile
constexpr uint32_t kNone = 0xFFFFFFFFu;
constexpr uint32_t kHotWord = 40;               // misc[] word of the hot digit

// Pages written by one pass for one relation.
struct PageSet {
    uint64_t *pages;     // pool pages x 64 tuples
    uint32_t *log;       // output digit of each pool page
    uint8_t *pcount;     // tuples in each pool page
    uint32_t *nlog;      // [G] pages used by each CTA
    uint32_t *doff;      // its place among digit d's pages at doff_at(CTA) + d
    uint2 *udesc;        // [G] each CTA's first output digit and digit count
    uint32_t *plist;     // page list grouped by output digit (filled by page_place)
    uint64_t *pstart;    // [Fout + 1] page-list starts
};

// Result of the paged partitioning front end: both relations' final pages,
// page lists per output partition, pstart = [2][Fout + 1] list starts.
struct PartOut {
    PageSet R, S;
    uint32_t Fout;
    uint64_t *pstart;
    uint64_t pool_pages;
};

struct PassIn {
    // flat input (pass 1): the relation, and the CTAs that share it (the
    // others of the launch idle)
    const uint64_t *in;
    uint64_t n;
    int G;
    // paged input (pass 2): the previous pass's pages, grouped by its digit
    const uint64_t *pages;
    const uint8_t *pcount;
    const uint32_t *plist;
    const uint64_t *pstart;   // [F1 + 1]
    const uint32_t *uoff;     // [F1 + 1] first work unit of each input partition (segments: of each segment)
    // segmented flat input (batched windows): segment w is in[seg_off[w] .. seg_off[w+1]),
    // partitioned 2^seg_bits[w] ways into output partitions seg_dbase[w] + d
    const uint64_t *seg_off;
    const uint8_t *seg_bits;
    const uint32_t *seg_dbase;
    const uint32_t *unit_pool;   // segmented input: first pool page of each unit ([G + 1])
};

struct PassArgs {
    PassIn in[2];
    PageSet out[2];
    DigitFn df;          // this pass's digit (F = df.mask + 1 <= 512)
    uint32_t F1;         // input partitions (1 for flat input)
    int G;               // CTAs per relation, the larger bound: flat chunks, or work units
    uint32_t pool_cap;   // pages per CTA pool
    uint32_t unit_pages; // paged input: pages per work unit
    uint64_t unit_tuples;// segmented input: tuples per work unit
    int paged;           // 0 = flat input, 1 = paged input, 2 = segmented flat input
    uint32_t *totals;    // [2][Dtot] pages per output partition (atomic sums, zeroed before the pass)
    uint32_t Dtot;
    int *err;
};

// Where CTA g's doff entries begin: F per CTA, or for segmented input, where F
// differs, at the CTA's first pool page (a pool has more pages than digits).
__device__ __forceinline__ uint32_t doff_at(int mode, uint32_t g, uint32_t F, uint32_t pool_base) {
    return mode == 2 ? pool_base : g * F;
}

__host__ __device__ __forceinline__ uint32_t flat_pool_cap(uint64_t n, int G, uint32_t F) {
    return (uint32_t)((chunk_of(n, G) + kPageTuples - 1) / kPageTuples + F + 1);
}
__host__ __device__ __forceinline__ uint32_t unit_pool_cap(uint32_t F, uint32_t unit_pages) { return unit_pages + F + 1; }

// Pass-2 work-unit size: about four waves of the resident CTAs over both
// relations (units never cross a pass-1 partition, so there are a few more).
__host__ __device__ __forceinline__ uint32_t unit_pages_for(uint64_t pages1_both, int num_sms) {
    uint64_t u = pages1_both / (4ull * kPassMinBlocks * num_sms) + 1;
    if (u < kMinUnitPages) u = kMinUnitPages;
    if (u > kMaxUnitPages) u = kMaxUnitPages;
    return (uint32_t)u;
}

// Shared memory of one pass:
//   stage[tile] u64 | cnt[2][F] u32 | toff[F] u16 (in F words) | lim[F] | b1[F] | b2[F] | npos[F] | npages[F] u32
//   | misc[48] u32
//   | paged input only: upage[kMaxUnitPages] u32
__host__ __device__ __forceinline__ size_t pass_smem(int tile, uint32_t F, bool paged) {
    return (size_t)tile * 8 + (size_t)F * 4 * 8 + 48 * 4 +
           (paged ? (size_t)kMaxUnitPages * 4 : 0);
}

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t x, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    return x;
}

// One pass over one input unit (a flat chunk, a unit of input pages, or a
// unit of a segment).  Per tile of up to kTile tuples:
//   A  every thread ranks its tuples within their digit (shared atomics on
//      cnt[tile parity][d]);
//   B  warp 0 (up to 32 digits, one per lane) or warps 0 .. F/32 - 1 (one
//      digit per lane) turn the counts into the tile's digit runs (toff), take
//      the pages each digit's stream needs from the CTA's pool, and advance
//      the streams (npos = next free slot of the digit's current page, kNone
//      when there is none);
//   C  every thread puts its tuples into the stage, grouped by digit;
//   D  every thread copies stage slots to their pages: slot i of digit d goes
//      to i + b1[d] while i < lim[d] (the rest of the current page), else to
//      i + b2[d] (the pages taken in B, consecutive in the pool); the thread
//      that writes a page's first slot also writes the page's log entry.
// Consecutive stage slots of a digit go to consecutive addresses, so warps
// store contiguous runs; a run's partial first and last 32-byte sectors are
// completed by the neighbouring tiles of the same stream while the line is
// still in L2.  Three barriers per tile (four above 32 digits); the next
// tile's loads are in flight during D.  kMode: 0 flat input, 1 paged input
// (pass 2), 2 segmented flat input (batched windows).  kHashed: the digit is
// taken from key * kHashMul instead of the key.
//
// Bound: shared-memory data wavefronts (about 23 per 32 tuples, the pipe 73 %
// busy in pass 1 with 4096-tuple tiles) and, between them, the barriers around
// B.  Larger tiles give B more tuples to share and D longer runs, so each kind
// takes the largest tile whose tuples, kTile / kThreads 64-bit registers, leave
// 64 registers enough for the rest.  Two passes of 2^7 digits, 2^27 x 2^27, ms
// at tiles of 4096 / 6144 / 8192: pass 1 0.991 / 0.953 / 0.966, pass 2 1.162 /
// 1.096 / 1.069 (10240: 1.186, spills); 512 batched windows of 2^10 .. 2^22
// tuples, whole call 5.94 / 5.67 / 5.51 (10240: 5.78).  Run starts (toff) of 16
// bits instead of 32, so that two share a bank: pass 1 0.944 -> 0.927, pass 2 1.062
// -> 1.040.
template <int kMode, int kThreads, int kTile, bool kHashed = false>
__global__ void __launch_bounds__(kThreads, kThreads == kWideThreads ? 1 : kPassMinBlocks)
partition_pass(PassArgs a) {
    constexpr bool kPaged = kMode == 1;
    constexpr int kPer = kTile / kThreads;
    constexpr uint32_t kHotRun = kTile / 2;   // a digit above this many tuples of a tile is hot
    constexpr uint32_t kAll = (1u << kPer) - 1u;
    static_assert(kPer % 2 == 0 && kThreads % 32 == 0 && (kTile / kPageTuples) % (kThreads / 32) == 0, "tile shape");
    static_assert((1u << kMaxPassBits) <= (uint32_t)kThreads, "one digit per thread in step B");
    extern __shared__ __align__(16) unsigned char smem[];
    const int relidx = blockIdx.y, g = blockIdx.x;
    const PassIn &in = relidx ? a.in[1] : a.in[0];

    // ---- this CTA's input: a flat chunk, a unit of input pages, or a unit of a segment
    uint64_t b = 0, e = 0;        // flat / segmented: tuple range; paged: page-list range
    uint32_t p1 = 0;              // paged: input partition; segmented: segment
    DigitFn df = a.df;
    if (kMode == 0) {
        const uint64_t chunk = chunk_of(in.n, in.G);
        b = min(in.n, (uint64_t)g * chunk);
        e = min(in.n, b + chunk);
    } else if ((uint32_t)g < in.uoff[a.F1]) {
        uint32_t lo = 0, hi = a.F1;   // largest p with uoff[p] <= g
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (in.uoff[mid] <= (uint32_t)g) lo = mid; else hi = mid;
        }
        p1 = lo;
        if (kMode == 1) {
            b = in.pstart[p1] + (uint64_t)(g - in.uoff[p1]) * a.unit_pages;
            e = min(in.pstart[p1 + 1], b + a.unit_pages);
        } else {
            b = in.seg_off[p1] + (uint64_t)(g - in.uoff[p1]) * a.unit_tuples;
            e = min(in.seg_off[p1 + 1], b + a.unit_tuples);
            df = DigitFn{0u, (1u << in.seg_bits[p1]) - 1u};
        }
    }
    const uint32_t F = df.mask + 1;
    auto dig = [&](uint64_t w) { return df(kHashed ? tkey(w) * kHashMul : tkey(w)); };
    uint64_t *stage = reinterpret_cast<uint64_t *>(smem);
    uint32_t *cnt = reinterpret_cast<uint32_t *>(stage + kTile);   // [2][F]
    uint16_t *toff = reinterpret_cast<uint16_t *>(cnt + 2 * F);   // 16 bits: half the banks' conflicts in C
    uint32_t *lim = cnt + 3 * F;
    uint32_t *b1 = lim + F;
    uint32_t *b2 = b1 + F;
    uint32_t *npos = b2 + F;
    uint32_t *npages = npos + F;        // pages the digit has taken
    uint32_t *misc = npages + F;        // [0] pool pages taken, [1] tuples in the tile,
                                        // [8..24) per-warp totals of the digit scan,
                                        // [kHotWord] hot digit
    uint32_t *upage = misc + 48;        // paged input: this unit's pages, id << 6 | tuples - 1

    const PageSet &o = relidx ? a.out[1] : a.out[0];
    const int tid = threadIdx.x, lane = tid & 31;
    const uint32_t pool_base = kMode == 2 ? in.unit_pool[g] : (uint32_t)g * a.pool_cap;
    const uint32_t pool_cap = kMode == 2 ? in.unit_pool[g + 1] - pool_base : a.pool_cap;
    const uint32_t dbase = kMode == 2 ? in.seg_dbase[p1] : p1 * F;   // output digit = dbase + d

    for (uint32_t d = tid; d < F; d += kThreads) {
        cnt[d] = 0;
        cnt[F + d] = 0;
        npos[d] = kNone;
        npages[d] = 0;
    }
    if (tid == 0) {
        misc[0] = 0;
        misc[kHotWord] = kNone;
    }
    if (kPaged)
        for (uint64_t i = b + tid; i < e; i += kThreads) {
            const uint32_t pg = in.plist[i];
            upage[i - b] = pg << 6 | (in.pcount[pg] - 1u);
        }
    __syncthreads();

    // ---- tiles: kTile flat tuples, or kTile / 64 input pages.  Whole flat
    // tiles take loads, ranks and staging without bounds checks (pass 1 at 2^27:
    // 1.033 -> 0.988 ms; the same for paged tiles made pass 2 slower, 1.059 -> 1.124).
    constexpr uint64_t kStep = kPaged ? (uint64_t)(kTile / kPageTuples) : (uint64_t)kTile;
    const bool vec = !kPaged && ((reinterpret_cast<uintptr_t>(in.in + b) & 15) == 0);
    uint64_t w[kPer];
    uint32_t valid = 0;   // bit k: w[k] holds a tuple
    auto load_tile = [&](uint64_t t0) {
        if (kPaged) {
            // tuple pair k of this thread: slots 2 (tid % 32), +1 of the tile's page k * (kThreads / 32) + tid / 32
            valid = 0;
            const uint32_t slot = 2 * (tid & 31);
#pragma unroll
            for (int k = 0; k < kPer / 2; k++) {
                const uint64_t li = t0 + (uint64_t)k * (kThreads / 32) + tid / 32;
                const uint32_t v = li < e ? upage[li - b] : 0u;
                const uint32_t c = li < e ? (v & 63u) + 1u : 0u;
                const uint64_t *src = in.pages + (uint64_t)(v >> 6) * kPageTuples + slot;
                if (slot + 1 < c) {
                    const ulonglong2 x = __ldcs(reinterpret_cast<const ulonglong2 *>(src));
                    w[2 * k] = x.x;
                    w[2 * k + 1] = x.y;
                    valid |= 3u << (2 * k);
                } else {
                    const bool ok = slot < c;
                    w[2 * k] = ok ? ld_stream(src) : 0;
                    w[2 * k + 1] = 0;
                    valid |= (ok ? 1u : 0u) << (2 * k);
                }
            }
        } else if (vec && t0 + kStep <= e) {
            valid = kAll;
            const ulonglong2 *src = reinterpret_cast<const ulonglong2 *>(in.in + t0) + tid;
#pragma unroll
            for (int k = 0; k < kPer / 2; k++) {
                const ulonglong2 v = __ldcs(src + k * kThreads);
                w[2 * k] = v.x;
                w[2 * k + 1] = v.y;
            }
        } else {
            const uint64_t *src = in.in + t0 + tid;
            const int left = (int)min(kStep, e - t0) - tid;
            valid = 0;
#pragma unroll
            for (int k = 0; k < kPer; k++) {
                const bool ok = k * kThreads < left;
                w[k] = ok ? ld_stream(src + k * kThreads) : 0;
                valid |= (ok ? 1u : 0u) << k;
            }
        }
    };

    // L2 prefetch of a tile: flat input one bulk prefetch of the whole tile;
    // paged input one 128-byte line prefetch per thread, four per page (a bulk
    // prefetch per 512-byte page costs the SM's bulk-copy unit more than the
    // latency it hides)
    auto prefetch_tile = [&](uint64_t t0) {
        if (t0 >= e) return;
        if (!kPaged && vec && tid == 0) {
            const uint64_t n = min(kStep, e - t0) & ~1ull;   // 16-byte multiple
            if (n) prefetch_l2(in.in + t0, (uint32_t)(n * 8));
        }
        if (kPaged && tid < (int)(kStep * 4)) {
            const uint64_t li = t0 + (uint64_t)(tid >> 2);
            if (li < e) {
                const uint64_t *line = in.pages + (uint64_t)(upage[li - b] >> 6) * kPageTuples + (tid & 3) * 16;
                asm volatile("prefetch.global.L2 [%0];" ::"l"(line));
            }
        }
    };

    if (b < e) {
        prefetch_tile(b + kStep);
        load_tile(b);
    }
    uint32_t par = 0;
    for (uint64_t t0 = b; t0 < e; t0 += kStep, par ^= F) {
        uint32_t *c = cnt + par;
        // A. rank each tuple within its digit.  A digit that held more than
        //    half of the previous tile (a hot key under skew) takes its ranks
        //    from one atomic per warp and tuple slot, by ballot: its increments
        //    would otherwise serialise on one shared counter.
        uint32_t rk[kPer / 2];   // two 16-bit ranks per word
        const uint32_t hot = misc[kHotWord];   // block-uniform
        if (!kPaged && hot == kNone && valid == kAll) {
#pragma unroll
            for (int k = 0; k < kPer; k++) {
                const uint32_t r = atomicAdd(&c[dig(w[k])], 1u);
                if (k & 1) rk[k / 2] |= r << 16; else rk[k / 2] = r;
            }
        } else if (hot == kNone) {
#pragma unroll
            for (int k = 0; k < kPer; k++) {
                const uint32_t r = (valid >> k) & 1 ? atomicAdd(&c[dig(w[k])], 1u) : 0u;
                if (k & 1) rk[k / 2] |= r << 16; else rk[k / 2] = r;
            }
        } else {
            uint32_t lt;
            asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
#pragma unroll
            for (int k = 0; k < kPer; k++) {
                const bool ok = (valid >> k) & 1;
                const uint32_t d = ok ? dig(w[k]) : kNone;
                const uint32_t m = __ballot_sync(0xffffffffu, d == hot);
                uint32_t r = 0;
                if (d == hot) r = (uint32_t)__popc(m & lt);
                else if (ok) r = atomicAdd(&c[d], 1u);
                if (m) {   // warp-uniform
                    const int leader = __ffs(m) - 1;
                    uint32_t base = 0;
                    if (lane == leader) base = atomicAdd(&c[hot], (uint32_t)__popc(m));
                    base = __shfl_sync(0xffffffffu, base, leader);
                    if (d == hot) r += base;
                }
                if (k & 1) rk[k / 2] |= r << 16; else rk[k / 2] = r;
            }
        }
        __syncthreads();
        // B. digit runs of the tile, pages, stream positions.  Up to 32 digits
        //    warp 0 alone, one per lane; above that warp w < F / 32 takes digits
        //    32w .. 32w + 31, one per lane, and the warps' totals are combined
        //    through shared memory (one extra barrier, which costs less than warp
        //    0 walking 2 or 4 digits per lane while the CTA waits: at 2^27 both
        //    passes of PRO gain, pass 2 1.232 -> 1.170 ms).  New pages get their
        //    log entry in D, from the thread that writes their first slot.
        auto run_digit = [&](uint32_t d, uint32_t L, uint32_t p, uint32_t off, uint32_t first) {
            const uint32_t room = p == kNone ? 0u : kPageTuples - (p & (kPageTuples - 1));
            c[d] = 0;
            toff[d] = (uint16_t)off;
            lim[d] = off + (L < room ? L : room);
            b1[d] = p - off;
            uint32_t np = p + L;
            if (L > room) {
                const uint32_t need = (L - room + kPageTuples - 1) / kPageTuples;
                if (first + need > pool_cap) {   // cannot happen: the pool covers the input
                    atomicExch(a.err, kErrPagesUsedUp);
                    first = pool_cap - need;
                }
                const uint32_t nx = (pool_base + first) * kPageTuples - room;
                b2[d] = nx - off;
                np = nx + L;
                npages[d] += need;
            }
            if (L && (np & (kPageTuples - 1)) == 0) np = kNone;   // page exactly full
            npos[d] = np;
        };
        auto pages_for = [&](uint32_t L, uint32_t p) {
            const uint32_t room = p == kNone ? 0u : kPageTuples - (p & (kPageTuples - 1));
            return L > room ? (L - room + kPageTuples - 1) / kPageTuples : 0u;
        };
        if (F <= 32) {
            // (one digit per lane; without the loops ptxas schedules the paged pass of
            // 2^7 digits, which does not come here, 2.7 % slower: 1.040 -> 1.068 ms)
            constexpr int kQ = 1;
            const uint32_t q = (F + 31) / 32;
            if (tid < 32) {
                uint32_t Ls[kQ], Ps[kQ], sumL = 0, sumN = 0;
#pragma unroll
                for (int j = 0; j < kQ; j++) {
                    const uint32_t d = (uint32_t)lane * q + j;
                    Ls[j] = 0;
                    Ps[j] = kNone;
                    if ((uint32_t)j < q && d < F) {
                        Ls[j] = c[d];
                        Ps[j] = npos[d];
                        sumL += Ls[j];
                        sumN += pages_for(Ls[j], Ps[j]);
                    }
                }
                const uint32_t v = sumL | (sumN << 16);   // L <= kTile, pages < 2^16
                const uint32_t inc = warp_incl_scan(v, lane);
                const uint32_t all = __shfl_sync(0xffffffffu, inc, 31);
                const uint32_t pool0 = misc[0];
                uint32_t off = (inc - v) & 0xFFFFu, first = pool0 + ((inc - v) >> 16);
#pragma unroll
                for (int j = 0; j < kQ; j++) {
                    const uint32_t d = (uint32_t)lane * q + j;
                    if ((uint32_t)j < q && d < F) {
                        run_digit(d, Ls[j], Ps[j], off, first);
                        off += Ls[j];
                        first += pages_for(Ls[j], Ps[j]);
                    }
                }
                // the largest run (one digit per lane here): the next tile's hot digit
                const uint32_t mx = __reduce_max_sync(0xffffffffu, (Ls[0] << 16) | (uint32_t)lane);
                __syncwarp();
                if (lane == 0) {
                    misc[0] = pool0 + (all >> 16);
                    misc[1] = all & 0xFFFFu;
                    misc[kHotWord] = (mx >> 16) > kHotRun ? (mx & 0xFFFFu) : kNone;
                }
            }
        } else {
            const uint32_t nbw = (F + 31) / 32;                 // B warps
            const int bw = tid >> 5;
            const uint32_t d = (uint32_t)tid;                   // this lane's digit
            uint32_t L = 0, p = kNone, need = 0, inc = 0, pool0 = 0, mx = 0;
            if (bw < (int)nbw) {
                if (d < F) {
                    L = c[d];
                    p = npos[d];
                    need = pages_for(L, p);
                }
                inc = warp_incl_scan(L | (need << 16), lane);   // L <= kTile, pages of 32 digits < 2^16
                mx = __reduce_max_sync(0xffffffffu, (L << 16) | d);   // this warp's largest run, its digit
                pool0 = misc[0];
                if (lane == 31) misc[8 + bw] = inc;
                if (tid == 0) misc[kHotWord] = kNone;   // all of this tile's readers are past step A
            }
            __syncthreads();   // every B warp has read misc[0] and written its total
            if (bw < (int)nbw) {
                // totals of the warps before this one, and of all of them: by a
                // shuffle scan, in the paged pass one by one (2^22 x 2^22, 16 warps:
                // pass 1 58.6 -> 56.3 us; 512 batched windows 5.275 -> 5.255 ms; 2^27 x
                // 2^27, four warps: pass 1 0.926 either way, pass 2 1.038 -> 1.057 ms)
                uint32_t before_t = 0, before_p = 0, all_t = 0, all_p = 0;
                if (!kPaged) {
                    const uint32_t tv = lane < (int)nbw ? misc[8 + lane] : 0u;
                    const uint32_t sums = warp_incl_scan(tv, lane);   // both halves stay below 2^16
                    const uint32_t all = __shfl_sync(0xffffffffu, sums, 31);
                    const uint32_t before = __shfl_sync(0xffffffffu, sums - tv, bw);
                    before_t = before & 0xFFFFu;
                    before_p = before >> 16;
                    all_t = all & 0xFFFFu;
                    all_p = all >> 16;
                } else {
                    for (uint32_t k = 0; k < nbw; k++) {
                        const uint32_t tv = misc[8 + k];
                        if ((int)k < bw) { before_t += tv & 0xFFFFu; before_p += tv >> 16; }
                        all_t += tv & 0xFFFFu;
                        all_p += tv >> 16;
                    }
                }
                const uint32_t ex = inc - (L | (need << 16));
                if (d < F) run_digit(d, L, p, before_t + (ex & 0xFFFFu), pool0 + before_p + (ex >> 16));
                if (bw == 0 && lane == 0) {   // warp 0 read misc[0] before the shuffle above
                    misc[0] = pool0 + all_p;
                    misc[1] = all_t;
                }
                // the next tile's hot digit: a run above half a tile (at most one)
                if (lane == 0 && (mx >> 16) > kHotRun) misc[kHotWord] = mx & 0xFFFFu;
            }
        }
        __syncthreads();
        // C. stage the tile grouped by digit
        if (!kPaged && valid == kAll) {
#pragma unroll
            for (int k = 0; k < kPer; k++)
                stage[toff[dig(w[k])] + ((rk[k / 2] >> ((k & 1) * 16)) & 0xFFFFu)] = w[k];
        } else {
#pragma unroll
            for (int k = 0; k < kPer; k++)
                if ((valid >> k) & 1)
                    stage[toff[dig(w[k])] + ((rk[k / 2] >> ((k & 1) * 16)) & 0xFFFFu)] = w[k];
        }
        const uint32_t tile_n = misc[1];
        if (t0 + kStep < e) {   // in flight during D; the tile after that into L2
            prefetch_tile(t0 + 2 * kStep);
            load_tile(t0 + kStep);
        }
        __syncthreads();
        // D. stage slots to their pages
        auto copy = [&](uint32_t i0, auto n) {   // slots i0, i0 + kThreads, ..: n of them
            constexpr int U = decltype(n)::value;
            uint64_t v[U];
            uint32_t d[U], dst[U];
#pragma unroll
            for (int u = 0; u < U; u++) v[u] = stage[i0 + u * kThreads];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const uint32_t i = i0 + u * kThreads;
                d[u] = dig(v[u]);
                dst[u] = i + (i < lim[d[u]] ? b1 : b2)[d[u]];
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                o.pages[dst[u]] = v[u];
                if ((dst[u] & (kPageTuples - 1)) == 0) {   // first slot of a page taken in B
                    o.log[dst[u] / kPageTuples] = dbase + d[u];
                    o.pcount[dst[u] / kPageTuples] = kPageTuples;
                }
            }
        };
        // two at a time, so that one's look-ups overlap the other's (2^27 x 2^27,
        // ms, one / two / four / eight: pass 1 0.954 / 0.948 / 0.946 / 1.085, pass 2
        // 1.068 / 1.065 / 1.073 / 1.514)
        uint32_t i = tid;
        for (; i + kThreads < tile_n; i += 2 * kThreads) copy(i, std::integral_constant<int, 2>());
        if (i < tile_n) copy(i, std::integral_constant<int, 1>());
        // the next tile's A uses the other counter array and registers only;
        // its B / C run after the next barrier, when every thread is past D
    }
    __syncthreads();
    // E. fill of each digit's last page (every other page of a stream is full); a
    //    page's readers take tuples two at a time and leave out what is past its count
    for (uint32_t d = tid; d < F; d += kThreads) {
        const uint32_t p = npos[d];
        if (p != kNone && (p & (kPageTuples - 1))) o.pcount[p / kPageTuples] = (uint8_t)(p & (kPageTuples - 1));
    }
    // F. pages per digit of this CTA
    uint32_t *tot = a.totals + (size_t)relidx * a.Dtot;
    for (uint32_t d = tid; d < F; d += kThreads)
        if (npages[d]) o.doff[doff_at(kMode, g, F, pool_base) + d] = atomicAdd(&tot[dbase + d], npages[d]);
    if (tid == 0) {
        o.nlog[g] = misc[0];
        o.udesc[g] = make_uint2(dbase, F);
    }
}

// Exclusive scan of t[0..n) into out[0..n], out[n] = *total = the sum: block b
// takes elements 1024 b .. + 1023 and sums everything before them itself
// (16-byte loads; n is at most 2^16 here, so at most 256 KB from L2), so one
// launch does it: 65,536 elements 4 us, 55 us with one block walking them.
// t is 16-byte aligned.
constexpr uint32_t kScanThreads = 1024;
template <class T>
__device__ __forceinline__ void scan_list(const uint32_t *t, uint32_t n, uint32_t b, T *out, uint32_t *total,
                                          uint32_t *tmp) {
    const uint4 *t4 = reinterpret_cast<const uint4 *>(t);
    uint32_t before = 0, tot;
    for (uint32_t i = threadIdx.x; i < b * (kScanThreads / 4); i += kScanThreads) {
        const uint4 v = ld_done(t4 + i);
        before += v.x + v.y + v.z + v.w;
    }
    block_exclusive_scan(before, tmp, &before);
    const uint32_t i = b * kScanThreads + threadIdx.x;
    const uint32_t v = i < n ? ld_done(t + i) : 0u;
    const uint32_t ex = block_exclusive_scan(v, tmp, &tot);
    if (i < n) out[i] = before + ex;
    if (i + 1 == n) {
        out[n] = before + ex + v;
        if (total) *total = before + ex + v;
    }
}

// Page-list starts of every output partition (grid.y = relation).
static __global__ void __launch_bounds__(kScanThreads) list_starts(PassArgs a) {
    __shared__ uint32_t tmp[32];
    scan_list(a.totals + (size_t)blockIdx.y * a.Dtot, a.Dtot, blockIdx.x, (blockIdx.y ? a.out[1] : a.out[0]).pstart,
              nullptr, tmp);
}

// Groups the CTAs' page logs into one page list per output partition: CTA g's
// pages of digit d go to pstart[D] + doff[d], +1, ...  Flat input (up to 512
// digits, one per thread): every block scans the totals for itself, so no
// launch comes between the pass and this one, and block 0 of each relation
// writes pstart and, with unit_pages, the next pass's work units
// (uoff[p] = first unit of input partition p).
constexpr int kPlaceThreads = 512;
static __global__ void __launch_bounds__(kPlaceThreads)
page_place(PassArgs a, uint32_t unit_pages, uint32_t *uoff0, uint32_t *uoff1) {
    __shared__ uint32_t base[1u << kMaxPassBits];
    __shared__ uint32_t tmp[32];
    static_assert((1u << kMaxPassBits) <= (uint32_t)kPlaceThreads, "one digit per thread");
    const int relidx = blockIdx.y, g = blockIdx.x;
    const uint32_t tid = threadIdx.x;
    const PageSet &o = relidx ? a.out[1] : a.out[0];
    const uint32_t used = o.nlog[g];
    const uint2 ud = o.udesc[g];   // first output digit, digits
    const uint32_t pool_base = a.paged == 2 ? (relidx ? a.in[1] : a.in[0]).unit_pool[g] : (uint32_t)g * a.pool_cap;
    if (a.paged == 0) {
        const uint32_t F = a.Dtot;
        const uint32_t v = tid < F ? a.totals[(size_t)relidx * F + tid] : 0u;
        uint32_t tot;
        const uint32_t ex = block_exclusive_scan(v, tmp, &tot);
        if (tid < F) base[tid] = ex + o.doff[doff_at(0, g, F, pool_base) + tid];   // (an absent digit's is not used)
        if (g == 0) {
            if (tid < F) o.pstart[tid] = ex;
            if (tid == 0) o.pstart[F] = tot;
            if (unit_pages) {
                uint32_t *uo = relidx ? uoff1 : uoff0;
                const uint32_t ue = block_exclusive_scan((v + unit_pages - 1) / unit_pages, tmp, &tot);
                if (tid < F) uo[tid] = ue;
                if (tid == 0) uo[F] = tot;
            }
        }
    } else {
        if (!used) return;
        for (uint32_t d = tid; d < ud.y; d += kPlaceThreads)
            base[d] = (uint32_t)o.pstart[ud.x + d] + o.doff[doff_at(a.paged, g, ud.y, pool_base) + d];
    }
    __syncthreads();
    for (uint32_t k = tid; k < used; k += kPlaceThreads)
        o.plist[atomicAdd(&base[o.log[pool_base + k] - ud.x], 1u)] = pool_base + k;
}

}  // namespace adb
