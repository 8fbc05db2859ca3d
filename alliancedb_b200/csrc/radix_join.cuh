// radix_join.cuh -- per-partition build/probe of the partitioned hash joins.
//
// Replaces, per partition pair (R_p, S_p) produced by paged.cuh:
//   bucket_chaining_join   hashing/joins/parallel_radix_join.cpp:291-354   (PRO, RJ_st)
//   histogram_join         hashing/joins/parallel_radix_join.cpp:373-432   (PRH, PRHO)
//   sorting and merge phases  sorting/joins/sortmergejoin_multiway.cpp:499-660, merge_join
//                          sorting/joins/common_functions.cpp:298-372      (m-way, m-pass, m-way+skew)
// (one chained table for all four: a histogram table, built with two passes
// over R and a scan, took 0.35 ms where the chained one took 0.15 at 2^24)
// and the task-queue loop of prj_thread (:1409-1416) with a persistent kernel
// that takes work items from a global counter (work stealing).  A work item is
// (partition p, R chunk, S chunk): an R chunk is a run of R_p's pages packed
// greedily up to kRSlots tuples (part_chunks), read page by page and linked
// into a chained table in shared memory, and up to kSPages pages of S_p are
// streamed from global memory and probed, one warp per page.  Large R
// partitions (duplicate or skewed build keys, or |R| beyond 2^15 * 8K) take
// several R chunks; large S partitions (skewed probe keys) several S chunks.
#pragma once

#include "adb_common.cuh"
#include "engine.cuh"
#include "paged.cuh"

namespace adb {

constexpr int kJoinThreads = 512;
constexpr int kJoinMinBlocks = 2;                          // CTAs per SM: one's copies and build hide behind the other's probe
constexpr uint32_t kRSlots = 8704;                         // R tuples a CTA holds (68 KB)
constexpr uint32_t kChunkW = kRSlots - kPageTuples;        // chunk weight budget
constexpr uint32_t kMinPageW = 32;                         // weight floor of a page
constexpr uint32_t kRMaxPages = kChunkW / kMinPageW + 16;  // pages of one R chunk (bound)
constexpr int kProbeWarps = kJoinThreads / 32 - 1;        // the last warp is the control warp
constexpr uint32_t kSPages = kProbeWarps * 32;             // S pages per item: <= 32 per probing warp (one per lane)
constexpr uint32_t kMaxHeadsLog2 = 13;                     // bucket heads: one per slot up to 2^13

__device__ __forceinline__ uint32_t page_weight(uint32_t cnt) {
    const uint32_t e = (cnt + 1) & ~1u;                    // slots a page occupies (16-byte copies)
    return e > kMinPageW ? e : kMinPageW;
}

// The work items of a join: partition p's items are (R chunk, S chunk) pairs
// items_off[p] .. items_off[p + 1); its R chunks start at pages
// cstart[chunk_off[p]], +1, .. (page-list indexes), rch[p] of them.
struct WorkList {
    uint32_t *rch, *chunk_off, *items, *items_off;   // [F], [F], [F], [F + 1]
    uint32_t *spp;                                   // [F] pages per S chunk
    uint64_t *cstart;
    uint32_t ctas;                                   // CTAs of the join
    uint32_t *ctr;                                   // items, work counter, blocks done (zeroed before part_chunks)
    // A partition's chunks weigh more than chunk_w but for the last, so at
    // most 64 x pages / chunk_w + 1 of them: chunk_off needs no scan.
    static size_t chunks(uint64_t F, uint64_t pages, uint32_t chunk_w) { return pages * kPageTuples / chunk_w + F + 1; }
    static size_t bytes(uint64_t F, uint64_t pages, uint32_t chunk_w) {
        return 4 * Workspace::need(F, 4) + Workspace::need(F + 1, 4) + Workspace::need(chunks(F, pages, chunk_w), 8) +
               Workspace::need(3, 4);
    }
    void take(Workspace &ws, uint64_t F, uint64_t pages, uint32_t chunk_w, int num_sms, uint32_t *counters = nullptr) {
        ctas = (uint32_t)(num_sms * kJoinMinBlocks);
        rch = ws.take<uint32_t>(F);
        chunk_off = ws.take<uint32_t>(F);
        items = ws.take<uint32_t>(F);
        spp = ws.take<uint32_t>(F);
        items_off = ws.take<uint32_t>(F + 1);
        cstart = ws.take<uint64_t>(chunks(F, pages, chunk_w));
        ctr = counters ? counters : ws.take<uint32_t>(3);
    }
};

// Pages per S chunk of a partition with nsp of all the S pages in F partitions, and
// rch R chunks: up to kSPages, but where the partition has more than twice the
// mean, no more than makes a CTA's share of the join's items.  A few hot keys on
// both sides would else be a few items, each with all the pairs of a key, while the
// other CTAs have none.  300,007 x 300,007 tuples, 4,096 / 16,384 of each key, ms:
// sorted 8.4 / 58.7 -> 4.2 / 8.3, chained 9.9 / 70 -> 5.0 / 9.8.  (From 1.25 times the
// mean on: 2^20 x 2^22, theta 1, 0.149 -> 0.166, its items no longer one wave of CTAs.)
__device__ __forceinline__ uint32_t s_chunk_pages(uint32_t nsp, uint32_t rch, uint32_t all, uint32_t F, uint32_t ctas) {
    if ((uint64_t)nsp * F <= 2ull * all) return kSPages;
    const uint32_t share = (min(all / ctas, kSPages) + 1) * min(rch, kSPages);
    const uint32_t most = max(max(share, 2 * (all / F)), (uint32_t)kProbeWarps + 1);
    if (most >= kSPages || nsp <= most) return kSPages;
    const uint32_t chunks = (nsp + most - 1) / most, per = (nsp + chunks - 1) / chunks;   // of like size
    return per <= 4 * kProbeWarps ? per : (per + kProbeWarps - 1) / kProbeWarps * kProbeWarps;
}

__device__ __forceinline__ uint32_t s_chunks(uint32_t nsp, uint32_t per) {
    return per == kSPages ? (nsp + kSPages - 1) / kSPages : (nsp + per - 1) / per;   // (the usual divisor is a constant)
}

// R chunks and item counts, one warp per partition: chunk c of a partition
// starts at the first page whose preceding weight reaches c * kChunkW (greedy
// by page weight); S chunks are spp[p] pages each.  With `scan` (F <= 1024) the
// last block to finish also makes items_off and the item count, so that one
// launch stands between the passes and the join.
static __global__ void __launch_bounds__(1024)
part_chunks(const uint64_t *pstart, const uint32_t *Rlist, const uint8_t *Rcount, uint32_t F, WorkList wl,
            bool scan) {
    const int lane = threadIdx.x & 31;
    const uint32_t p = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (p < F) {
        const uint64_t *pS = pstart + (F + 1);
        const uint64_t r0 = pstart[p], r1 = pstart[p + 1];
        const uint32_t nsp = (uint32_t)(pS[p + 1] - pS[p]), all = (uint32_t)pS[F];
        const uint64_t cid = r0 * kPageTuples / kChunkW + p;
        uint64_t carry = 0;                 // weight before this round
        uint32_t prev_chunk = 0xFFFFFFFFu;  // chunk of the page before this round
        constexpr int U = 4;                // rounds of 32 pages loaded together
        for (uint64_t base = r0; base < r1; base += 32 * U) {
            uint32_t w[U];
#pragma unroll
            for (int u = 0; u < U; u++) w[u] = base + 32 * u + lane < r1 ? Rlist[base + 32 * u + lane] : kNone;
#pragma unroll
            for (int u = 0; u < U; u++) w[u] = w[u] != kNone ? page_weight(Rcount[w[u]]) : 0u;
#pragma unroll
            for (int u = 0; u < U; u++) {
                const uint64_t k = base + 32 * u + lane;
                const uint32_t x = warp_incl_scan(w[u], lane);
                const uint32_t ch = (uint32_t)((carry + x - w[u]) / kChunkW);
                uint32_t before = __shfl_up_sync(0xffffffffu, ch, 1);
                if (lane == 0) before = prev_chunk;
                if (k < r1 && ch != before) wl.cstart[cid + ch] = k;
                carry += __shfl_sync(0xffffffffu, x, 31);
                // the chunk of the last page so far (pages past the end weigh nothing and do not move it)
                const uint32_t last = __ballot_sync(0xffffffffu, k < r1);
                if (last) prev_chunk = __shfl_sync(0xffffffffu, ch, 31 - __clz(last));
            }
        }
        if (lane == 0) {
            const uint32_t rc = r1 > r0 ? prev_chunk + 1 : 0u;
            const uint32_t per = s_chunk_pages(nsp, rc, all, F, wl.ctas);
            const uint32_t sc = s_chunks(nsp, per);
            wl.rch[p] = rc;
            wl.spp[p] = per;
            wl.chunk_off[p] = (uint32_t)cid;
            wl.items[p] = rc * sc;
        }
    }
    if (!scan) return;
    __shared__ uint32_t tmp[32];
    __shared__ bool last_block;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last_block = atomicAdd(&wl.ctr[2], 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last_block) return;
    __threadfence();
    scan_list(wl.items, F, 0, wl.items_off, &wl.ctr[0], tmp);
}

static __global__ void __launch_bounds__(kScanThreads) items_scan(WorkList wl, uint32_t F) {
    __shared__ uint32_t tmp[32];
    scan_list(wl.items, F, blockIdx.x, wl.items_off, &wl.ctr[0], tmp);
}

// The work list of F partitions; returns the launches it took.
static int make_work_list(cudaStream_t st, const uint64_t *pstart, const uint32_t *Rlist, const uint8_t *Rcount,
                          uint32_t F, const WorkList &wl) {
    part_chunks<<<(F + 31) / 32, 1024, 0, st>>>(pstart, Rlist, Rcount, F, wl, F <= kScanThreads);
    if (F <= kScanThreads) return 1;
    items_scan<<<(F + kScanThreads - 1) / kScanThreads, kScanThreads, 0, st>>>(wl, F);
    return 2;
}

// Search by one warp, 32 probes per round: the largest i in [0, n)
// with off[i] <= v (off non-decreasing, off[0] <= v).  Three dependent rounds
// for 2^14 entries instead of fourteen.
__device__ __forceinline__ uint32_t warp_find(const uint32_t *off, uint32_t n, uint32_t v, int lane) {
    uint32_t lo = 0, hi = n;
    while (hi - lo > 1) {
        const uint32_t step = (hi - lo + 31) / 32;
        const uint32_t idx = lo + (uint32_t)lane * step;
        const bool le = idx < hi && off[idx] <= v;
        const uint32_t m = __ballot_sync(0xffffffffu, le);
        lo += (31u - __clz(m)) * step;   // lane 0 always qualifies
        hi = min(hi, lo + step);
    }
    return lo;
}

// Page ranges of one work item (R chunk pages [rb, rb + nrpg) and S pages
// [sb, sb + nspg) of its partition's page lists), kept in shared memory so the
// whole CTA reads them once warp 0 has taken the item.
struct ItemGeo {
    uint64_t rb, sb;
    uint32_t nrpg, nspg;
};

template <typename Args>
__device__ __forceinline__ ItemGeo item_geo(const Args &a, uint32_t item, uint32_t p) {
    const uint64_t *pR = a.pstart, *pS = a.pstart + (a.F + 1);
    const uint64_t r0 = pR[p], nrp = pR[p + 1] - r0;
    const uint64_t s0 = pS[p], nsp = pS[p + 1] - s0;
    const uint32_t local = item - a.wl.items_off[p], rch = a.wl.rch[p], s_pages = a.wl.spp[p];
    const uint32_t sch = s_chunks((uint32_t)nsp, s_pages);
    const uint32_t rc = local / sch, sc = local % sch;
    const uint32_t cid = a.wl.chunk_off[p] + rc;
    ItemGeo g;
    g.rb = a.wl.cstart[cid];
    const uint64_t re = rc + 1 < rch ? a.wl.cstart[cid + 1] : r0 + nrp;
    g.nrpg = (uint32_t)(re - g.rb);
    g.sb = s0 + (uint64_t)sc * s_pages;
    g.nspg = (uint32_t)min((uint64_t)s_pages, nsp - (uint64_t)sc * s_pages);
    return g;
}

// Shared memory: tup[kRSlots] u64 | heads[2^kMaxHeadsLog2] u32 | two page tables
// {pg[kRMaxPages + 1] u32, dst << 8 | count [kRMaxPages + 1] u32} | reduction and
// two item records.
constexpr size_t kPageTabBytes = ((size_t)kRMaxPages + 1) * 4 * 2;
constexpr size_t kJoinSmem = (size_t)kRSlots * 8 + ((size_t)4 << kMaxHeadsLog2) + 2 * kPageTabBytes + 1024;
static_assert(((size_t)kRSlots * 8 + 2 * kPageTabBytes) % 8 == 0, "reduction words must be 8-byte aligned");
static_assert(kJoinMinBlocks * (kJoinSmem + 1024) <= 233472, "join CTAs exceed the SM's shared memory");
static_assert(kRSlots <= (2u << kMaxHeadsLog2), "a slot index must fit the key bits a bucket shares");

struct JoinArgs {
    const uint64_t *Rpages, *Spages;
    const uint8_t *Rcount, *Scount;
    const uint32_t *Rlist, *Slist;   // page lists grouped by digit
    const uint64_t *pstart;          // [2][F+1] page-list starts
    WorkList wl;
    unsigned long long *acc;         // [0] count, [1] checksum
    unsigned long long *out;         // pinned host copy of acc[0 .. 3], written by the last CTA (null: none)
    uint32_t F;
    uint32_t bits;                   // bits the partitioning consumed (the hash skips them)
    uint64_t *mat;                   // optional <S-key, S-payload> output
    unsigned long long *mat_n;
    uint64_t mat_cap;
    // batched windows: partition p belongs to window w with wbase[w] <= p < wbase[w + 1];
    // each item's count and checksum go to wacc[2w], wacc[2w + 1] (null: to acc)
    const uint32_t *wbase;
    const uint8_t *wbits;            // fan-out bits of each window (its in-partition hash skips them)
    uint32_t nwin;
    unsigned long long *wacc;
};

// One work item as the control warp publishes it.
struct ItemRec {
    uint64_t rb, sb;          // first page-list index of the R chunk / S chunk
    uint32_t item, p, win;    // item (>= n_items: none), partition, window
    uint32_t nrpg, nspg;      // pages of the R chunk / S chunk
    uint32_t lnb;             // log2 of the bucket heads: one per slot of the R chunk (pages rounded up to even counts)
    uint32_t shift;           // key bits the partitioning consumed
};

// The items of one CTA form a pipeline run by its last warp (the control
// warp), so that no dependent global load sits between two items:
//   while item i is probed, the control warp builds the page table of item
//   i + 1 (page ids, 16-byte aligned shared-memory destinations), takes item
//   i + 2 from the work counter and prefetches item i + 1's R pages to L2; the
//   probing warps load their S page ids of item i + 1.
// Per item: the table build by all warps (a page per warp, kB pages' loads in
// flight), then the probe by warps 0 .. kProbeWarps - 1, each with one S page
// in flight ahead of the one it probes.
//
// The table: bucket heads indexed by the lnb key bits above the b bits the
// partitioning consumed (kHashed: the lnb bits of key * kHashMul below the b
// highest), one head per R slot (up to 2^13), and chains through the tuples
// themselves.  All keys of a bucket share their low b + lnb bits, so a linked
// tuple's key holds the next slot of its chain there (its own slot: the end);
// the bits above stay for the comparison.  One 8-byte read per
// visited tuple gives payload, comparison bits and link.
//
// Bound: instruction issue and the ALU pipe (60 % busy), not DRAM.  |R| = |S| =
// 2^27, ms, dense keys / keys spread over 32 bits:
//   one 1024-thread CTA per SM, two slots per head, a
//   separate next array, bulk-copied pages                  1.05  / 1.74
//   two CTAs, so that one builds while the other probes    -0.08  / -0.05
//   one head per slot, links in the tuples                 -0.13  / -0.5
//   pages read straight into the build, without the copy's
//   issue cost of about 58 cycles a page and its wait      -0.03
//   the probe's half of the checksum before the walk       -0.05  / -0.07
//   the next item's R pages in L2 before its build          0.740 / 1.315
//   one S page in flight instead of two and three R pages
//   instead of four: room within 64 registers               0.678 / 1.230
// The sorted form, with two R pages in flight (four spilled), 1.308 -> 1.168;
// 512 batched windows (2^10 .. 2^22 tuples), the whole call 5.50 -> 5.29 ms.
// Not kept: adding a warp's matches together after the walk instead of as they
// are found, 0.744 / 1.013, and batched windows 3 % slower; choosing between
// the two by item, by the tuples that share a bucket, 0.694 / 1.025, windows
// 2 % slower.
template <bool kMat, bool kHashed = false, bool kSorted = false>
__global__ void __launch_bounds__(kJoinThreads, kJoinMinBlocks)
radix_join_items(JoinArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    uint64_t *tup = reinterpret_cast<uint64_t *>(smem);
    uint32_t *heads = reinterpret_cast<uint32_t *>(tup + kRSlots);
    uint32_t *ptab = heads + (1u << kMaxHeadsLog2);                      // [2] x {pg[], dst << 8 | cnt []}
    uint64_t *red = reinterpret_cast<uint64_t *>(ptab + 4 * (kRMaxPages + 1));
    ItemRec *rec = reinterpret_cast<ItemRec *>(red + 64);                // [2]

    const uint32_t n_items = a.wl.ctr[0];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int kWarps = kJoinThreads / 32;
    constexpr int kCtl = kWarps - 1;
    const uint32_t F = a.F;

    // control warp: take the next item from the work counter into r
    auto take = [&](ItemRec *r) {
        uint32_t item = 0;
        if (lane == 0) item = atomicAdd(&a.wl.ctr[1], 1u);
        item = __shfl_sync(0xffffffffu, item, 0);
        uint32_t p = 0, w = 0;
        if (item < n_items) {
            p = warp_find(a.wl.items_off, F, item, lane);
            if (a.wacc) w = warp_find(a.wbase, a.nwin, p, lane);
        }
        if (lane == 0) {
            r->item = item;
            if (item < n_items) {
                const ItemGeo g = item_geo(a, item, p);
                r->p = p;
                r->win = w;
                r->shift = a.wacc ? a.wbits[w] : a.bits;
                r->rb = g.rb;
                r->sb = g.sb;
                r->nrpg = g.nrpg;
                r->nspg = g.nspg;
            }
        }
        __syncwarp();
    };
    // control warp: page table of item r (page ids, packed destination and count)
    auto table = [&](ItemRec *r, uint32_t *pt) {
        if (r->item >= n_items) return;
        const uint64_t rb = r->rb;
        const uint32_t nrpg = r->nrpg;
        uint32_t *tpg = pt, *tpk = pt + kRMaxPages + 1;
        uint32_t carry = 0;
        constexpr int U = 4;
        for (uint32_t base = 0; base < nrpg; base += 32 * U) {
            uint32_t pg[U], cnt[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const uint32_t k = base + 32 * u + lane;
                pg[u] = k < nrpg ? a.Rlist[rb + k] : kNone;
            }
#pragma unroll
            for (int u = 0; u < U; u++) cnt[u] = pg[u] != kNone ? a.Rcount[pg[u]] : 0u;
#pragma unroll
            for (int u = 0; u < U; u++) {
                const uint32_t k = base + 32 * u + lane;
                const uint32_t e = (cnt[u] + 1) & ~1u;
                const uint32_t inc = warp_incl_scan(e, lane);
                if (k < nrpg) {
                    tpg[k] = pg[u];
                    tpk[k] = ((carry + inc - e) << 8) | cnt[u];
                }
                carry += __shfl_sync(0xffffffffu, inc, 31);
            }
        }
        if (lane == 0) {
            uint32_t l = carry > 1 ? 32u - __clz(carry - 1) : 0u;
            r->lnb = l < kMaxHeadsLog2 ? l : kMaxHeadsLog2;
        }
        __syncwarp();
    };

    if (warp == kCtl) {
        take(&rec[0]);
        table(&rec[0], ptab);
        take(&rec[1]);
    }
    __syncthreads();

    // S pages of a probing warp for item r: lane i holds page warp + kProbeWarps * i
    // as id << 6 | count - 1 (kNone: no page)
    auto s_ids = [&](const ItemRec &r) {
        uint32_t v = kNone;
        if (warp < kProbeWarps && r.item < n_items) {
            const uint32_t i = (uint32_t)warp + (uint32_t)kProbeWarps * lane;
            if (i < r.nspg) {
                const uint32_t pg = a.Slist[r.sb + i];
                v = pg << 6 | (a.Scount[pg] - 1u);
            }
        }
        return v;
    };
    uint32_t my_pg = s_ids(rec[0]);

    int cur = 0;
    Acc acc;
    while (true) {
        const ItemRec C = rec[cur];
        if (C.item >= n_items) break;
        const uint32_t *tpg = ptab + cur * 2 * (kRMaxPages + 1);
        const uint32_t *tpk = tpg + kRMaxPages + 1;
        const uint32_t shift = C.shift;
        const uint32_t nrpg = C.nrpg, nspg = C.nspg;

        // --- the probing warp's first S page (ids loaded during the
        //     previous item): lane l holds tuples 2l, 2l + 1 of a page, cn the
        //     page's count (0: none)
        const uint32_t npw = warp < kProbeWarps && (uint32_t)warp < nspg
                                 ? (nspg - warp + kProbeWarps - 1) / kProbeWarps : 0u;
        auto load_page = [&](uint32_t i, ulonglong2 &x, uint32_t &cn) {
            const uint32_t v = __shfl_sync(0xffffffffu, my_pg, i & 31);
            cn = i < npw ? (v & 63u) + 1u : 0u;
            // an odd page's pad word is read with its last tuple
            if (2 * lane < (int)cn)
                x = __ldcs(reinterpret_cast<const ulonglong2 *>(a.Spages + (uint64_t)(v >> 6) * kPageTuples) + lane);
        };
        ulonglong2 x0 = make_ulonglong2(0, 0);
        uint32_t n0 = 0;
        if (warp < kProbeWarps) {
            load_page(0, x0, n0);
        }

        // the bits of x (the key, or its hash) that a bucket shares: the lowest
        // `link` ones, or the highest
        const uint32_t lnb = C.lnb, link = shift + lnb;
        const uint32_t bmask = (1u << lnb) - 1;
        const uint32_t lim = 1u << link, lmask = lim - 1;
        auto hash = [&](uint64_t t) { return kHashed ? tkey(t) * kHashMul : tkey(t); };
        auto bucket = [&](uint32_t x) { return kHashed ? x >> (32 - link) & bmask : x >> shift & bmask; };
        auto linked = [&](uint32_t x, uint32_t next) {
            return kHashed ? next << (32 - link) | (x << link) >> link : (x & ~lmask) | next;
        };
        auto next_of = [&](uint32_t w) { return kHashed ? w >> (32 - link) : w & lmask; };
        auto same = [&](uint32_t w, uint32_t x) { return kHashed ? (w ^ x) << link == 0 : (w ^ x) < lim; };
        for (uint32_t i = threadIdx.x; i < ((1u << lnb) + 3) / 4; i += kJoinThreads)
            reinterpret_cast<uint4 *>(heads)[i] = kSorted ? make_uint4(0, 0, 0, 0) : make_uint4(kNone, kNone, kNone, kNone);
        __syncthreads();

        // --- build: a warp per page, two tuples per lane, kB pages in flight
        auto enter = [&](uint32_t s, uint64_t t) {
            const uint32_t x = hash(t), old = atomicExch(&heads[bucket(x)], s);
            return tword(linked(x, old == kNone ? s : old), tpay(t));
        };
        constexpr int kB = kSorted ? 2 : 3;
        // f(slot, the lane's two tuples, whether the second is one) for every page of the chunk
        auto each_page = [&](auto f) {
            for (uint32_t k0 = warp; k0 < nrpg; k0 += kB * kWarps) {
                ulonglong2 r[kB];
                uint32_t v[kB];
#pragma unroll
                for (int j = 0; j < kB; j++) {
                    const uint32_t k = k0 + j * kWarps;
                    v[j] = k < nrpg ? tpk[k] : 0u;
                    if (2 * lane < (int)(v[j] & 0xFFu))
                        r[j] = __ldcs(reinterpret_cast<const ulonglong2 *>(a.Rpages + (uint64_t)tpg[k] * kPageTuples) +
                                      lane);
                }
#pragma unroll
                for (int j = 0; j < kB; j++)
                    if (2 * lane < (int)(v[j] & 0xFFu))
                        f((v[j] >> 8) + 2 * lane, r[j], 2 * lane + 1 < (int)(v[j] & 0xFFu));
            }
        };
        if (kSorted) {
            each_page([&](uint32_t, const ulonglong2 &r, bool two) {
                atomicAdd(&heads[bucket(hash(r.x))], 1u);
                if (two) atomicAdd(&heads[bucket(hash(r.y))], 1u);
            });
            __syncthreads();
            {   // bucket starts << 16: thread t's buckets t, t + 512, .. follow one another (any
                // order of the buckets will do, and this one has no bank conflicts)
                uint32_t loc = 0, tot;
                for (uint32_t d = threadIdx.x; d <= bmask; d += kJoinThreads) loc += heads[d];
                uint32_t at = block_exclusive_scan(loc, reinterpret_cast<uint32_t *>(red), &tot);
                for (uint32_t d = threadIdx.x; d <= bmask; d += kJoinThreads) {
                    const uint32_t n = heads[d];
                    heads[d] = at << 16;
                    at += n;
                }
            }
            __syncthreads();
            each_page([&](uint32_t, const ulonglong2 &r, bool two) {
                auto place = [&](uint64_t t) {
                    const uint32_t h = atomicAdd(&heads[bucket(hash(t))], 1u);   // start << 16 | placed
                    tup[(h >> 16) + (h & 0xFFFFu)] = t;
                };
                place(r.x);
                if (two) place(r.y);
            });
        } else {
            each_page([&](uint32_t s, ulonglong2 &r, bool two) {
                r.x = enter(s, r.x);
                if (two) r.y = enter(s + 1, r.y);
                *reinterpret_cast<ulonglong2 *>(tup + s) = r;
            });
        }
        __syncthreads();

        if (warp == kCtl) {
            // the next item's page table, then the item after it (rec[cur] is
            // free: every thread copied it before the barriers above)
            ItemRec *nx = &rec[cur ^ 1];
            uint32_t *npt = ptab + (cur ^ 1) * 2 * (kRMaxPages + 1);
            table(nx, npt);
            take(&rec[cur]);
            if (nx->item < n_items)   // and the table's pages into L2, a line per lane
                for (uint32_t i = lane; i < 4 * nx->nrpg; i += 32)
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(a.Rpages + (uint64_t)npt[i >> 2] * kPageTuples +
                                                                  (i & 3) * 16));
        } else {
            // the next item's S page ids, in flight during this probe
            const uint32_t nx_pg = s_ids(rec[cur ^ 1]);
            uint32_t matches = 0;
            auto probe = [&](uint64_t s) {
                const uint32_t key = tkey(s), x = hash(s);
                uint32_t at = heads[bucket(x)];
                if (at == (kSorted ? 0u : kNone)) return;
                const uint64_t sh = s_half(key, tpay(s));
                auto add = [&](uint64_t r) {
                    acc.sum += pair_hash_pre(key, tpay(r), sh);
                    matches++;
                };
                if (kSorted) {
                    uint32_t n = at & 0xFFFFu;
                    for (at >>= 16; n; n--, at++) {
                        const uint64_t r = tup[at];
                        if (tkey(r) == key) add(r);
                    }
                    return;
                }
                while (true) {
                    const uint64_t r = tup[at];
                    const uint32_t nx = next_of(tkey(r));
                    if (same(tkey(r), x)) add(r);
                    if (nx == at) break;
                    at = nx;
                }
            };
            for (uint32_t i = 0; i < npw; i++) {
                const ulonglong2 c = x0;
                const uint32_t n = n0;
                n0 = 0;
                if (i + 1 < npw) load_page(i + 1, x0, n0);
                const uint32_t m0 = matches;
                if (2 * lane < (int)n) probe(c.x);
                __syncwarp();
                const uint32_t m1 = matches;
                if (2 * lane + 1 < (int)n) probe(c.y);
                __syncwarp();
                if (kMat) {
                    mat_rows(a.mat, a.mat_cap, a.mat_n, c.x, m1 - m0);
                    mat_rows(a.mat, a.mat_cap, a.mat_n, c.y, matches - m1);
                }
            }
            acc.count += matches;
            my_pg = nx_pg;
        }
        if (a.wacc) {   // batched windows: this item's sums to its window
            block_flush(acc, a.wacc + 2 * C.win, red);
            acc = Acc();
        }
        __syncthreads();   // the next item rebuilds the table; rec / page tables published
        cur ^= 1;
    }
    block_flush(acc, a.acc, red);
    if (a.out && threadIdx.x == 0) finish_call(a.acc, a.out);
}

}  // namespace adb
