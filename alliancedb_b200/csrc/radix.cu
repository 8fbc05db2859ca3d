// radix.cu -- paged partitioning front end and the partitioned joins (PRO, RJ_st,
// PRH, PRHO; NPO beyond L2; m-way, m-pass, m-way+skew).
//
// Reference flow: join_init_run (hashing/joins/parallel_radix_join.cpp:1488-1701)
// spawns prj_thread (:981-1473): parallel pass-1 partitioning, task-queued
// pass-2 partitioning, then a task-queued join per partition pair.  Here:
//   pass 1        partition_pass (flat input)  + page lists
//   pass 2        partition_pass (paged input, work units) + page lists  [fan-out > 2^9]
//   R chunks      part_chunks
//   join          radix_join_items: persistent, work-stealing build + probe
// The fan-out 2^bits is chosen so an R partition fills about one CTA's
// shared-memory table (8704 tuples).
#include <algorithm>

#include "joins.cuh"
#include "paged.cuh"
#include "radix_join.cuh"

namespace adb {

// CTAs of a flat pass, split over the relations by size, at most one per tile.
// Every (CTA, digit) stream ends in a partial page, which the join reads and
// copies like a full one, so the fewer streams the better where they are short:
//   * inputs below 2^27 tuples get one wave of CTAs (2^22 x 2^22, two waves of
//     1024-thread CTAs: 138 us instead of 118).  From 2^27 on the partial pages
//     no longer count and a second wave evens out skewed digits (2^27 x 2^27,
//     pass 1: theta 0 1.057 -> 1.046 ms, theta 1.5 1.154 -> 1.088 ms);
//   * wide: a single pass, whose pages go to the join, runs as one 1024-thread
//     CTA per SM, so half as many streams as two of 512 threads.  PRO, us, two
//     CTAs / one: 2^20 x 2^20 68 / 59, 2^22 x 2^22 134 / 117, the same with four of
//     each key 101 / 80 and 223 / 193, 2^22 x 2^26 (512 digits) 1669 / 1570; 2^20 x
//     2^25 854 / 867 (0.99, the one size where it was slower).  A first pass with
//     a second to follow keeps two CTAs, one of which loads and stores while
//     the other waits at a barrier (2^27 x 2^27: 0.953 ms, one CTA 1.033).
// The smaller relation's share is rounded up: rounded down, its chunks, and with
// them every CTA's page pool, would be up to 1.5 times the larger one's.
static void flat_ctas(uint64_t nR, uint64_t nS, int num_sms, bool wide, int G[2]) {
    const uint64_t all = (uint64_t)num_sms * (wide ? 1 : kPassMinBlocks) * (nR + nS >= (1ull << 27) ? 2 : 1);
    const uint64_t n[2] = {nR, nS}, tile = wide ? kWideTile : kFlatTile;
    const int small = nS < nR;
    auto at_most = [](uint64_t g, uint64_t a, uint64_t b) { return std::max<uint64_t>(1, std::min({g, a, b})); };
    const uint64_t share = nR + nS ? (all * n[small] + nR + nS - 1) / (nR + nS) : 1;
    const uint64_t gs = at_most(share, all - 1, (n[small] + tile - 1) / tile);
    G[small] = (int)gs;   // not more than all together: one CTA over would be a wave of its own
    G[!small] = (int)at_most(all - gs, all - gs, (n[!small] + tile - 1) / tile);
}

// Launches one partition pass (both relations: grid.y = relation).
static void launch_pass(const PassArgs &a, uint32_t F, int G, bool wide, cudaStream_t st) {
    const dim3 grid(G, 2);
    const bool h = a.df.hashed;
    auto go = [&](auto kernel, int threads, int tile) {
        kernel<<<grid, threads, pass_smem(tile, F, a.paged == 1), st>>>(a);
    };
    if (a.paged) go(h ? partition_pass<1, kPassThreads, kPagedTile, true> : partition_pass<1, kPassThreads, kPagedTile>,
                    kPassThreads, kPagedTile);
    else if (wide) go(h ? partition_pass<0, kWideThreads, kWideTile, true> : partition_pass<0, kWideThreads, kWideTile>,
                      kWideThreads, kWideTile);
    else go(h ? partition_pass<0, kPassThreads, kFlatTile, true> : partition_pass<0, kPassThreads, kFlatTile>,
            kPassThreads, kFlatTile);
}

// ---------------------------------------------------------------------------
// Paged partitioning front end
// ---------------------------------------------------------------------------
struct PartPlan {
    int passes;
    bool wide;                 // pass 1 in 1024-thread CTAs
    uint32_t F1, F2, Fout;
    int g1[2], g2[2];          // CTAs of R, S in pass 1, and in pass 2 (bounds)
    int G1, G2;                // the larger of the two
    uint32_t pool1, pool2;
    uint32_t unit_pages;       // pass-2 work unit
    uint64_t pages1[2], pages2[2];   // pool pages of R, S
    const uint64_t *pages() const { return passes == 2 ? pages2 : pages1; }   // of the output
    // slot numbers (page x 64 + place) are 32 bits
    bool fits() const {
        return std::max({pages1[0], pages1[1], pages2[0], pages2[1]}) * kPageTuples < (uint64_t)kNone;
    }
};

static PartPlan plan_partition(uint64_t nR, uint64_t nS, uint32_t b1, uint32_t b2, int num_sms) {
    PartPlan p{};
    p.passes = b2 ? 2 : 1;
    p.F1 = 1u << b1;
    p.F2 = b2 ? 1u << b2 : 1u;
    p.Fout = p.F1 * p.F2;
    p.wide = !b2;
    flat_ctas(nR, nS, num_sms, p.wide, p.g1);
    p.pool1 = std::max(flat_pool_cap(nR, p.g1[0], p.F1), flat_pool_cap(nS, p.g1[1], p.F1));
    // units from the tuples actually present (the pass-1 pool has slack)
    const uint64_t pages_in = (nR + kPageTuples - 1) / kPageTuples + (nS + kPageTuples - 1) / kPageTuples;
    p.unit_pages = unit_pages_for(pages_in, num_sms);
    p.pool2 = unit_pool_cap(p.F2, p.unit_pages);
    for (int r = 0; r < 2; r++) {
        p.pages1[r] = (uint64_t)p.g1[r] * p.pool1;
        if (b2) {
            p.g2[r] = (int)((p.pages1[r] + p.unit_pages - 1) / p.unit_pages + p.F1);
            p.pages2[r] = (uint64_t)p.g2[r] * p.pool2;
        }
    }
    p.G1 = std::max(p.g1[0], p.g1[1]);
    p.G2 = std::max(p.g2[0], p.g2[1]);
    return p;
}

static void split_bits(int bits, uint32_t *b1, uint32_t *b2) {
    // one pass up to 2^9 partitions; two passes of at most 2^8 each above
    if (bits <= (int)kMaxPassBits) {
        *b1 = bits;
        *b2 = 0;
    } else {
        *b1 = bits / 2;
        *b2 = bits - bits / 2;
    }
}

bool radix_fits(uint64_t nR, uint64_t nS, int bits, int num_sms) {
    uint32_t b1, b2;
    split_bits(bits, &b1, &b2);
    return plan_partition(nR, nS, b1, b2, num_sms).fits();
}

// Fan-out bits: partitions of at most 2^13 tuples (one R chunk), and below that
// size up to 2^8 partitions, down to 256 tuples each, so that the join's items
// fill the SMs.  Device time of PRO / m-way, us, four of each key on both sides,
// at these bits (and at 2^12 tuples a partition, or one bit less): 2^16 - / 53
// (4 bits 72), 2^18 64 / 71 (6 bits 73 / 83), 2^20 102 / 110 (7 bits 108 / 118), 2^21 133 /
// 167 (9 bits 166 / 186), 2^22 228 / 256 (8 bits 223 / 273), 2^23 - / 410 (9 bits 450).
// The largest relations leave 32-bit slot numbers less room for partial pages:
// where 2^b partitions do not fit them there are fewer, down to four R chunks per
// partition (2^13 partitions above 2^27 tuples).
static int partition_bits(uint64_t nR, uint64_t nS, int requested, int most, int num_sms) {
    int b = requested, least = requested;
    if (requested <= 0) {
        const int full = (int)ceil_log2_u64((nR + 8191) / 8192), fill = (int)ceil_log2_u64((nR + 255) / 256);
        least = full;
        b = std::max(full, std::min(fill, 8));
        most = 15;
    }
    b = std::max(1, std::min(b, most));
    least = std::max(1, std::min(least, 15) - 2);
    while (b > least && !radix_fits(nR, nS, b, num_sms)) b--;
    return b;
}

int radix_bits_for(uint64_t nR, uint64_t nS, int requested, int num_sms) {
    return partition_bits(nR, nS, requested, 15, num_sms);
}

// m-way / m-pass: the fan-out joinconfig_t.PARTFANOUT asks for, rounded up to a
// power of two (at most 2^16, two passes of 2^8), else as above.
int sort_bits_for(uint64_t nR, uint64_t nS, int part_fanout, int num_sms) {
    return partition_bits(nR, nS, part_fanout > 1 ? (int)ceil_log2_u64((uint64_t)part_fanout) : 0, 16, num_sms);
}

static size_t pageset_bytes(uint64_t pages, uint32_t G, uint32_t F) {
    return Workspace::need(pages * kPageTuples, 8) + 2 * Workspace::need(pages, 4) + Workspace::need(pages, 1) +
           Workspace::need(G, 4) + Workspace::need((uint64_t)G * F, 4) + Workspace::need(G, 8);
}

static size_t partition_bytes(const PartPlan &p) {
    size_t s = Workspace::need(2ull * (p.F1 + p.Fout) + 4, 4) + Workspace::need(2ull * (p.F1 + 1), 8);
    for (int r = 0; r < 2; r++) s += pageset_bytes(p.pages1[r], p.G1, p.F1);
    if (p.passes == 2) {
        s += Workspace::need(2ull * (p.Fout + 1), 8) + 2 * Workspace::need(p.F1 + 1, 4);
        for (int r = 0; r < 2; r++) s += pageset_bytes(p.pages2[r], p.G2, p.F2);
    }
    return s;
}

size_t paged_partition_scratch(uint64_t nR, uint64_t nS, uint32_t b1, uint32_t b2, int num_sms) {
    return partition_bytes(plan_partition(nR, nS, b1, b2, num_sms));
}

static void take_pageset(Context *ctx, PageSet &ps, uint64_t pages, int G, uint32_t F) {
    ps.pages = ctx->ws.take<uint64_t>(pages * kPageTuples);
    ps.log = ctx->ws.take<uint32_t>(pages);
    ps.pcount = ctx->ws.take<uint8_t>(pages);
    ps.nlog = ctx->ws.take<uint32_t>(G);
    ps.doff = ctx->ws.take<uint32_t>((uint64_t)G * F);
    ps.udesc = ctx->ws.take<uint2>(G);
    ps.plist = ctx->ws.take<uint32_t>(pages);
}

// Partitions R and S by d1 (and then d2) into page lists per output partition
// D = p1 * F2 + p2.  out->pstart = [2][Fout + 1] page-list starts.
int run_paged_partition(Context *ctx, const DevJoin &j, DigitFn d1, const DigitFn *d2, PartOut *out,
                        unsigned long long *acc, uint32_t **ctr) {
    cudaStream_t st = ctx->stream;
    const uint32_t b1 = ceil_log2_u64((uint64_t)d1.mask + 1), b2 = d2 ? ceil_log2_u64((uint64_t)d2->mask + 1) : 0;
    const PartPlan p = plan_partition(j.nR, j.nS, b1, b2, ctx->num_sms);
    if (!p.fits()) {
        set_error("relations too large for one partitioned join (%llu and %llu pool pages)",
                  (unsigned long long)p.pages()[0], (unsigned long long)p.pages()[1]);
        return ADB_ERR_ARG;
    }
    int *err = reinterpret_cast<int *>(acc + 2);

    // ---- pass 1
    PassArgs a1{};
    for (int r = 0; r < 2; r++) {
        a1.in[r].in = r ? j.S : j.R;
        a1.in[r].n = r ? j.nS : j.nR;
        a1.in[r].G = p.g1[r];
        take_pageset(ctx, a1.out[r], p.pages1[r], p.G1, p.F1);
    }
    a1.df = d1;
    a1.F1 = 1;
    a1.G = p.G1;
    a1.pool_cap = p.pool1;
    a1.paged = 0;
    a1.err = err;
    // the work counters and both passes' totals, cleared by one launch
    uint32_t *zeros = ctx->ws.take<uint32_t>(2ull * (p.F1 + p.Fout) + 4);
    uint32_t *totals1 = zeros + 4, *totals2 = totals1 + 2ull * p.F1;
    ADB_CK(cudaMemsetAsync(zeros, 0, 16 + 8ull * (p.F1 + (p.passes == 2 ? p.Fout : 0)), st));
    if (ctr) *ctr = zeros;
    a1.totals = totals1;
    a1.Dtot = p.F1;
    uint64_t *pstart1 = ctx->ws.take<uint64_t>(2ull * (p.F1 + 1));
    a1.out[0].pstart = pstart1;
    a1.out[1].pstart = pstart1 + (p.F1 + 1);

    launch_pass(a1, p.F1, p.G1, p.wide, st);
    uint32_t *uoff0 = nullptr, *uoff1 = nullptr;
    if (p.passes == 2) {
        uoff0 = ctx->ws.take<uint32_t>(p.F1 + 1);
        uoff1 = ctx->ws.take<uint32_t>(p.F1 + 1);
    }
    page_place<<<dim3(p.G1, 2), kPlaceThreads, 0, st>>>(a1, p.passes == 2 ? p.unit_pages : 0u, uoff0, uoff1);
    ADB_CK(cudaGetLastError());
    ADB_CK(mark(ctx, 1));   // end of pass 1
    ctx->kernels += 2;
    if (p.passes == 1) {
        out->R = a1.out[0];
        out->S = a1.out[1];
        out->Fout = p.F1;
        out->pstart = pstart1;
        out->pool_pages = p.pages1[0];
        return ADB_OK;
    }

    // ---- pass 2: work units over pass-1 partitions
    PassArgs a2{};
    for (int r = 0; r < 2; r++) {
        PassIn &in = a2.in[r];
        in.pages = a1.out[r].pages;
        in.pcount = a1.out[r].pcount;
        in.plist = a1.out[r].plist;
        in.pstart = a1.out[r].pstart;
        in.uoff = r ? uoff1 : uoff0;
        take_pageset(ctx, a2.out[r], p.pages2[r], p.G2, p.F2);
    }
    a2.df = *d2;
    a2.F1 = p.F1;
    a2.G = p.G2;
    a2.pool_cap = p.pool2;
    a2.unit_pages = p.unit_pages;
    a2.paged = 1;
    a2.err = err;
    a2.totals = totals2;
    a2.Dtot = p.Fout;
    uint64_t *pstart2 = ctx->ws.take<uint64_t>(2ull * (p.Fout + 1));
    a2.out[0].pstart = pstart2;
    a2.out[1].pstart = pstart2 + (p.Fout + 1);

    launch_pass(a2, p.F2, p.G2, false, st);
    list_starts<<<dim3((p.Fout + kScanThreads - 1) / kScanThreads, 2), kScanThreads, 0, st>>>(a2);
    page_place<<<dim3(p.G2, 2), kPlaceThreads, 0, st>>>(a2, 0u, nullptr, nullptr);
    ADB_CK(cudaGetLastError());
    ctx->kernels += 3;
    out->R = a2.out[0];
    out->S = a2.out[1];
    out->Fout = p.Fout;
    out->pstart = pstart2;
    out->pool_pages = p.pages2[0];
    return ADB_OK;
}

// ---------------------------------------------------------------------------
// Partitioned hash joins
// ---------------------------------------------------------------------------
size_t radix_scratch(uint64_t nR, uint64_t nS, int bits, int num_sms) {
    uint32_t b1, b2;
    split_bits(bits, &b1, &b2);
    const PartPlan p = plan_partition(nR, nS, b1, b2, num_sms);
    return partition_bytes(p) + WorkList::bytes(p.Fout, p.pages()[0], kChunkW);
}

int run_radix(Context *ctx, const DevJoin &j, int bits, PartJoin kind, unsigned long long *acc) {
    const bool hashed = kind != PartJoin::Chain;
    cudaStream_t st = ctx->stream;
    uint32_t b1, b2;
    split_bits(bits, &b1, &b2);
    // the key's low bits, or the high bits of key * kHashMul
    const DigitFn d1{hashed ? 32u - b1 : 0u, (1u << b1) - 1, hashed};
    const DigitFn d2{hashed ? 32u - b1 - b2 : b1, (1u << b2) - 1, hashed};
    PartOut po;
    uint32_t *ctr;
    ADB_TRY(run_paged_partition(ctx, j, d1, b2 ? &d2 : nullptr, &po, acc, &ctr));
    if (b2) ADB_CK(mark(ctx, 2));   // phases: pass 1 | pass 2 | work list | join

    const uint32_t F = po.Fout;
    WorkList wl;
    wl.take(ctx->ws, F, po.pool_pages, kChunkW, ctx->num_sms, ctr);
    ctx->kernels += make_work_list(st, po.pstart, po.R.plist, po.R.pcount, F, wl);
    ADB_CK(cudaGetLastError());
    ADB_CK(mark(ctx, 3));

    JoinArgs a;
    a.Rpages = po.R.pages; a.Spages = po.S.pages;
    a.Rcount = po.R.pcount; a.Scount = po.S.pcount;
    a.Rlist = po.R.plist; a.Slist = po.S.plist;
    a.pstart = po.pstart; a.wl = wl;
    a.acc = acc; a.out = ctx->h_res;
    a.F = F; a.bits = (uint32_t)bits;
    a.mat = j.mat; a.mat_n = acc + 3; a.mat_cap = j.mat_cap;
    a.wbase = nullptr; a.wbits = nullptr; a.nwin = 0; a.wacc = nullptr;
    const int grid = ctx->num_sms * kJoinMinBlocks;
    auto launch = [&](auto kernel) { kernel<<<grid, kJoinThreads, kJoinSmem, st>>>(a); };
    switch (kind) {
        case PartJoin::Chain: j.mat ? launch(radix_join_items<true>) : launch(radix_join_items<false>); break;
        case PartJoin::HashedChain:
            j.mat ? launch(radix_join_items<true, true>) : launch(radix_join_items<false, true>);
            break;
        case PartJoin::Sorted:
            j.mat ? launch(radix_join_items<true, true, true>) : launch(radix_join_items<false, true, true>);
            break;
    }
    ADB_CK(cudaGetLastError());
    ctx->kernels += 1;
    return ADB_OK;
}

int radix_set_attrs() {
    const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    auto pass_attr = [&](auto kernel, int tile, bool paged) {
        return cudaFuncSetAttribute(kernel, attr, (int)pass_smem(tile, 1u << kMaxPassBits, paged));
    };
    ADB_CK(pass_attr(partition_pass<0, kPassThreads, kFlatTile>, kFlatTile, false));
    ADB_CK(pass_attr(partition_pass<0, kPassThreads, kFlatTile, true>, kFlatTile, false));
    ADB_CK(pass_attr(partition_pass<0, kWideThreads, kWideTile>, kWideTile, false));
    ADB_CK(pass_attr(partition_pass<0, kWideThreads, kWideTile, true>, kWideTile, false));
    ADB_CK(pass_attr(partition_pass<1, kPassThreads, kPagedTile>, kPagedTile, true));
    ADB_CK(pass_attr(partition_pass<1, kPassThreads, kPagedTile, true>, kPagedTile, true));
    ADB_CK(cudaFuncSetAttribute(radix_join_items<false>, attr, (int)kJoinSmem));
    ADB_CK(cudaFuncSetAttribute(radix_join_items<true>, attr, (int)kJoinSmem));
    ADB_CK(cudaFuncSetAttribute(radix_join_items<false, true>, attr, (int)kJoinSmem));
    ADB_CK(cudaFuncSetAttribute(radix_join_items<true, true>, attr, (int)kJoinSmem));
    ADB_CK(cudaFuncSetAttribute(radix_join_items<false, true, true>, attr, (int)kJoinSmem));
    ADB_CK(cudaFuncSetAttribute(radix_join_items<true, true, true>, attr, (int)kJoinSmem));
    return ADB_OK;
}

}  // namespace adb
