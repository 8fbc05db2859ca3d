// small.cu -- the hash joins of a small build side: one launch, no partitioning.
//
// Up to 2^13 build tuples fit one CTA's shared memory, so a CTA builds the
// table of one such chunk of R for itself (R is read from L2) and probes its
// share of S straight from the input: grid.x shares of S times grid.y chunks of
// R.  The last CTA to finish hands the totals to the host's result words and
// clears them for the next call, so a call is this launch and a wait.  Used by
// every hash-join name (PRO, RJ_st, PRH, PRHO, NPO, NPO_st): their results are
// the same join.
//
// The table is radix_join.cuh's, over hk = key * kHashMul instead of the key (a
// bijection): bucket = the top lnb bits of hk, so that keys with equal low bits
// spread; a linked tuple holds its chain's next slot (its own: the end) in
// those bits and the rest of hk below them.
#include <algorithm>

#include "joins.cuh"

namespace adb {

constexpr uint32_t kSmallLog2 = 13;                    // log2 of the most build tuples
constexpr int kSmallThreads = 512;
constexpr int kSmallBlocks = 2;                        // CTAs per SM
constexpr int kSmallU = 4;                             // S tuples per lane in flight
constexpr uint64_t kSmallMaxChunks = 65535;            // grid.y
constexpr uint64_t kSmallMaxProbes = 1ull << 23;
constexpr uint32_t kSmallNone = 0xFFFFFFFFu;
constexpr size_t kSmallSmem = ((size_t)12 << kSmallLog2) + 64 * 8;
static_assert(kSmallBlocks * (kSmallSmem + 1024) <= 233472, "small_join CTAs exceed the SM's shared memory");

// acc: [0] count, [1] checksum, [3] materialised tuples; out: the host's copy.
template <bool kMat>
__global__ void __launch_bounds__(kSmallThreads, kSmallBlocks)
small_join(const uint64_t *__restrict__ R, uint64_t allR, uint32_t lnb, const uint64_t *__restrict__ S, uint64_t nS,
           uint64_t per_cta, unsigned long long *acc, unsigned long long *out, uint64_t *mat, uint64_t mat_cap) {
    extern __shared__ __align__(16) unsigned char smem[];
    uint64_t *tup = reinterpret_cast<uint64_t *>(smem);
    uint32_t *heads = reinterpret_cast<uint32_t *>(tup + (1u << kSmallLog2));
    uint64_t *red = reinterpret_cast<uint64_t *>(heads + (1u << kSmallLog2));
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t rest = 32u - lnb;                   // bits of hk below the bucket's
    R += (uint64_t)blockIdx.y << kSmallLog2;           // this CTA's chunk
    const uint32_t nR = (uint32_t)min(allR - ((uint64_t)blockIdx.y << kSmallLog2), (uint64_t)1 << kSmallLog2);

    // the warp's first S tuples, in flight during the build
    const uint64_t b = (uint64_t)blockIdx.x * per_cta, e = min(nS, b + per_cta);
    uint64_t s[kSmallU];
    uint64_t i0 = b + (uint64_t)warp * (32 * kSmallU) + lane;
#pragma unroll
    for (int u = 0; u < kSmallU; u++)
        s[u] = i0 + 32 * u < e ? __ldcs(reinterpret_cast<const unsigned long long *>(S) + i0 + 32 * u) : 0ULL;

    for (uint32_t i = threadIdx.x; i < 1u << lnb; i += kSmallThreads) heads[i] = kSmallNone;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < nR; i += 4 * kSmallThreads) {
        uint64_t r[4];
#pragma unroll
        for (int j = 0; j < 4; j++) r[j] = i + j * kSmallThreads < nR ? R[i + j * kSmallThreads] : 0ULL;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const uint32_t k = i + j * kSmallThreads;
            if (k < nR) {
                const uint32_t hk = tkey(r[j]) * kHashMul;
                const uint32_t old = atomicExch(&heads[hk >> rest], k);
                tup[k] = tword((old == kSmallNone ? k : old) << rest | (hk << lnb) >> lnb, tpay(r[j]));
            }
        }
    }
    __syncthreads();

    Acc a;
    while (i0 < e + lane) {   // warp-uniform: the warp's first tuple
        const uint64_t i1 = i0 + kSmallThreads * kSmallU;
        uint64_t n[kSmallU];
#pragma unroll
        for (int u = 0; u < kSmallU; u++)
            n[u] = i1 + 32 * u < e ? __ldcs(reinterpret_cast<const unsigned long long *>(S) + i1 + 32 * u) : 0ULL;
#pragma unroll
        for (int u = 0; u < kSmallU; u++) {
            uint32_t rows = 0;
            if (i0 + 32 * u < e) {
                const uint32_t key = tkey(s[u]), hk = key * kHashMul;
                uint32_t at = heads[hk >> rest];
                if (at != kSmallNone) {
                    const uint64_t sh = s_half(key, tpay(s[u]));
                    while (true) {
                        const uint64_t r = tup[at];
                        if ((tkey(r) ^ hk) << lnb == 0) {
                            a.count++;
                            a.sum += pair_hash_pre(key, tpay(r), sh);
                            if (kMat) rows++;
                        }
                        const uint32_t nx = tkey(r) >> rest;
                        if (nx == at) break;
                        at = nx;
                    }
                }
            }
            __syncwarp();
            if (kMat) mat_rows(mat, mat_cap, acc + 3, s[u], rows);
        }
#pragma unroll
        for (int u = 0; u < kSmallU; u++) s[u] = n[u];
        i0 = i1;
    }
    block_flush(a, acc, red);
    if (threadIdx.x == 0) finish_call(acc, out);
}

// One chunk of R at any |S|; several while the probes, one per S tuple and
// chunk, stay within 2^23.  Device time, us, here / partitioned / NPO's global
// table (keys over 32 bits; four of each key on both sides): 2^14 x 2^18 20 / 162 /
// 51, 2^16 x 2^16 20 / 79 / 47, 2^17 x 2^18 38 / 96 / 63, 2^18 x 2^18 (2^23 probes) 54 /
// 76 / 55 (64 / 91 / 67), and past it 2^18 x 2^19 90 / 90 / 62, 2^19 x 2^18 (110 / 86 / 86).
// With one chunk: 2^13 x 2^23 79 / 196 / 223, 2^13 x 2^27 1007 / 1895 / 2796.
// With many and a short S, whole calls, us, here / partitioned: 2^22 x 2^11 41 / 165,
// 2^24 x 2^11 82 / 356, 2^26 x 2^8 229 / 735, 2^27.5 x 2^8 578 / 1793.
bool small_fits(uint64_t nR, uint64_t nS) {
    const uint64_t chunks = (nR + (1u << kSmallLog2) - 1) >> kSmallLog2;
    return chunks <= 1 || (chunks <= kSmallMaxChunks && chunks * nS <= kSmallMaxProbes);
}

// One launch; the result is in ctx->h_res once the stream has passed it.
int run_small(Context *ctx, const DevJoin &j) {
    const uint64_t chunks = (j.nR + (1u << kSmallLog2) - 1) >> kSmallLog2;
    const uint32_t lnb = j.nR <= 2 ? 1u : chunks > 1 ? kSmallLog2 : ceil_log2_u64(j.nR);
    // a CTA takes at least one round of S tuples; every CTA resident at once
    const uint64_t round = (uint64_t)kSmallThreads * kSmallU;
    const uint64_t most = std::max<uint64_t>(1, (uint64_t)ctx->num_sms * kSmallBlocks / chunks);
    const uint64_t gx = std::min((j.nS + round - 1) / round, most);
    const uint64_t per = ((j.nS + gx - 1) / gx + 127) & ~127ULL;
    const dim3 grid((unsigned)gx, (unsigned)chunks);
    if (j.mat)
        small_join<true><<<grid, kSmallThreads, kSmallSmem, ctx->stream>>>(
            j.R, j.nR, lnb, j.S, j.nS, per, ctx->d_acc, ctx->h_res, j.mat, j.mat_cap);
    else
        small_join<false><<<grid, kSmallThreads, kSmallSmem, ctx->stream>>>(
            j.R, j.nR, lnb, j.S, j.nS, per, ctx->d_acc, ctx->h_res, nullptr, 0);
    ADB_CK(cudaGetLastError());
    ctx->kernels++;
    return ADB_OK;
}

int small_set_attrs() {
    ADB_CK(cudaFuncSetAttribute(small_join<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmallSmem));
    ADB_CK(cudaFuncSetAttribute(small_join<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmallSmem));
    return ADB_OK;
}

}  // namespace adb
