// joins.cuh -- device-resident join drivers shared by the C ABI and the
// batched/served paths.  Each driver: scratch size for a call, then the
// launch sequence on ctx->stream.  Results land in acc[0] (count) and acc[1]
// (checksum) of a device accumulator that is 0 at the start; acc[2] is the error
// word (a timed-out device wait sets it), acc[3] the materialised count, acc[4]
// NPO's build tuples equal to its empty marker, acc[5] the CTAs done.  All but
// the eager drivers end with a kernel that moves acc[0 .. 3] to ctx->h_res and
// clears acc (finish_call); run_eager leaves that to its caller.  After a driver
// that failed half-way, the caller waits for the stream and clears acc.
#pragma once

#include "engine.cuh"

namespace adb {

struct DevJoin {
    const uint64_t *R;
    uint64_t nR;
    const uint64_t *S;
    uint64_t nS;
    uint64_t *mat = nullptr;      // optional <S-key, S-payload> output
    uint64_t mat_cap = 0;
    int test_flags = 0;           // adb_join_params.test_flags
};

enum class Family { Radix, RadixHist, Npo, SortMerge, Shj, Pmj, Unsupported };

// ---- paged partitioning front end (radix and sort-merge joins), paged.cuh ----
struct PartOut;
struct DigitFn;
size_t paged_partition_scratch(uint64_t nR, uint64_t nS, uint32_t b1, uint32_t b2, int num_sms);
int run_paged_partition(Context *ctx, const DevJoin &j, DigitFn d1, const DigitFn *d2, PartOut *out,
                        unsigned long long *acc, uint32_t **ctr = nullptr);

// ---- hash joins of a small build side, small.cu ----
bool small_fits(uint64_t nR, uint64_t nS);
int run_small(Context *ctx, const DevJoin &j);

// ---- partitioned joins (PRO / RJ_st / PRH / PRHO, large NPO, m-way / m-pass / m-way+skew) ----
int radix_bits_for(uint64_t nR, uint64_t nS, int requested, int num_sms);
int sort_bits_for(uint64_t nR, uint64_t nS, int part_fanout, int num_sms);   // joinconfig_t.PARTFANOUT, 0 = chosen
size_t radix_scratch(uint64_t nR, uint64_t nS, int bits, int num_sms);
bool radix_fits(uint64_t nR, uint64_t nS, int bits, int num_sms);   // the slot numbers' 32 bits
// How a partition is joined: a chained table over digits of the key's low bits
// or of its hash, or a counting sort (the sort-merge names).
enum class PartJoin { Chain, HashedChain, Sorted };
int run_radix(Context *ctx, const DevJoin &j, int bits, PartJoin kind, unsigned long long *acc);

// ---- NPO / NPO_st ----
bool npo_partitioned(uint64_t nR, uint64_t nS, int requested, int num_sms);
uint32_t npo_region_bits(uint64_t nR, int requested);
size_t npo_scratch(uint64_t nR, uint64_t nS, int region_bits, int num_sms);
int run_npo(Context *ctx, const DevJoin &j, int region_bits, unsigned long long *acc);

// ---- eager SHJ / PMJ over one window given as arrival-ordered relations ----
size_t eager_scratch(uint64_t nR, uint64_t nS, Family fam, int model, int nthreads, int group_size);
int run_eager(Context *ctx, const DevJoin &j, Family fam, int model, uint64_t batch, int nthreads,
              int group_size, int progressive_step, uint64_t seed, unsigned long long *acc);
int stream_join(Context *ctx, Family fam, int model, const adb_stream_tuple *R, uint64_t nR,
                const adb_stream_tuple *S, uint64_t nS, const adb_join_params *p, adb_window_result *out,
                adb_window_progress *progress, uint64_t max_windows, uint64_t *n_windows);

}  // namespace adb
