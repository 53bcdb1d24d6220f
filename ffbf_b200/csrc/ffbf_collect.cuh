// ffbf_collect.cuh -- results of ordinary size (up to kSmallResults records) finished by one launch each, written
// straight to pinned host memory in their final order, so a call waits for the device once.
#pragma once
#include "ffbf_kernels.cuh"

namespace ffbf {

constexpr uint32_t kSmallResults = 16384;  // hit windows or matches the single-launch paths order

// Head of a pinned result buffer. `done` is 1 when the arrays behind it hold the whole result; `error` holds the scan's
// or the verification's error flags.
struct ResultHead {
    unsigned long long n, n_lines, error, done;
    unsigned long long at;  // where the arrays start in the job's words: n window starts, n line starts, n line ends
};
constexpr size_t result_bytes(uint32_t cap) { return 64 + 3 * 8 * (size_t)cap; }  // a head and three arrays

// What the hit collection of one scan reads and writes.
struct CollectJob {
    const uint8_t* text;
    uint64_t n;
    uint32_t len;
    uint32_t hits_cap;
    const HitRec* hits;
    HitLine* lines;
    uint32_t* counters;  // CNT_HITS in; CNT_MATCHES counts finished CTAs (zero before and after)
    const long long* tile_first_nl;
    const long long* tile_last_nl;
    uint32_t tile_bytes;
    uint64_t ntiles;
    ResultHead* head;  // pinned
    uint64_t* words;   // pinned: the arrays (ResultHead::at)
    uint64_t n_words;  // room there: three per window
    unsigned long long* used;  // words taken so far where several jobs share them (zero at first); null: all are this job's
    uint32_t cap;              // most windows
    uint32_t per_cta;  // windows per CTA and round
    uint32_t ctas;     // CTAs launched for the job; more windows than they take in a round need further ones
};
// A scan alone on the GPU spreads its windows over the SMs; among many jobs a CTA takes more of one.
constexpr uint32_t kCollectAlone = 128, kCollectBatch = 1024;

// Lines of a scan's hits, the hits in text order and their distinct lines. Leaves head->done 0 when there are more
// hits than job.cap or than shared room is left for, or a line reaches over more than kWalkTiles tiles: resolve_lines and
// order_hits then do it.
cudaError_t collect_hits(const CollectJob& job, cudaStream_t st);
// The same for jobs in device memory: items {job, CTA}, each job's CTAs 0 .. ctas - 1.
cudaError_t collect_hits_multi(const CollectJob* d_jobs, const uint2* d_items, uint32_t n_items, cudaStream_t st);

// Feed-forward prune of npat patterns: a bit per pattern in d_bits, counts per kPruneBlock patterns in d_counts (beyond
// kPrefixBlocks of them the sums of the counts before), the ascending ids in d_ids (the first ids_cap) and in host_ids
// (the first host_cap), their number in head->n.
constexpr uint32_t kPruneBlock = 1024;
constexpr uint64_t kPrefixBlocks = 8192;
inline uint64_t prune_blocks(uint64_t npat) { return (npat + kPruneBlock - 1) / kPruneBlock; }
cudaError_t prune_count(const uint64_t* d_start, const uint64_t* d_end, const uint64_t* d_hash, uint64_t npat,
                        const Geom& g, const uint32_t* d_ff, uint32_t* d_bits, uint32_t* d_counts, cudaStream_t st);
cudaError_t prune_emit(const uint32_t* d_bits, const uint32_t* d_counts, uint64_t npat, uint64_t* d_ids,
                       uint64_t ids_cap, ResultHead* head, uint64_t* host_ids, uint64_t host_cap, cudaStream_t st);

// (start, end) of the lines `ids`, and their bytes, line i's to out + at[i].
cudaError_t gather_spans(const uint64_t* d_ids, uint64_t n, const uint64_t* d_start, const uint64_t* d_end,
                         uint64_t* d_spans, cudaStream_t st);
cudaError_t gather_lines(const uint8_t* d_file, const uint64_t* d_spans, const uint64_t* d_at, uint64_t n,
                         uint8_t* d_out, cudaStream_t st);

// Exact matches of nhits hit records (verify_window), ordered by (offset, pattern id) and written to host memory
// when there are at most out_cap and kSmallResults of them; head->n is their number in any case. d_counters must be zero;
// CNT_QUEUE counts finished CTAs.
struct VerifyJob {
    const HitRec* hits;
    uint32_t nhits, match_cap;
    const uint8_t* text;
    uint64_t n;
    const uint64_t* keys;
    const uint32_t* vals;
    uint64_t mask;
    const uint8_t* pat;
    const uint64_t *pstart, *pend;
    uint64_t* m_off;
    uint32_t* m_pid;
    uint32_t* counters;
    ResultHead* head;
    uint64_t* out_off;
    uint64_t* out_pid;
    uint32_t out_cap;
};
cudaError_t verify_collect(const VerifyJob& job, cudaStream_t st);

}  // namespace ffbf
