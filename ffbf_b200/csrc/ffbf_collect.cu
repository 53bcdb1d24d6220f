// ffbf_collect.cu -- single-launch collection of scan results, matches and pruned ids (see ffbf_collect.cuh).
//
// A call on an ordinary text spends its time between kernels: the general path (tile scan, line resolution, radix
// sorts, selection, copies) is about fifteen launches and three waits for the device, 130 us for 500 hit windows.
// Here the records are finished by one launch that reads their number from the device: its CTAs share the
// windows, and the last CTA to finish sorts them in its shared memory and writes the result to pinned host memory. The
// sort is a bucket sort over the text's span, about two buckets per record, each then sorted by one thread (records of
// one bucket are few unless a text is very uneven, which takes a bitonic network instead: for 8000 windows about 120 us
// against 10). What bounds it is latency: the dependent loads of a line search, then four passes over the records.
// Whole calls, 500 windows of a 64 MiB text: 132 -> 39 us, 8000 of 1 GiB: 276 -> 89.
#include <climits>

#include "ffbf_collect.cuh"
#include "ffbf_text.cuh"

namespace ffbf {

namespace {

constexpr int kThreads = 1024;
constexpr uint64_t kWalkTiles = 64;              // tile summaries a line's end is searched in
// bitonic keys: the offset above the record's index
constexpr int kIndexBits = 14;
static_assert(kSmallResults == 1u << kIndexBits, "an index fits beside an offset below 2^50");

// Exclusive sum of v over the CTA; *total is the whole sum.
__device__ __forceinline__ uint32_t block_sum(uint32_t v, uint32_t* s_warp, uint32_t* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
        if (lane >= d) x += y;
    }
    __syncthreads();
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < (int)(blockDim.x >> 5) ? s_warp[lane] : 0u;
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, w, d);
            if (lane >= d) w += y;
        }
        s_warp[lane] = w;
    }
    __syncthreads();
    *total = s_warp[31];
    return x - v + (warp ? s_warp[warp - 1] : 0u);
}

// True in the last of the launch's (or the job's) `ctas` CTAs to get here, which then sees the others' writes.
__device__ __forceinline__ bool last_cta(uint32_t* ticket, uint32_t ctas, uint32_t* s_flag) {
    if (ctas == 1) {  // nobody to wait for
        __syncthreads();
        return true;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) *s_flag = atomicAdd(ticket, 1u) == ctas - 1;
    __syncthreads();
    __threadfence();
    return *s_flag != 0;
}

__device__ __forceinline__ uint32_t pow2_at_least(uint32_t n) { return n < 2 ? 1u : 1u << (32 - __clz(n - 1)); }

// Sorts s_key[0, n) ascending (n <= kSmallResults), where offset(q) is record q's offset, below 2^50, and its key is the
// offset above q's 14 bits; less orders two keys. s_bucket holds kBuckets words. All of the CTA's threads call it.
constexpr uint32_t kBuckets = 2 * kSmallResults;
constexpr uint32_t kMaxBucket = 24;  // records one thread sorts by insertion

template <class Offset, class Less>
__device__ void sort_records(uint32_t n, uint64_t span, uint64_t* s_key, uint16_t* s_bucket, uint32_t* s_warp,
                             Offset offset, Less less) {
    // buckets of 2^shift offsets, more of them than records and a multiple of the threads
    const uint32_t nb = max(2 * pow2_at_least(n), (uint32_t)kThreads);
    uint32_t shift = 0;
    while ((span >> shift) >= nb) shift++;
    uint32_t* s_pair = reinterpret_cast<uint32_t*>(s_bucket);  // two 16-bit counts per word
    for (uint32_t b = threadIdx.x; b < nb / 2; b += kThreads) s_pair[b] = 0;
    __syncthreads();
    uint32_t most = 0;
    for (uint32_t q = threadIdx.x; q < n; q += kThreads) {
        const uint32_t b = (uint32_t)(offset(q) >> shift);
        const uint32_t old = atomicAdd(&s_pair[b >> 1], (b & 1) ? 0x10000u : 1u);
        most = max(most, ((b & 1) ? old >> 16 : old & 0xffffu) + 1);
    }
    most = (uint32_t)__syncthreads_or((int)(most > kMaxBucket));
    if (most) {
        // uneven: a bitonic network over the next power of two
        const uint32_t n2 = pow2_at_least(n);
        for (uint32_t q = threadIdx.x; q < n2; q += kThreads) s_key[q] = q < n ? offset(q) << kIndexBits | q : ~0ull;
        for (uint32_t k = 2; k <= n2; k <<= 1) {
            for (uint32_t j = k >> 1; j > 0; j >>= 1) {
                __syncthreads();
                for (uint32_t t = threadIdx.x; t < n2 / 2; t += kThreads) {
                    const uint32_t lo = 2 * t - (t & (j - 1)), hi = lo + j;  // bit j of lo is clear
                    const uint64_t x = s_key[lo], y = s_key[hi];
                    if (less(y, x) == ((lo & k) == 0)) {
                        s_key[lo] = y;
                        s_key[hi] = x;
                    }
                }
            }
        }
        __syncthreads();
        return;
    }
    // each thread's consecutive buckets: counts to starts
    const uint32_t per = nb / kThreads, b0 = threadIdx.x * per;
    uint32_t mine = 0;
    for (uint32_t b = b0; b < b0 + per; b++) mine += s_bucket[b];
    uint32_t total;
    uint32_t at = block_sum(mine, s_warp, &total);
    for (uint32_t b = b0; b < b0 + per; b++) {
        const uint32_t c = s_bucket[b];
        s_bucket[b] = (uint16_t)at;
        at += c;
    }
    __syncthreads();
    // a bucket's word counts up to the next bucket's start while its records are placed
    for (uint32_t q = threadIdx.x; q < n; q += kThreads) {
        const uint64_t o = offset(q);
        const uint32_t b = (uint32_t)(o >> shift);
        const uint32_t old = atomicAdd(&s_pair[b >> 1], (b & 1) ? 0x10000u : 1u);
        s_key[(b & 1) ? old >> 16 : old & 0xffffu] = o << kIndexBits | q;
    }
    __syncthreads();
    for (uint32_t b = threadIdx.x; b < nb; b += kThreads) {
        const uint32_t lo = b ? s_bucket[b - 1] : 0u, hi = s_bucket[b];
        for (uint32_t x = lo + 1; x < hi; x++) {
            const uint64_t v = s_key[x];
            uint32_t y = x;
            for (; y > lo && less(v, s_key[y - 1]); y--) s_key[y] = s_key[y - 1];
            s_key[y] = v;
        }
    }
    __syncthreads();
}

__device__ void collect_one(const CollectJob& a, uint32_t cta) {
    extern __shared__ uint64_t s_key[];
    __shared__ uint32_t s_warp[32], s_flag;
    __shared__ unsigned long long s_at;
    const uint32_t nh = a.counters[CNT_HITS];
    if (nh > a.cap || nh > a.hits_cap) {  // the general path takes over
        if (cta == 0 && threadIdx.x == 0) {
            a.head->n = nh;
            a.head->error = a.counters[CNT_ERROR];
            a.head->done = 0;
        }
        return;
    }
    const uint32_t ctas = min(a.ctas, nh ? (nh + a.per_cta - 1) / a.per_cta : 1u);
    if (cta >= ctas) return;
    // Eight lanes per window; every lane of a warp takes part in every round. A CTA's next windows follow those of all.
    uint32_t end = min(nh, (cta + 1) * a.per_cta);
    for (uint32_t i0 = cta * a.per_cta; i0 < nh; i0 += kThreads / 8) {
        if (i0 >= end) {
            i0 = end + (ctas - 1) * a.per_cta;
            end = min(nh, i0 + a.per_cta);
            if (i0 >= nh) break;
        }
        const uint32_t i = i0 + threadIdx.x / 8;
        const uint64_t w = i < end ? a.hits[i].off : 0u;
        const long long found = line_end_of_window(a.text, a.n, a.len, a.tile_bytes, w, i < end);
        const long long sp = __shfl_sync(0xffffffffu, found, threadIdx.x & 24);
        const long long ep = __shfl_sync(0xffffffffu, found, (threadIdx.x & 24) + 4);
        if (i < end && (threadIdx.x & 7) == 0) {
            long long s = sp, e = ep;
            if (s < 0) {
                long long t = (long long)((w - 1) / a.tile_bytes) - 1;
                for (uint64_t k = 0; k < kWalkTiles && s < 0 && t >= 0; k++, t--) {
                    const long long l = a.tile_last_nl[t];
                    if (l >= 0) s = l + 1;
                }
                if (t < 0 && s < 0) s = 0;
            }
            if (e < 0) {
                uint64_t t = (w + a.len) / a.tile_bytes + 1;
                for (uint64_t k = 0; k < kWalkTiles && e < 0 && t < a.ntiles; k++, t++) {
                    const long long f = a.tile_first_nl[t];
                    if (f != LLONG_MAX) e = f;
                }
                if (t >= a.ntiles && e < 0) e = (long long)a.n;
            }
            a.lines[i] = HitLine{(uint64_t)s, (uint64_t)e};  // ~0: not found in the tiles walked
        }
    }
    if (!last_cta(a.counters + CNT_MATCHES, ctas, &s_flag)) return;
    if (threadIdx.x == 0) a.counters[CNT_MATCHES] = 0;
    uint32_t open = 0;
    for (uint32_t q = threadIdx.x; q < nh; q += kThreads)
        open |= __ldcg(&a.lines[q].start) == ~0ull || __ldcg(&a.lines[q].end) == ~0ull;
    open = (uint32_t)__syncthreads_or((int)open);
    if (!open) {
        if (threadIdx.x == 0) s_at = a.used ? atomicAdd(a.used, 3ull * nh) : 0ull;
        __syncthreads();
    }
    if (open || s_at + 3ull * nh > a.n_words) {
        if (threadIdx.x == 0) {
            a.head->n = nh;
            a.head->error = a.counters[CNT_ERROR];
            a.head->done = 0;
        }
        return;
    }
    uint64_t *const off = a.words + s_at, *const line_start = off + nh, *const line_end = line_start + nh;
    sort_records(
        nh, a.n, s_key, reinterpret_cast<uint16_t*>(s_key + kSmallResults), s_warp,
        [&](uint32_t q) { return a.hits[q].off; }, [](uint64_t x, uint64_t y) { return x < y; });
    // lines are disjoint and windows sorted by start, so equal lines are adjacent
    uint32_t n_lines = 0;
    for (uint32_t q0 = 0; q0 < nh; q0 += kThreads) {
        const uint32_t q = q0 + threadIdx.x;
        uint32_t flag = 0;
        uint64_t ls = 0, le = 0;
        if (q < nh) {
            const uint32_t idx = (uint32_t)s_key[q] & (kSmallResults - 1);
            ls = __ldcg(&a.lines[idx].start);
            le = __ldcg(&a.lines[idx].end);
            flag = q == 0 || __ldcg(&a.lines[(uint32_t)s_key[q - 1] & (kSmallResults - 1)].start) != ls;
            off[q] = s_key[q] >> kIndexBits;
        }
        uint32_t total;
        const uint32_t at = n_lines + block_sum(flag, s_warp, &total);
        if (flag) {
            line_start[at] = ls;
            line_end[at] = le;
        }
        n_lines += total;
    }
    if (threadIdx.x == 0) {
        a.head->n = nh;
        a.head->n_lines = n_lines;
        a.head->error = a.counters[CNT_ERROR];
        a.head->at = s_at;
        a.head->done = 1;
    }
}

__global__ void __launch_bounds__(kThreads) k_collect(CollectJob a) { collect_one(a, blockIdx.x); }

__global__ void __launch_bounds__(kThreads) k_collect_multi(const CollectJob* jobs, const uint2* items) {
    collect_one(jobs[items[blockIdx.x].x], items[blockIdx.x].y);
}

// One bit and one ballot per pattern (filterPhrases, ffbf.cpp:394-485, as k_prune), counts per block.
__global__ void __launch_bounds__(kPruneBlock) k_prune_count(const uint64_t* start, const uint64_t* end,
                                                             const uint64_t* hash, uint64_t npat, Geom g,
                                                             const uint32_t* ff, uint32_t* bits, uint32_t* counts) {
    const uint64_t i = blockIdx.x * (uint64_t)kPruneBlock + threadIdx.x;
    const bool keep = i < npat && end[i] - start[i] >= g.len && check_all<2>(g, ff, hash[i]);
    const unsigned m = __ballot_sync(0xffffffffu, keep);
    if ((threadIdx.x & 31) == 0 && i < npat) bits[i >> 5] = m;
    const int n = __syncthreads_count(keep);
    if (threadIdx.x == 0) counts[blockIdx.x] = (uint32_t)n;
}

// Counts to the sums of those before them, in place, by one CTA.
__global__ void __launch_bounds__(kThreads) k_prune_prefix(uint32_t* counts, uint64_t n) {
    __shared__ uint32_t s_warp[32];
    constexpr uint32_t kPer = 16;  // consecutive counts per thread and round
    uint32_t before = 0;
    for (uint64_t first = 0; first < n; first += kPer * kThreads) {
        const uint64_t i = first + kPer * threadIdx.x;
        uint32_t v[kPer], mine = 0, total;
#pragma unroll
        for (uint32_t q = 0; q < kPer; q++) {
            v[q] = i + q < n ? counts[i + q] : 0u;
            mine += v[q];
        }
        uint32_t at = before + block_sum(mine, s_warp, &total);
#pragma unroll
        for (uint32_t q = 0; q < kPer; q++) {
            if (i + q < n) counts[i + q] = at;
            at += v[q];
        }
        before += total;
    }
}

// Block b writes its patterns' ids behind those of the blocks before it, whose counts it sums (a few coalesced loads
// per thread, in place of a scan launch).
__global__ void __launch_bounds__(kPruneBlock) k_prune_emit(const uint32_t* bits, const uint32_t* counts,
                                                            uint64_t npat, uint64_t* ids, uint64_t ids_cap,
                                                            ResultHead* head, uint64_t* host_ids, uint64_t host_cap) {
    __shared__ uint32_t s_warp[32];
    uint32_t before = 0;
    for (uint32_t b = threadIdx.x; b < blockIdx.x; b += kPruneBlock) before += counts[b];
    uint32_t base, total;
    block_sum(before, s_warp, &base);
    const uint64_t i = blockIdx.x * (uint64_t)kPruneBlock + threadIdx.x;
    const uint32_t keep = i < npat ? bits[i >> 5] >> (threadIdx.x & 31) & 1u : 0u;
    const uint64_t at = base + block_sum(keep, s_warp, &total);
    if (keep) {
        if (at < ids_cap) ids[at] = i;
        if (at < host_cap) host_ids[at] = i;
    }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) head->n = (unsigned long long)base + total;
}

// The same behind k_prune_prefix, a warp per block of patterns and a lane per word of bits. The sums that k_prune_emit's
// blocks make grow with the square of their number, and their barriers cost as much: 128M patterns, whole
// prune 3.0 -> 1.5 ms, 64M 1.35 -> 0.83, 16M 0.41 -> 0.32; 4M take 0.20 the other way and do not reach it.
__global__ void __launch_bounds__(256) k_prune_emit_prefixed(const uint32_t* bits, const uint32_t* sums, uint64_t npat,
                                                             uint64_t* ids, uint64_t ids_cap, ResultHead* head,
                                                             uint64_t* host_ids, uint64_t host_cap) {
    static_assert(kPruneBlock == 32 * 32, "a lane per word");
    const uint64_t block = (blockIdx.x * (uint64_t)256 + threadIdx.x) / 32, word = 32 * block + (threadIdx.x & 31);
    if (block * kPruneBlock >= npat) return;
    uint32_t m = word < (npat + 31) / 32 ? bits[word] : 0u;
    uint32_t before = __popc(m);
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, before, d);
        if ((threadIdx.x & 31) >= d) before += y;
    }
    uint64_t at = (uint64_t)sums[block] + before - __popc(m);
    if ((threadIdx.x & 31) == 31 && (block + 1) * kPruneBlock >= npat) head->n = at + __popc(m);
    for (; m; m &= m - 1, at++) {
        const uint64_t i = 32 * word + (__ffs(m) - 1);
        if (at < ids_cap) ids[at] = i;
        if (at < host_cap) host_ids[at] = i;
    }
}

__global__ void k_gather_spans(const uint64_t* ids, uint64_t n, const uint64_t* start, const uint64_t* end,
                               uint64_t* spans) {
    const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    spans[2 * i] = start[ids[i]];
    spans[2 * i + 1] = end[ids[i]];
}

// A warp per line.
__global__ void k_gather_lines(const uint8_t* file, const uint64_t* spans, const uint64_t* at, uint64_t n,
                               uint8_t* out) {
    const uint64_t i = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) / 32;
    if (i >= n) return;
    const uint64_t s = spans[2 * i], len = spans[2 * i + 1] - s;
    for (uint64_t b = threadIdx.x & 31; b < len; b += 32) out[at[i] + b] = file[s + b];
}

// Orders the matches (offset, then pattern id) of a.counters when shared memory holds them: one CTA.
__device__ void order_matches_small(const VerifyJob& a, uint32_t* s_warp) {
    extern __shared__ uint64_t s_key[];
    const uint32_t nm = __ldcg(a.counters + CNT_MATCHES);
    const bool small = nm <= kSmallResults && nm <= a.match_cap && nm <= a.out_cap;
    if (small) {
        auto pid = [&](uint64_t key) { return __ldcg(a.m_pid + ((uint32_t)key & (kSmallResults - 1))); };
        sort_records(
            nm, a.n, s_key, reinterpret_cast<uint16_t*>(s_key + kSmallResults), s_warp,
            [&](uint32_t q) { return __ldcg(a.m_off + q); },
            [&](uint64_t x, uint64_t y) {
                const uint64_t ox = x >> kIndexBits, oy = y >> kIndexBits;
                // a network pads with ~0, above every record
                return ox != oy ? ox < oy : x != ~0ull && pid(x) < pid(y);
            });
        for (uint32_t q = threadIdx.x; q < nm; q += kThreads) {
            a.out_off[q] = s_key[q] >> kIndexBits;
            a.out_pid[q] = pid(s_key[q]);
        }
    }
    if (threadIdx.x == 0) {
        a.head->n = nm;
        a.head->error = a.counters[CNT_ERROR];
        a.head->done = small;
    }
}

// Matches of a few windows, ordered by the last CTA to finish.
__global__ void __launch_bounds__(kThreads) k_verify_collect(VerifyJob a) {
    __shared__ uint32_t s_warp[32], s_flag;
    // neighbouring windows go to different CTAs: a few hundred windows then wait on as many SMs' memory pipes
    for (uint64_t j = blockIdx.x + (uint64_t)gridDim.x * threadIdx.x; j < a.nhits; j += (uint64_t)gridDim.x * kThreads)
        verify_window(a.hits[j], a.text, a.n, a.keys, a.vals, a.mask, a.pat, a.pstart, a.pend, a.m_off, a.m_pid,
                      a.match_cap, a.counters);
    if (last_cta(a.counters + CNT_QUEUE, gridDim.x, &s_flag)) order_matches_small(a, s_warp);
}

__global__ void __launch_bounds__(256) k_verify(VerifyJob a) {
    const uint64_t j = blockIdx.x * (uint64_t)256 + threadIdx.x;
    if (j < a.nhits)
        verify_window(a.hits[j], a.text, a.n, a.keys, a.vals, a.mask, a.pat, a.pstart, a.pend, a.m_off, a.m_pid,
                      a.match_cap, a.counters);
}

__global__ void __launch_bounds__(kThreads) k_order_matches(VerifyJob a) {
    __shared__ uint32_t s_warp[32];
    order_matches_small(a, s_warp);
}

constexpr size_t kSmem = (8 + 2 * (kBuckets / kSmallResults)) * (size_t)kSmallResults;  // keys, 16-bit bucket counts

}  // namespace

cudaError_t collect_hits(const CollectJob& job, cudaStream_t st) {
    cudaError_t e = cudaFuncSetAttribute(k_collect, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
    if (e != cudaSuccess) return e;
    k_collect<<<job.ctas, kThreads, kSmem, st>>>(job);
    note_launches(1);
    return cudaGetLastError();
}

cudaError_t collect_hits_multi(const CollectJob* d_jobs, const uint2* d_items, uint32_t n_items, cudaStream_t st) {
    if (!n_items) return cudaSuccess;
    cudaError_t e =
        cudaFuncSetAttribute(k_collect_multi, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
    if (e != cudaSuccess) return e;
    k_collect_multi<<<n_items, kThreads, kSmem, st>>>(d_jobs, d_items);
    note_launches(1);
    return cudaGetLastError();
}

cudaError_t prune_count(const uint64_t* d_start, const uint64_t* d_end, const uint64_t* d_hash, uint64_t npat,
                        const Geom& g, const uint32_t* d_ff, uint32_t* d_bits, uint32_t* d_counts, cudaStream_t st) {
    k_prune_count<<<(unsigned)prune_blocks(npat), kPruneBlock, 0, st>>>(d_start, d_end, d_hash, npat, g, d_ff, d_bits,
                                                                      d_counts);
    note_launches(1);
    if (prune_blocks(npat) > kPrefixBlocks) {
        k_prune_prefix<<<1, kThreads, 0, st>>>(d_counts, prune_blocks(npat));
        note_launches(1);
    }
    return cudaGetLastError();
}

cudaError_t prune_emit(const uint32_t* d_bits, const uint32_t* d_counts, uint64_t npat, uint64_t* d_ids,
                       uint64_t ids_cap, ResultHead* head, uint64_t* host_ids, uint64_t host_cap, cudaStream_t st) {
    const uint64_t blocks = prune_blocks(npat);
    if (blocks > kPrefixBlocks)
        k_prune_emit_prefixed<<<(unsigned)((blocks + 7) / 8), 256, 0, st>>>(d_bits, d_counts, npat, d_ids, ids_cap, head,
                                                                            host_ids, host_cap);
    else
        k_prune_emit<<<(unsigned)blocks, kPruneBlock, 0, st>>>(d_bits, d_counts, npat, d_ids, ids_cap, head, host_ids,
                                                               host_cap);
    note_launches(1);
    return cudaGetLastError();
}

cudaError_t gather_spans(const uint64_t* d_ids, uint64_t n, const uint64_t* d_start, const uint64_t* d_end,
                         uint64_t* d_spans, cudaStream_t st) {
    if (!n) return cudaSuccess;
    k_gather_spans<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(d_ids, n, d_start, d_end, d_spans);
    note_launches(1);
    return cudaGetLastError();
}

cudaError_t gather_lines(const uint8_t* d_file, const uint64_t* d_spans, const uint64_t* d_at, uint64_t n,
                         uint8_t* d_out, cudaStream_t st) {
    if (!n) return cudaSuccess;
    k_gather_lines<<<(unsigned)((n + 7) / 8), 256, 0, st>>>(d_file, d_spans, d_at, n, d_out);
    note_launches(1);
    return cudaGetLastError();
}

cudaError_t verify_collect(const VerifyJob& job, cudaStream_t st) {
    cudaError_t e =
        cudaFuncSetAttribute(k_verify_collect, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_order_matches, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
    if (e != cudaSuccess) return e;
    if (job.nhits > 2 * kSmallResults) {
        // many windows: as many threads as the SMs hold, which the fused kernel's shared memory would halve (356k
        // windows: 299 us against 218), then one CTA orders what is few
        k_verify<<<(job.nhits + 255) / 256, 256, 0, st>>>(job);
        k_order_matches<<<1, kThreads, kSmem, st>>>(job);
        note_launches(2);
        return cudaGetLastError();
    }
    const uint32_t ctas = job.nhits / 32 + 1;
    k_verify_collect<<<ctas > 148 ? 148 : ctas, kThreads, kSmem, st>>>(job);
    note_launches(1);
    return cudaGetLastError();
}

}  // namespace ffbf
