// ffbf_capi.cu -- host side of the C ABI declared in include/ffbf.h.
//
// Owns the per-context device state (the two bit arrays, the pattern file image and its line table, the
// scan/prune/verify buffers) and sequences the kernels on the context's stream. Host work is limited to
// argument checks, sorting the (few) hit and match records, and formatting the reference's output files.
#include <cuda_runtime.h>

#include <algorithm>
#include <charconv>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <new>
#include <string>
#include <vector>

#include "../../include/ffbf.h"
#include "ffbf_kernels.cuh"
#include "ffbf_scan_fast.cuh"

#include "ffbf_collect.cuh"
#include "ffbf_ctx.cuh"
#include "ffbf_order.cuh"

using ffbf::Geom;
using ffbf::HitLine;
using ffbf::HitRec;

namespace ffbf_host {

ffbf_status fail(ffbf_ctx* c, ffbf_status s, const char* fmt, ...) {
    if (c) {
        char buf[512];
        va_list ap;
        va_start(ap, fmt);
        vsnprintf(buf, sizeof buf, fmt, ap);
        va_end(ap);
        c->err = buf;
    }
    return s;
}


// What an entry point returns when a host allocation throws; the message fits a string without one.
ffbf_status no_host_memory(ffbf_ctx* c) { return fail(c, FFBF_ENOMEM_HOST, "no host memory"); }

ffbf_status dalloc(ffbf_ctx* c, void** p, size_t bytes) {
    *p = nullptr;
    if (bytes == 0) bytes = 16;
    if (c->budget && c->used + bytes > c->budget)
        return fail(c, FFBF_ENOMEM_DEVICE, "device allocation of %zu bytes exceeds the HBM budget (%llu of %llu used)",
                    bytes, (unsigned long long)c->used, (unsigned long long)c->budget);
    cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaSuccess) {
        cudaGetLastError();
        *p = nullptr;
        return fail(c, FFBF_ENOMEM_DEVICE, "cudaMalloc(%zu): %s", bytes, cudaGetErrorString(e));
    }
    c->used += bytes;
    c->allocs[*p] = bytes;
    return FFBF_OK;
}

ffbf_status ensure_tmp(ffbf_ctx* c, size_t words) {
    if (c->tmp_words >= words) return FFBF_OK;
    dfree(c, c->d_tmp);
    c->tmp_words = 0;
    TRY(dalloc_t(c, &c->d_tmp, words));
    c->tmp_words = words;
    return FFBF_OK;
}

// Grows the result-ordering scratch to at least `bytes`.
ffbf_status ensure_order(ffbf_ctx* c, size_t bytes) {
    if (c->order_bytes >= bytes) return FFBF_OK;
    dfree(c, c->d_order);
    c->order_bytes = 0;
    TRY(dalloc_t(c, &c->d_order, bytes));
    c->order_bytes = bytes;
    return FFBF_OK;
}

// Pinned room for `cap` single-launch results. The first kFirstResults come with the context's counters (pinning
// memory costs a call up to a millisecond); a larger result gets the full size once.
constexpr uint32_t kFirstResults = 2048;

ffbf_status ensure_results(ffbf_ctx* c, uint32_t cap) {
    if (c->res_cap >= cap) return FFBF_OK;
    uint8_t* p = nullptr;
    if (cudaMallocHost(&p, ffbf::result_bytes(ffbf::kSmallResults)) != cudaSuccess) {
        cudaGetLastError();
        return fail(c, FFBF_ENOMEM_HOST, "pinned result buffer");
    }
    if (c->h_res_own) cudaFreeHost(c->h_res_own);
    c->h_res = c->h_res_own = p;
    c->res_cap = ffbf::kSmallResults;
    return FFBF_OK;
}

ffbf::ResultHead* result_head(ffbf_ctx* c) { return reinterpret_cast<ffbf::ResultHead*>(c->h_res); }

uint64_t* result_array(ffbf_ctx* c, int i) {
    return reinterpret_cast<uint64_t*>(c->h_res + 64) + (size_t)i * c->res_cap;
}

constexpr uint32_t kUploads = 8;          // blocks of the upload ring, taken in halves
constexpr size_t kUploadBytes = 768;      // zero counters, then a descriptor

// The pinned block for the next upload on the context's stream; nothing that was enqueued earlier still reads it.
ffbf_status upload_block(ffbf_ctx* c, uint8_t** block) {
    cudaStreamCaptureStatus capture;
    CUDA_TRY(c, cudaStreamIsCapturing(c->st, &capture));
    if (capture != cudaStreamCaptureStatusNone) {
        // each replay reads the block again, so no other scan may use it while the context lives
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        CUDA_TRY(c, cudaThreadExchangeStreamCaptureMode(&mode));
        const cudaError_t e = cudaMallocHost(block, kUploadBytes);
        cudaThreadExchangeStreamCaptureMode(&mode);
        if (e != cudaSuccess) {
            cudaGetLastError();
            return fail(c, FFBF_ENOMEM_HOST, "pinned upload block");
        }
        memset(*block, 0, kUploadBytes);
        c->captured_uploads.push_back(*block);
        return FFBF_OK;
    }
    constexpr uint32_t half = kUploads / 2;
    if (c->uploads % half == 0 && c->uploads) {
        // the half just used up is behind this event; the other one, if it was used, is taken again
        cudaEvent_t* ev = c->upload_done;
        const uint32_t used = (c->uploads / half - 1) % 2;
        if (!ev[used]) CUDA_TRY(c, cudaEventCreateWithFlags(&ev[used], cudaEventDisableTiming));
        CUDA_TRY(c, cudaEventRecord(ev[used], c->st));
        if (c->uploads >= kUploads) CUDA_TRY(c, cudaEventSynchronize(ev[1 - used]));
    }
    *block = c->h_uploads + c->uploads++ % kUploads * kUploadBytes;
    return FFBF_OK;
}

// A context's small memory in one allocation each: pinning costs a call one to two milliseconds, a device allocation
// 0.6, whatever its size. Pinned: counters, the upload ring, the first results. Device (behind `front_bytes` of the
// caller's): counters, the job descriptor, the fill counts.
ffbf_status alloc_small(ffbf_ctx* c, size_t front_bytes, uint8_t** front) {
    static_assert(ffbf::CNT_WORDS * sizeof(uint32_t) <= 256 && sizeof(ffbf::FastJob) <= 512 &&
                      ffbf::kJobOffset + sizeof(ffbf::FastJob) <= kUploadBytes,
                  "sections of the blocks");
    constexpr size_t kBeforeResults = 256 + kUploads * kUploadBytes;
    uint8_t *h = nullptr, *d = nullptr;
    TRY(dalloc_t(c, &d, front_bytes + 1024));
    *front = d;
    c->d_counters = reinterpret_cast<uint32_t*>(d + front_bytes);
    c->d_job = reinterpret_cast<ffbf::FastJob*>(d + front_bytes + ffbf::kJobOffset);
    c->d_popc = reinterpret_cast<unsigned long long*>(d + front_bytes + 768);
    if (cudaMallocHost(&h, kBeforeResults + ffbf::result_bytes(kFirstResults)) != cudaSuccess) {
        cudaGetLastError();
        return fail(c, FFBF_ENOMEM_HOST, "pinned context block");
    }
    c->h_counters = reinterpret_cast<uint32_t*>(h);
    c->h_uploads = h + 256;
    memset(c->h_uploads, 0, kUploads * kUploadBytes);  // the counters in each stay zero
    c->h_res = h + kBeforeResults;
    c->res_cap = kFirstResults;
    return FFBF_OK;
}

// Room for cap hit records and their lines, in one allocation.
ffbf_status alloc_hits(ffbf_ctx* c, uint64_t cap) {
    dfree(c, c->d_hits);
    c->d_hitlines = nullptr;
    c->hits_cap = 0;
    uint8_t* d = nullptr;
    TRY(dalloc_t(c, &d, cap * (sizeof(HitRec) + sizeof(HitLine))));
    c->d_hits = reinterpret_cast<HitRec*>(d);
    c->d_hitlines = reinterpret_cast<HitLine*>(d + cap * sizeof(HitRec));
    c->hits_cap = (uint32_t)cap;
    return FFBF_OK;
}

// Room for cap verified matches, in one allocation.
ffbf_status alloc_matches(ffbf_ctx* c, uint64_t cap) {
    dfree(c, c->d_moff);
    c->d_mpid = nullptr;
    c->match_cap = 0;
    uint8_t* d = nullptr;
    TRY(dalloc_t(c, &d, cap * 12));
    c->d_moff = reinterpret_cast<uint64_t*>(d);
    c->d_mpid = reinterpret_cast<uint32_t*>(d + cap * 8);
    c->match_cap = (uint32_t)cap;
    return FFBF_OK;
}

ffbf_status enter(ffbf_ctx* c) {
    if (!c) return FFBF_EINVAL;
    c->err.clear();
    CUDA_TRY(c, cudaSetDevice(c->device));
    return FFBF_OK;
}

ffbf_status sync(ffbf_ctx* c) {
    CUDA_TRY(c, cudaStreamSynchronize(c->st));
    c->uploads = 0;  // every upload has been read
    return FFBF_OK;
}

bool is_pow2(uint64_t x) { return x && !(x & (x - 1)); }

ffbf_status check_params(ffbf_ctx* c, const ffbf_params* p) {
    if (!p) return fail(c, FFBF_EINVAL, "params is NULL");
    if (p->len < 1 || p->len > 63) return fail(c, FFBF_EINVAL, "len must be in 1..63 (got %u)", p->len);
    if (p->k < 1 || p->k > 11) return fail(c, FFBF_EINVAL, "k must be in 1..11 (got %u)", p->k);
    if (p->s > p->k) return fail(c, FFBF_EINVAL, "s must be <= k (got s=%u k=%u)", p->s, p->k);
    if (p->reserved) return fail(c, FFBF_EINVAL, "reserved must be 0");
    if (!is_pow2(p->cache_bits) || !is_pow2(p->ext_bits))
        return fail(c, FFBF_EINVAL, "cache_bits and ext_bits must be powers of two");
    if (p->cache_bits < 32 || p->ext_bits < 32)
        return fail(c, FFBF_EINVAL, "cache_bits and ext_bits must be at least 32");
    if (p->cache_bits + p->ext_bits > (1ull << 31))
        return fail(c, FFBF_EINVAL, "cache_bits + ext_bits must be <= 2^31");
    return FFBF_OK;
}

// The reference prints a line as C strings (cut at the first NUL) and its carry buffer holds only the
// line's part in the previous read() chunk; see ffbf_format_lines in include/ffbf.h.
void put_cstr(std::vector<uint8_t>& out, const uint8_t* s, size_t n) {
    const void* z = memchr(s, 0, n);
    size_t m = z ? (size_t)((const uint8_t*)z - s) : n;
    out.insert(out.end(), s, s + m);
}

void format_line(std::vector<uint8_t>& out, const uint8_t* buf, uint64_t n, uint64_t s, uint64_t e, uint64_t chunk) {
    if (e < n) {
        // line ends with the '\n' at e, read in chunk ce
        uint64_t ce = e / chunk, cs = ce * chunk;
        if (s < cs) {
            uint64_t ps = std::max(s, cs - chunk);
            put_cstr(out, buf + ps, cs - ps);  // carry: the part in chunk ce-1
            put_cstr(out, buf + cs, e - cs);
        } else {
            put_cstr(out, buf + s, e - s);
        }
    } else {
        // final line without '\n': only the carry of the last chunk is printed (ffbf.cpp:385-388)
        uint64_t cl = (n - 1) / chunk, cs = cl * chunk;
        uint64_t ps = std::max(s, cs);
        put_cstr(out, buf + ps, n - ps);
    }
    out.push_back('\n');
}

ffbf_status to_host_buffer(ffbf_ctx* c, const std::vector<uint8_t>& v, uint8_t** out, size_t* out_len) {
    *out = (uint8_t*)malloc(v.size() ? v.size() : 1);
    if (!*out) return fail(c, FFBF_ENOMEM_HOST, "malloc(%zu) failed", v.size());
    if (!v.empty()) memcpy(*out, v.data(), v.size());
    *out_len = v.size();
    return FFBF_OK;
}

void order_hits(const HitRec* hr, const HitLine* hl, uint32_t nh, Words& hits, Words& ls, Words& le) {
    std::vector<uint32_t> order(nh);
    for (uint32_t i = 0; i < nh; i++) order[i] = i;
    std::sort(order.begin(), order.end(), [&](uint32_t a, uint32_t b) { return hr[a].off < hr[b].off; });
    hits.resize(nh);
    ls.clear();
    le.clear();
    for (uint32_t i = 0; i < nh; i++) {
        const uint32_t j = order[i];
        hits[i] = hr[j].off;
        if (ls.empty() || ls.back() != hl[j].start) {
            ls.push_back(hl[j].start);
            le.push_back(hl[j].end);
        }
    }
}

void reset_scan(ffbf_ctx* c) {
    ++*c->scan_no;
    c->have_scan = false;
    c->scan_pending = false;
    c->ready = nullptr;
    c->ready_block.reset();
    c->have_prune = false;
    c->r_hits.clear();
    c->r_ls.clear();
    c->r_le.clear();
    c->r_moff.clear();
    c->r_mpid.clear();
}

const uint64_t kInitialHitsCap = 1u << 16;

// Builds the stage-1 table for a CTA size unless the table on the device already is that one.
ffbf_status ensure_stage1(ffbf_ctx* c, int threads, bool force) {
    if (!force && c->d_stage1 && c->stage1_threads == threads) return FFBF_OK;
    const uint32_t nw = ffbf::stage1_words_for(c->g, threads);
    if (c->d_stage1 && c->stage1_words != nw) dfree(c, c->d_stage1);
    if (!c->d_stage1) TRY(dalloc_t(c, &c->d_stage1, ffbf::table_halves(c->g) ? 2 * nw : nw));
    c->stage1_words = nw;
    c->stage1_threads = threads;
    CUDA_TRY(c, ffbf::build_stage1(c->d_main, c->g, threads, c->d_stage1, c->st));
    return FFBF_OK;
}

// Makes the tuned scan ready for this context's filter: the stage-1 table the configured kernel reads and,
// unless the autotuner or the environment fixed them, the probe mode and the dense mode's probe order (from the
// fills of the stage-1 table and of the filter's regions).
ffbf_status prepare_fast(ffbf_ctx* c) {
    if (c->borrowed) return FFBF_OK;  // the filter's owner built the table and chose the configuration
    if (c->stage1_dirty || !c->d_stage1) {
        TRY(ensure_stage1(c, 384, true));  // the table of mode 3 and of the prefiltered dense kernel
        CUDA_TRY(c, ffbf::popcount_words(c->d_stage1, c->stage1_words, c->d_popc, c->st));
        const uint32_t cw = c->g.cache_bits / 32, ew = (uint32_t)(((uint64_t)c->g.ext_mask + 1) / 32);
        CUDA_TRY(c, ffbf::popcount_words(c->d_main, cw, c->d_popc + 1, c->st));
        CUDA_TRY(c, ffbf::popcount_words(c->d_main + cw, ew, c->d_popc + 2, c->st));
        unsigned long long ones[3] = {0, 0, 0};
        CUDA_TRY(c, cudaMemcpyAsync(ones, c->d_popc, sizeof ones, cudaMemcpyDeviceToHost, c->st));
        TRY(sync(c));
        c->stage1_fill = (double)ones[0] / (32.0 * c->stage1_words);
        const ffbf::ScanChoice best = ffbf::choose_scan(c->g, c->stage1_fill, (double)ones[1] / (32.0 * cw),
                                                        (double)ones[2] / (32.0 * ew));
        c->probe_order = best.order;
        if (!c->cfg_tuned) {
            c->cfg.mode = c->force_mode >= 0 ? c->force_mode : best.mode;
            // default CTA sizes (measured best on the 10k- and 1M-pattern workloads): 512 threads for the
            // shared-memory stage (launch_config fits it to each text), 2 x 192 per SM for dense filters, 384 with their prefilter
            c->cfg.threads = c->threads_env ? c->threads_env : c->cfg.mode == 1 ? 192 : c->cfg.mode == 2 ? 256 : 512;
        }
        c->stage1_dirty = false;
    }
    if (c->force_mode >= 0) c->cfg.mode = c->force_mode;
    if (c->cfg.mode == 3) c->cfg.threads = 512;  // launch_config picks the size for each text
    // the dense mode probes distinct index functions: with K = 1 only the sparse mode applies; with S = 0 no probe
    // falls in the cache region, and only the dense mode without its table does
    if (c->g.k < 2 && c->cfg.mode == 1) c->cfg.mode = 0;
    if (c->g.s < 1 && c->cfg.mode != 1) {
        c->cfg.mode = 1;
        c->cfg.threads = 192;
    }
    // the dense mode's probe order is the filter's, unless the environment fixes it (orders 1 and 3 need f2 and f3)
    c->cfg.order = c->force_order >= 0 ? c->force_order : c->probe_order;
    if (c->g.s < 1 && c->cfg.order >= 2) c->cfg.order = 1;
    if (c->g.k < 4 && c->cfg.order == 1) c->cfg.order = 0;
    if (c->g.k >= 4 && c->cfg.order == 2) c->cfg.order = 3;
    c->cfg.halves = c->cfg.mode == 3 && ffbf::table_halves(c->g);
    // the table the configured kernel reads (a dense kernel without prefilter reads none)
    if (c->cfg.mode != 1 || c->cfg.order >= 2) TRY(ensure_stage1(c, ffbf::table_threads(c->cfg), false));
    return FFBF_OK;
}


ffbf::ScanArgs make_scan_args(ffbf_ctx* c) {
    ffbf::ScanArgs a{};
    a.text = c->d_text;
    a.n = c->text_len;
    a.g = c->g;
    a.main_words = c->d_main;
    a.ff_words = c->d_ff;
    a.hits = c->d_hits;
    a.hits_cap = c->hits_cap;
    a.counters = c->d_counters;
    a.tile_first_nl = c->d_tiles;
    a.tile_last_nl = c->d_tiles + c->tiles_cap;
    a.tile_bytes = c->tile_bytes;
    a.ntiles = scan_tiles(c);
    a.cache_in_smem = c->g.cache_bits <= ffbf::kSmemCacheMaxBits;
    return a;
}

ffbf::CollectJob collect_job(const ffbf::ScanArgs& a, HitLine* lines, uint8_t* res, uint32_t cap, uint32_t per_cta,
                             uint32_t windows) {
    return ffbf::CollectJob{a.text, a.n, a.g.len, a.hits_cap, a.hits, lines, a.counters, a.tile_first_nl, a.tile_last_nl,
                            a.tile_bytes, a.ntiles, reinterpret_cast<ffbf::ResultHead*>(res),
                            reinterpret_cast<uint64_t*>(res + 64), 3ull * cap, nullptr, cap, per_cta,
                            std::max(1u, (std::min(cap, windows) + per_cta - 1) / per_cta)};
}

void take_results(const ffbf::ResultHead* head, const uint64_t* words, Words& hits, Words& ls, Words& le) {
    const uint64_t* a = words + head->at;
    hits.assign(a, a + head->n);
    ls.assign(a + head->n, a + head->n + head->n_lines);
    le.assign(a + 2 * head->n, a + 2 * head->n + head->n_lines);
}

bool tunable(const ffbf_ctx* c, uint64_t n) {
    return use_fast(c, n) && ffbf::compiled_len(c->g.len) && c->g.s >= 1;
}

bool use_fast(const ffbf_ctx* c, uint64_t n) { return ffbf::fast_scan_supported(c->g, n) && !c->force_generic; }

ffbf_status launch_scan(ffbf_ctx* c) {
    const uint64_t n = c->text_len;
    if (n && use_fast(c, n)) {
        c->scan_path = 1;
        TRY(prepare_fast(c));
        const ffbf::FastConfig cfg = ffbf::launch_config(c->cfg, c->g.len, n, c->num_sms, c->as_batch);
        c->tile_bytes = ffbf::fast_tile_bytes(cfg.rows);
        uint8_t* block;
        TRY(upload_block(c, &block));
        CUDA_TRY(c, ffbf::scan_fast(make_scan_args(c), c->d_stage1, cfg, c->num_sms, block, c->st));
    } else {
        CUDA_TRY(c, cudaMemsetAsync(c->d_counters, 0, ffbf::CNT_WORDS * sizeof(uint32_t), c->st));
        if (n == 0) return FFBF_OK;
        c->scan_path = 0;
        c->tile_bytes = ffbf::kScanTile;
        const ffbf::ScanArgs a = make_scan_args(c);
        int grid = ffbf::scan_generic_grid(c->g, a.cache_in_smem, a.ntiles);
        if (grid <= 0) return fail(c, FFBF_ECUDA, "scan kernel cannot be launched (occupancy query failed)");
        CUDA_TRY(c, ffbf::scan_generic(a, grid, c->st));
    }
    return FFBF_OK;
}

// Scan state for a text already on the device, without launching: buffers sized, results reset.
ffbf_status setup_scan_state(ffbf_ctx* c, const uint8_t* d_text, size_t len) {
    if (!d_text && len) return fail(c, FFBF_EINVAL, "text pointer is NULL");
    if (((uintptr_t)d_text & 15) != 0) return fail(c, FFBF_EINVAL, "device text must be 16-byte aligned");
    reset_scan(c);
    if (!c->keep_records) {  // a scan of one device text ends any segmented scan's state
        c->segmented = false;
        c->segs.clear();
        c->seg_hr.clear();
    }
    const uint64_t ntiles = tiles_for(len);
    if (c->tiles_cap < ntiles) {
        dfree(c, c->d_tiles);
        c->tiles_cap = 0;
        // first, last, prev, next per tile, then the two-pass scan's block aggregates
        TRY(dalloc_t(c, &c->d_tiles, 4 * ntiles + 2 * ffbf::tile_agg_words(ntiles)));
        c->tiles_cap = ntiles;
    }
    if (!c->d_hits) TRY(alloc_hits(c, kInitialHitsCap));
    c->d_text = d_text;
    c->text_len = len;
    c->tile_bytes = ffbf::kScanTile;
    return FFBF_OK;
}

// A scan whose kernel raised error flags has no results: some of its windows may not have been tested.
ffbf_status scan_failed(ffbf_ctx* c, uint32_t flags) {
    reset_scan(c);
    return fail(c, flags & 4u ? FFBF_ETIMEOUT : FFBF_ECUDA,
                "scan error flags 0x%x (4: a bounded wait gave up; others: self-checks)", flags);
}

cudaError_t resolve_scan_lines(ffbf_ctx* c, uint32_t nh) {
    if (scan_tiles(c) > c->tiles_cap) return cudaErrorInvalidValue;  // the summaries are of another scan
    return ffbf::resolve_lines(c->d_text, c->text_len, c->g.len, c->d_hits, nh, c->d_tiles, c->d_tiles + c->tiles_cap,
                               c->d_tiles + 2 * c->tiles_cap, c->d_tiles + 3 * c->tiles_cap, c->tile_bytes,
                               scan_tiles(c), c->d_hitlines, c->st, c->d_tiles + 4 * c->tiles_cap);
}

uint64_t tiles_for(uint64_t len) {
    // tiles are 16 KiB or more, but 4 KiB where a small text's scan may use streams of less than four rows
    const uint64_t tile = len < ffbf::kShortRowsText ? 4096 : ffbf::kScanTile;
    return (len + tile - 1) / tile;
}

}  // namespace ffbf_host

using namespace ffbf_host;

extern "C" {

const char* ffbf_status_string(ffbf_status s) {
    switch (s) {
        case FFBF_OK: return "ok";
        case FFBF_EINVAL: return "invalid argument";
        case FFBF_ENOMEM_DEVICE: return "out of device memory";
        case FFBF_EIO: return "i/o error";
        case FFBF_ETIMEOUT: return "device wait timed out";
        case FFBF_ECUDA: return "CUDA error";
        case FFBF_ESTATE: return "call out of order";
        case FFBF_ENOMEM_HOST: return "out of host memory";
    }
    return "unknown status";
}

ffbf_status ffbf_params_default(ffbf_params* p) {
    if (!p) return FFBF_EINVAL;
    p->len = 19;
    p->k = 5;
    p->s = 2;
    p->reserved = 0;
    p->cache_bits = 0x1000000ull;
    p->ext_bits = 0x10000000ull;
    return FFBF_OK;
}

ffbf_status ffbf_create(const ffbf_params* p, int device, ffbf_ctx** out) {
    if (!out) return FFBF_EINVAL;
    *out = nullptr;
    ffbf_ctx* c = new (std::nothrow) ffbf_ctx();
    if (!c) return FFBF_ENOMEM_HOST;
    ffbf_status s = check_params(c, p);
    if (s != FFBF_OK) {
        delete c;
        return s;
    }
    int ndev = 0;
    cudaError_t e = cudaGetDeviceCount(&ndev);
    if (e != cudaSuccess || device < 0 || device >= ndev) {
        cudaGetLastError();
        delete c;
        return FFBF_ECUDA;
    }
    c->prm = *p;
    c->device = device;
    c->g.len = p->len;
    c->g.k = p->k;
    c->g.s = p->s;
    c->g.cache_bits = (uint32_t)p->cache_bits;
    c->g.cache_mask = (uint32_t)(p->cache_bits - 1);
    c->g.ext_mask = (uint32_t)(p->ext_bits - 1);
    c->g.nbits = (uint32_t)(p->cache_bits + p->ext_bits);
    c->filter_bytes = (p->cache_bits + p->ext_bits) / 8;
    auto bail = [&](ffbf_status st) {
        ffbf_destroy(c);
        return st;
    };
    if ((e = cudaSetDevice(device)) != cudaSuccess || (e = cudaStreamCreateWithFlags(&c->st, cudaStreamNonBlocking)) != cudaSuccess ||
        (e = cudaDeviceGetAttribute(&c->num_sms, cudaDevAttrMultiProcessorCount, device)) != cudaSuccess) {
        cudaGetLastError();
        return bail(FFBF_ECUDA);
    }
    {
        size_t fr = 0, tot = 0;
        if (cudaMemGetInfo(&fr, &tot) != cudaSuccess) {
            cudaGetLastError();
            return bail(FFBF_ECUDA);
        }
        c->device_mem = tot;
    }
    const size_t room = (c->filter_bytes + 255) / 256 * 256;
    uint8_t* filters = nullptr;
    if ((s = alloc_small(c, 2 * room, &filters)) != FFBF_OK) return bail(s);
    c->d_main = reinterpret_cast<uint32_t*>(filters);
    c->d_ff = reinterpret_cast<uint32_t*>(filters + room);
    if (cudaMemsetAsync(filters, 0, 2 * room, c->st) != cudaSuccess ||
        cudaStreamSynchronize(c->st) != cudaSuccess) {
        cudaGetLastError();
        return bail(FFBF_ECUDA);
    }
    const char* th = getenv("FFBF_SCAN_THREADS");
    if (th && (atoi(th) == 192 || atoi(th) == 256 || atoi(th) == 384 || atoi(th) == 512))
        c->cfg.threads = c->threads_env = atoi(th);
    const char* fm = getenv("FFBF_SCAN_MODE");
    if (fm && fm[0] >= '0' && fm[0] <= '3') c->force_mode = fm[0] - '0';
    const char* fo = getenv("FFBF_SCAN_ORDER");
    if (fo && fo[0] >= '0' && fo[0] <= '2') c->force_order = fo[0] - '0';
    const char* fg = getenv("FFBF_FORCE_GENERIC_SCAN");
    c->force_generic = fg && fg[0] == '1';
    const char* ho = getenv("FFBF_HOST_ORDER");
    c->host_order = ho && ho[0] == '1';
    *out = c;
    return FFBF_OK;
}

}  // extern "C"

namespace ffbf_host {

ffbf_status create_scan_slot(int device, ffbf_ctx** out) {
    *out = nullptr;
    ffbf_ctx* c = new (std::nothrow) ffbf_ctx();
    if (!c) return FFBF_ENOMEM_HOST;
    c->device = device;
    c->borrowed = true;
    if (cudaSetDevice(device) != cudaSuccess || cudaStreamCreateWithFlags(&c->st, cudaStreamNonBlocking) != cudaSuccess ||
        cudaDeviceGetAttribute(&c->num_sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) {
        cudaGetLastError();
        ffbf_destroy(c);
        return FFBF_ECUDA;
    }
    uint8_t* none = nullptr;
    const ffbf_status st = alloc_small(c, 0, &none);
    if (st != FFBF_OK) {
        ffbf_destroy(c);
        return st;
    }
    *out = c;
    return FFBF_OK;
}

void attach_filters(ffbf_ctx* slot, const ffbf_ctx* owner) {
    slot->prm = owner->prm;
    slot->g = owner->g;
    slot->filter_bytes = owner->filter_bytes;
    slot->d_main = owner->d_main;
    slot->d_ff = owner->d_ff;
    slot->d_stage1 = owner->d_stage1;
    slot->stage1_threads = owner->stage1_threads;
    slot->stage1_words = owner->stage1_words;
    slot->stage1_fill = owner->stage1_fill;
    slot->stage1_dirty = false;
    slot->cfg = owner->cfg;
    slot->cfg_tuned = true;
    slot->force_mode = owner->force_mode;
    slot->force_generic = owner->force_generic;
}

}  // namespace ffbf_host

extern "C" {

void ffbf_destroy(ffbf_ctx* c) {
    if (!c) return;
    cudaSetDevice(c->device);
    if (c->st) cudaStreamSynchronize(c->st);
    ++*c->scan_no;
    for (auto& kv : c->allocs) cudaFree(kv.first);
    c->allocs.clear();
    if (c->h_counters) cudaFreeHost(c->h_counters);
    for (void* p : c->captured_uploads) cudaFreeHost(p);
    for (cudaEvent_t ev : c->upload_done)
        if (ev) cudaEventDestroy(ev);
    if (c->h_res_own) cudaFreeHost(c->h_res_own);
    if (c->h_jobs) cudaFreeHost(c->h_jobs);
    for (auto ev : c->pipe_events) cudaEventDestroy(ev);
    if (c->st_copy) {
        cudaStreamSynchronize(c->st_copy);
        cudaStreamDestroy(c->st_copy);
    }
    if (c->st) cudaStreamDestroy(c->st);
    cudaGetLastError();
    delete c;
}

const char* ffbf_last_error(const ffbf_ctx* c) { return c ? c->err.c_str() : "null context"; }

uint64_t ffbf_filter_bytes(const ffbf_ctx* c) { return c ? c->filter_bytes : 0; }

void ffbf_free(void* p) { free(p); }

void* ffbf_host_alloc(size_t bytes) {
    void* p = nullptr;
    if (cudaMallocHost(&p, bytes ? bytes : 1) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return p;
}

void ffbf_host_free(void* p) {
    if (p) cudaFreeHost(p);
}

void* ffbf_stream(ffbf_ctx* c) { return c ? (void*)c->st : nullptr; }

uint64_t ffbf_kernel_launches(void) { return ffbf::launches_total(); }

ffbf_status ffbf_set_hbm_budget(ffbf_ctx* c, uint64_t bytes) {
    if (!c) return FFBF_EINVAL;
    c->budget = bytes;
    return FFBF_OK;
}

}  // extern "C"

namespace {

// Copies a pattern file to the device, finds its lines and hashes their prefixes; with set_bits the hash pass also sets
// the main filter's bits.
ffbf_status set_patterns(ffbf_ctx* c, const uint8_t* file, size_t len, int set_bits) {
    TRY(enter(c));
    if (!file && len) return fail(c, FFBF_EINVAL, "pattern buffer is NULL");
    c->have_patterns = false;
    c->have_prune = false;
    dfree(c, c->d_pat);
    dfree(c, c->d_pstart);
    c->d_pend = c->d_phash = nullptr;
    c->npat = 0;
    c->pat_len = len;
    c->h_pat = {};
    TRY(dalloc_t(c, &c->d_pat, len + 16));
    if (len) CUDA_TRY(c, cudaMemcpyAsync(c->d_pat, file, len, cudaMemcpyHostToDevice, c->st));
    const uint64_t nb = ffbf::compact_blocks(len);
    TRY(ensure_tmp(c, nb + 1));
    CUDA_TRY(c, ffbf::count_bytes(c->d_pat, len, '\n', c->d_tmp, c->st));
    uint64_t m = 0;
    CUDA_TRY(c, cudaMemcpyAsync(&m, c->d_tmp + nb, sizeof m, cudaMemcpyDeviceToHost, c->st));
    TRY(sync(c));
    const int tail = len > 0 && file[len - 1] != '\n';
    const uint64_t npat = m + (tail ? 1 : 0);
    // one allocation for starts, ends and hashes; the newline positions use the hashes' room until those are written
    TRY(dalloc_t(c, &c->d_pstart, 3 * (npat + 1)));
    c->d_pend = c->d_pstart + (npat + 1);
    c->d_phash = c->d_pend + (npat + 1);
    if (ffbf::emit_bytes(c->d_pat, len, '\n', c->d_phash, c->d_tmp, c->st) != cudaSuccess ||
        ffbf::lines_from_newlines(c->d_phash, m, len, tail, c->d_pstart, c->d_pend, c->st) != cudaSuccess ||
        ffbf::hash_patterns(c->d_pat, c->d_pstart, c->d_pend, npat, c->g, c->d_phash, c->d_main, set_bits, c->st) !=
            cudaSuccess)
        return fail(c, FFBF_ECUDA, "pattern hashing failed: %s", cudaGetErrorString(cudaGetLastError()));
    if (set_bits) c->stage1_dirty = true;
    TRY(sync(c));
    c->npat = npat;
    c->have_patterns = true;
    return FFBF_OK;
}

}  // namespace

extern "C" {

ffbf_status ffbf_set_patterns(ffbf_ctx* c, const uint8_t* file, size_t len) { return set_patterns(c, file, len, 0); }

ffbf_status ffbf_build(ffbf_ctx* c) {
    NvtxRange nvtx_("ffbf_build");
    TRY(enter(c));
    if (!c->have_patterns) return fail(c, FFBF_ESTATE, "ffbf_build needs ffbf_set_patterns first");
    CUDA_TRY(c, ffbf::hash_patterns(c->d_pat, c->d_pstart, c->d_pend, c->npat, c->g, c->d_phash, c->d_main, 1, c->st));
    c->stage1_dirty = true;
    return sync(c);
}

ffbf_status ffbf_add_patterns(ffbf_ctx* c, const uint8_t* file, size_t len) {
    return set_patterns(c, file, len, 1);
}

ffbf_status ffbf_load_filter(ffbf_ctx* c, const uint8_t* data, size_t len) {
    TRY(enter(c));
    if (!data && len) return fail(c, FFBF_EINVAL, "filter buffer is NULL");
    const uint64_t nd = len / 4;
    if (!nd) return FFBF_OK;
    uint32_t *d_d = nullptr, *d_idx = nullptr;
    TRY(dalloc_t(c, &d_d, nd));
    ffbf_status s = dalloc_t(c, &d_idx, nd);
    if (s == FFBF_OK) s = ensure_tmp(c, ffbf::decode_blocks(nd) + 1);
    if (s == FFBF_OK) {
        uint32_t err = 0;
        if (cudaMemcpyAsync(d_d, data, nd * 4, cudaMemcpyHostToDevice, c->st) != cudaSuccess ||
            cudaMemsetAsync(c->d_counters, 0, ffbf::CNT_WORDS * 4, c->st) != cudaSuccess ||
            ffbf::filter_decode(d_d, nd, c->g.nbits, d_idx, c->d_tmp, c->d_counters, c->st) != cudaSuccess ||
            cudaMemcpyAsync(&err, c->d_counters + ffbf::CNT_ERROR, 4, cudaMemcpyDeviceToHost, c->st) != cudaSuccess ||
            cudaStreamSynchronize(c->st) != cudaSuccess) {
            s = fail(c, FFBF_ECUDA, "filter decode failed: %s", cudaGetErrorString(cudaGetLastError()));
        } else if (err) {
            s = fail(c, FFBF_EINVAL, "filter file holds a bit index at or beyond N = %u", c->g.nbits);
        } else if ((c->stage1_dirty = true, ffbf::filter_set_indices(d_idx, nd, c->d_main, c->st) != cudaSuccess) ||
                   cudaStreamSynchronize(c->st) != cudaSuccess) {
            s = fail(c, FFBF_ECUDA, "filter load failed: %s", cudaGetErrorString(cudaGetLastError()));
        }
    }
    dfree(c, d_d);
    dfree(c, d_idx);
    return s;
}

ffbf_status ffbf_save_filter(ffbf_ctx* c, uint8_t** data, size_t* len) {
    TRY(enter(c));
    if (!data || !len) return fail(c, FFBF_EINVAL, "NULL output pointer");
    *data = nullptr;
    *len = 0;
    const uint32_t nwords = c->g.nbits / 32;
    const uint64_t nb = ffbf::enc_blocks(nwords);
    TRY(ensure_tmp(c, nb + 1));
    CUDA_TRY(c, ffbf::filter_count(c->d_main, nwords, c->d_tmp, c->st));
    uint64_t total = 0;
    CUDA_TRY(c, cudaMemcpyAsync(&total, c->d_tmp + nb, 8, cudaMemcpyDeviceToHost, c->st));
    TRY(sync(c));
    uint8_t* h = (uint8_t*)malloc(total * 4 + 1);
    if (!h) return fail(c, FFBF_ENOMEM_HOST, "malloc(%llu) failed", (unsigned long long)(total * 4));
    if (total) {
        uint32_t *d_idx = nullptr, *d_del = nullptr;
        ffbf_status s = dalloc_t(c, &d_idx, total);
        if (s == FFBF_OK) s = dalloc_t(c, &d_del, total);
        if (s == FFBF_OK && (ffbf::filter_encode(c->d_main, nwords, c->d_tmp, d_idx, c->st) != cudaSuccess ||
                             ffbf::filter_deltas(d_idx, total, d_del, c->st) != cudaSuccess ||
                             cudaMemcpyAsync(h, d_del, total * 4, cudaMemcpyDeviceToHost, c->st) != cudaSuccess ||
                             cudaStreamSynchronize(c->st) != cudaSuccess))
            s = fail(c, FFBF_ECUDA, "filter encode failed: %s", cudaGetErrorString(cudaGetLastError()));
        dfree(c, d_idx);
        dfree(c, d_del);
        if (s != FFBF_OK) {
            free(h);
            return s;
        }
    }
    *data = h;
    *len = total * 4;
    return FFBF_OK;
}

ffbf_status ffbf_load_filter_file(ffbf_ctx* c, const char* path) try {
    if (!c) return FFBF_EINVAL;
    if (!path) return fail(c, FFBF_EINVAL, "path is NULL");
    std::unique_ptr<FILE, int (*)(FILE*)> f(fopen(path, "rb"), fclose);
    if (!f) return fail(c, FFBF_EIO, "cannot open %s", path);
    std::vector<uint8_t> buf;
    uint8_t tmp[1 << 16];
    size_t r;
    while ((r = fread(tmp, 1, sizeof tmp, f.get())) > 0) buf.insert(buf.end(), tmp, tmp + r);
    const bool bad = ferror(f.get());
    f.reset();
    if (bad) return fail(c, FFBF_EIO, "error while reading the filter file %s", path);
    return ffbf_load_filter(c, buf.data(), buf.size());
} catch (...) {
    return no_host_memory(c);
}

ffbf_status ffbf_save_filter_file(ffbf_ctx* c, const char* path) {
    if (!c) return FFBF_EINVAL;
    if (!path) return fail(c, FFBF_EINVAL, "path is NULL");
    uint8_t* data = nullptr;
    size_t len = 0;
    TRY(ffbf_save_filter(c, &data, &len));
    FILE* f = fopen(path, "wb");
    if (!f) {
        ffbf_free(data);
        return fail(c, FFBF_EIO, "cannot create %s", path);
    }
    bool ok = fwrite(data, 1, len, f) == len;
    ok = (fclose(f) == 0) && ok;
    ffbf_free(data);
    if (!ok) return fail(c, FFBF_EIO, "error while writing to the filter file %s", path);
    return FFBF_OK;
}

ffbf_status ffbf_scan_device(ffbf_ctx* c, const uint8_t* d_text, size_t len) try {
    NvtxRange nvtx_("ffbf_scan_device");
    TRY(enter(c));
    TRY(setup_scan_state(c, d_text, len));
    TRY(launch_scan(c));
    c->scan_pending = true;
    return FFBF_OK;
} catch (...) {
    return no_host_memory(c);
}

ffbf_status ffbf_scan_collect(ffbf_ctx* c, ffbf_scan_result* out) try {
    NvtxRange nvtx_("ffbf_scan_collect");
    TRY(enter(c));
    if (!c->scan_pending && !c->have_scan) return fail(c, FFBF_ESTATE, "no scan to collect");
    if (c->scan_pending && !c->host_order && !c->keep_records) {
        // one launch finishes a result of up to kSmallResults windows, unless the scan's batch has done it already;
        // the general path below takes the others
        const ffbf::ResultHead* head = c->ready;
        const uint64_t* words = c->ready_words;
        const bool collected = head && (head->done || head->error || head->n > ffbf::kSmallResults);
        for (int attempt = 0; !collected && attempt < 2; attempt++) {
            const uint32_t cap = c->res_cap;
            head = result_head(c);
            words = result_array(c, 0);
            CUDA_TRY(c, ffbf::collect_hits(collect_job(make_scan_args(c), c->d_hitlines, c->h_res, cap,
                                                       ffbf::kCollectAlone, cap),
                                           c->st));
            TRY(sync(c));
            if (head->n <= cap || head->n > ffbf::kSmallResults || head->n > c->hits_cap) break;
            TRY(ensure_results(c, ffbf::kSmallResults));
        }
        if (head->error) return scan_failed(c, (uint32_t)head->error);
        if (head->done) {
            c->nhits = (uint32_t)head->n;
            take_results(head, words, c->r_hits, c->r_ls, c->r_le);
            c->ready = nullptr;
            c->ready_block.reset();
            c->scan_pending = false;
            c->have_scan = true;
        }
    }
    if (c->scan_pending) {
        CUDA_TRY(c, cudaMemcpyAsync(c->h_counters, c->d_counters, ffbf::CNT_WORDS * 4, cudaMemcpyDeviceToHost, c->st));
        TRY(sync(c));
        if (c->h_counters[ffbf::CNT_ERROR]) return scan_failed(c, c->h_counters[ffbf::CNT_ERROR]);
        uint32_t nh = c->h_counters[ffbf::CNT_HITS];
        if (nh > c->hits_cap) {
            // Too many hits for the buffer: grow it and scan again. Setting feed-forward bits is
            // idempotent, so the second pass leaves the same filter.
            uint64_t cap = (uint64_t)nh + nh / 4 + 1024;
            if (cap > 0xffffffffull) return fail(c, FFBF_EINVAL, "more than 2^32 hit windows in one scan");
            TRY(alloc_hits(c, cap));
            TRY(launch_scan(c));
            CUDA_TRY(c, cudaMemcpyAsync(c->h_counters, c->d_counters, ffbf::CNT_WORDS * 4, cudaMemcpyDeviceToHost, c->st));
            TRY(sync(c));
            if (c->h_counters[ffbf::CNT_ERROR]) return scan_failed(c, c->h_counters[ffbf::CNT_ERROR]);
            nh = c->h_counters[ffbf::CNT_HITS];
        }
        c->nhits = nh;
        CUDA_TRY(c, resolve_scan_lines(c, nh));
        // Text order on the device: sorted window starts, then the distinct lines of the sorted windows. When
        // the device has no room for the sort's scratch (about 60 bytes per hit window), or FFBF_HOST_ORDER is
        // set, the records are ordered on the host instead; the results are the same.
        const int kb = ffbf::key_bits_for(c->text_len);
        const size_t scratch = ffbf::order_hits_scratch(nh, kb);
        const size_t off_bytes = ((size_t)nh * 8 + 255) / 256 * 256, line_bytes = ((size_t)nh * 16 + 255) / 256 * 256;
        const bool on_device = !c->host_order && ensure_order(c, off_bytes + line_bytes + 256 + scratch) == FFBF_OK;
        if (!on_device) c->err.clear();
        std::vector<HitRec> hr;
        if (nh && (c->keep_records || !on_device)) {
            hr.resize(nh);
            CUDA_TRY(c, cudaMemcpyAsync(hr.data(), c->d_hits, nh * sizeof(HitRec), cudaMemcpyDeviceToHost, c->st));
            TRY(sync(c));
        }
        if (c->keep_records)  // a segment of a larger text: ffbf_verify needs its records again
            for (uint32_t i = 0; i < nh; i++) c->seg_hr.push_back(HitRec{hr[i].off + c->seg_base, hr[i].h});
        if (!on_device) {
            std::vector<HitLine> hl(nh);
            if (nh)
                CUDA_TRY(c, cudaMemcpyAsync(hl.data(), c->d_hitlines, nh * sizeof(HitLine), cudaMemcpyDeviceToHost,
                                            c->st));
            TRY(sync(c));
            order_hits(hr.data(), hl.data(), nh, c->r_hits, c->r_ls, c->r_le);
        } else {
            uint64_t* d_off = reinterpret_cast<uint64_t*>(c->d_order);
            HitLine* d_lu = reinterpret_cast<HitLine*>(c->d_order + off_bytes);
            uint64_t* d_nl = reinterpret_cast<uint64_t*>(c->d_order + off_bytes + line_bytes);
            uint64_t *d_ls, *d_le;
            CUDA_TRY(c, ffbf::order_hits(c->d_hits, c->d_hitlines, nh, kb, c->d_order + off_bytes + line_bytes + 256,
                                         scratch, d_off, d_lu, &d_ls, &d_le, d_nl, c->st));
            uint64_t n_lines = 0;
            c->r_hits.resize(nh);
            CUDA_TRY(c, cudaMemcpyAsync(&n_lines, d_nl, 8, cudaMemcpyDeviceToHost, c->st));
            if (nh)
                CUDA_TRY(c, cudaMemcpyAsync(c->r_hits.data(), d_off, nh * 8ull, cudaMemcpyDeviceToHost, c->st));
            TRY(sync(c));
            if (n_lines > nh) return fail(c, FFBF_ECUDA, "line reduction returned %llu lines for %u hits",
                                          (unsigned long long)n_lines, nh);
            c->r_ls.resize(n_lines);
            c->r_le.resize(n_lines);
            if (n_lines) {
                CUDA_TRY(c, cudaMemcpyAsync(c->r_ls.data(), d_ls, n_lines * 8, cudaMemcpyDeviceToHost, c->st));
                CUDA_TRY(c, cudaMemcpyAsync(c->r_le.data(), d_le, n_lines * 8, cudaMemcpyDeviceToHost, c->st));
                TRY(sync(c));
            }
        }
        c->scan_pending = false;
        c->have_scan = true;
    }
    if (out) {
        out->text_len = c->text_len;
        out->n_hits = c->r_hits.size();
        out->hit_offsets = c->r_hits.data();
        out->n_lines = c->r_ls.size();
        out->line_start = c->r_ls.data();
        out->line_end = c->r_le.data();
    }
    return FFBF_OK;
} catch (...) {
    return no_host_memory(c);
}

}  // extern "C"

namespace {

// Host texts of kPipeMinText bytes or more are copied in chunks that the scan follows; a chunk is about an
// eighth of the text, between 8 and 128 MiB.
constexpr uint64_t kPipeMinText = 32ull << 20;
constexpr uint64_t kPipeChunkMin = 8ull << 20, kPipeChunkMax = 128ull << 20;

uint64_t pipe_chunk(uint64_t len) {
    return std::min(kPipeChunkMax, std::max(kPipeChunkMin, len / 8 >> 20 << 20));
}

// The scan of a host text whose copy to the device overlaps the scan: the text goes over in chunks of
// about pipe_chunk(len) bytes on the context's copy stream, and after each chunk the tuned kernel runs over
// the work items whose bytes (and halos) have landed. The rows per stream suit one chunk, whose launch
// then spreads over the SMs and ends soon after its copy; the copy is the bound. Every chunk's launch uses
// the whole text's tensor map and absolute positions; its descriptor only shifts the item numbering
// (item_begin = -first item).
ffbf_status scan_host_pipelined(ffbf_ctx* c, const uint8_t* text, size_t len) {
    TRY(setup_scan_state(c, c->d_text_own, len));
    CUDA_TRY(c, cudaMemsetAsync(c->d_counters, 0, ffbf::CNT_WORDS * sizeof(uint32_t), c->st));
    TRY(prepare_fast(c));
    c->scan_path = 1;
    const uint64_t chunk = pipe_chunk(len);
    ffbf::FastConfig cfg = ffbf::launch_config(c->cfg, c->g.len, chunk, c->num_sms, false);
    if (len >= ffbf::kShortRowsText && cfg.rows < 4) cfg.rows = 4;
    c->tile_bytes = ffbf::fast_tile_bytes(cfg.rows);
    ffbf::FastJob job;
    CUDA_TRY(c, ffbf::fill_fast_job(make_scan_args(c), c->d_stage1, cfg, &job));
    const uint64_t item_bytes = (uint64_t)ffbf::config_threads(cfg) * cfg.rows * 128;
    const uint32_t per_chunk = (uint32_t)std::max<uint64_t>(1, chunk / item_bytes);
    const uint32_t n_chunks = (job.n_supertiles + per_chunk - 1) / per_chunk;
    if (!c->st_copy) CUDA_TRY(c, cudaStreamCreateWithFlags(&c->st_copy, cudaStreamNonBlocking));
    while (c->pipe_events.size() < (size_t)n_chunks + 1) {
        cudaEvent_t ev;
        CUDA_TRY(c, cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
        c->pipe_events.push_back(ev);
    }
    if (c->jobs_cap < n_chunks) {
        TRY(sync(c));  // the old staging may still feed a copy
        if (c->h_jobs) cudaFreeHost(c->h_jobs);
        c->h_jobs = nullptr;
        dfree(c, c->d_jobs);
        c->jobs_cap = 0;
        if (cudaMallocHost(&c->h_jobs, n_chunks * sizeof(ffbf::FastJob)) != cudaSuccess) {
            cudaGetLastError();
            c->h_jobs = nullptr;
            return fail(c, FFBF_ENOMEM_HOST, "pinned chunk descriptors");
        }
        TRY(dalloc_t(c, &c->d_jobs, n_chunks));
        c->jobs_cap = n_chunks;
    }
    TRY(sync(c));  // the staging array is rewritten below; earlier uploads must be done
    for (uint32_t i = 0; i < n_chunks; i++) {
        c->h_jobs[i] = job;
        c->h_jobs[i].item_begin = 0u - i * per_chunk;  // item k of chunk i is supertile i * per_chunk + k
    }
    CUDA_TRY(c, cudaMemcpyAsync(c->d_jobs, c->h_jobs, n_chunks * sizeof(ffbf::FastJob), cudaMemcpyHostToDevice,
                                c->st));
    // the copies overwrite the text buffer: start them after what the context's stream already holds
    CUDA_TRY(c, cudaEventRecord(c->pipe_events[n_chunks], c->st));
    CUDA_TRY(c, cudaStreamWaitEvent(c->st_copy, c->pipe_events[n_chunks], 0));
    uint64_t copied = 0;
    for (uint32_t i = 0; i < n_chunks; i++) {
        const uint32_t first = i * per_chunk;
        const uint32_t count = std::min(per_chunk, job.n_supertiles - first);
        // the last item's launch also scans the bytes after the last whole stream
        const uint64_t end = i + 1 == n_chunks ? len : std::min<uint64_t>(len, (uint64_t)(first + count) * item_bytes);
        CUDA_TRY(c, cudaMemcpyAsync(c->d_text_own + copied, text + copied, end - copied, cudaMemcpyHostToDevice,
                                    c->st_copy));
        copied = end;
        CUDA_TRY(c, cudaEventRecord(c->pipe_events[i], c->st_copy));
        CUDA_TRY(c, cudaStreamWaitEvent(c->st, c->pipe_events[i], 0));
        CUDA_TRY(c, cudaMemsetAsync(c->d_counters + ffbf::CNT_QUEUE, 0, sizeof(uint32_t), c->st));
        CUDA_TRY(c, ffbf::launch_fast_jobs(c->g.len, cfg, c->d_jobs + i, 1, count, job.stage1_nwords,
                                           c->d_counters + ffbf::CNT_ERROR, c->num_sms, c->st));
    }
    return FFBF_OK;
}

// One host text that fits the device: copied (overlapped with the scan when large) and scanned.
ffbf_status scan_one(ffbf_ctx* c, const uint8_t* text, size_t len, ffbf_scan_result* out) {
    if (c->text_cap < len + 64) {
        dfree(c, c->d_text_own);
        c->text_cap = 0;
        TRY(dalloc_t(c, &c->d_text_own, len + 64));
        c->text_cap = len + 64;
    }
    if (len >= kPipeMinText && use_fast(c, len)) {
        TRY(scan_host_pipelined(c, text, len));
        c->scan_pending = true;
        return ffbf_scan_collect(c, out);
    }
    if (len) CUDA_TRY(c, cudaMemcpyAsync(c->d_text_own, text, len, cudaMemcpyHostToDevice, c->st));
    TRY(ffbf_scan_device(c, c->d_text_own, len));
    return ffbf_scan_collect(c, out);
}

// Device bytes a scan of `len` text bytes needs beyond what the context holds: the text buffer, the tile
// summaries and, the first time, the hit buffers.
uint64_t scan_need(const ffbf_ctx* c, uint64_t len) {
    const uint64_t ntiles = tiles_for(len);
    uint64_t need = len + 64 + 8 * (4 * ntiles + 2 * ffbf::tile_agg_words(ntiles));
    if (!c->d_hits) need += 2 * kInitialHitsCap * 16;
    return need;
}

// The largest segment a scan may put on the device: what the HBM budget (or the device's free memory, less
// 1 GiB) leaves after everything but the text buffer, three quarters of it; 0 when the whole text fits.
ffbf_status segment_size(ffbf_ctx* c, uint64_t len, uint64_t* seg) {
    *seg = 0;
    uint64_t avail;
    if (c->budget) {
        avail = c->budget > c->used ? c->budget - c->used : 0;
    } else {
        // asking the driver for free memory costs about a millisecond: only texts of a quarter of the
        // device or more can fail to fit, so smaller ones skip the query
        if (scan_need(c, len) < c->device_mem / 4) return FFBF_OK;
        size_t fr = 0, tot = 0;
        CUDA_TRY(c, cudaMemGetInfo(&fr, &tot));
        avail = fr > (1ull << 30) ? fr - (1ull << 30) : 0;
    }
    avail += c->text_cap;  // the current text buffer is given back first
    if (scan_need(c, len) <= avail) return FFBF_OK;
    *seg = avail / 4 * 3 / 65536 * 65536;
    if (*seg < (1u << 20)) return fail(c, FFBF_ENOMEM_DEVICE, "no room on the device for a 1 MiB text segment");
    return FFBF_OK;
}

}  // namespace

extern "C" {

ffbf_status ffbf_scan(ffbf_ctx* c, const uint8_t* text, size_t len, ffbf_scan_result* out) try {
    NvtxRange nvtx_("ffbf_scan");
    TRY(enter(c));
    if (!text && len) return fail(c, FFBF_EINVAL, "text is NULL");
    c->segmented = false;
    c->keep_records = false;
    c->segs.clear();
    c->seg_hr.clear();
    uint64_t seg = 0;
    TRY(segment_size(c, len, &seg));
    if (seg == 0) return scan_one(c, text, len, out);
    // A text larger than the device holds: scan it in segments that end just after a '\n'. A valid window
    // never spans a '\n', so the segments' scans are independent; their results are offset and joined, and
    // the feed-forward filter accumulates over them as over successive scans.
    dfree(c, c->d_text_own);
    c->text_cap = 0;
    Words hits, ls, le;
    c->keep_records = true;
    for (uint64_t pos = 0; pos < len;) {
        uint64_t end = std::min<uint64_t>(len, pos + seg);
        if (end < len) {
            const void* nl = memrchr(text + pos, '\n', end - pos);
            if (!nl) {
                c->keep_records = false;
                return fail(c, FFBF_EINVAL, "a line longer than the device's text segment (%llu bytes) at offset %llu",
                            (unsigned long long)seg, (unsigned long long)pos);
            }
            end = (uint64_t)((const uint8_t*)nl - text) + 1;
        }
        c->seg_base = pos;
        c->segs.push_back({pos, end - pos, (uint64_t)c->seg_hr.size(), 0});
        ffbf_scan_result r{};
        ffbf_status st = scan_one(c, text + pos, end - pos, &r);
        if (st != FFBF_OK) {
            c->keep_records = false;
            return st;
        }
        c->segs.back().hr_end = c->seg_hr.size();
        for (uint64_t i = 0; i < r.n_hits; i++) hits.push_back(r.hit_offsets[i] + pos);
        for (uint64_t i = 0; i < r.n_lines; i++) {
            ls.push_back(r.line_start[i] + pos);
            le.push_back(r.line_end[i] + pos);
        }
        pos = end;
    }
    c->keep_records = false;
    c->segmented = true;
    c->seg_text = text;
    c->r_hits.swap(hits);
    c->r_ls.swap(ls);
    c->r_le.swap(le);
    c->nhits = (uint32_t)c->r_hits.size();
    c->text_len = len;
    c->have_scan = true;
    c->scan_pending = false;
    if (out) {
        out->text_len = len;
        out->n_hits = c->r_hits.size();
        out->hit_offsets = c->r_hits.data();
        out->n_lines = c->r_ls.size();
        out->line_start = c->r_ls.data();
        out->line_end = c->r_le.data();
    }
    return FFBF_OK;
} catch (...) {
    c->keep_records = false;
    return no_host_memory(c);
}

ffbf_status ffbf_format_lines(ffbf_ctx* c, const uint8_t* text, size_t len, size_t chunk, uint8_t** out,
                              size_t* out_len) try {
    if (!c) return FFBF_EINVAL;
    if (!out || !out_len || (!text && len)) return fail(c, FFBF_EINVAL, "NULL argument");
    if (!c->have_scan) return fail(c, FFBF_ESTATE, "ffbf_format_lines needs a collected scan");
    if (len != c->text_len) return fail(c, FFBF_EINVAL, "text length differs from the scanned text");
    if (chunk == 0) return fail(c, FFBF_EINVAL, "chunk must be > 0");
    std::vector<uint8_t> v;
    for (size_t i = 0; i < c->r_ls.size(); i++) format_line(v, text, len, c->r_ls[i], c->r_le[i], chunk);
    return to_host_buffer(c, v, out, out_len);
} catch (...) {
    return no_host_memory(c);
}

ffbf_status ffbf_format_spans(const uint8_t* buf, size_t len, const uint64_t* start, const uint64_t* end, size_t n,
                              size_t chunk, uint8_t** out, size_t* out_len) {
    if (!out || !out_len || (!buf && len) || (n && (!start || !end)) || chunk == 0) return FFBF_EINVAL;
    *out = nullptr;
    *out_len = 0;
    for (size_t i = 0; i < n; i++)
        if (start[i] > end[i] || end[i] > len || (i && start[i] <= end[i - 1]))
            return FFBF_EINVAL;
    std::vector<uint8_t> v;
    try {
        for (size_t i = 0; i < n; i++) format_line(v, buf, len, start[i], end[i], chunk);
    } catch (...) {
        return FFBF_ENOMEM_HOST;
    }
    return to_host_buffer(nullptr, v, out, out_len);
}

ffbf_status ffbf_prune(ffbf_ctx* c, ffbf_prune_result* out) try {
    NvtxRange nvtx_("ffbf_prune");
    TRY(enter(c));
    if (!c->have_patterns) return fail(c, FFBF_ESTATE, "ffbf_prune needs ffbf_set_patterns first");
    if (c->scan_pending) TRY(ffbf_scan_collect(c, nullptr));
    const uint64_t n = c->npat;
    uint64_t cnt = 0;
    c->have_prune = false;
    if (n) {
        TRY(ensure_tmp(c, ffbf::prune_blocks(n)));
        uint32_t* counts = reinterpret_cast<uint32_t*>(c->d_tmp);
        // the bit and id buffers are kept between calls: a cudaFree would wait for the whole device
        const uint64_t words = (n + 31) / 32;
        if (c->pbits_cap < words) {
            dfree(c, c->d_pbits);
            c->pbits_cap = 0;
            TRY(dalloc_t(c, &c->d_pbits, words));
            c->pbits_cap = words;
        }
        auto ids_room = [&](uint64_t want) -> ffbf_status {
            dfree(c, c->d_ids);
            c->ids_cap = 0;
            TRY(dalloc_t(c, &c->d_ids, want));
            c->ids_cap = want;
            return FFBF_OK;
        };
        if (!c->d_ids && ids_room(std::min<uint64_t>(n, ffbf::kSmallResults)) != FFBF_OK) c->err.clear();
        const uint64_t host_cap = 3ull * c->res_cap;
        CUDA_TRY(c, ffbf::prune_count(c->d_pstart, c->d_pend, c->d_phash, n, c->g, c->d_ff, c->d_pbits, counts, c->st));
        CUDA_TRY(c, ffbf::prune_emit(c->d_pbits, counts, n, c->d_ids, c->ids_cap, result_head(c), result_array(c, 0),
                                     host_cap, c->st));
        TRY(sync(c));
        cnt = result_head(c)->n;
        if (c->ids_cap < cnt) {
            TRY(ids_room(cnt));
            CUDA_TRY(c, ffbf::prune_emit(c->d_pbits, counts, n, c->d_ids, c->ids_cap, result_head(c),
                                         result_array(c, 0), host_cap, c->st));
            TRY(sync(c));  // it writes the pinned room again
        }
        if (cnt <= host_cap) {
            c->r_ids.assign(result_array(c, 0), result_array(c, 0) + cnt);
        } else {
            c->r_ids.resize(cnt);
            CUDA_TRY(c, cudaMemcpyAsync(c->r_ids.data(), c->d_ids, cnt * 8, cudaMemcpyDeviceToHost, c->st));
            TRY(sync(c));
        }
    } else {
        c->r_ids.clear();
    }
    c->nids = cnt;
    c->have_prune = true;
    if (out) {
        out->n_ids = cnt;
        out->ids = c->r_ids.data();
    }
    return FFBF_OK;
} catch (...) {
    return no_host_memory(c);
}

}  // extern "C"

namespace {

// The pattern file on the host: brought back by the first call that needs it, kept until the patterns change.
ffbf_status host_patterns(ffbf_ctx* c) {
    if (c->h_pat.size() == c->pat_len) return FFBF_OK;
    c->h_pat.resize(c->pat_len);
    const cudaError_t e =
        cudaMemcpyAsync(c->h_pat.data(), c->d_pat, c->pat_len, cudaMemcpyDeviceToHost, c->st);
    const ffbf_status s = e == cudaSuccess ? sync(c) : fail(c, FFBF_ECUDA, "pattern file read failed: %s", cudaGetErrorString(e));
    if (s != FFBF_OK) c->h_pat.clear();
    return s;
}

// The pruned lines' (start, end) pairs and their bytes, line i at bytes[at[i]], gathered on the device. False where its
// memory is short or the lines make up half the file.
ffbf_status gather_pruned(ffbf_ctx* c, std::vector<uint64_t>& spans, std::vector<uint8_t>& bytes,
                          std::vector<uint64_t>& at, bool* gathered) {
    const uint64_t cnt = c->r_ids.size();
    *gathered = ensure_order(c, 16 * cnt) == FFBF_OK;
    if (*gathered) {
        uint64_t* d_spans = reinterpret_cast<uint64_t*>(c->d_order);
        CUDA_TRY(c, ffbf::gather_spans(c->d_ids, cnt, c->d_pstart, c->d_pend, d_spans, c->st));
        CUDA_TRY(c, cudaMemcpyAsync(spans.data(), d_spans, 16 * cnt, cudaMemcpyDeviceToHost, c->st));
        TRY(sync(c));
        for (uint64_t i = 0; i < cnt; i++) at[i + 1] = at[i] + spans[2 * i + 1] - spans[2 * i];
        // spans, places and bytes share the scratch
        *gathered = 2 * at[cnt] < c->pat_len && ensure_order(c, 24 * cnt + at[cnt]) == FFBF_OK;
    }
    c->err.clear();
    if (!*gathered) return FFBF_OK;
    uint64_t* d_spans = reinterpret_cast<uint64_t*>(c->d_order);
    uint64_t* d_at = d_spans + 2 * cnt;
    uint8_t* d_bytes = reinterpret_cast<uint8_t*>(d_at + cnt);
    bytes.resize(at[cnt]);
    CUDA_TRY(c, cudaMemcpyAsync(d_spans, spans.data(), 16 * cnt, cudaMemcpyHostToDevice, c->st));
    CUDA_TRY(c, cudaMemcpyAsync(d_at, at.data(), 8 * cnt, cudaMemcpyHostToDevice, c->st));
    CUDA_TRY(c, ffbf::gather_lines(c->d_pat, d_spans, d_at, cnt, d_bytes, c->st));
    CUDA_TRY(c, cudaMemcpyAsync(bytes.data(), d_bytes, bytes.size(), cudaMemcpyDeviceToHost, c->st));
    return sync(c);
}

}  // namespace

extern "C" {

ffbf_status ffbf_format_pruned(ffbf_ctx* c, size_t chunk, uint8_t** out, size_t* out_len, uint8_t** index,
                               size_t* index_len) {
    if (!c) return FFBF_EINVAL;
    if (!out || !out_len || !index || !index_len) return fail(c, FFBF_EINVAL, "NULL argument");
    if (!c->have_prune) return fail(c, FFBF_ESTATE, "ffbf_format_pruned needs ffbf_prune first");
    if (chunk == 0) return fail(c, FFBF_EINVAL, "chunk must be > 0");
    TRY(enter(c));
    std::vector<uint8_t> o, ix;
    try {
        // A few lines of a large file come back by themselves. For a small file, or many lines, the whole file does, once:
        // 1M lines of 1M took 182 ms with their spans and places, 125 by a walk over the file.
        const uint64_t cnt = c->r_ids.size();
        char num[32];
        auto put = [&](const uint8_t* file, uint64_t s, uint64_t e, uint64_t id) {
            format_line(o, file, c->pat_len, s, e, chunk);
            char* end = std::to_chars(num, num + sizeof num, id).ptr;
            *end++ = '\n';
            ix.insert(ix.end(), num, end);
        };
        bool gathered = false;
        if (cnt && c->h_pat.empty() && c->pat_len > (256u << 10) && 4 * cnt < c->npat) {
            std::vector<uint64_t> spans(2 * cnt), at(cnt + 1, 0);
            std::vector<uint8_t> bytes;
            TRY(gather_pruned(c, spans, bytes, at, &gathered));
            for (uint64_t i = 0; i < cnt && gathered; i++) {
                // format_line addresses the line by its place in the file
                const uint8_t* file = reinterpret_cast<const uint8_t*>((uintptr_t)bytes.data() + at[i] - spans[2 * i]);
                put(file, spans[2 * i], spans[2 * i + 1], c->r_ids[i]);
            }
        }
        if (cnt && !gathered) {
            TRY(host_patterns(c));
            const uint8_t* f = c->h_pat.data();
            uint64_t line = 0, pos = 0;
            auto line_end = [&] {
                const void* nl = memchr(f + pos, '\n', c->pat_len - pos);
                return nl ? (uint64_t)((const uint8_t*)nl - f) : c->pat_len;
            };
            for (uint64_t id : c->r_ids) {  // ascending
                for (; line < id; line++) pos = line_end() + 1;
                const uint64_t e = line_end();
                put(f, pos, e, id);
                pos = e + 1;
                line++;
            }
        }
    } catch (...) {
        return fail(c, FFBF_ENOMEM_HOST, "out of host memory for the pruned patterns");
    }
    TRY(to_host_buffer(c, o, out, out_len));
    ffbf_status s = to_host_buffer(c, ix, index, index_len);
    if (s != FFBF_OK) {
        free(*out);
        *out = nullptr;
    }
    return s;
}

}  // extern "C"

namespace {

// Verifies nh hit records already in c->d_hits against a device text, appending (offset + base, pattern)
// pairs. The match buffers grow and the pass reruns when they overflow. The counters are zero but for the table
// build's error flags, which come back with the first pass.
ffbf_status verify_pass(ffbf_ctx* c, uint32_t nh, const uint8_t* d_text, uint64_t text_len, uint64_t tsize,
                        uint64_t base, std::vector<uint64_t>& off_out, std::vector<uint32_t>& pid_out) {
    if (c->match_cap < std::max<uint32_t>(1024, nh)) TRY(alloc_matches(c, std::max<uint32_t>(1024, nh)));
    for (int attempt = 0; attempt < 3; attempt++) {
        CUDA_TRY(c, ffbf::verify_collect(ffbf::VerifyJob{c->d_hits, nh, c->match_cap, d_text, text_len, c->d_keys,
                                                         c->d_vals, tsize - 1, c->d_pat, c->d_pstart, c->d_pend,
                                                         c->d_moff, c->d_mpid, c->d_counters, result_head(c),
                                                         result_array(c, 0), result_array(c, 1), c->res_cap},
                                         c->st));
        CUDA_TRY(c, cudaMemsetAsync(c->d_counters, 0, ffbf::CNT_WORDS * 4, c->st));
        TRY(sync(c));
        if (result_head(c)->error) return fail(c, FFBF_ECUDA, "verification table overflow");
        const uint64_t nm = result_head(c)->n;
        if (nm <= c->match_cap && (nm <= c->res_cap || nm > ffbf::kSmallResults || c->host_order)) break;
        if (nm <= ffbf::kSmallResults) TRY(ensure_results(c, ffbf::kSmallResults));
        if (nm <= c->match_cap) continue;
        uint64_t cap = nm + nm / 4 + 1024;
        if (cap > 0xffffffffull) return fail(c, FFBF_EINVAL, "more than 2^32 matches");
        TRY(alloc_matches(c, cap));
    }
    const uint32_t nm = (uint32_t)result_head(c)->n;
    if (result_head(c)->done && !c->host_order) {
        for (uint32_t i = 0; i < nm; i++) off_out.push_back(result_array(c, 0)[i] + base);
        for (uint32_t i = 0; i < nm; i++) pid_out.push_back((uint32_t)result_array(c, 1)[i]);
        return FFBF_OK;
    }
    // (offset, pattern id) order on the device, or on the host as the hits' order is (see ffbf_scan_collect)
    const int kb = ffbf::key_bits_for(text_len);
    const size_t scratch = ffbf::order_matches_scratch(nm, kb);
    const bool on_device = !c->host_order && ensure_order(c, scratch) == FFBF_OK;
    if (!on_device) c->err.clear();
    if (on_device) CUDA_TRY(c, ffbf::order_matches(c->d_moff, c->d_mpid, nm, kb, c->d_order, scratch, c->st));
    const size_t at = off_out.size();
    off_out.resize(at + nm);
    pid_out.resize(at + nm);
    if (nm) {
        CUDA_TRY(c, cudaMemcpyAsync(off_out.data() + at, c->d_moff, nm * 8ull, cudaMemcpyDeviceToHost, c->st));
        CUDA_TRY(c, cudaMemcpyAsync(pid_out.data() + at, c->d_mpid, nm * 4ull, cudaMemcpyDeviceToHost, c->st));
    }
    TRY(sync(c));
    if (!on_device) {
        std::vector<std::pair<uint64_t, uint32_t>> m(nm);
        for (size_t i = 0; i < nm; i++) m[i] = {off_out[at + i], pid_out[at + i]};
        std::sort(m.begin(), m.end());
        for (size_t i = 0; i < nm; i++) {
            off_out[at + i] = m[i].first;
            pid_out[at + i] = m[i].second;
        }
    }
    for (size_t i = at; i < off_out.size(); i++) off_out[i] += base;
    return FFBF_OK;
}

}  // namespace

extern "C" {

ffbf_status ffbf_verify(ffbf_ctx* c, ffbf_matches* out) try {
    NvtxRange nvtx_("ffbf_verify");
    TRY(enter(c));
    if (c->scan_pending) TRY(ffbf_scan_collect(c, nullptr));
    if (!c->have_scan) return fail(c, FFBF_ESTATE, "ffbf_verify needs a scan first");
    if (!c->have_prune) TRY(ffbf_prune(c, nullptr));
    uint64_t tsize = 64;
    while (tsize < 2 * c->nids + 2) tsize <<= 1;
    if (c->table_cap < tsize) {
        dfree(c, c->d_keys);
        c->table_cap = 0;
        uint8_t* d = nullptr;
        TRY(dalloc_t(c, &d, tsize * 12));
        c->d_keys = reinterpret_cast<uint64_t*>(d);
        c->d_vals = reinterpret_cast<uint32_t*>(d + tsize * 8);
        c->table_cap = tsize;
    }
    CUDA_TRY(c, cudaMemsetAsync(c->d_vals, 0xff, tsize * 4, c->st));
    CUDA_TRY(c, cudaMemsetAsync(c->d_counters, 0, ffbf::CNT_WORDS * 4, c->st));
    CUDA_TRY(c, ffbf::table_build(c->d_ids, c->nids, c->d_phash, c->d_keys, c->d_vals, tsize - 1, c->d_counters, c->st));
    std::vector<uint64_t> off;
    std::vector<uint32_t> pid;
    if (!c->segmented) {
        TRY(verify_pass(c, c->nhits, c->d_text, c->text_len, tsize, 0, off, pid));
    } else {
        // the text was scanned in segments: each segment's text goes back to the device with its hit records
        for (const auto& sg : c->segs) {
            const uint64_t nh = sg.hr_end - sg.hr_begin;
            if (!nh) continue;
            if (c->hits_cap < nh) TRY(alloc_hits(c, nh));
            if (c->text_cap < sg.len + 64) {
                dfree(c, c->d_text_own);
                c->text_cap = 0;
                TRY(dalloc_t(c, &c->d_text_own, sg.len + 64));
                c->text_cap = sg.len + 64;
            }
            std::vector<HitRec> rel(c->seg_hr.begin() + sg.hr_begin, c->seg_hr.begin() + sg.hr_end);
            for (auto& h : rel) h.off -= sg.pos;
            CUDA_TRY(c, cudaMemcpyAsync(c->d_text_own, c->seg_text + sg.pos, sg.len, cudaMemcpyHostToDevice, c->st));
            CUDA_TRY(c, cudaMemcpyAsync(c->d_hits, rel.data(), nh * sizeof(HitRec), cudaMemcpyHostToDevice, c->st));
            TRY(verify_pass(c, (uint32_t)nh, c->d_text_own, sg.len, tsize, sg.pos, off, pid));
        }
    }
    // each pass's matches come sorted, and segments follow one another in the text
    const size_t nm = off.size();
    c->r_moff.swap(off);
    c->r_mpid.resize(nm);
    for (size_t i = 0; i < nm; i++) c->r_mpid[i] = pid[i];
    if (out) {
        out->n = nm;
        out->offsets = c->r_moff.data();
        out->pattern_ids = c->r_mpid.data();
    }
    return FFBF_OK;
} catch (...) {
    return no_host_memory(c);
}

ffbf_status ffbf_test_line(ffbf_ctx* c, const uint8_t* line, size_t len, int* hit) {
    TRY(enter(c));
    if (!hit || (!line && len)) return fail(c, FFBF_EINVAL, "NULL argument");
    // a short line is read by the kernel from the pinned result room, a longer one is copied to the device
    unsigned long long* found = &result_head(c)->n;
    const uint8_t* src = c->h_res + 64;
    *found = 0;
    if (len <= 3 * 8 * (size_t)c->res_cap) {
        if (len) memcpy(c->h_res + 64, line, len);
    } else {
        if (c->small_cap < len + 16) {
            dfree(c, c->d_small);
            c->small_cap = 0;
            TRY(dalloc_t(c, &c->d_small, len + 16));
            c->small_cap = len + 16;
        }
        CUDA_TRY(c, cudaMemcpyAsync(c->d_small, line, len, cudaMemcpyHostToDevice, c->st));
        src = c->d_small;
    }
    CUDA_TRY(c, ffbf::test_line(src, len, c->g, c->d_main, found, c->st));
    TRY(sync(c));
    const bool r = *found != 0;
    *hit = r ? 1 : 0;
    return FFBF_OK;
}

ffbf_status ffbf_debug_scan_unpublished(ffbf_ctx* c, const uint8_t* d_text, size_t len, uint32_t spins) {
    TRY(enter(c));
    if (!tunable(c, len)) return fail(c, FFBF_EINVAL, "the tuned scan does not cover this geometry or size");
    TRY(setup_scan_state(c, d_text, len));
    if (!c->d_gate) TRY(dalloc_t(c, &c->d_gate, 1));
    CUDA_TRY(c, cudaMemsetAsync(c->d_gate, 0, sizeof(uint32_t), c->st));  // never published
    CUDA_TRY(c, cudaMemsetAsync(c->d_counters, 0, ffbf::CNT_WORDS * sizeof(uint32_t), c->st));
    TRY(prepare_fast(c));
    const ffbf::FastConfig cfg = ffbf::launch_config(c->cfg, c->g.len, len, c->num_sms, false);
    c->tile_bytes = ffbf::fast_tile_bytes(cfg.rows);
    uint8_t* block;
    TRY(upload_block(c, &block));
    auto* job = reinterpret_cast<ffbf::FastJob*>(block + ffbf::kJobOffset);
    CUDA_TRY(c, ffbf::fill_fast_job(make_scan_args(c), c->d_stage1, cfg, job));
    job->ready = c->d_gate;
    job->ready_spins = spins;
    CUDA_TRY(c, cudaMemcpyAsync(c->d_job, job, sizeof *job, cudaMemcpyHostToDevice, c->st));
    CUDA_TRY(c, ffbf::launch_fast_jobs(c->g.len, cfg, c->d_job, 1, job->n_supertiles, job->stage1_nwords,
                                       c->d_counters + ffbf::CNT_ERROR, c->num_sms, c->st));
    CUDA_TRY(c, cudaMemcpyAsync(c->h_counters, c->d_counters, ffbf::CNT_WORDS * 4, cudaMemcpyDeviceToHost, c->st));
    TRY(sync(c));
    reset_scan(c);
    if (c->h_counters[ffbf::CNT_ERROR] & 4u)
        return fail(c, FFBF_ETIMEOUT, "the scan's publication gate stayed closed for %u polls", spins);
    return fail(c, FFBF_ESTATE, "the unpublished scan did not time out");
}

ffbf_status ffbf_get_scan_config(const ffbf_ctx* c, int* threads, int* mode) {
    if (!c) return FFBF_EINVAL;
    if (threads) *threads = ffbf::config_threads(c->cfg);
    if (mode) *mode = c->cfg.mode;
    return FFBF_OK;
}

ffbf_status ffbf_get_probe_order(const ffbf_ctx* c, int* order) {
    if (!c || !order) return FFBF_EINVAL;
    *order = c->cfg.order == 3 ? 2 : c->cfg.order;
    return FFBF_OK;
}

ffbf_status ffbf_clear_ff(ffbf_ctx* c) {
    TRY(enter(c));
    CUDA_TRY(c, cudaMemsetAsync(c->d_ff, 0, c->filter_bytes, c->st));
    c->have_prune = false;
    return FFBF_OK;
}

ffbf_status ffbf_get_filters(ffbf_ctx* c, uint8_t* main_bits, uint8_t* ff_bits) {
    TRY(enter(c));
    if (c->scan_pending) TRY(ffbf_scan_collect(c, nullptr));
    if (main_bits) CUDA_TRY(c, cudaMemcpyAsync(main_bits, c->d_main, c->filter_bytes, cudaMemcpyDeviceToHost, c->st));
    if (ff_bits) CUDA_TRY(c, cudaMemcpyAsync(ff_bits, c->d_ff, c->filter_bytes, cudaMemcpyDeviceToHost, c->st));
    return sync(c);
}

}  // extern "C"

