// ffbf_scan_fast.cuh -- the tuned sm_100a scan (see ffbf_scan_fast.cu): job descriptors, configuration, launch.
#pragma once
#include <cuda.h>

#include "ffbf_kernels.cuh"

namespace ffbf {

// One scan job of the tuned kernel (a text, its filter, its outputs). Jobs live in device memory; a plain
// scan is a batch of one. The tensor map is the first member (64-byte alignment).
struct alignas(64) FastJob {
    CUtensorMap tmap;        // the text as {128 bytes, rows, n_streams}
    uint64_t n_streams;      // streams covered by the tensor map
    uint32_t rows;           // rows per stream (tile size: a supertile is THREADS * rows * 128 bytes)
    uint32_t n_supertiles;   // ceil(n_streams / THREADS)
    uint32_t item_begin;     // first work item of this job; the next job's item_begin ends it
    uint32_t streams_per_tile_log2;  // streams per newline tile (fast_tile_bytes)
    Geom g;
    const uint32_t* main_words;
    uint32_t* ff_words;
    const uint8_t* text;     // the text's first byte (the sparse modes read candidate windows back)
    const uint32_t* stage1_words;  // sparse mode: cache region copy or its fold (global), copied into smem
    uint32_t stage1_nwords;
    uint32_t stage1_shift;         // the table holds C >> shift bits (0: exact copy of the cache region)
    // dense mode: the regions of its two pipelined probes (bit = (f & mask) + add for index functions f0/f1,
    // or f2/f3 when the configuration's probe order is 1)
    uint32_t a_mask, a_add, b_mask, b_add;
    HitRec* hits;
    uint32_t hits_cap;
    uint32_t ready_spins;  // polls of *ready before the launch gives up (about 1 us each)
    uint32_t* counters;
    long long* tile_first_nl;
    long long* tile_last_nl;
    uint64_t n;        // text bytes; those after the last whole stream are scanned with the last work item
    uint64_t n_tiles;  // tiles of the newline summaries (bounds their writes)
    // 1: the text's TMA loads carry an L2 evict-first policy (every text byte is read once, so its lines
    // should leave L2 before the filter's do); 0: the default policy
    uint32_t text_evict_first;
    // Optional publication gate of the launch (read from its first job): no load is issued until *ready is
    // non-zero; a gate still closed after ready_spins polls ends the launch with the timeout flag.
    const uint32_t* ready;
};

// How a job is scanned: CTA size, probe mode, rows per stream (which launch_config sets; 0 before), and in the dense mode
// the probe order. Modes 0, 2 and 3 are the sparse kernel (shared-memory stage 1) at 256/384/512, 192/256/384 and 512
// threads, the last from 192 to 512 as each text's size asks (launch_config); mode 1 is the dense one (pipelined L2 probes). Orders:
// 0: the pipelined probes are index functions f0 = h1 and f1 = h2; 1: f2 = rot16(h1) and f3 = rot16(h2), the better
// pair when their region is sparser; 2 and 3: f0 and f1 are tested against the stage-1 table first, and f0 (order 2)
// or f2 (order 3) is then probed for the windows that pass. The order only changes which bits are tested first: a
// window hits iff all K bits are set, in any order.
struct FastConfig {
    int threads;
    int mode;
    uint32_t rows;
    int order;
    bool halves = false;  // mode 3: the kernel that reads the table's 16-bit entries (table_halves)
};

// Mode (1 or 3) and dense probe order with the least expected time per window, from the fills (fraction of set bits)
// of the 384-thread kernel's stage-1 table, of the cache region and of the external region. Orders 1 and 3 need f2
// and f3 among the K index functions (K >= 4).
struct ScanChoice {
    int mode, order;
};
ScanChoice choose_scan(const Geom& g, double table_fill, double cache_fill, double ext_fill);

// True when the tuned kernel handles this geometry and text size; otherwise the generic scan runs.
bool fast_scan_supported(const Geom& g, uint64_t n);
// LENs the tuned kernel is compiled for; it takes the others as an argument.
bool compiled_len(uint32_t len);

int config_threads(const FastConfig& cfg);
// The CTA size whose shared memory the configuration's stage-1 table is sized for.
int table_threads(const FastConfig& cfg);

// The configuration a text of n bytes is launched with, alone on the GPU or in a batch: rows per stream, and in mode 3
// the CTA size.
FastConfig launch_config(const FastConfig& cfg, uint32_t len, uint64_t n, int num_sms, bool batch);
// Bytes per tile of the newline summaries of a scan with that many rows per stream: as many streams as reach 16 KiB, a
// power of two of at most 32. Texts below kShortRowsText may be scanned with less than four rows.
uint32_t fast_tile_bytes(uint32_t rows);
constexpr uint64_t kShortRowsText = 64ull << 20;

// Stage-1 table for a CTA size: a copy of the cache region when it fits in the shared memory the kernel
// leaves over, otherwise its fold to C >> shift bits.
uint32_t stage1_shift_for(const Geom& g, int threads);
uint32_t stage1_words_for(const Geom& g, int threads);
// Whether mode 3 reads the table as 16-bit entries, which lie behind its words on the device.
bool table_halves(const Geom& g);
cudaError_t build_stage1(const uint32_t* main_words, const Geom& g, int threads, uint32_t* out, cudaStream_t st);

// CTAs of the tuned kernel resident per SM for a configuration (two for the 192-thread dense kernel).
int fast_ctas_per_sm(const FastConfig& cfg);

// Rows per stream for a text of n bytes: a power of two, from 4 to 16, in a batch, or alone on the GPU where only those
// are compared (launch_config takes every row count and CTA size for a lone text).
uint32_t fast_rows(uint64_t n, const FastConfig& cfg, int num_sms, bool batch);

// Fills *job (host memory) for a.text, whose a.tile_bytes is fast_tile_bytes(cfg.rows); the caller sets item_begin.
cudaError_t fill_fast_job(const ScanArgs& a, const uint32_t* stage1_words, const FastConfig& cfg, FastJob* job);

// One launch of the tuned kernel over n_jobs device-resident jobs sharing LEN and configuration.
// d_ctl[0] collects error flags; d_ctl[1] is the work-queue counter and must be zero at launch.
cudaError_t launch_fast_jobs(uint32_t len, const FastConfig& cfg, const FastJob* d_jobs, uint32_t n_jobs,
                             uint32_t n_items, uint32_t max_s1_words, uint32_t* d_ctl, int num_sms, cudaStream_t st);

// A plain scan: one job, whose descriptor lies kJobOffset bytes behind the counters. One copy zeroes the counters and
// brings the descriptor, from pinned h_block (kJobOffset zero bytes, then room for the descriptor). The caller leaves the
// block as it is until the copy has run, and where the stream is being captured, for as long as the graph may be replayed.
constexpr size_t kJobOffset = 256;
cudaError_t scan_fast(const ScanArgs& a, const uint32_t* stage1_words, const FastConfig& cfg, int num_sms,
                      uint8_t* h_block, cudaStream_t st);

// Number of set bits in n words, written to *d_out (device).
cudaError_t popcount_words(const uint32_t* w, uint32_t n, unsigned long long* d_out, cudaStream_t st);

}  // namespace ffbf
