// ffbf_scan_fast.cu -- the tuned sm_100a scan of processFile (src/rabin-karp/ffbf.cpp:310-392).
//
// Work decomposition. The text is cut into streams of SLEN = rows * 128 bytes. A CTA of THREADS threads
// owns THREADS consecutive streams (a "supertile") at a time, one stream per thread, and walks them in parts of 64
// bytes. Each thread rolls the hash over its stream without restarting, so the LEN-byte warm-up is paid once
// per stream (from a 32-byte halo) instead of once per tile.
//
// Staging. Part p of the CTA's streams is loaded by TMA as 3-D boxes {64 bytes, 1 row, <=256 streams}
// (cp.async.bulk.tensor, 64B swizzle, one CTA per load) into one of two shared-memory stages. A "full" mbarrier
// completes when the load lands, an "empty" one when every warp has left the stage, so warps run up to a stage
// apart. The swizzle XORs a 16-byte chunk's index with bits of its thread's number, so the 16-byte reads of a
// quarter-warp hit eight different bank groups.
//
// Hash. h <- rol64(h,1) ^ S[in] ^ rol64(S[out], LEN) (hash_rot_sbox_pre_2.h:42-51 without its ring of bytes), on two
// 32-bit halves. S sits in shared memory as 16 interleaved copies of 8-byte entries, so the 16 lanes of each half-warp
// read disjoint banks whatever their bytes, and a byte's entry address is one byte-wise dot product (dp4a) of the text
// word, off the ALU pipe that the rest of the hash fills. The sparse kernel keeps the last LEN entries in registers and
// rotates the one that leaves; the others look the leaving byte, still in registers, up in a second table of rotated
// entries. Bytes with the high bit set hash as byte 0 (ffbf.cpp:127-130).
//
// Probes. Sparse filters test the first two index functions against a shared-memory table: the cache region itself
// when it fits, else its fold (bit j = OR of the cache bits i with i mod T == j), which only rejects windows the full
// test rejects. Dense filters probe the global filter, in L2, through register rings. Surviving windows are
// queued by position per warp; a full queue, or the stream's end, is flushed by the whole warp, each lane hashing
// its queued windows again and running the full K-bit test on the global filter in the reference order (checkInFilter,
// ffbf.cpp:214-239). The bytes after the last whole stream are scanned by the CTA of the last work item.
//
// Validity. A window is tested only when its LEN bytes hold no '\n' (processFile resets the hash at '\n'), from a
// newline mask per 32-byte block. Each stream's first and last '\n' feed the newline summaries, per tile of 16
// KiB or a little more, that the line resolver reads.
//
// What bounds it. Sparse: of the 9 clocks that a warp spends on a byte the ALU pipe is busy for 7.3, the shared-memory
// pipe for 7.1 (wavefronts: 2 for the S-box entry, 3.5 for the first table probe's random words, the rest for the
// predicated second probe and the text) and the issue slots for 6.4, at 12 to 16 warps per SM. Dense:
// the L1TEX unit, which looks up one random sector per clock and SM (words, 1M patterns: 0.93 of that). On one B200,
// before -> now, GB/s of text: 10k patterns, 4 GiB 662 -> 1067, 64 MiB 443 -> 799, 8 MiB 69 -> 292; LEN 24, 8k patterns in
// 2^20 + 2^24 bits, 2 GiB 487 -> 1017 and 40k in 2^22 + 2^26 299 -> 645; LEN 19, 50k in 2^24 + 2^28, 256 MiB 350 -> 714; LEN
// 24, 150k in 2^23 + 2^27, 256 MiB 295 -> 547; LEN 40, 8k in 2^20 + 2^24, 2 GiB 168 -> 805; words, 1M patterns 311 -> 351;
// 4M 16-byte signatures 245 -> 275.
//
// Every mbarrier wait is bounded; on timeout the CTA records an error flag and stops.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdlib>
#include <cstring>

#include "ffbf_scan_fast.cuh"
#include "ffbf_text.cuh"

namespace ffbf {

namespace {

constexpr int kRowBytes = 128;
constexpr int kTabBytes = 256 * 16 * 8;  // 16 copies of the 256-entry S-box
constexpr int kHalfTabBytes = kTabBytes / 2;
constexpr int kQueueCap = 64;            // candidates per warp queue
constexpr uint32_t kWaitLimit = 1u << 24;
constexpr size_t kSmemLimit = 232448;    // opt-in shared memory per block on sm_100

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// Waits for the phase of the given parity, at most kWaitLimit polls; false when it gave up.
__device__ __noinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity);

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

__device__ __noinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity) {
    for (uint32_t it = 0; it < kWaitLimit; it++)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
        "[%5];" ::"r"(dst),
        "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar)
        : "memory");
}

// The same load with an L2 cache policy (createpolicy): the text streams through L2 once.
__device__ __forceinline__ void tma_load_3d_hint(uint32_t dst, const CUtensorMap* map, int x, int y, int z,
                                                 uint32_t bar, uint64_t policy) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint "
        "[%0], [%1, {%2, %3, %4}], [%5], %6;" ::"r"(dst),
        "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar), "l"(policy)
        : "memory");
}

// Before a thread's first load through a tensor map that a host copy has written to global memory: the map may still be
// cached as it was for an earlier launch, with another text or another box.
__device__ __forceinline__ void acquire_map(const CUtensorMap* map) {
    asm volatile("fence.proxy.tensormap::generic.acquire.sys [%0], 128;" ::"l"(map) : "memory");
}

// An untiled copy of `bytes` (a multiple of 16, both addresses 16-byte aligned) completed on an mbarrier.
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

__device__ __forceinline__ uint64_t l2_evict_first_policy() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}

// Shared-memory loads of the read-only tables, which the compiler may schedule freely (a table is
// rewritten only between block barriers, at a change of job).
__device__ __forceinline__ uint2 lds64(uint32_t addr) {
    uint2 v;
    asm("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
    return v;
}
// The same at a constant distance, which the load's own offset takes.
template <int OFFSET>
__device__ __forceinline__ uint2 lds64_at(uint32_t addr) {
    uint2 v;
    asm("ld.shared.v2.u32 {%0, %1}, [%2+%3];" : "=r"(v.x), "=r"(v.y) : "r"(addr), "n"(OFFSET));
    return v;
}
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
    uint32_t v;
    asm("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}

// The same load for memory that changes between reads.
__device__ __forceinline__ uint32_t lds32_volatile(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}
// The same load where `pred` holds; 0 elsewhere.
__device__ __forceinline__ uint32_t lds32_if(uint32_t addr, bool pred) {
    uint32_t v;
    asm("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\tmov.u32 %0, 0;\n\t@q ld.shared.u32 %0, [%1];\n\t}"
        : "=r"(v)
        : "r"(addr), "r"((uint32_t)pred));
    return v;
}

// A 16-bit entry, zero-extended, and the same where `pred` holds (0 elsewhere).
__device__ __forceinline__ uint32_t lds16(uint32_t addr) {
    uint32_t v;
    asm("{\n\t.reg .u16 t;\n\tld.shared.u16 t, [%1];\n\tcvt.u32.u16 %0, t;\n\t}" : "=r"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint32_t lds16_if(uint32_t addr, bool pred) {
    uint32_t v;
    asm("{\n\t.reg .pred q;\n\t.reg .u16 t;\n\tsetp.ne.u32 q, %2, 0;\n\tmov.u16 t, 0;\n\t@q ld.shared.u16 t, [%1];\n\t"
        "cvt.u32.u16 %0, t;\n\t}"
        : "=r"(v)
        : "r"(addr), "r"((uint32_t)pred));
    return v;
}
// base + 2 * the upper half of w in one dot product: the address of a 16-bit entry
__device__ __forceinline__ uint32_t half_addr(uint32_t w, uint32_t base) { return __dp2a_lo(w, 0x0200u, base); }

// Global load of one filter word when `pred` holds (0 otherwise); read-only path.
__device__ __forceinline__ uint32_t ldg_if(const uint32_t* p, bool pred) {
    uint32_t v;
    asm("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\tmov.u32 %0, 0;\n\t@q ld.global.nc.u32 %0, [%1];\n\t}"
        : "=r"(v)
        : "l"(p), "r"((uint32_t)pred));
    return v;
}

// base + 128 * byte i (0..3) of w: the address of a byte's S-box entry in one byte-wise dot product, which runs
// beside the ALU pipe that bounds the hash
__device__ __forceinline__ uint32_t entry_addr(uint32_t w, int i, uint32_t base) {
    return __dp4a(w, 128u << (8 * i), base);
}

// Zeroes the bytes of w that have their high bit set: they hash as byte 0 (ffbf.cpp:127-130).
__device__ __forceinline__ uint32_t clear_high_bytes(uint32_t w) {
    const uint32_t hb = w & 0x80808080u;
    return w & ~((hb >> 7) * 255u);
}

// rol32 by a compile-time amount (0: identity)
template <int N>
__device__ __forceinline__ uint32_t rot_const(uint32_t x) {
    if constexpr (N == 0) return x;
    else return __funnelshift_l(x, x, N);
}

// Full test from probe FROM on (reference order, early exit); probes before FROM are known to be set.
__device__ __forceinline__ bool full_check_from(const Geom& g, const uint32_t* __restrict__ words, uint64_t h,
                                                uint32_t from) {
    for (uint32_t i = from; i < g.k; i++) {
        uint32_t b = bit_index<1>(g, h, i);
        if (!((__ldg(words + (b >> 5)) >> (b & 31)) & 1u)) return false;
    }
    return true;
}

// LEN as the kernels' template parameter: the common lengths are compiled in; kShort stands for any other one up to 32
// and kLong for 33 to 63, which the kernel then takes as an argument.
constexpr int kShort = 0, kLong = -1;
template <int L>
__device__ __forceinline__ int len_of(uint32_t len) {
    return L > 0 ? L : (int)len;
}

// Mode 5 keeps the hash rotated by this (its S-box entries are), so that the upper half of each word of it is the low
// 16 bits of one index function and the other word's low bits follow them.
constexpr uint32_t kHalvesRot = 48;

// The hash of the window of LEN bytes at `start`, its bytes read from the text's aligned words that hold them and no
// others. *newline tells whether one of them is '\n'.
template <int L, bool HALVES>
__device__ __forceinline__ uint64_t text_window_hash(const uint8_t* __restrict__ text, uint64_t start, uint32_t rt_len,
                                                     uint32_t lane_tab, bool* newline) {
    const int len = len_of<L>(rt_len);
    const uint32_t* src = reinterpret_cast<const uint32_t*>(text + (start & ~3ull));
    const uint32_t off = (uint32_t)start & 3u;
    constexpr int kWords = L > 0 ? (L + 3) / 4 : 1;
    uint32_t w[kWords + 1];
    if constexpr (L > 0) {  // all loads before the first use
#pragma unroll
        for (int q = 0; q <= kWords; q++) w[q] = 4u * q < off + L ? __ldg(src + q) : 0u;
    } else {
        w[1] = __ldg(src);
    }
    uint32_t hl = 0, hh = 0, found = 0;
    auto word = [&](int q, uint32_t lo, uint32_t hi) {
        const uint32_t v = __funnelshift_r(lo, hi, 8 * off);
        const uint32_t c = clear_high_bytes(v);
        found |= nl_bytes(v) & (4 * q + 4 <= len ? 0xffffffffu : 0xffffffffu >> (8 * (4 * q + 4 - len)));
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if (4 * q + j >= len) continue;
            const uint2 sv = lds64(entry_addr(c, j, lane_tab));
            const uint32_t nl = __funnelshift_l(hh, hl, 1) ^ sv.x, nh = __funnelshift_l(hl, hh, 1) ^ sv.y;
            hl = nl;
            hh = nh;
        }
    };
    if constexpr (L > 0) {
#pragma unroll
        for (int q = 0; q < kWords; q++) word(q, w[q], w[q + 1]);
    } else {
        for (int q = 0; 4 * q < len; q++) {
            w[0] = w[1];
            w[1] = 4u * (q + 1) < off + len ? __ldg(src + q + 1) : 0u;
            word(q, w[0], w[1]);
        }
    }
    *newline = found != 0;
    const uint64_t h = ((uint64_t)hh << 32) | hl;
    return HALVES ? rol64(h, 64 - kHalvesRot) : h;
}

__device__ __forceinline__ void record_hit(const FastJob* J, const Geom& g, uint64_t start, uint64_t h) {
    set_all<2>(g, J->ff_words, h);
    const uint32_t slot = atomicAdd(J->counters + CNT_HITS, 1u);
    if (slot < J->hits_cap) J->hits[slot] = HitRec{start, h};
}

// The whole warp drains its candidate queue: lane i takes entries i, i + 32, ... (PER_LANE at most). An entry is a
// window's end, {position in the stream | lane << 16}. Each lane reads its windows' bytes back from the text (still in
// L2), hashes them and runs the full K-bit test: few windows get here, so this costs less than carrying every
// window's hash to its test in the byte loop. All of a lane's first probes are issued before any is used.
template <int L, bool HALVES, int PER_LANE>
__device__ __noinline__ void flush_queue(const FastJob* J, uint32_t qaddr, int qn, uint64_t warp_pos0, uint64_t stride,
                                         int lane, uint32_t lane_tab) {
    const int len = len_of<L>(J->g.len);
    // the job's fields are read here rather than passed: the caller's loop keeps only its hot values live
    const Geom g = J->g;
    const uint32_t* __restrict__ main_words = J->main_words;
    const uint8_t* __restrict__ text = J->text;
    uint64_t start[PER_LANE], h[PER_LANE];
    uint32_t v[PER_LANE], bi[PER_LANE];
#pragma unroll
    for (int t = 0; t < PER_LANE; t++) {
        const int i = lane + 32 * t;
        v[t] = bi[t] = 0;
        if (i >= qn) continue;
        const uint32_t e = lds32_volatile(qaddr + 4u * (uint32_t)i);
        start[t] = warp_pos0 + (e >> 16) * stride + (e & 0xFFFFu) + 1 - len;
        bool newline;
        h[t] = text_window_hash<L, HALVES>(text, start[t], len, lane_tab, &newline);  // windows with a '\n' are not queued
        bi[t] = bit_index<1>(g, h[t], 0);
        v[t] = __ldg(main_words + (bi[t] >> 5));
    }
#pragma unroll
    for (int t = 0; t < PER_LANE; t++) {
        if (!((v[t] >> (bi[t] & 31)) & 1u)) continue;
        if (full_check_from(g, main_words, h[t], 1)) record_hit(J, g, start[t], h[t]);
    }
    __syncwarp();
}

// What a warp does when its streams are done: their newline summary, and in the CTA of the job's last work item the
// text's end after its last whole stream (less than one stream), a window per thread, where a launch of its own took 60
// us for 12 KB. z is the thread's stream, nl_span its first '\n' (low half, 0xffff: none) and its last. One function,
// so that the byte loop keeps its registers.
template <int L, bool HALVES>
__device__ __noinline__ void finish_streams(const FastJob* J, uint64_t z, uint32_t nl_span, int threads, uint32_t lane_tab,
                                            uint32_t* error_flag) {
    const int lane = threadIdx.x & 31;
    const uint64_t n = J->n, n_streams = J->n_streams, slen = (uint64_t)J->rows * kRowBytes;
    const uint64_t pos = z * slen;
    const bool active = z < n_streams, any = active && (nl_span & 0xffffu) != 0xffffu;
    long long f = any ? (long long)(pos + (nl_span & 0xffffu)) : LLONG_MAX;
    long long l = any ? (long long)(pos + (nl_span >> 16)) : -1;
    // reduce over the lanes whose streams share a tile
    const uint32_t spt_log2 = J->streams_per_tile_log2;
    const int G = 1 << spt_log2;
    for (int o = 1; o < G; o <<= 1) {
        f = min(f, __shfl_xor_sync(0xffffffffu, f, o));
        l = max(l, __shfl_xor_sync(0xffffffffu, l, o));
    }
    uint64_t tile = z >> spt_log2;
    bool write = active && (lane & (G - 1)) == 0;
    const uint64_t covered = n_streams * slen;
    if (covered < n && z / threads == J->n_supertiles - 1) {
        const Geom g = J->g;
        for (uint64_t p = covered + threadIdx.x; p < n; p += threads) {
            const int len = len_of<L>(g.len);
            if (p + 1 < len) continue;
            bool newline;
            const uint64_t h = text_window_hash<L, HALVES>(J->text, p + 1 - len, len, lane_tab, &newline);
            if (!newline && full_check_from(g, J->main_words, h, 0)) record_hit(J, g, p + 1 - len, h);
        }
        __syncwarp();
        // the last stream's warp adds the newlines of the text's end to the tile it falls in, which may be a new one
        const uint64_t z0 = z - lane;
        if (z0 < n_streams && n_streams <= z0 + 32) {
            long long tf = LLONG_MAX, tl = -1;
            for (long long c = (long long)covered + 16 * lane; c < (long long)n; c += 512) {
                const uint4 v = chunk16(J->text, c, (long long)n);
                const uint32_t w[4] = {nl_bytes(v.x), nl_bytes(v.y), nl_bytes(v.z), nl_bytes(v.w)};
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    if (!w[q]) continue;
                    tf = min(tf, c + 4 * q + (__ffs(w[q]) - 1) / 8);
                    tl = max(tl, c + 4 * q + (31 - __clz(w[q])) / 8);
                }
            }
            for (int o = 16; o; o >>= 1) {
                tf = min(tf, __shfl_xor_sync(0xffffffffu, tf, o));
                tl = max(tl, __shfl_xor_sync(0xffffffffu, tl, o));
            }
            const uint64_t end_tile = n_streams >> spt_log2;
            if (tile == end_tile) {
                f = min(f, tf);
                l = max(l, tl);
            }
            if (n_streams % G == 0 && lane == 31) {
                // no stream is in that tile; lane 31 writes no other one (G is at least 8)
                tile = end_tile;
                f = tf;
                l = tl;
                write = true;
            }
        }
    }
    if (write) {
        if (tile < J->n_tiles) {
            J->tile_first_nl[tile] = f;
            J->tile_last_nl[tile] = l;
        } else {
            atomicOr(error_flag, 0x200u);
        }
    }
}

// The current job as the byte loop reads it, once per part: kept in shared memory, so that it holds no registers.
struct JobState {
    int job;
    uint32_t rows;  // 0: the job's table does not fit or did not arrive, and its parts fail the self-check
    uint32_t n_supertiles;
    uint32_t s1_bmask;      // byte offset of the stage-1 table word of bit (h & (T-1)): (h >> 3) & s1_bmask
    uint32_t s2, s2_bmask;  // the second probe's table: the same, or with S = 1 a word of ones
    uint32_t twice;  // 0x10001: repeats a 16-bit entry in both halves, by a multiplication that the ALU pipe is spared
    uint32_t a_mask, b_mask;  // dense modes: the regions of the two pipelined probes
    const uint32_t *a_words, *b_words;
    uint64_t n_streams;
    uint32_t tables;  // tables loaded so far: the parity of their barrier
    int started;      // the job whose table was sent for at the kernel's start
};

// Sends for a job's stage-1 table (thread 0): its words, or 0 where it does not fit or is too small for a bulk copy.
__device__ __forceinline__ uint32_t start_table(const FastJob* J, uint32_t s1, uint32_t max_s1_words, uint32_t tbar) {
    const uint32_t nw = J->stage1_nwords;  // a power of two
    if (nw > max_s1_words || nw < 4) return 0;
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // after plain stores to a table
    mbar_expect_tx(tbar, 4 * nw);
    bulk_load(s1, J->stage1_words, 4 * nw, tbar);
    return nw;
}

// Makes job `job` current: all threads of the CTA call it at the same stage, where every warp is done with the job
// before. With `s1` its stage-1 table (T = C >> shift bits) is loaded there.
__device__ __noinline__ void change_job(const FastJob* jobs, int job, JobState* s, uint32_t s1, uint32_t* s1p,
                                        uint32_t max_s1_words, uint32_t ones, uint32_t tbar, uint32_t* error_flag) {
    const FastJob* J = jobs + job;
    const uint32_t tid = threadIdx.x;
    __syncthreads();
    const bool fits = !s1 || J->stage1_nwords <= max_s1_words;
    const uint32_t nw = s1 && fits ? J->stage1_nwords : 0u;
    const uint32_t parity = s->tables & 1u;
    if (tid == 0) {
        const uint32_t bmask = ((J->g.cache_mask >> J->stage1_shift) >> 3) & ~3u;
        s->job = job;
        s->rows = fits ? J->rows : 0u;
        s->n_supertiles = J->n_supertiles;
        s->s1_bmask = bmask;
        s->twice = 0x10001u;
        s->s2 = J->g.s > 1 ? s1 : ones;
        s->s2_bmask = J->g.s > 1 ? bmask : 0u;
        s->a_mask = J->a_mask;
        s->b_mask = J->b_mask;
        s->a_words = J->main_words + J->a_add / 32;
        s->b_words = J->main_words + J->b_add / 32;
        s->n_streams = J->n_streams;
        if (s1 && s->started != job) start_table(J, s1, max_s1_words, tbar);
        s->started = -1;
    }
    if (nw >= 4) {
        if (!mbar_wait_bounded(tbar, parity)) {
            atomicOr(error_flag, 4u);
            s->rows = 0;
        }
    } else if (tid < nw) {
        s1p[tid] = J->stage1_words[tid];  // regions of 32 and 64 bits
    }
    __syncthreads();
    if (tid == 0 && nw >= 4) s->tables++;  // read next after the barrier of the next change
}

template <int N>
__device__ __forceinline__ void shl64_or(uint32_t& lo, uint32_t& hi) {
    // (hi:lo) |= (hi:lo) << N, 0 < N < 32
    hi |= __funnelshift_l(lo, hi, N);
    lo |= lo << N;
}

// Bit j set when the window of L bytes ending at byte j of a 32-byte block holds a '\n'. `prev` and `cur`
// are the newline masks (bit i = byte i is '\n') of the previous block and of this one.
template <int L>
__device__ __forceinline__ uint32_t window_has_newline(uint32_t prev, uint32_t cur) {
    static_assert(L >= 1 && L <= 32, "windows reach back at most one block");
    // OR of (cur:prev) << k for k in [0, L), high word: (cur:prev) << k covers [0, w) after the doubling
    // steps below; the set bits of L add shifted copies of it
    uint32_t lo = prev, hi = cur;
    uint32_t rhi = 0;
    int covered = 0;
#pragma unroll
    for (int m = 0; m < 6; m++) {
        const int w = 1 << m;
        if (L & w) {
            if (covered == 0) rhi |= hi;
            else if (covered < 32) rhi |= __funnelshift_l(lo, hi, covered);
            else rhi |= lo << (covered - 32);
            covered += w;
        }
        if (2 * w <= L) {
            switch (w) {
                case 1: shl64_or<1>(lo, hi); break;
                case 2: shl64_or<2>(lo, hi); break;
                case 4: shl64_or<4>(lo, hi); break;
                case 8: shl64_or<8>(lo, hi); break;
                case 16: shl64_or<16>(lo, hi); break;
                default: break;
            }
        }
    }
    return rhi;
}

// The same for a length given at run time, up to 32 or, with the mask `prev2` of the block before `prev`, to 63.
template <bool LONG>
__device__ __forceinline__ uint32_t window_has_newline(int len, uint32_t prev2, uint32_t prev, uint32_t cur) {
    uint32_t m0 = cur, m1 = prev, m2 = prev2;
    int w = 1;  // m0 covers shifts [0, w)
    for (; 2 * w <= (LONG ? 32 : len); w *= 2) {
        m0 |= __funnelshift_l(m1, m0, w);
        m1 |= LONG ? __funnelshift_l(m2, m1, w) : m1 << w;
        if (LONG) m2 |= m2 << w;
    }
    return len > w ? m0 | __funnelshift_l(m1, m0, len - w) : m0;
}

// The 32 bytes that leave the window as the block `c` enters it: the bytes LEN before c's, of which p holds the 32
// before c and pp the 32 before those; K = LEN / 4, and shift 32 - 8 * (LEN % 4) bits.
template <int K>
__device__ __forceinline__ void leaving_words(const uint32_t (&pp)[8], const uint32_t (&p)[8], const uint32_t (&c)[8],
                                              uint32_t shift, uint32_t (&out)[8]) {
    auto word = [&](int i) { return i >= 0 ? c[i & 7] : i >= -8 ? p[(i + 8) & 7] : pp[(i + 16) & 7]; };
#pragma unroll
    for (int q = 0; q < 8; q++) out[q] = __funnelshift_rc(word(q - K - 1), word(q - K), shift);
}

template <int L>
__device__ __forceinline__ void leaving_block(const uint32_t (&pp)[8], const uint32_t (&p)[8], const uint32_t (&c)[8],
                                              int len, uint32_t (&out)[8]) {
    const uint32_t shift = 32u - 8u * ((uint32_t)len & 3u);
    switch (len >> 2) {
#define FFBF_LEAVING(K) \
    case K: leaving_words<K>(pp, p, c, shift, out); break
        case 0:
        default:
            if constexpr (L == kShort) leaving_words<0>(pp, p, c, shift, out);
            break;
        FFBF_LEAVING(8);
        FFBF_LEAVING(L == kShort ? 1 : 9);
        FFBF_LEAVING(L == kShort ? 2 : 10);
        FFBF_LEAVING(L == kShort ? 3 : 11);
        FFBF_LEAVING(L == kShort ? 4 : 12);
        FFBF_LEAVING(L == kShort ? 5 : 13);
        FFBF_LEAVING(L == kShort ? 6 : 14);
        FFBF_LEAVING(L == kShort ? 7 : 15);
#undef FFBF_LEAVING
    }
}

// Newline mask of a block's 32 bytes: bit i set when byte i is '\n' (exact). Each word's zero-byte mask keeps
// its high bits (0x80 per '\n'); byte-wise dot products with weights 1, 2, 4, 8 (and 16, 32, 64, 128 for the
// next word) gather two words' eight bits into bits 7..14 without shifts.
__device__ __forceinline__ uint32_t newline_mask32(const uint32_t (&w)[8]) {
    uint32_t f[4];
#pragma unroll
    for (int q = 0; q < 8; q++) {
        const uint32_t z = ((w[q] ^ 0x0A0A0A0Au) & 0x7F7F7F7Fu) + 0x7F7F7F7Fu;
        const uint32_t zb = ~(z | w[q]) & 0x80808080u;
        f[q >> 1] = __dp4a(zb, (q & 1) ? 0x80402010u : 0x08040201u, (q & 1) ? f[q >> 1] : 0u);
    }
    return ((f[0] + (f[1] << 8)) >> 7) | ((f[2] + (f[3] << 8)) << 9);
}

// Kernel modes.
// MODE 0 (sparse filters): both first index functions are tested against a shared-memory table, the cache region
// itself when it fits, else its fold, which only rejects windows the full test rejects.
// MODE 5: MODE 0 for a table of exactly 2^20 bits (any cache region from 2^20 bits on), S >= 2 and the lengths that keep
// their entries. The table is 65536 entries of 16 bits, and the hash is kept rotated by 48 (a rotation of the S-box), so
// that each word's upper half is the low 16 bits of one index function: an entry's address is one dot product, without
// the shift, the mask and the sum, and the other word's low bits choose the bit. That takes 4 instructions per byte
// off the ALU pipe: 10k patterns, 4 GiB 992 -> 1067 GB/s, 64 MiB 762 -> 799; 8k in 2^20 + 2^24, 2 GiB 957 -> 1017.
// MODE 1 (dense filters, where a shared-memory table would pass most windows): the exact probes of the first two
// index functions are global loads, the first issued per valid window, the second for the windows that pass it;
// both are consumed kRing bytes later from register rings, so L2 latency overlaps the hashing of the next windows.
// MODE 2: MODE 1 with the pipelined probes on index functions f2 = rot16(h1) and f3 = rot16(h2) (the
// external region for S <= 2, usually much sparser than the cache region, so fewer windows need a second probe).
// MODE 3: a window's f0 and f1 are tested against the shared-memory table as in MODE 0, and for the windows that
// pass, one exact probe of f0 is pipelined as in MODE 1; MODE 4 pipelines f2 instead. They suit filters whose table
// passes too many windows for MODE 0's queue (above about 2 %) but still rejects most.
//
// In every mode the byte loop over a 32-byte block is one branch-free stretch: a window's verdict is shifted into a
// 32-bit register mask, and only after the block do the lanes with surviving windows queue their positions. Against
// a warp vote and a queue append per byte this took the sparse scan of a 4 GiB text from 662 to 749 GB/s.
__host__ __device__ constexpr bool sparse_mode(int mode) { return mode == 0 || mode == 5; }

// Whether the byte loop keeps the window's LEN S-box entries in registers and rotates the leaving one there, instead of
// reading it from the rotated table: the sparse mode at the compiled lengths but 32, whose 64 registers spill beside the
// loop's at 384 threads (92 bytes). Two shifts per byte take the place of 2 of 9.2 shared-memory wavefronts and of a dp4a,
// and the table's other half makes room for a 2^20-bit stage-1 table beside 512 threads: 1 GiB, 10k patterns, 822 ->
// 850 GB/s from the registers alone (512 threads, 2^19 bits), 964 with both; 2 GiB in 2^20 + 2^24 bits 789 -> 955.
__host__ __device__ constexpr bool keeps_entries(int mode, int len) { return sparse_mode(mode) && len > 0 && len != 32; }
__host__ __device__ constexpr int tab_bytes(int mode, int len) { return keeps_entries(mode, len) ? kHalfTabBytes : kTabBytes; }

// CTAs per SM: dense modes 1 and 2 at 192 threads run two CTAs per SM (12 warps, as one 384-thread CTA, but two
// independent pipelines); every other configuration runs one.
__host__ __device__ constexpr int ctas_per_sm(int threads, int mode) {
    return threads == 192 && (mode == 1 || mode == 2) ? 2 : 1;
}
// Bytes of each stream that a stage holds. Half a row leaves shared memory for a stage-1 table of twice the size
// (prefiltered dense scan of 150k patterns: 343 -> 406 GB/s) and more often lets a warp leave a stage (dense scan of
// 1M patterns: 343 -> 353 GB/s).
constexpr int kPart = 64;
constexpr int kParts = kRowBytes / kPart;
// Streams per TMA box (<= 256), a divisor of the CTA's threads.
__host__ __device__ constexpr int box_streams_for(int threads) {
    return threads <= 256 ? threads : threads <= 512 ? threads / 2 : threads % 3 == 0 ? threads / 3 : threads / 4;
}

// Work items. Job j owns items [item_begin_j, item_begin_{j+1}), one per supertile of THREADS streams; CTA b starts
// with item b and takes the next ones from the work queue. Each item is one TMA load of the last part of the
// streams before (the halo) followed by the loads of its streams' parts. Thread 0 issues load k+1 while the CTA
// consumes load k and records in meta[] which job, item and part each stage holds.
template <int L, int THREADS, int MODE>
__global__ void __launch_bounds__(THREADS, ctas_per_sm(THREADS, MODE)) k_scan_fast(const FastJob* __restrict__ jobs, uint32_t n_jobs,
                                                          uint32_t n_items, uint32_t max_s1_words, uint32_t rt_len,
                                                          uint32_t* __restrict__ ctl) {
    // ctl[0]: error flags; ctl[1]: the work queue, the count of items handed out past the first wave
    uint32_t* const error_flag = ctl;
    constexpr int kStageBytes = THREADS * kPart;
    // dense modes: ring depth per probe (divides 32); 384-thread CTAs trade depth for warps (more L2 probes
    // in flight per SM within the register file)
    constexpr int kRing = THREADS >= 384 || ctas_per_sm(THREADS, MODE) == 2 ? 4 : 8;
    constexpr int kBox = box_streams_for(THREADS);
    constexpr bool kSparse = sparse_mode(MODE);
    constexpr bool kPre = MODE == 3 || MODE == 4;  // dense with the shared-memory prefilter and one pipelined probe
    constexpr int kLag = kPre ? kRing : 2 * kRing;  // bytes from a window's first probe to its verdict
    constexpr bool kTable = kSparse || kPre;  // reads the stage-1 table
    // S-box layout: 16 bank-private copies of S[0..127] and, where the leaving byte is looked up, of rol64(S[0..127],
    // LEN), so that it needs no rotation; a block's high bytes are cleared beforehand (they hash as byte 0). With LEN =
    // 32 the rotation only swaps the halves, and the table holds all 256 bytes once.
    constexpr bool kTwoTables = L != 32;
    constexpr bool kHalves = MODE == 5;
    constexpr bool kEntries = keeps_entries(MODE, L);
    constexpr int kTab = tab_bytes(MODE, L);
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t* smem = smem_raw + (base - raw);
    // layout: [stage 0][stage 1][S tables][mbarriers, meta, a word of ones (128 B)][warp queues][stage-1 table]
    const uint32_t stage0 = base;
    const uint32_t tab = base + 2 * kStageBytes;
    const uint32_t bar0 = tab + kTab;
    // Stage k & 1's "full" barrier completes when load k lands, its "empty" barrier when every warp is done reading
    // it; load k + 2 reuses the stage only after that, and warps otherwise run apart by up to a stage.
    auto fbar = [&](uint32_t k) { return bar0 + 8u * (k & 1u); };
    auto ebar = [&](uint32_t k) { return bar0 + 16u + 8u * (k & 1u); };
    int* meta = reinterpret_cast<int*>(smem + 2 * kStageBytes + kTab + 32);  // [stage][4]: job, item, part, valid
    const uint32_t ones = bar0 + 64u, tbar = bar0 + 72u;  // the table's load completes on tbar
    const uint32_t queues = bar0 + 128u;
    const uint32_t s1 = queues + (THREADS / 32) * 4u * kQueueCap;
    uint32_t* s1p = reinterpret_cast<uint32_t*>(smem + (s1 - base));
    // the load sequencer's state (thread 0 only) and each warp's first text position
    __shared__ int s_abort;
    __shared__ uint32_t s_ni, s_nj;
    __shared__ JobState s_job;
    __shared__ int s_nr, s_map;  // s_map: the job whose tensor map thread 0 has acquired
    __shared__ uint64_t s_wpos[THREADS / 32];

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // Load sequencer, run by thread 0: the next load is part nr (-1: halo) of item ni, which belongs to job nj.
    // Load k waits (bounded) until every warp has released load k - 2's stage; with no item left it completes
    // the stage's full barrier without a load and marks the end in meta. Returns false when the wait gave up.
    auto issue = [&](uint32_t k) -> bool {
        if (k >= 2 && !mbar_wait_bounded(ebar(k), ((k - 2) >> 1) & 1u)) {
            atomicOr(error_flag, 4u);
            return false;
        }
        int* m = meta + 4 * (k & 1);
        uint32_t ni = s_ni, nj = s_nj;
        int nr = s_nr;
        if (ni >= n_items) {
            m[3] = 0;
            mbar_arrive(fbar(k));
            return true;
        }
        while (nj + 1 < n_jobs && __ldg(&jobs[nj + 1].item_begin) <= ni) nj++;
        const FastJob* J = jobs + nj;
        if (s_map != (int)nj) {
            acquire_map(&J->tmap);
            s_map = (int)nj;
        }
        const uint32_t R = __ldg(&J->rows);
        const uint32_t st = ni - __ldg(&J->item_begin);
        const int y = nr < 0 ? (int)R - 1 : nr / kParts;
        const int x = nr < 0 ? kRowBytes - kPart : nr % kParts * kPart;
        const int z = (int)(st * THREADS) + (nr < 0 ? -1 : 0);
        const uint32_t bar = fbar(k);
        const uint32_t dst = stage0 + (k & 1) * kStageBytes;
        m[0] = (int)nj;
        m[1] = (int)st;
        m[2] = nr;
        m[3] = 1;
        mbar_expect_tx(bar, kStageBytes);
        if (__ldg(&J->text_evict_first)) {
            const uint64_t pol = l2_evict_first_policy();
            for (int b = 0; b < THREADS / kBox; b++)
                tma_load_3d_hint(dst + b * kBox * kPart, &J->tmap, x, y, z + b * kBox, bar, pol);
        } else {
            for (int b = 0; b < THREADS / kBox; b++)
                tma_load_3d(dst + b * kBox * kPart, &J->tmap, x, y, z + b * kBox, bar);
        }
        if (++nr == (int)R * kParts) {
            nr = -1;
            ni = gridDim.x + atomicAdd(ctl + 1, 1u);  // next item from the queue
        }
        s_ni = ni;
        s_nj = nj;
        s_nr = nr;
        return true;
    };
    if (tid == 0) {
        s_abort = 0;
        s_job.job = -1;
        s_job.tables = 0;
        s_job.started = -1;
        s_ni = blockIdx.x;
        s_nj = 0;
        s_nr = -1;
        s_map = -1;
        for (uint32_t b = 0; b < 2; b++) {
            mbar_init(fbar(b), 1);
            mbar_init(ebar(b), THREADS / 32);
        }
        mbar_init(tbar, 1);
        *reinterpret_cast<uint32_t*>(smem + (ones - base)) = 0xFFFFFFFFu;  // the S = 1 second-probe word
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        // publication gate: a bounded poll, and no load in flight if it gives up
        bool open = true;
        if (const uint32_t* rw = jobs[0].ready) {
            const uint32_t spins = jobs[0].ready_spins;
            for (uint32_t i = 0;; i++) {
                if (*reinterpret_cast<const volatile uint32_t*>(rw) != 0u) break;
                if (i >= spins) {
                    atomicOr(error_flag, 4u);
                    open = false;
                    break;
                }
                __nanosleep(1000);
            }
        }
        if (open) {
            // the first job's table travels while the S-box is laid out
            if constexpr (kTable) {
                if (s_ni < n_items) {
                    while (s_nj + 1 < n_jobs && __ldg(&jobs[s_nj + 1].item_begin) <= s_ni) s_nj++;
                    if (start_table(jobs + s_nj, s1, max_s1_words, tbar)) s_job.started = (int)s_nj;
                }
            }
            issue(0);
        } else {
            meta[3] = 0;
            mbar_arrive(fbar(0));
        }
    }
    // a thread per byte value, its 16 copies stored in an order that keeps the lanes on different banks
    for (int c = tid; c < kTab / 128; c += THREADS) {
        uint64_t* tp = reinterpret_cast<uint64_t*>(smem + 2 * kStageBytes) + 16 * c;
        const uint64_t v = kHalves ? rol64(c_sbox[c], kHalvesRot)
                           : kTwoTables ? (c < 128 ? c_sbox[c] : rol64(c_sbox[c - 128], (uint32_t)len_of<L>(rt_len)))
                                      : c_sbox[(c & 0x80) ? 0 : c];
#pragma unroll
        for (int q = 0; q < 16; q++) tp[(q + lane) & 15] = v;
    }
    __syncthreads();

    const uint32_t lane_tab = tab + (uint32_t)(lane & 15) * 8u;  // entry c of this lane's copy: + c * 128
    // S-box entry of byte i of the 64-byte span (p, c): as it enters the window, and rotated by LEN as it leaves
    auto sbox_in = [&](const uint32_t (&c)[8], int i) { return lds64(entry_addr(c[i >> 2], i & 3, lane_tab)); };
    uint32_t leaving[8] = {0, 0, 0, 0, 0, 0, 0, 0};  // with a run-time LEN, the block of leaving bytes
    auto sbox_out = [&](const uint32_t (&p)[8], const uint32_t (&c)[8], int i) {
        if constexpr (L <= 0) return lds64_at<128 * 128>(entry_addr(leaving[i >> 2], i & 3, lane_tab));
        const uint2 o = lds64_at<kTwoTables ? 128 * 128 : 0>(
            i >= L ? entry_addr(c[(i - L) >> 2], (i - L) & 3, lane_tab)
                   : entry_addr(p[(i - L + 32) >> 2], (i - L + 32) & 3, lane_tab));
        return kTwoTables ? o : make_uint2(o.y, o.x);
    };
    // Zeroes the block's high bytes where the table does not map them (rare in text: one test per block).
    auto map_high_bytes = [&](uint32_t (&w)[8]) {
        if constexpr (kTwoTables) {
            if (((w[0] | w[1] | w[2]) | (w[3] | w[4] | w[5]) | (w[6] | w[7])) & 0x80808080u) {
#pragma unroll
                for (int q = 0; q < 8; q++) w[q] = clear_high_bytes(w[q]);
            }
        }
    };
    const uint32_t qaddr = queues + (uint32_t)warp * 4u * kQueueCap;
    const unsigned lt_mask = (1u << lane) - 1u;

    auto job_desc = [&]() { return jobs + s_job.job; };

    int qn = 0;  // warp-uniform queue fill
    auto flush = [&]() {
        __syncwarp();
        flush_queue<L, kHalves, kQueueCap / 32>(job_desc(), qaddr, qn, s_wpos[warp], (uint64_t)s_job.rows * kRowBytes, lane,
                                         lane_tab);
        qn = 0;
    };
    // Queues the windows whose bits are set in each lane's mask; bit i is the window ending at pos + i in the lane's
    // stream. Every round takes one window of each lane that has any.
    auto enqueue = [&](uint32_t cand, uint32_t pos) {
        while (__any_sync(0xffffffffu, cand != 0u)) {
            const unsigned m = __ballot_sync(0xffffffffu, cand != 0u);
            if (cand) {
                // qn <= kQueueCap - 32 holds on entry (the queue flushes above that)
                asm volatile("st.shared.u32 [%0], %1;" ::"r"(qaddr + 4u * (uint32_t)(qn + __popc(m & lt_mask))),
                             "r"((pos + (uint32_t)__ffs(cand) - 1u) | ((uint32_t)lane << 16))
                             : "memory");
                cand &= cand - 1;
            }
            qn += __popc(m);
            if (qn > kQueueCap - 32) flush();
        }
    };
    // dense-mode rings. Stage A: the first probe's word (0 when the window was not valid, so its test fails) and the
    // window's two index functions. Stage B: the second probe's word (0 when stage A failed) and its index function.
    constexpr int kR = kSparse ? 1 : kRing;
    constexpr int kRot = MODE == 2 || MODE == 4 ? 16 : 0;  // rotation of h1/h2 giving the pipelined probes' index functions
    uint32_t ring_v[kR], ring_a[kR], ring_b[kR], ring2_v[kR], ring2_b[kR];
#pragma unroll
    for (int q = 0; q < kR; q++) ring_v[q] = ring_a[q] = ring_b[q] = ring2_v[q] = ring2_b[q] = 0;

    uint32_t hl = 0, hh = 0;
    uint32_t el[kEntries ? L : 1], eh[kEntries ? L : 1];  // the S-box entries of the LEN bytes before the block
#pragma unroll
    for (int q = 0; q < (kEntries ? L : 1); q++) el[q] = eh[q] = 0;
    uint32_t prev[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    uint32_t prev2[8] = {0, 0, 0, 0, 0, 0, 0, 0}, nl_prev2 = 0;  // the block before prev (kLong)
    // newline mask of the previous block (bit 31 forced at the text's start, where nothing precedes offset 0)
    uint32_t nl_prev = 0;
    uint32_t nl_span = 0xffffu;  // first (low half, 0xffff: none) and last '\n' of the stream so far

    for (uint32_t k = 0;; k++) {
        {
            uint32_t it = 0;
            while (!mbar_try_wait(fbar(k), (k >> 1) & 1u)) {
                if (++it >= kWaitLimit) {
                    atomicOr(error_flag, 4u);
                    s_abort = 1;
                    break;
                }
            }
        }
        if (s_abort) {
            // Give the loads still in flight a bounded chance to land before the shared memory goes away.
            if (tid == 0 && meta[4 * (k & 1) + 3])
                for (uint32_t j = 0; j < kWaitLimit && !mbar_try_wait(fbar(k), (k >> 1) & 1u); j++) {
                }
            if (tid == 0 && s_job.started >= 0) mbar_wait_bounded(tbar, s_job.tables & 1u);
            break;
        }
        // the stage's meta is written before its full barrier completes, so it is read after the wait
        const int* m = meta + 4 * (k & 1);
        if (!m[3]) break;
        const int job = m[0], r = m[2];
        const uint32_t st = (uint32_t)m[1];
        if (tid == 0 && !issue(k + 1)) s_abort = 1;
        if (job != s_job.job) change_job(jobs, job, &s_job, kTable ? s1 : 0u, s1p, max_s1_words, ones, tbar, error_flag);
        const uint32_t R = s_job.rows;

        // self-checks: a bad descriptor or sequencing records a code and skips the work
        if ((uint32_t)job >= n_jobs || st >= s_job.n_supertiles || r < -1 || r >= (int)R * kParts) {
            if (tid == 0) atomicOr(error_flag, 0x100u);
            __syncwarp();
            if (lane == 0) mbar_arrive(ebar(k));
            continue;
        }
        const bool active = (uint64_t)st * THREADS + tid < s_job.n_streams;
        const uint8_t* row = smem + (k & 1) * kStageBytes + tid * kPart;
        const int sw = (tid >> 1) & 3;  // the 64-byte swizzle XORs a 16-byte chunk's index with its address bits 7 and 8

        if (r < 0) {
            // halo: the last 32 bytes before the stream
            const uint4 c6 = *reinterpret_cast<const uint4*>(row + (((kPart / 16 - 2) ^ sw) << 4));
            const uint4 c7 = *reinterpret_cast<const uint4*>(row + (((kPart / 16 - 1) ^ sw) << 4));
            prev[0] = c6.x; prev[1] = c6.y; prev[2] = c6.z; prev[3] = c6.w;
            prev[4] = c7.x; prev[5] = c7.y; prev[6] = c7.z; prev[7] = c7.w;
            map_high_bytes(prev);
            hl = 0;
            hh = 0;
            // the hash of the halo's last LEN bytes, from a zero state: nothing leaves the window
            const int from = 32 - len_of<L>(rt_len);
            auto enter = [&](const uint32_t (&w)[8], int j) {
                const uint2 sv = sbox_in(w, j);
                const uint32_t nl = __funnelshift_l(hh, hl, 1) ^ sv.x, nh = __funnelshift_l(hl, hh, 1) ^ sv.y;
                hl = nl;
                hh = nh;
                if constexpr (kEntries) {
                    el[j >= 32 - L ? j - (32 - L) : 0] = sv.x;
                    eh[j >= 32 - L ? j - (32 - L) : 0] = sv.y;
                }
            };
            if constexpr (L == kLong) {
                const uint4 c4 = *reinterpret_cast<const uint4*>(row + ((0 ^ sw) << 4));
                const uint4 c5 = *reinterpret_cast<const uint4*>(row + ((1 ^ sw) << 4));
                prev2[0] = c4.x; prev2[1] = c4.y; prev2[2] = c4.z; prev2[3] = c4.w;
                prev2[4] = c5.x; prev2[5] = c5.y; prev2[6] = c5.z; prev2[7] = c5.w;
                map_high_bytes(prev2);
                nl_prev2 = newline_mask32(prev2);
#pragma unroll
                for (int j = 0; j < 32; j++)
                    if (j - 32 >= from) enter(prev2, j);
            }
#pragma unroll
            for (int j = 0; j < 32; j++)
                if (j >= from) enter(prev, j);
            nl_prev = newline_mask32(prev) | (st == 0 && tid == 0 ? 0x80000000u : 0u);  // text start: nothing before offset 0
            nl_span = 0xffffu;
            if (lane == 0) s_wpos[warp] = ((uint64_t)st * THREADS + (uint64_t)warp * 32) * R * kRowBytes;
        } else {
            const uint32_t pos0 = (uint32_t)r * kPart;  // this part's first byte in the stream
            const uint32_t s1_bmask = s_job.s1_bmask, s2 = s_job.s2, s2_bmask = s_job.s2_bmask;
            const uint32_t twice = s_job.twice;
            const uint32_t a_mask = s_job.a_mask, b_mask = s_job.b_mask;
            const uint32_t *const a_words = s_job.a_words, *const b_words = s_job.b_words;
#pragma unroll 1
            for (int b = 0; b < kPart / 32; b++) {
                uint32_t cur[8];
                {
                    const uint4 v0 = *reinterpret_cast<const uint4*>(row + (((2 * b) ^ sw) << 4));
                    const uint4 v1 = *reinterpret_cast<const uint4*>(row + (((2 * b + 1) ^ sw) << 4));
                    cur[0] = v0.x; cur[1] = v0.y; cur[2] = v0.z; cur[3] = v0.w;
                    cur[4] = v1.x; cur[5] = v1.y; cur[6] = v1.z; cur[7] = v1.w;
                }
                map_high_bytes(cur);
                const uint32_t nlm = newline_mask32(cur);
                // valid windows hold no '\n' (processFile resets the hash there); a stream past the job's end,
                // which reads zero-filled rows, has none
                uint32_t crossed;
                if constexpr (L > 0) {
                    crossed = window_has_newline<L>(nl_prev, nlm);
                } else {
                    crossed = window_has_newline<L == kLong>((int)rt_len, nl_prev2, nl_prev, nlm);
                    leaving_block<L>(prev2, prev, cur, (int)rt_len, leaving);
                }
                const uint32_t valid = active ? ~crossed : 0u;
                uint32_t pass = 0;
                uint32_t cl[kEntries ? 32 : 1], ch[kEntries ? 32 : 1];  // the block's S-box entries
#pragma unroll
                for (int j = 0; j < 32; j++) {
                    const uint2 sv = sbox_in(cur, j);
                    uint2 o;
                    if constexpr (kEntries) {
                        const uint32_t pl = j < L ? el[j < L ? j : 0] : cl[j < L ? 0 : j - L];
                        const uint32_t ph = j < L ? eh[j < L ? j : 0] : ch[j < L ? 0 : j - L];
                        o = make_uint2(__funnelshift_l(ph, pl, L), __funnelshift_l(pl, ph, L));
                        cl[j] = sv.x;
                        ch[j] = sv.y;
                    } else {
                        o = sbox_out(prev, cur, j);
                    }
                    const uint32_t nl = __funnelshift_l(hh, hl, 1), nh = __funnelshift_l(hl, hh, 1);
                    hl = nl ^ sv.x ^ o.x;
                    hh = nh ^ sv.y ^ o.y;
                    if constexpr (kSparse) {
                        // the second probe is loaded only where the first passes: its random words would cost the
                        // shared-memory pipe, which bounds this loop, another 3.5 wavefronts per warp
                        uint32_t w0, w1;
                        if constexpr (kHalves) {
                            w0 = lds16(half_addr(hh, s1)) * twice;
                            w1 = lds16_if(half_addr(hl, s1), (__funnelshift_r(w0, w0, hl) & 1u) != 0) * twice;
                            pass = __funnelshift_r(pass, __funnelshift_r(w1, w1, hh), 1);
                            continue;
                        }
                        w0 = lds32(s1 + ((hl >> 3) & s1_bmask));
                        w1 = lds32_if(s2 + ((hh >> 3) & s2_bmask), (__funnelshift_r(w0, w0, hl) & 1u) != 0);
                        pass = __funnelshift_r(pass, __funnelshift_r(w1, w1, hh), 1);  // the bit enters at bit 31
                    } else {
                        const int slot = j % kRing;
                        // The window that entered stage A kLag bytes ago leaves its last stage (a probe's bit sits
                        // at f & 31 in its word: region offsets are multiples of 32).
                        if constexpr (kPre) {
                            pass = __funnelshift_r(pass, __funnelshift_r(ring_v[slot], ring_v[slot], ring_a[slot]), 1);
                        } else {
                            pass = __funnelshift_r(pass, __funnelshift_r(ring2_v[slot], ring2_v[slot], ring2_b[slot]),
                                                   1);
                            // stage A: the window issued kRing bytes ago; its word has arrived by now
                            const bool pass1 = (__funnelshift_r(ring_v[slot], ring_v[slot], ring_a[slot]) & 1u) != 0;
                            ring2_b[slot] = ring_b[slot];
                            ring2_v[slot] = ldg_if(b_words + ((ring_b[slot] & b_mask) >> 5), pass1);
                        }
                        bool issue = (valid & (1u << j)) != 0;
                        if constexpr (kPre) {
                            // the table's bits: a clear one means the cache bit of f0 or f1 is clear too
                            const uint32_t w0 = lds32(s1 + ((hl >> 3) & s1_bmask));
                            const uint32_t w1 =
                                lds32_if(s2 + ((hh >> 3) & s2_bmask), (__funnelshift_r(w0, w0, hl) & 1u) != 0);
                            issue = issue && (__funnelshift_r(w1, w1, hh) & 1u) != 0;
                        }
                        ring_a[slot] = rot_const<kRot>(hl);
                        ring_b[slot] = rot_const<kRot>(hh);
                        ring_v[slot] = ldg_if(a_words + ((ring_a[slot] & a_mask) >> 5), issue);
                    }
                }
                if constexpr (kEntries) {
#pragma unroll
                    for (int q = 0; q < L; q++) {
                        el[q] = cl[32 - L + q];
                        eh[q] = ch[32 - L + q];
                    }
                }
                if constexpr (kSparse) enqueue(pass & valid, pos0 + (uint32_t)(32 * b));
                else enqueue(pass, pos0 + (uint32_t)(32 * b - kLag));
                if (nlm) {
                    const uint32_t at = pos0 + (uint32_t)(32 * b);
                    nl_span = min(nl_span & 0xffffu, at + (uint32_t)__ffs(nlm) - 1u) | (at + 31u - __clz(nlm)) << 16;
                }
                if constexpr (L == kLong) {
                    nl_prev2 = nl_prev;
#pragma unroll
                    for (int q = 0; q < 8; q++) prev2[q] = prev[q];
                }
                nl_prev = nlm;
#pragma unroll
                for (int q = 0; q < 8; q++) prev[q] = cur[q];
            }
            if (r == (int)R * kParts - 1) {
                if constexpr (!kSparse) {
                    // The rings carry over between a stream's parts and drain at its end: the last stage's slot q
                    // holds the window kLag - q bytes before the end; with two stages, stage A's survivors are queued
                    // with only their first probe known.
                    uint32_t rest = 0;
#pragma unroll
                    for (int q = 0; q < kRing; q++) {
                        const uint32_t a = (__funnelshift_r(ring_v[q], ring_v[q], ring_a[q]) & 1u) << q;
                        rest |= kPre ? a : (a << kRing) | (__funnelshift_r(ring2_v[q], ring2_v[q], ring2_b[q]) & 1u) << q;
                        ring_v[q] = 0;
                        ring2_v[q] = 0;
                    }
                    enqueue(rest, pos0 + (uint32_t)(kPart - kLag));
                }
                if (qn) flush();  // the queue keeps its candidates across the stream's parts, not across streams
                finish_streams<L, kHalves>(job_desc(), (uint64_t)st * THREADS + tid, nl_span, THREADS, lane_tab, error_flag);
            }
        }
        // this warp is done reading the stage
        __syncwarp();
        if (lane == 0) mbar_arrive(ebar(k));
    }
}

PFN_cuTensorMapEncodeTiled_v12000 encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    }
    return fn;
}

// static shared memory of k_scan_fast<., THREADS, .> (sequencer, current job, warp positions)
constexpr size_t static_smem(int threads) { return 8 * (size_t)(threads / 32) + 176; }

constexpr size_t fixed_smem(int threads, int table_bytes = kTabBytes) {
    return 1024 + 2 * (size_t)threads * kPart + table_bytes + 128 + (threads / 32) * 4 * (size_t)kQueueCap;
}

template <int L, int THREADS, int MODE>
cudaError_t launch_cfg(uint32_t len, const FastJob* d_jobs, uint32_t n_jobs, uint32_t n_items, uint32_t max_s1_words,
                       uint32_t* d_ctl, int num_sms, cudaStream_t st) {
    const size_t smem =
        fixed_smem(THREADS, tab_bytes(MODE, L)) + (sparse_mode(MODE) || MODE >= 3 ? 4 * (size_t)max_s1_words : 0);
    // the limit is the function's, not the launch's: one value, so that threads launching with different tables agree
    cudaError_t e = cudaFuncSetAttribute(k_scan_fast<L, THREADS, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)(kSmemLimit - static_smem(THREADS)));
    if (e != cudaSuccess) return e;
    const uint32_t slots = (uint32_t)num_sms * (uint32_t)ctas_per_sm(THREADS, MODE);
    const int grid = (int)(n_items < slots ? n_items : slots);
    if (grid == 0) return cudaSuccess;
    k_scan_fast<L, THREADS, MODE><<<grid, THREADS, smem, st>>>(d_jobs, n_jobs, n_items, max_s1_words, len, d_ctl);
    note_launches(1);
    return cudaGetLastError();
}

// The kernel of a configuration: its CTA size is config_threads(cfg), the size its descriptors' TMA boxes and work
// items were made for.
template <int L>
cudaError_t launch_len(uint32_t len, const FastConfig& cfg, const FastJob* d_jobs, uint32_t n_jobs, uint32_t n_items,
                       uint32_t max_s1_words, uint32_t* d_ctl, int num_sms, cudaStream_t st) {
    // kernel mode: 0 and 5 sparse, 1..4 dense in probe order 0..3
    const int mode = cfg.mode == 1 ? 1 + cfg.order : cfg.mode == 3 && cfg.halves ? 5 : 0;
    if constexpr (keeps_entries(5, L)) {
        if (mode == 5) switch (config_threads(cfg)) {
            case 192: return launch_cfg<L, 192, 5>(len, d_jobs, n_jobs, n_items, max_s1_words, d_ctl, num_sms, st);
            case 256: return launch_cfg<L, 256, 5>(len, d_jobs, n_jobs, n_items, max_s1_words, d_ctl, num_sms, st);
            case 384: return launch_cfg<L, 384, 5>(len, d_jobs, n_jobs, n_items, max_s1_words, d_ctl, num_sms, st);
            case 512: return launch_cfg<L, 512, 5>(len, d_jobs, n_jobs, n_items, max_s1_words, d_ctl, num_sms, st);
        }
    }
    switch (16 * config_threads(cfg) + mode) {
#define FFBF_CASE(T, M) \
    case 16 * T + M: return launch_cfg<L, T, M>(len, d_jobs, n_jobs, n_items, max_s1_words, d_ctl, num_sms, st)
        FFBF_CASE(192, 0);
        FFBF_CASE(256, 0);
        FFBF_CASE(384, 0);
        FFBF_CASE(512, 0);
        FFBF_CASE(192, 1);
        FFBF_CASE(256, 1);
        FFBF_CASE(384, 1);
        FFBF_CASE(192, 2);
        FFBF_CASE(256, 2);
        FFBF_CASE(384, 2);
        FFBF_CASE(256, 3);
        FFBF_CASE(384, 3);
        FFBF_CASE(256, 4);
        FFBF_CASE(384, 4);
#undef FFBF_CASE
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace

bool compiled_len(uint32_t len) { return len == 16 || len == 19 || len == 20 || len == 24 || len == 32; }

bool fast_scan_supported(const Geom& g, uint64_t n) {
    if (g.s < 1 && g.k < 2) return false;  // neither a cache-region probe nor two pipelined ones
    return n >= (uint64_t)kScanTile && encoder() != nullptr;
}

// Largest power-of-two stage-1 table (in bits, <= C) that fits beside the fixed shared-memory layout.
uint32_t stage1_shift_for(const Geom& g, int threads) {
    const size_t room = kSmemLimit - fixed_smem(threads) - static_smem(threads) - 64;
    uint32_t sh = 0;
    while (((uint64_t)g.cache_bits >> sh) / 8 > room) sh++;
    return sh;
}
// mode 3's table fits beside its largest CTAs (launch_config)
static_assert(kSmemLimit - fixed_smem(384) - static_smem(384) - 64 >= 131072, "384 threads: a 2^20-bit table");
static_assert(kSmemLimit - fixed_smem(512, kHalfTabBytes) - static_smem(512) - 64 >= 131072, "512: a 2^20-bit table");

// mode 3 reads the 384-thread table at every CTA size it takes
int table_threads(const FastConfig& cfg) { return cfg.mode == 3 ? 384 : config_threads(cfg); }

bool table_halves(const Geom& g) {
    return g.s >= 2 && compiled_len(g.len) && keeps_entries(0, (int)g.len) &&
           g.cache_bits >> stage1_shift_for(g, 384) == 1u << 20;
}

uint32_t stage1_words_for(const Geom& g, int threads) {
    return (uint32_t)(((uint64_t)g.cache_bits >> stage1_shift_for(g, threads)) / 32);
}

ScanChoice choose_scan(const Geom& g, double table_fill, double cache_fill, double ext_fill) {
    // Costs per window in units of one L2 probe per window (3.1 ps on the whole GPU: 148 SMs, each looking up one
    // random sector per clock). Measured against the model: words, 1M patterns, order 1: 354 GB/s; 150k printable
    // patterns in 2^23 + 2^27 bits, order 3: 547 GB/s (order 1: 323, mode 3: 309); 40k in 2^22 + 2^26, mode 3: 625,
    // order 3: 637; 50k in 2^24 + 2^28 (LEN 19), mode 3: 688, order 3: 601; 8k in 2^20 + 2^24, mode 3: 955, order 3:
    // 653 (before mode 3 read 16-bit entries, which gains it 4 to 8 %).
    // Orders 0 and 1: the first probe always, the second when the first passes, and a queued window's full test
    // (about three probes' worth of issue and flush work) when both pass. A probe of a region that the L1 left
    // beside the shared memory can largely hold (about 64 KiB) mostly hits there.
    const double c_bytes = g.cache_bits / 8.0, e_bytes = (g.ext_mask + 1.0) / 8.0;
    auto fill = [&](uint32_t i) { return i < g.s ? cache_fill : ext_fill; };
    auto miss = [&](uint32_t i) { return 1.0 - std::min(1.0, 65536.0 / (i < g.s ? c_bytes : e_bytes)); };
    auto cost = [&](uint32_t a, uint32_t b) {
        return std::max(0.45, miss(a) + fill(a) * miss(b) + 3.0 * fill(a) * fill(b));
    };
    ScanChoice best{1, 0};
    double best_cost = cost(0, 1);
    if (g.k >= 4 && cost(2, 3) < best_cost) {
        best.order = 1;
        best_cost = cost(2, 3);
    }
    // Orders 2 and 3: both table bits, then one L2 probe for the windows that pass. A bit of the prefiltered dense
    // kernel's table ORs C/T cache bits, so it is set with probability 1 - (1 - fill)^(C/T).
    auto both = [&](double f) { return g.s > 1 ? f * f : f; };
    const double pre_fill = 1.0 - std::pow(1.0 - cache_fill, (double)(1u << stage1_shift_for(g, 384)));
    const double pre = 0.48 + 1.45 * both(pre_fill);
    if (g.s > 0 && pre < best_cost) {
        best.order = g.k >= 4 ? 3 : 2;
        best_cost = pre;
    }
    // Sparse: both table bits; a window that passes costs its lane's queue append and its share of a flush, much more
    // of it where its exact first probe passes too (cache_fill / table_fill of them) and others follow.
    const double base = compiled_len(g.len) && keeps_entries(0, (int)g.len) ? 0.325 : 0.38;
    const double per_pass = 13.0 + 70.0 * cache_fill / std::max(table_fill, 1e-9);
    if (g.s > 0 && (g.k < 2 || base + both(table_fill) * per_pass <= best_cost)) best.mode = 3;
    return best;
}

int config_threads(const FastConfig& cfg) {
    if (cfg.mode == 1) return cfg.threads == 256 ? 256 : cfg.threads == 192 && cfg.order < 2 ? 192 : 384;
    if (cfg.mode == 2) return cfg.threads == 192 || cfg.threads == 384 ? cfg.threads : 256;
    if (cfg.mode == 3)  // launch_config fits the size to the text
        return cfg.threads == 192 || cfg.threads == 256 || cfg.threads == 384 ? cfg.threads : 512;
    return cfg.threads == 384 || cfg.threads == 512 ? cfg.threads : 256;
}

int fast_ctas_per_sm(const FastConfig& cfg) { return cfg.mode == 1 && config_threads(cfg) == 192 ? 2 : 1; }

uint32_t fast_tile_bytes(uint32_t rows) {
    uint32_t streams = 1;
    while (streams < 32 && streams * rows * kRowBytes < (uint32_t)kScanTile) streams *= 2;
    return streams * rows * kRowBytes;
}

FastConfig launch_config(const FastConfig& cfg, uint32_t len, uint64_t n, int num_sms, bool batch) {
    // Mode 3's CTA sizes, the largest first, and the time of a step in which each of its threads takes a byte (ns; 4
    // GiB plain text, and 2 GiB at LEN 21 and 32; with 16-bit entries about 7 % less, all sizes alike). The kernel that
    // keeps its S-box entries in registers leaves room for its table beside 512 threads; the others take 384 at most:
    // with half the table 640 threads scanned 2 GiB at 712 GB/s (LEN 21) and 840 (32), 384 with the whole one at 803 and
    // 887.
    struct Size {
        int threads;
        double tau;
    };
    static const Size kept[] = {{512, 76.3}, {384, 59.1}, {256, 46.3}, {192, 45.1}};
    static const Size read[] = {{384, 68.0}, {256, 52.0}, {192, 49.0}};
    const bool keeps = compiled_len(len) && keeps_entries(0, (int)len);
    const Size* sizes = keeps ? kept : read;
    FastConfig best = cfg;
    if (batch) {
        // other jobs fill the GPU
        if (cfg.mode == 3) best.threads = sizes[0].threads;
        best.rows = fast_rows(n, best, num_sms, true);
        return best;
    }
    // Alone, the scan lasts as many waves of equal items as the busiest CTA slot takes; an item costs its rows and
    // about 16 steps more. With powers of two from 4 rows and 512 or 768 threads only, 64 MiB took 131 us (now 84), 8
    // MiB 114 (29).
    constexpr double kItemBytes = 16.0;
    double best_cost = 0;
    const uint32_t min_rows = n < kShortRowsText ? 1 : 4;
    for (int i = 0; i < (cfg.mode != 3 ? 1 : keeps ? 4 : 3); i++) {
        FastConfig c = cfg;
        if (cfg.mode == 3) c.threads = sizes[i].threads;
        const uint64_t threads = config_threads(c), slots = (uint64_t)num_sms * fast_ctas_per_sm(c);
        for (uint32_t rows = 16; rows >= min_rows; rows--) {
            const uint64_t items = (n / (rows * kRowBytes) + threads - 1) / threads;
            const double cost = (double)((items + slots - 1) / slots) * (rows * kRowBytes + kItemBytes) * sizes[i].tau;
            if (best_cost == 0 || cost < best_cost) {
                best_cost = cost;
                best = c;
                best.rows = rows;
            }
        }
    }
    return best;
}

uint32_t fast_rows(uint64_t n, const FastConfig& cfg, int num_sms, bool batch) {
    const int threads = config_threads(cfg);
    const uint64_t tiles_bytes = n / kScanTile * kScanTile;
    if (batch) {
        // in a batch other jobs fill the GPU: the largest tile this job still fills four times over
        uint32_t rows = 16;
        while (rows > 4 && tiles_bytes < 4ull * rows * kRowBytes * threads) rows >>= 1;
        return rows;
    }
    // alone: waves of equal items over the CTA slots, an item its rows and a quarter row for its halo; the row count
    // with the least work wins, ties go to the longer items
    const uint64_t slots = (uint64_t)num_sms * (uint64_t)fast_ctas_per_sm(cfg);
    uint32_t best = 16;
    uint64_t best_cost = ~0ull;
    for (uint32_t rows = 16; rows >= 4; rows >>= 1) {
        const uint64_t items = (tiles_bytes / ((uint64_t)rows * kRowBytes) + threads - 1) / threads;
        const uint64_t cost = (items + slots - 1) / slots * (4 * rows + 1);  // in quarter rows
        if (cost < best_cost) {
            best_cost = cost;
            best = rows;
        }
    }
    return best;
}

cudaError_t fill_fast_job(const ScanArgs& a, const uint32_t* stage1_words, const FastConfig& cfg, FastJob* job) {
    const int threads = config_threads(cfg);
    const uint32_t rows = cfg.rows;
    const uint64_t slen = (uint64_t)rows * kRowBytes;
    const uint64_t n_streams = rows ? a.n / slen : 0;
    if (n_streams == 0 || a.tile_bytes != fast_tile_bytes(rows)) return cudaErrorInvalidValue;
    memset(job, 0, sizeof *job);
    job->n_streams = n_streams;
    job->rows = rows;
    job->n_supertiles = (uint32_t)((n_streams + threads - 1) / threads);
    while ((slen << job->streams_per_tile_log2) < a.tile_bytes) job->streams_per_tile_log2++;
    job->g = a.g;
    job->main_words = a.main_words;
    job->ff_words = a.ff_words;
    job->text = a.text;
    // the table the kernel reads: the sparse mode's, or the dense mode's prefilter (order 2)
    const bool reads_table = cfg.mode != 1 || cfg.order >= 2;
    job->stage1_shift = reads_table ? stage1_shift_for(a.g, table_threads(cfg)) : 0;
    job->stage1_nwords = reads_table ? (uint32_t)(((uint64_t)a.g.cache_bits >> job->stage1_shift) / 32) : 0;
    job->stage1_words = stage1_words + (cfg.mode == 3 && cfg.halves ? job->stage1_nwords : 0u);
    {
        // dense mode: regions of the pipelined probes, index functions f0/f1 (order 0) or f2/f3 (order 1,
        // which only K >= 4 filters set)
        if (cfg.mode < 0 || cfg.mode > 3 ||
            (cfg.mode == 1 && (a.g.k < 2 || ((cfg.order & 1) && a.g.k < 4) || cfg.order < 0 || cfg.order > 3)))
            return cudaErrorInvalidValue;
        const uint32_t fa = (cfg.order & 1) ? 2u : 0u, fb = fa + 1;
        job->a_mask = fa < a.g.s ? a.g.cache_mask : a.g.ext_mask;
        job->a_add = fa < a.g.s ? 0u : a.g.cache_bits;
        job->b_mask = fb < a.g.s ? a.g.cache_mask : a.g.ext_mask;
        job->b_add = fb < a.g.s ? 0u : a.g.cache_bits;
    }
    job->hits = a.hits;
    job->hits_cap = a.hits_cap;
    job->counters = a.counters;
    job->tile_first_nl = a.tile_first_nl;
    job->tile_last_nl = a.tile_last_nl;
    job->n = a.n;
    job->n_tiles = a.ntiles;
    // FFBF_TEXT_L2=normal keeps the default L2 policy for the text's loads (for comparisons)
    static const bool evict_first = [] {
        const char* v = getenv("FFBF_TEXT_L2");
        return !(v && strcmp(v, "normal") == 0);
    }();
    job->text_evict_first = evict_first ? 1u : 0u;
    cuuint64_t dims[3] = {(cuuint64_t)kRowBytes, (cuuint64_t)rows, (cuuint64_t)n_streams};
    cuuint64_t strides[2] = {(cuuint64_t)kRowBytes, (cuuint64_t)slen};
    cuuint32_t box[3] = {(cuuint32_t)kPart, 1u, (cuuint32_t)box_streams_for(threads)};
    cuuint32_t estr[3] = {1u, 1u, 1u};
    const CUresult cr = encoder()(&job->tmap, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, (void*)a.text, dims, strides, box, estr,
                                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B,
                                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return cr == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

cudaError_t launch_fast_jobs(uint32_t len, const FastConfig& cfg, const FastJob* d_jobs, uint32_t n_jobs,
                             uint32_t n_items, uint32_t max_s1_words, uint32_t* d_ctl, int num_sms,
                             cudaStream_t st) {
    switch (len) {
        case 16: return launch_len<16>(len, cfg, d_jobs, n_jobs, n_items, max_s1_words, d_ctl, num_sms, st);
        case 19: return launch_len<19>(len, cfg, d_jobs, n_jobs, n_items, max_s1_words, d_ctl, num_sms, st);
        case 20: return launch_len<20>(len, cfg, d_jobs, n_jobs, n_items, max_s1_words, d_ctl, num_sms, st);
        case 24: return launch_len<24>(len, cfg, d_jobs, n_jobs, n_items, max_s1_words, d_ctl, num_sms, st);
        case 32: return launch_len<32>(len, cfg, d_jobs, n_jobs, n_items, max_s1_words, d_ctl, num_sms, st);
    }
    if (len < 1 || len > 63) return cudaErrorInvalidValue;
    if (len < 32) return launch_len<kShort>(len, cfg, d_jobs, n_jobs, n_items, max_s1_words, d_ctl, num_sms, st);
    return launch_len<kLong>(len, cfg, d_jobs, n_jobs, n_items, max_s1_words, d_ctl, num_sms, st);
}

cudaError_t scan_fast(const ScanArgs& a, const uint32_t* stage1_words, const FastConfig& cfg, int num_sms,
                      uint8_t* h_block, cudaStream_t st) {
    FastJob* h_job = reinterpret_cast<FastJob*>(h_block + kJobOffset);
    cudaError_t e = fill_fast_job(a, stage1_words, cfg, h_job);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(a.counters, h_block, kJobOffset + sizeof(FastJob), cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) return e;
    const FastJob* d_job = reinterpret_cast<const FastJob*>(reinterpret_cast<uint8_t*>(a.counters) + kJobOffset);
    return launch_fast_jobs(a.g.len, cfg, d_job, 1, h_job->n_supertiles, h_job->stage1_nwords, a.counters + CNT_ERROR,
                            num_sms, st);  // ctl = {CNT_ERROR, CNT_QUEUE}
}

// Stage-1 table of T = C >> sh bits for the sparse mode: bit j = OR of the cache bits i with i mod T == j
// (a fold, so the table index of a window is just h & (T-1)). A window passes the reference test only if
// its cache bit is set, which sets its table bit: the table rejects only windows the full test rejects.
__global__ void k_stage1_fold(const uint32_t* main_words, uint32_t sh, uint32_t* out, uint32_t nwords) {
    uint32_t w = blockIdx.x * blockDim.x + threadIdx.x;
    if (w >= nwords) return;
    uint32_t v = 0;
    const uint32_t folds = 1u << sh;
    for (uint32_t m = 0; m < folds; m++) v |= main_words[w + m * nwords];
    out[w] = v;
}

// The same 2^20 bits as 65536 entries of 16: bit i of the table is bit i >> 16 of entry i & 0xFFFF. A warp turns 64
// entries: lane l reads the words of 32 of them in one sixteenth of the table, and 32 votes collect the entries.
__global__ void k_stage1_halves(const uint32_t* table, uint32_t* out) {
    const uint32_t lane = threadIdx.x & 31, k = 2 * (blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32);
    const uint32_t w = table[(lane & 15) * 2048 + k + (lane >> 4)];
    uint32_t v = 0;
#pragma unroll
    for (uint32_t t = 0; t < 32; t++) {
        const uint32_t m = __ballot_sync(0xffffffffu, (w >> t) & 1u);
        const uint32_t e = lane < 16 ? m & 0xffffu : m >> 16;
        if ((lane & 15) == t / 2) v |= t & 1 ? e << 16 : e;
    }
    out[(k + (lane >> 4)) * 16 + (lane & 15)] = v;
}

cudaError_t build_stage1(const uint32_t* main_words, const Geom& g, int threads, uint32_t* out, cudaStream_t st) {
    const uint32_t sh = stage1_shift_for(g, threads);
    const uint32_t nwords = (uint32_t)(((uint64_t)g.cache_bits >> sh) / 32);
    if (sh == 0) {
        cudaError_t e = cudaMemcpyAsync(out, main_words, 4ull * nwords, cudaMemcpyDeviceToDevice, st);
        if (e != cudaSuccess) return e;
    } else {
        k_stage1_fold<<<(nwords + 255) / 256, 256, 0, st>>>(main_words, sh, out, nwords);
        note_launches(1);
    }
    if (threads == 384 && table_halves(g)) {
        k_stage1_halves<<<128, 256, 0, st>>>(out, out + nwords);  // 1024 warps
        note_launches(1);
    }
    return cudaGetLastError();
}

}  // namespace ffbf

namespace ffbf {

__global__ void k_popcount(const uint32_t* w, uint32_t n, unsigned long long* out) {
    unsigned long long c = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) c += __popc(w[i]);
    for (int o = 16; o; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(out, c);
}

cudaError_t popcount_words(const uint32_t* w, uint32_t n, unsigned long long* d_out, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(d_out, 0, sizeof(unsigned long long), st);
    if (e != cudaSuccess || n == 0) return e;
    k_popcount<<<(n + 255) / 256 < 1024 ? (n + 255) / 256 : 1024, 256, 0, st>>>(w, n, d_out);
    note_launches(1);
    return cudaGetLastError();
}

}  // namespace ffbf
