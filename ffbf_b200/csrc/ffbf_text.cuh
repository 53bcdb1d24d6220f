// ffbf_text.cuh -- device helpers on text bytes: the search for a window's line ends and the exact byte compare of a
// hit window with its candidate patterns.
#pragma once
#include "ffbf_kernels.cuh"

namespace ffbf {

// Byte masks of '\n' in a 32-bit word (0x80 in each byte that is '\n'; no false positives).
__device__ __forceinline__ uint32_t nl_bytes(uint32_t w) {
    const uint32_t t = w ^ 0x0A0A0A0Au;
    return ~(((t & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | t) & 0x80808080u;
}

// The aligned 16 bytes of `text` at c (c a multiple of 16, c < n). The last, partial chunk of a text whose
// length is not a multiple of 16 is read byte by byte, zero-filled past n, so nothing beyond the text is read.
__device__ __forceinline__ uint4 chunk16(const uint8_t* text, long long c, long long n) {
    if (c + 16 <= n) return __ldg(reinterpret_cast<const uint4*>(text + c));
    uint32_t w[4] = {0u, 0u, 0u, 0u};
    for (int i = 0; i < 16 && c + i < n; i++) w[i >> 2] |= (uint32_t)__ldg(text + c + i) << (8 * (i & 3));
    return make_uint4(w[0], w[1], w[2], w[3]);
}

// Last '\n' in [lo, p] (lo <= p < n), or -1: aligned 16-byte chunks from p down to lo.
__device__ __forceinline__ long long last_nl_back(const uint8_t* text, long long n, long long lo, long long p) {
    while (p >= lo) {
        const long long c = p & ~15LL;
        const uint4 v = chunk16(text, c, n);
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
        // bytes of the chunk at offsets max(lo - c, 0) .. p - c
        const int hi = (int)(p - c), low = (int)max(lo - c, 0LL);
        for (int q = hi >> 2; q >= (low >> 2); q--) {
            uint32_t m = nl_bytes(w[q]);
            // keep byte positions 4q + b with low <= 4q + b <= hi
            const int b_hi = min(hi - 4 * q, 3), b_lo = max(low - 4 * q, 0);
            m &= (0xFFFFFFFFu >> (8 * (3 - b_hi))) & (0xFFFFFFFFu << (8 * b_lo));
            if (m) return c + 4 * q + (31 - __clz(m)) / 8;
        }
        p = c - 1;
    }
    return -1;
}

// First '\n' in [q, hi) (q < hi <= n), or -1: aligned 16-byte chunks from q up to hi.
__device__ __forceinline__ long long first_nl_fwd(const uint8_t* text, long long n, long long q, long long hi) {
    while (q < hi) {
        const long long c = q & ~15LL;
        const uint4 v = chunk16(text, c, n);
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
        const int low = (int)(q - c), top = (int)min(hi - c, 16LL) - 1;  // offsets low .. top
        for (int k = low >> 2; k <= (top >> 2); k++) {
            uint32_t m = nl_bytes(w[k]);
            const int b_lo = max(low - 4 * k, 0), b_hi = min(top - 4 * k, 3);
            m &= (0xFFFFFFFFu << (8 * b_lo)) & (0xFFFFFFFFu >> (8 * (3 - b_hi)));
            if (m) return c + 4 * k + (__ffs(m) - 1) / 8;
        }
        q = c + 16;
    }
    return -1;
}

// Start of the line that holds offset w: one past the last '\n' before w in that '\n's tile, 0 at the text's start, or -1
// when the tile of w - 1 holds none before w.
__device__ __forceinline__ long long line_start_in_tile(const uint8_t* text, uint64_t n, uint64_t w,
                                                        uint32_t tile_bytes) {
    if (w == 0) return 0;
    const long long p =
        last_nl_back(text, (long long)n, (long long)((w - 1) / tile_bytes * tile_bytes), (long long)w - 1);
    return p >= 0 ? p + 1 : -1;
}

// End of the line whose bytes before q hold no '\n' back to the window: the first '\n' at or after q in q's tile, n
// when q is the text's end, or -1 when that tile holds none.
__device__ __forceinline__ long long line_end_in_tile(const uint8_t* text, uint64_t n, uint64_t q,
                                                      uint32_t tile_bytes) {
    if (q >= n) return (long long)n;
    const uint64_t hi = min(n, (q / tile_bytes + 1) * (uint64_t)tile_bytes);
    return first_nl_fwd(text, (long long)n, (long long)q, (long long)hi);
}

// Slot hash of the verification multimap.
__device__ __forceinline__ uint64_t mix64(uint64_t x) {
    x ^= x >> 33;
    x *= 0xff51afd7ed558ccdull;
    x ^= x >> 33;
    x *= 0xc4ceb9fe1a85ec53ull;
    return x ^ (x >> 33);
}

// The 16 bytes at p (any alignment), of which the first `need` (1..16) are used, read as aligned 16-byte
// loads: the chunk holding p, and the next one only when the bytes reach into it. An aligned chunk that holds a
// needed byte never crosses a page, so no load leaves the buffer's pages.
__device__ __forceinline__ uint4 load16_unaligned(const uint8_t* p, uint32_t need) {
    const uintptr_t a = (uintptr_t)p;
    const uint4* base = reinterpret_cast<const uint4*>(a & ~(uintptr_t)15);
    const uint32_t off = (uint32_t)(a & 15);
    const uint4 x0 = __ldg(base);
    const uint4 x1 = off + need > 16 ? __ldg(base + 1) : make_uint4(0, 0, 0, 0);
    const uint32_t ws = off >> 2, bs = (off & 3) * 8;
    // words ws .. ws + 4 of x0:x1, selected without a runtime-indexed array
    uint32_t w0, w1, w2, w3, w4;
    if (ws == 0) { w0 = x0.x; w1 = x0.y; w2 = x0.z; w3 = x0.w; w4 = x1.x; }
    else if (ws == 1) { w0 = x0.y; w1 = x0.z; w2 = x0.w; w3 = x1.x; w4 = x1.y; }
    else if (ws == 2) { w0 = x0.z; w1 = x0.w; w2 = x1.x; w3 = x1.y; w4 = x1.z; }
    else { w0 = x0.w; w1 = x1.x; w2 = x1.y; w3 = x1.z; w4 = x1.w; }
    return make_uint4(__funnelshift_r(w0, w1, bs), __funnelshift_r(w1, w2, bs), __funnelshift_r(w2, w3, bs),
                      __funnelshift_r(w3, w4, bs));
}

// mask of the bytes of 32-bit word i that fall within the first `need` bytes of a 16-byte block
__device__ __forceinline__ uint32_t word_mask(uint32_t need, uint32_t i) {
    const uint32_t v = need > 4 * i ? min(need - 4 * i, 4u) : 0u;
    return v >= 4 ? 0xffffffffu : (1u << (8 * v)) - 1u;
}

// Looks one hit window's hash up in the pruned patterns' multimap (open addressing, empty value 0xffffffff) and
// appends (offset, pattern id) for every candidate whose bytes occur at the window's start.
__device__ __forceinline__ void verify_window(const HitRec& hit, const uint8_t* text, uint64_t n, const uint64_t* keys,
                                              const uint32_t* vals, uint64_t mask, const uint8_t* pat,
                                              const uint64_t* pstart, const uint64_t* pend, uint64_t* m_off,
                                              uint32_t* m_pid, uint32_t cap, uint32_t* counters) {
    const uint64_t w = hit.off, h = hit.h;
    uint64_t slot = mix64(h) & mask;
    for (uint64_t probe = 0; probe <= mask; probe++) {
        uint32_t id = vals[slot];
        if (id == 0xffffffffu) break;
        if (keys[slot] == h) {
            uint64_t ps = pstart[id], pl = pend[id] - ps;
            if (w + pl <= n) {
                const uint8_t* t = text + w;
                const uint8_t* q = pat + ps;
                // byte compare, 16 bytes per step from aligned 16-byte loads of both sides
                bool same = true;
                for (uint64_t k = 0; k < pl && same; k += 16) {
                    const uint32_t need = pl - k < 16 ? (uint32_t)(pl - k) : 16u;
                    const uint4 x = load16_unaligned(t + k, need), y = load16_unaligned(q + k, need);
                    same = (((x.x ^ y.x) & word_mask(need, 0)) | ((x.y ^ y.y) & word_mask(need, 1)) |
                            ((x.z ^ y.z) & word_mask(need, 2)) | ((x.w ^ y.w) & word_mask(need, 3))) == 0;
                }
                if (same) {
                    uint32_t o = atomicAdd(counters + CNT_MATCHES, 1u);
                    if (o < cap) {
                        m_off[o] = w;
                        m_pid[o] = id;
                    }
                }
            }
        }
        slot = (slot + 1) & mask;
    }
}

}  // namespace ffbf
