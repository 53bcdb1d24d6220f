// ffbf_text.cuh -- device helpers on text bytes: the search for a window's line ends and the exact byte compare of a
// hit window with its candidate patterns.
#pragma once
#include <climits>

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

// The ends of the line of the window at w, searched by eight lanes of a warp: lanes 0-3 go back from the byte before
// the window, 64 bytes a step, and return the line's start; lanes 4-7 go forward from the byte behind it and return its
// end. -1 when the tile of that first byte holds no '\n' on that side. One thread per window took 16-byte steps, each a
// memory latency, and its warp as long as its longest line.
__device__ __forceinline__ long long line_end_of_window(const uint8_t* text, uint64_t text_len, uint32_t len,
                                                        uint32_t tile_bytes, uint64_t w, bool active) {
    const bool back = (threadIdx.x & 4) == 0;
    const long long n = (long long)text_len;
    const long long pos = back ? (long long)w - 1 : (long long)(w + len);
    const long long tile = pos / tile_bytes * tile_bytes;
    const long long stop = back ? tile : min(n, tile + tile_bytes);
    long long res = -1, c = (pos & ~63LL) + 16 * (threadIdx.x & 3);
    bool busy = active;
    if (back ? pos < 0 : pos >= n) {  // the text's first and last byte end a line
        res = back ? 0 : n;
        busy = false;
    }
    while (__any_sync(0xffffffffu, busy)) {
        long long at = back ? -1 : LLONG_MAX;
        if (busy && c < n) {
            const uint4 v = chunk16(text, c, n);
            const uint32_t m8 = __dp4a(nl_bytes(v.y), 0x80402010u, __dp4a(nl_bytes(v.x), 0x08040201u, 0u)) >> 7;
            const uint32_t m16 = __dp4a(nl_bytes(v.w), 0x80402010u, __dp4a(nl_bytes(v.z), 0x08040201u, 0u)) << 1;
            uint32_t m = m8 | m16;
            // bytes on the searched side of pos, and before `stop` going forward
            if (back) m &= pos - c >= 15 ? 0xffffu : pos < c ? 0u : (2u << (pos - c)) - 1u;
            else m &= (pos <= c ? 0xffffu : pos - c >= 16 ? 0u : 0xffffu << (pos - c)) &
                      (stop - c >= 16 ? 0xffffu : stop <= c ? 0u : (1u << (stop - c)) - 1u);
            if (m) at = c + (back ? 31 - __clz(m) : __ffs(m) - 1);
        }
        for (int d = 1; d < 4; d <<= 1) {
            const long long o = __shfl_xor_sync(0xffffffffu, at, d);
            at = back ? max(at, o) : min(at, o);
        }
        if (busy) {
            if (back ? at >= 0 : at != LLONG_MAX) {
                res = back ? at + 1 : at;
                busy = false;
            } else {
                c += back ? -64 : 64;
                busy = back ? (c & ~63LL) >= stop : (c & ~63LL) < stop;
            }
        }
    }
    // a last line without '\n' ends with the text
    return !back && res < 0 && stop == n ? n : res;
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
