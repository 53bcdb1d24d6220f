// Host-only checks of the rules that size a tuned scan's launch (no device is touched): the CTA size and rows that
// launch_config gives a lone text and a batch's job, the newline tile that follows from them and the room for its
// summaries, and the refusal of a descriptor without rows. Prints each failure and exits non-zero on any.
#include <cstdio>

#include "ffbf_ctx.cuh"

namespace {

int failures = 0;

void expect(const char* what, unsigned long long n, unsigned long long got, unsigned long long want) {
    if (got != want) {
        std::printf("FAIL %s (%llu): got %llu, want %llu\n", what, n, got, want);
        failures++;
    }
}

}  // namespace

int main() {
    using ffbf::FastConfig;
    const int sms = 148;
    const FastConfig sparse{512, 3, 0, 0}, fixed{384, 0, 0, 0}, dense{192, 1, 0, 1}, prefiltered{384, 1, 0, 3};
    // lone texts: the least waves x (item + 16 steps) x time of a step, worked out by hand
    expect("1 GiB, threads", 0, ffbf::launch_config(sparse, 20, 1ull << 30, sms, false).threads, 512);
    expect("64 MiB, threads", 0, ffbf::launch_config(sparse, 20, 64ull << 20, sms, false).threads, 512);
    expect("64 MiB, rows", 0, ffbf::launch_config(sparse, 20, 64ull << 20, sms, false).rows, 7);
    expect("16 KiB, threads", 0, ffbf::launch_config(sparse, 20, 16384, sms, false).threads, 192);
    expect("16 KiB, rows", 0, ffbf::launch_config(sparse, 20, 16384, sms, false).rows, 1);
    expect("run-time LEN, threads", 0, ffbf::launch_config(sparse, 21, 1ull << 30, sms, false).threads, 384);
    expect("batch, threads", 0, ffbf::launch_config(sparse, 20, 1 << 20, sms, true).threads, 512);
    expect("batch, run-time LEN", 0, ffbf::launch_config(sparse, 21, 1 << 20, sms, true).threads, 384);
    expect("batch, rows", 0, ffbf::launch_config(sparse, 20, 64ull << 20, sms, true).rows, 16);
    // every size: a stream at least, no more rows than a tile is made for, and room for the tiles' summaries
    for (const FastConfig& cfg : {sparse, fixed, dense, prefiltered})
        for (uint32_t len : {16u, 20u, 32u, 1u, 63u})
            for (unsigned long long n = 16384; n < 10ull << 30; n += n / 7 + 1)
                for (bool batch : {false, true}) {
                    const FastConfig c = ffbf::launch_config(cfg, len, n, sms, batch);
                    expect("rows in range", n, c.rows >= 1 && c.rows <= 16, 1);
                    expect("mode kept", n, c.mode == cfg.mode && c.order == cfg.order, 1);
                    if (cfg.mode != 3) expect("threads kept", n, c.threads, cfg.threads);
                    const uint64_t tile = ffbf::fast_tile_bytes(c.rows);
                    expect("whole streams per tile", n, tile % (c.rows * 128), 0);
                    expect("room for the tiles", n, (n + tile - 1) / tile <= ffbf_host::tiles_for(n), 1);
                }
    ffbf::ScanArgs a{};
    a.n = 1 << 20;
    ffbf::FastJob job;
    for (uint32_t tile : {uint32_t(ffbf::kScanTile), ffbf::fast_tile_bytes(0)}) {
        a.tile_bytes = tile;
        expect("no rows", tile, ffbf::fill_fast_job(a, nullptr, sparse, &job), cudaErrorInvalidValue);
    }
    if (failures == 0) std::printf("launch rules: all checks passed\n");
    return failures ? 1 : 0;
}
