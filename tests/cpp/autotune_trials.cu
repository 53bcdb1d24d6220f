// The autotuner's trial scans run as what they are for runs: with a batch's rows per stream in ffbf_batch_autotune, with a
// lone scan's in ffbf_autotune. A 1 MiB sample tells them apart by the newline tile of the last trial. Prints each failure
// and exits non-zero on any.
#include <cstdio>
#include <string>

#include "ffbf_ctx.cuh"

namespace {

int failures = 0;

void expect(const char* what, long long got, long long want) {
    if (got != want) {
        std::printf("FAIL %s: got %lld, want %lld\n", what, got, want);
        failures++;
    }
}

}  // namespace

int main() {
    const size_t n = 1 << 20;
    const std::string pattern = "a pattern of thirty characters", text(n, '.');
    const ffbf_params prm{20, 5, 2, 0, 1 << 20, 1 << 24};
    ffbf_ctx* c = nullptr;
    ffbf_batch* b = nullptr;
    expect("create", ffbf_create(&prm, 0, &c), FFBF_OK);
    expect("create batch", ffbf_batch_create(0, &b), FFBF_OK);
    if (failures) return 1;
    expect("patterns", ffbf_add_patterns(c, (const uint8_t*)pattern.data(), pattern.size()), FFBF_OK);
    uint8_t* d_text = nullptr;
    cudaMalloc(&d_text, n);
    cudaMemcpy(d_text, text.data(), n, cudaMemcpyHostToDevice);
    const auto tile = [&](bool batch) {
        const ffbf::FastConfig last{256, 1, 0, 0};  // the last configuration tried; its rows follow CTA size and text
        return ffbf::fast_tile_bytes(ffbf::launch_config(last, 20, n, c->num_sms, batch).rows);
    };
    expect("the tiles differ", tile(true) != tile(false), 1);
    int threads, mode;
    uint32_t classes;
    expect("autotune", ffbf_autotune(c, d_text, n, &threads, &mode), FFBF_OK);
    expect("tile of a lone trial", c->tile_bytes, tile(false));
    expect("add", ffbf_batch_add(b, c, d_text, n), FFBF_OK);
    expect("batch autotune", ffbf_batch_autotune(b, n, &classes), FFBF_OK);
    expect("tile of a batch's trial", c->tile_bytes, tile(true));
    ffbf_batch_destroy(b);
    cudaFree(d_text);
    ffbf_destroy(c);
    if (failures == 0) std::printf("autotune trials: all checks passed\n");
    return failures ? 1 : 0;
}
