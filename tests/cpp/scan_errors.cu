// Error flags of a scan: whatever path collects it, a flag that its kernel raised is reported and no result is kept, and
// the context then scans as before. The flags are set here behind the scan, in the context's own counters. Prints each
// failure and exits non-zero on any.
#include <cstdio>
#include <string>
#include <vector>

#include "ffbf_ctx.cuh"

namespace {

int failures = 0;

void expect(const char* what, long long got, long long want) {
    if (got != want) {
        std::printf("FAIL %s: got %lld, want %lld\n", what, got, want);
        failures++;
    }
}

// Scans a text of n_hits lines, each holding the pattern, and collects it with `flag` raised.
void check(bool host_order, size_t n_hits) {
    const std::string pattern = "a pattern of thirty characters";
    std::string text;
    for (size_t i = 0; i < n_hits; i++) text += pattern + "\n";
    text.resize(std::max<size_t>(text.size(), 100000), '.');
    const ffbf_params prm{20, 5, 2, 0, 1 << 20, 1 << 24};
    ffbf_ctx* c = nullptr;
    expect("create", ffbf_create(&prm, 0, &c), FFBF_OK);
    if (!c) return;
    c->host_order = host_order;
    expect("patterns", ffbf_add_patterns(c, (const uint8_t*)pattern.data(), pattern.size()), FFBF_OK);
    uint8_t* d_text = nullptr;
    cudaMalloc(&d_text, text.size());
    cudaMemcpy(d_text, text.data(), text.size(), cudaMemcpyHostToDevice);
    for (const auto& [flag, status] : std::vector<std::pair<uint32_t, ffbf_status>>{
             {4u, FFBF_ETIMEOUT}, {0x100u, FFBF_ECUDA}, {0x200u, FFBF_ECUDA}, {0u, FFBF_OK}}) {
        ffbf_scan_result r{};
        expect("scan", ffbf_scan_device(c, d_text, text.size()), FFBF_OK);
        cudaStreamSynchronize(c->st);
        if (flag) cudaMemcpy(c->d_counters + ffbf::CNT_ERROR, &flag, 4, cudaMemcpyHostToDevice);
        expect("collect", ffbf_scan_collect(c, &r), status);
        if (flag) expect("collect again", ffbf_scan_collect(c, &r), FFBF_ESTATE);
        else expect("windows", (long long)r.n_hits, (long long)n_hits);
    }
    cudaFree(d_text);
    ffbf_destroy(c);
}

}  // namespace

int main() {
    for (bool host_order : {false, true})
        for (size_t n : {size_t(3), size_t(3000), size_t(20000), size_t(70000)})  // rooms: 2048, 16384, 65536
            check(host_order, n);
    if (failures == 0) std::printf("scan errors: all checks passed\n");
    return failures ? 1 : 0;
}
