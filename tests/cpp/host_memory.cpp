// Host memory that runs out inside an entry point: the call returns FFBF_ENOMEM_HOST instead of throwing through the C
// interface, and made again with memory at hand it gives the whole result. This program's operator new fails for blocks of
// `limit` bytes or more. Prints each failure and exits non-zero on any.
#include <cstdio>
#include <cstdlib>
#include <new>
#include <string>

#include <cuda_runtime.h>

#include "ffbf.h"

static size_t limit = ~size_t(0);

void* operator new(size_t n) {
    void* p = n < limit ? std::malloc(n ? n : 1) : nullptr;
    if (!p) throw std::bad_alloc();
    return p;
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

namespace {

int failures = 0;

void expect(const char* what, long long got, long long want) {
    if (got != want) {
        std::printf("FAIL %s: got %lld, want %lld\n", what, got, want);
        failures++;
    }
}

// Calls f once with blocks of 4 KiB and more refused, and once with memory.
template <class F>
void twice(const char* what, F f) {
    limit = 4096;
    const int first = f();
    limit = ~size_t(0);
    expect(what, first, FFBF_ENOMEM_HOST);
    expect(what, f(), FFBF_OK);
}

}  // namespace

int main() {
    const std::string pattern = "a pattern of thirty characters";
    const ffbf_params prm{20, 5, 2, 0, 1 << 20, 1 << 24};
    for (size_t n : {size_t(3000), size_t(40000)}) {  // results of one launch, and larger ones
        std::string text, patterns;
        for (size_t i = 0; i < n; i++) text += pattern + "\n";
        for (int i = 0; i < 1000; i++) patterns += pattern + "\n";
        ffbf_ctx* c = nullptr;
        expect("create", ffbf_create(&prm, 0, &c), FFBF_OK);
        if (!c) return 1;
        expect("patterns", ffbf_add_patterns(c, (const uint8_t*)patterns.data(), patterns.size()), FFBF_OK);
        uint8_t* d_text = nullptr;
        cudaMalloc(&d_text, text.size());
        cudaMemcpy(d_text, text.data(), text.size(), cudaMemcpyHostToDevice);
        ffbf_scan_result r{};
        ffbf_prune_result pr{};
        ffbf_matches m{};
        expect("scan", ffbf_scan_device(c, d_text, text.size()), FFBF_OK);
        twice("collect", [&] { return ffbf_scan_collect(c, &r); });
        expect("windows", (long long)r.n_hits, (long long)n);
        expect("lines", (long long)r.n_lines, (long long)n);
        text += text;  // more windows than the context's arrays have grown to
        twice("host scan", [&] { return ffbf_scan(c, (const uint8_t*)text.data(), text.size(), &r); });
        expect("windows", (long long)r.n_hits, 2 * (long long)n);
        twice("prune", [&] { return ffbf_prune(c, &pr); });
        expect("ids", (long long)pr.n_ids, 1000);
        if (n == 3000) {
            twice("verify", [&] { return ffbf_verify(c, &m); });
            expect("matches", (long long)m.n, 2 * (long long)n * 1000);
        }
        uint8_t* out = nullptr;
        size_t len = 0;
        twice("format", [&] {
            return ffbf_format_lines(c, (const uint8_t*)text.data(), text.size(), 1 << 19, &out, &len);
        });
        expect("bytes", (long long)len, (long long)text.size());
        ffbf_free(out);
        cudaFree(d_text);
        ffbf_destroy(c);
    }
    if (failures == 0) std::printf("host memory: all checks passed\n");
    return failures ? 1 : 0;
}
