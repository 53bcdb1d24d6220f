// ffbf_batch.cu -- many scans in one launch sequence: the job plan shared by the batch API and the server,
// the batch API (ffbf_batch_*: a fixed set of jobs captured once in a CUDA graph and launched repeatedly),
// and the autotuner of a context's scan configuration.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <memory>
#include <new>
#include <string>
#include <vector>

#include "ffbf_ctx.cuh"

using namespace ffbf_host;

struct ffbf_batch {
    int device = 0;
    int num_sms = 0;
    cudaStream_t st = nullptr;
    std::string err;
    struct Job {
        ffbf_ctx* c;
        const uint8_t* text;
        size_t len;
        uint32_t tile_bytes = 0;  // of the newline summaries that the prepared launch writes
        std::shared_ptr<uint64_t> scan_no;  // the context's, and its value for the batch's last launch
        uint64_t launched = 0;
        bool current() const { return scan_no && *scan_no == launched; }
    };
    // The device buffers and configuration each job's descriptors were built from. A context that has
    // since grown its hit buffer, reloaded its filter, added patterns or been retuned makes the batch
    // prepare again before its next launch.
    struct Key {
        const void *main, *ff, *hits, *counters, *tiles, *stage1;
        uint32_t hits_cap;
        uint64_t tiles_cap;
        int threads, mode, order;
        bool operator==(const Key& o) const {
            return main == o.main && ff == o.ff && hits == o.hits && counters == o.counters && tiles == o.tiles &&
                   stage1 == o.stage1 && hits_cap == o.hits_cap && tiles_cap == o.tiles_cap && threads == o.threads &&
                   mode == o.mode && order == o.order;
        }
    };
    std::vector<Key> keys;
    std::vector<Job> jobs;
    bool prepared = false;
    std::vector<void*> allocs;
    uint32_t* d_error = nullptr;  // n_ctl groups of 4 words: error flags, work-queue counter
    uint32_t n_ctl = 0;
    uint64_t graph_kernels = 0;  // kernel nodes of the graph
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    // Every job's results, collected by one launch after the graph (ffbf_batch_wait): a pinned block of a head per job,
    // words that the jobs share, and a copy of the control words. d_pool counts the words taken; a launch whose results
    // need more than there are makes the next one start with a larger block.
    std::shared_ptr<PinnedBlock> results;
    std::vector<ffbf::CollectJob> collect;
    uint64_t pool_words = 0, want_words = 0, max_words = 0;
    unsigned long long* d_pool = nullptr;
    ffbf::CollectJob* d_collect = nullptr;
    uint2* d_collect_items = nullptr;
    uint32_t n_collect_items = 0;
    bool uncollected = false;  // launched since the last collection
    uint32_t* h_ctl = nullptr;  // pinned copy of the control words, at the block's end
    // branch streams and events used while capturing the graph's parallel branches
    std::vector<cudaStream_t> branches;
    std::vector<cudaEvent_t> events;
};


namespace ffbf_host {

ffbf_status build_plan(const std::vector<PlanJob>& jobs, int num_sms, ScanPlan& plan, size_t* bad) {
    plan = ScanPlan{};
    struct Group {
        uint32_t len;
        ffbf::FastConfig cfg;
        std::vector<std::pair<uint64_t, ffbf::FastJob>> jobs;  // (bytes, descriptor)
    };
    std::vector<Group> groups;
    for (size_t i = 0; i < jobs.size(); i++) {
        ffbf_ctx* c = jobs[i].c;
        *bad = i;
        TRY(enter(c));
        TRY(setup_scan_state(c, jobs[i].text, jobs[i].len));
        if (use_fast(c, c->text_len)) {
            TRY(prepare_fast(c));
            // in a batch other jobs fill the GPU, so CTA size and rows per stream follow this job's size alone
            const ffbf::FastConfig cfg = ffbf::launch_config(c->cfg, c->g.len, c->text_len, num_sms, true);
            c->tile_bytes = ffbf::fast_tile_bytes(cfg.rows);
            const ffbf::ScanArgs a = make_scan_args(c);
            plan.args.push_back(a);
            ffbf::FastJob fj;
            if (ffbf::fill_fast_job(a, c->d_stage1, cfg, &fj) != cudaSuccess)
                return fail(c, FFBF_ECUDA, "tensor map encoding failed");
            Group* gp = nullptr;
            for (auto& g : groups)
                if (g.len == c->g.len && (g.cfg.mode == 1) == (cfg.mode == 1) &&
                    ffbf::config_threads(g.cfg) == ffbf::config_threads(cfg) &&
                    (cfg.mode != 1 || g.cfg.order == cfg.order) && g.cfg.halves == cfg.halves)
                    gp = &g;
            if (!gp) {
                groups.push_back(Group{c->g.len, cfg, {}});
                gp = &groups.back();
            }
            gp->jobs.push_back({a.n, fj});
        } else {
            plan.args.push_back(make_scan_args(c));
            for (uint64_t t = 0; t < scan_tiles(c); t++) plan.tail.push_back(make_uint2((uint32_t)i, (uint32_t)t));
        }
        CUDA_TRY(c, cudaStreamSynchronize(c->st));  // stage-1 tables built on the context's stream
        c->scan_pending = true;
    }
    // descriptors: groups contiguous, largest jobs first within a group (the work queue hands out the
    // largest items first, so the last wave is made of small ones)
    for (auto& g : groups) {
        std::stable_sort(g.jobs.begin(), g.jobs.end(), [](const auto& x, const auto& y) { return x.first > y.first; });
        PlanLaunch L{g.len, g.cfg, plan.fast.size(), (uint32_t)g.jobs.size(), 0, 0};
        for (auto& jb : g.jobs) {
            jb.second.item_begin = L.n_items;
            L.n_items += jb.second.n_supertiles;
            L.max_s1 = std::max(L.max_s1, jb.second.stage1_nwords);
            plan.fast.push_back(jb.second);
        }
        plan.launches.push_back(L);
    }
    return FFBF_OK;
}

cudaError_t launch_plan(const ScanPlan& p, const PlanDevice& d, int num_sms, cudaStream_t st,
                        const cudaStream_t* branches, const cudaEvent_t* events) {
    cudaError_t e = ffbf::zero_counters(d.counters, d.n_counters, st);
    const size_t nl = p.launches.size();
    if (!branches) {
        for (size_t li = 0; li < nl && e == cudaSuccess; li++) {
            const PlanLaunch& L = p.launches[li];
            e = ffbf::launch_fast_jobs(L.len, L.cfg, d.fast + L.off, L.n_jobs, L.n_items, L.max_s1, d.ctl + 4 * li,
                                       num_sms, st);
        }
        if (e == cudaSuccess) e = ffbf::scan_generic_multi(d.args, d.tail, (uint32_t)p.tail.size(), num_sms, st);
        return e;
    }
    // fork: each tuned launch and the generic launch on its own branch (they touch disjoint tiles), join
    // back on st; a branch's kernel takes SMs as the others' work queues drain
    if (e == cudaSuccess) e = cudaEventRecord(events[0], st);
    for (size_t li = 0; li <= nl && e == cudaSuccess; li++) {
        cudaStream_t bs = branches[li];
        e = cudaStreamWaitEvent(bs, events[0], 0);
        if (e == cudaSuccess && li < nl) {
            const PlanLaunch& L = p.launches[li];
            e = ffbf::launch_fast_jobs(L.len, L.cfg, d.fast + L.off, L.n_jobs, L.n_items, L.max_s1, d.ctl + 4 * li,
                                       num_sms, bs);
        } else if (e == cudaSuccess) {
            e = ffbf::scan_generic_multi(d.args, d.tail, (uint32_t)p.tail.size(), num_sms, bs);
        }
        if (e == cudaSuccess) e = cudaEventRecord(events[1 + li], bs);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(st, events[1 + li], 0);
    }
    return e;
}

}  // namespace ffbf_host

namespace {

ffbf_status autotune_impl(ffbf_ctx* c, const uint8_t* d_text, size_t sample_len, bool per_sm, int* threads,
                          int* mode);

ffbf_batch::Key batch_key(const ffbf_ctx* c) {
    return ffbf_batch::Key{c->d_main, c->d_ff,          c->d_hits,      c->d_counters, c->d_tiles,
                           c->d_stage1, c->hits_cap,    c->tiles_cap,   c->cfg.threads, c->cfg.mode,
                           c->cfg.order};
}

ffbf_status bfail(ffbf_batch* b, ffbf_status s, const std::string& msg) {
    b->err = msg;
    return s;
}

void batch_release(ffbf_batch* b) {
    if (b->exec) cudaGraphExecDestroy(b->exec);
    if (b->graph) cudaGraphDestroy(b->graph);
    for (auto s : b->branches) cudaStreamDestroy(s);
    for (auto e : b->events) cudaEventDestroy(e);
    b->branches.clear();
    b->events.clear();
    b->exec = nullptr;
    b->graph = nullptr;
    for (void* p : b->allocs) cudaFree(p);
    b->allocs.clear();
    b->d_error = nullptr;
    b->collect.clear();
    b->pool_words = b->want_words = 0;  // the block itself stays for the next preparation
    b->n_collect_items = 0;
    b->uncollected = false;
    b->prepared = false;
    b->keys.clear();
    cudaGetLastError();
}

template <class T>
ffbf_status balloc(ffbf_batch* b, T** p, size_t count) {
    void* v = nullptr;
    if (cudaMalloc(&v, count * sizeof(T) + 16) != cudaSuccess) {
        cudaGetLastError();
        return bfail(b, FFBF_ENOMEM_DEVICE, "batch table allocation failed");
    }
    b->allocs.push_back(v);
    *p = static_cast<T*>(v);
    return FFBF_OK;
}

// Pinning costs up to a millisecond per MiB and most jobs have few windows: the jobs share the words, 1 MiB of them at
// first, at most 32, and the block stays for the batch's next preparation. With room for each job of its own, preparing 48
// jobs of 64 MiB took 8.7 to 11.9 ms and 256 of 1 MiB 3.3 to 6.9; now 0.56 and 1.1 (with no such room: 0.50 and 0.95).
constexpr uint64_t kPoolWords = 1 << 17, kMaxPoolWords = 1 << 22;

// Makes the batch's pinned block with room for `words` and points the collection at it. Where they cannot be had, it keeps
// the block there is, or makes one without words: jobs that find no room are collected one by one.
ffbf_status make_results(ffbf_batch* b, uint64_t words) {
    const size_t heads = 64 * b->collect.size(), ctl = 16 * ((size_t)b->n_ctl + 1);
    auto block = b->results;
    if (!block || block->bytes < heads + 8 * words + ctl || block.use_count() > 2) {  // 2: no context holds it
        block = std::make_shared<PinnedBlock>();
        block->bytes = heads + 8 * words + ctl;
        if (cudaMallocHost(&block->p, block->bytes) != cudaSuccess) {
            cudaGetLastError();
            b->max_words = b->pool_words;
            if (b->pool_words) return FFBF_OK;
            words = 0;
            block->bytes = heads + ctl;
            if (cudaMallocHost(&block->p, block->bytes) != cudaSuccess) {
                cudaGetLastError();
                block->p = nullptr;
                return bfail(b, FFBF_ENOMEM_HOST, "pinned batch results");
            }
        }
    }
    for (size_t i = 0; i < b->collect.size(); i++) {
        b->collect[i].head = reinterpret_cast<ffbf::ResultHead*>(block->p + 64 * i);
        b->collect[i].words = reinterpret_cast<uint64_t*>(block->p + heads);
        b->collect[i].n_words = words;
    }
    if (!b->collect.empty() && cudaMemcpy(b->d_collect, b->collect.data(), b->collect.size() * sizeof(ffbf::CollectJob),
                                          cudaMemcpyHostToDevice) != cudaSuccess) {
        cudaGetLastError();
        return bfail(b, FFBF_ECUDA, "batch table upload failed");
    }
    b->h_ctl = reinterpret_cast<uint32_t*>(block->p + heads + 8 * words);
    b->results = block;
    b->pool_words = words;
    return FFBF_OK;
}

}  // namespace

extern "C" {

ffbf_status ffbf_batch_create(int device, ffbf_batch** out) {
    if (!out) return FFBF_EINVAL;
    *out = nullptr;
    ffbf_batch* b = new (std::nothrow) ffbf_batch();
    if (!b) return FFBF_ENOMEM_HOST;
    b->device = device;
    if (cudaSetDevice(device) != cudaSuccess || cudaStreamCreateWithFlags(&b->st, cudaStreamNonBlocking) != cudaSuccess ||
        cudaDeviceGetAttribute(&b->num_sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) {
        cudaGetLastError();
        delete b;
        return FFBF_ECUDA;
    }
    *out = b;
    return FFBF_OK;
}

void ffbf_batch_destroy(ffbf_batch* b) {
    if (!b) return;
    cudaSetDevice(b->device);
    if (b->st) cudaStreamSynchronize(b->st);
    batch_release(b);
    if (b->st) cudaStreamDestroy(b->st);
    delete b;
}

const char* ffbf_batch_last_error(const ffbf_batch* b) { return b ? b->err.c_str() : "null batch"; }

void* ffbf_batch_stream(ffbf_batch* b) { return b ? (void*)b->st : nullptr; }

ffbf_status ffbf_batch_add(ffbf_batch* b, ffbf_ctx* c, const uint8_t* d_text, size_t len) try {
    if (!b || !c) return FFBF_EINVAL;
    if (c->device != b->device) return bfail(b, FFBF_EINVAL, "context and batch are on different devices");
    if (((uintptr_t)d_text & 15) != 0 || (!d_text && len)) return bfail(b, FFBF_EINVAL, "device text must be 16-byte aligned");
    for (auto& j : b->jobs)
        if (j.c == c) return bfail(b, FFBF_EINVAL, "a context may appear only once in a batch");
    if (b->prepared) batch_release(b);
    b->jobs.push_back({c, d_text, len});
    return FFBF_OK;
} catch (...) {
    return FFBF_ENOMEM_HOST;
}

ffbf_status ffbf_batch_prepare(ffbf_batch* b) try {
    NvtxRange nvtx_("ffbf_batch_prepare");
    if (!b) return FFBF_EINVAL;
    if (cudaSetDevice(b->device) != cudaSuccess) return bfail(b, FFBF_ECUDA, "cudaSetDevice failed");
    batch_release(b);
    std::vector<PlanJob> pj;
    for (const auto& j : b->jobs) pj.push_back({j.c, j.text, j.len});
    ScanPlan plan;
    size_t bad = 0;
    ffbf_status s = build_plan(pj, b->num_sms, plan, &bad);
    if (s != FFBF_OK) return bfail(b, s, "job " + std::to_string(bad) + ": " + b->jobs[bad].c->err);
    std::vector<uint32_t*> counters;
    for (size_t i = 0; i < b->jobs.size(); i++) {
        auto& j = b->jobs[i];
        j.tile_bytes = plan.args[i].tile_bytes;
        b->keys.push_back(batch_key(j.c));
        counters.push_back(j.c->d_counters);
    }
    PlanDevice d{};
    TRY(balloc(b, &d.fast, plan.fast.size() + 1));
    TRY(balloc(b, &d.args, plan.args.size() + 1));
    TRY(balloc(b, &d.tail, plan.tail.size() + 1));
    // a group of control words per launch, and one whose first two count the results' words
    TRY(balloc(b, &b->d_error, 4 * (plan.launches.size() + 2)));
    b->n_ctl = (uint32_t)plan.launches.size() + 1;
    d.ctl = b->d_error;
    b->d_pool = reinterpret_cast<unsigned long long*>(b->d_error + 4 * b->n_ctl);
    for (uint32_t i = 0; i <= b->n_ctl; i++) counters.push_back(b->d_error + 4 * i);
    TRY(balloc(b, &d.counters, counters.size() + 1));
    d.n_counters = (uint32_t)counters.size();
    auto up = [](void* dst, const void* src, size_t bytes) {
        return bytes == 0 || cudaMemcpy(dst, src, bytes, cudaMemcpyHostToDevice) == cudaSuccess;
    };
    if (!up(d.fast, plan.fast.data(), plan.fast.size() * sizeof(ffbf::FastJob)) ||
        !up(d.args, plan.args.data(), plan.args.size() * sizeof(ffbf::ScanArgs)) ||
        !up(d.tail, plan.tail.data(), plan.tail.size() * sizeof(uint2)) ||
        !up(d.counters, counters.data(), counters.size() * sizeof(uint32_t*)) ||
        cudaMemset(b->d_error, 0, 16 * (b->n_ctl + 1)) != cudaSuccess) {
        cudaGetLastError();
        return bfail(b, FFBF_ECUDA, "batch table upload failed");
    }
    // the jobs' results: CTAs for one hit window per 8 KiB of text, at least 512
    {
        std::vector<uint2> items;
        uint64_t words = 0;
        for (size_t i = 0; i < b->jobs.size(); i++) {
            const uint32_t windows =
                (uint32_t)std::min<uint64_t>(ffbf::kSmallResults, std::max<uint64_t>(512, b->jobs[i].len / 8192));
            ffbf::CollectJob cj = collect_job(plan.args[i], b->jobs[i].c->d_hitlines, nullptr, ffbf::kSmallResults,
                                              ffbf::kCollectBatch, windows);
            cj.used = b->d_pool;
            for (uint32_t k = 0; k < cj.ctas; k++) items.push_back(make_uint2((uint32_t)i, k));
            b->collect.push_back(cj);
            words += 3 * windows;
        }
        b->n_collect_items = (uint32_t)items.size();
        TRY(balloc(b, &b->d_collect, b->collect.size() + 1));
        TRY(balloc(b, &b->d_collect_items, items.size() + 1));
        if (!up(b->d_collect_items, items.data(), items.size() * sizeof(uint2))) {
            cudaGetLastError();
            return bfail(b, FFBF_ECUDA, "batch table upload failed");
        }
        b->max_words = kMaxPoolWords;
        TRY(make_results(b, std::min(words, kPoolWords)));
    }
    // one graph: zero the jobs' counters, one tuned launch per group, one generic launch for all tail tiles
    if (cudaStreamBeginCapture(b->st, cudaStreamCaptureModeThreadLocal) != cudaSuccess)
        return bfail(b, FFBF_ECUDA, "stream capture failed to start");
    for (size_t i = 0; i <= plan.launches.size(); i++) {
        cudaStream_t bs;
        if (cudaStreamCreateWithFlags(&bs, cudaStreamNonBlocking) != cudaSuccess) {
            cudaGetLastError();
            return bfail(b, FFBF_ECUDA, "branch stream creation failed");
        }
        b->branches.push_back(bs);
    }
    for (size_t i = 0; i <= plan.launches.size() + 1; i++) {
        cudaEvent_t ev;
        if (cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) != cudaSuccess) {
            cudaGetLastError();
            return bfail(b, FFBF_ECUDA, "event creation failed");
        }
        b->events.push_back(ev);
    }
    const uint64_t launches0 = ffbf::launches_total();
    cudaError_t e = launch_plan(plan, d, b->num_sms, b->st, b->branches.data(), b->events.data());
    cudaError_t e2 = cudaStreamEndCapture(b->st, &b->graph);
    b->graph_kernels = ffbf::launches_total() - launches0;  // counted again at each graph launch
    ffbf::unnote_launches(b->graph_kernels);
    if (e != cudaSuccess || e2 != cudaSuccess || cudaGraphInstantiate(&b->exec, b->graph, 0) != cudaSuccess) {
        cudaGetLastError();
        return bfail(b, FFBF_ECUDA,
                     std::string("batch graph capture failed: ") + cudaGetErrorString(e != cudaSuccess ? e : e2));
    }
    b->prepared = true;
    return FFBF_OK;
} catch (...) {
    return FFBF_ENOMEM_HOST;
}

ffbf_status ffbf_batch_launch(ffbf_batch* b) try {
    NvtxRange nvtx_("ffbf_batch_launch");
    if (!b) return FFBF_EINVAL;
    bool stale = !b->prepared || b->keys.size() != b->jobs.size();
    for (size_t i = 0; i < b->jobs.size() && !stale; i++)
        stale = !(batch_key(b->jobs[i].c) == b->keys[i]) ||
                (use_fast(b->jobs[i].c, b->jobs[i].len) && b->jobs[i].c->stage1_dirty);
    if (stale) TRY(ffbf_batch_prepare(b));
    if (cudaSetDevice(b->device) != cudaSuccess) return bfail(b, FFBF_ECUDA, "cudaSetDevice failed");
    if (b->want_words > b->pool_words) {
        if (cudaStreamSynchronize(b->st) != cudaSuccess) {
            cudaGetLastError();
            return bfail(b, FFBF_ECUDA, "batch execution failed");
        }
        TRY(make_results(b, b->want_words));
        b->want_words = 0;
    }
    for (auto& j : b->jobs) {
        reset_scan(j.c);
        j.c->d_text = j.text;
        j.c->text_len = j.len;
        j.c->tile_bytes = j.tile_bytes;  // a scan of the context's own since may have had another
        j.c->scan_pending = true;
        j.c->segmented = false;  // nor is a host text scanned in segments the current one any more
        j.c->segs.clear();
        j.c->seg_hr.clear();
        j.scan_no = j.c->scan_no;
        j.launched = *j.scan_no;
    }
    if (cudaGraphLaunch(b->exec, b->st) != cudaSuccess) {
        cudaGetLastError();
        return bfail(b, FFBF_ECUDA, "graph launch failed");
    }
    ffbf::note_launches(b->graph_kernels);
    b->uncollected = true;
    return FFBF_OK;
} catch (...) {
    return FFBF_ENOMEM_HOST;
}

ffbf_status ffbf_batch_wait(ffbf_batch* b) {
    if (!b) return FFBF_EINVAL;
    cudaError_t e = cudaSetDevice(b->device);
    // Every job's results by one launch, and the control words, behind the graph: one wait for all of them. Where a
    // context has been used for another scan since the launch, or is gone, each of the others is collected by itself.
    const bool collect = b->prepared && b->uncollected &&
                         std::all_of(b->jobs.begin(), b->jobs.end(), [](const auto& j) { return j.current(); });
    if (e == cudaSuccess && collect)
        e = ffbf::collect_hits_multi(b->d_collect, b->d_collect_items, b->n_collect_items, b->st);
    if (e == cudaSuccess && b->prepared)
        e = cudaMemcpyAsync(b->h_ctl, b->d_error, 16 * (b->n_ctl + 1), cudaMemcpyDeviceToHost, b->st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(b->st);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return bfail(b, FFBF_ECUDA, std::string("batch execution failed: ") + cudaGetErrorString(e));
    }
    uint32_t flag = 0;
    if (b->prepared) {
        for (uint32_t i = 0; i < b->n_ctl; i++) flag |= b->h_ctl[4 * i];
        b->uncollected = false;
        for (size_t i = 0; i < b->jobs.size() && collect && !flag; i++) {
            ffbf_ctx* c = b->jobs[i].c;
            if (!c->scan_pending) continue;  // collected already
            c->ready_block = b->results;
            c->ready = b->collect[i].head;
            c->ready_words = b->collect[i].words;
        }
        if (collect) {
            unsigned long long used;
            memcpy(&used, b->h_ctl + 4 * b->n_ctl, 8);
            if (used > b->pool_words) b->want_words = std::min<uint64_t>(used + used / 4, b->max_words);
        }
    }
    if (flag) {
        char buf[96];
        snprintf(buf, sizeof buf, "batched scan error flags 0x%x (4: a bounded wait gave up; others: self-checks)", flag);
        return bfail(b, (flag & 4u) ? FFBF_ETIMEOUT : FFBF_ECUDA, buf);
    }
    return FFBF_OK;
}

ffbf_status ffbf_batch_autotune(ffbf_batch* b, size_t sample_bytes, uint32_t* n_classes) try {
    NvtxRange nvtx_("ffbf_batch_autotune");
    if (!b) return FFBF_EINVAL;
    if (n_classes) *n_classes = 0;
    // classes: jobs with the same geometry whose stage-1 tables are about as full (1/16 steps) scan alike
    struct Class {
        size_t rep;  // the class's largest job
        std::vector<size_t> members;
    };
    std::map<std::vector<uint64_t>, Class> classes;
    for (size_t i = 0; i < b->jobs.size(); i++) {
        ffbf_ctx* c = b->jobs[i].c;
        TRY(enter(c));
        if (!tunable(c, b->jobs[i].len)) continue;
        TRY(prepare_fast(c));  // builds the stage-1 table and measures its fill
        const std::vector<uint64_t> key = {c->g.len, c->g.k, c->g.s, c->g.cache_bits, c->g.nbits,
                                           (uint64_t)(c->stage1_fill * 16.0)};
        auto it = classes.find(key);
        if (it == classes.end()) {
            classes[key] = Class{i, {i}};
        } else {
            it->second.members.push_back(i);
            if (b->jobs[i].len > b->jobs[it->second.rep].len) it->second.rep = i;
        }
    }
    for (auto& kv : classes) {
        const auto& rep = b->jobs[kv.second.rep];
        size_t n = std::min(sample_bytes ? sample_bytes : (size_t)16 << 20, rep.len);
        n = n / ffbf::kScanTile * ffbf::kScanTile;
        if (n < ffbf::kScanTile) continue;
        int threads = 0, mode = 0;
        ffbf_status s = autotune_impl(rep.c, rep.text, n, true, &threads, &mode);
        if (s != FFBF_OK) return bfail(b, s, std::string("autotune: ") + rep.c->err);
        for (size_t m : kv.second.members) {
            ffbf_ctx* c = b->jobs[m].c;
            c->cfg = rep.c->cfg;
            c->cfg_tuned = true;
        }
    }
    if (n_classes) *n_classes = (uint32_t)classes.size();
    batch_release(b);  // the next launch prepares with the tuned configurations
    return FFBF_OK;
} catch (...) {
    return FFBF_ENOMEM_HOST;
}

}  // extern "C"

namespace {

// Times the tuned scan's configurations on a sample and keeps the best. per_sm scores by SM-seconds per
// byte (time x SMs the launch occupies), each trial with the CTA size and rows that a batch would give such a text: in a
// batch many jobs share the GPU, so a configuration whose items fill fewer SMs on a small sample must not win by wall time
// alone. Otherwise by wall time.
ffbf_status autotune_impl(ffbf_ctx* c, const uint8_t* d_text, size_t sample_len, bool per_sm, int* threads,
                          int* mode) {
    TRY(enter(c));
    if (!d_text || ((uintptr_t)d_text & 15)) return fail(c, FFBF_EINVAL, "device text must be 16-byte aligned");
    if (!tunable(c, sample_len)) return fail(c, FFBF_EINVAL, "the tuned scan does not cover this geometry or size");
    // keep the feed-forward filter: the trial scans set bits in it
    uint32_t* saved = nullptr;
    TRY(dalloc_t(c, &saved, c->filter_bytes / 4));
    CUDA_TRY(c, cudaMemcpyAsync(saved, c->d_ff, c->filter_bytes, cudaMemcpyDeviceToDevice, c->st));
    // the sparse kernel in mode 3 (whose CTA size launch_config picks and whose table may have 16-bit entries) and at three
    // fixed sizes, the dense one at three (its probe order follows the filter's fills; 192 runs two CTAs per SM, and
    // probe orders 2 and 3 run 192 as 384)
    const ffbf::FastConfig cands[] = {{512, 3, 0, 0}, {384, 0, 0, 0}, {256, 0, 0, 0}, {192, 2, 0, 0},
                                      {384, 1, 0, 0}, {192, 1, 0, 0}, {256, 1, 0, 0}};
    ffbf::FastConfig best = c->cfg;
    double best_score = 1e300;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    const int saved_force = c->force_mode;
    c->force_mode = -1;
    c->as_batch = per_sm;
    ffbf_status s = FFBF_OK;
    for (const auto& cand : cands) {
        c->cfg = cand;
        c->cfg_tuned = true;
        if ((s = setup_scan_state(c, d_text, sample_len)) != FFBF_OK) break;
        float ms = 1e30f;
        for (int rep = 0; rep < 3 && s == FFBF_OK; rep++) {
            cudaEventRecord(e0, c->st);
            s = launch_scan(c);
            cudaEventRecord(e1, c->st);
            if (cudaEventSynchronize(e1) != cudaSuccess) s = fail(c, FFBF_ECUDA, "autotune timing failed");
            float t = 0;
            cudaEventElapsedTime(&t, e0, e1);
            if (rep > 0) ms = std::min(ms, t);  // the first run also builds the stage-1 table
        }
        if (s != FFBF_OK) break;
        double score = ms;
        if (per_sm) {
            const ffbf::FastConfig run = ffbf::launch_config(cand, c->g.len, sample_len, c->num_sms, per_sm);
            const int t = ffbf::config_threads(run);
            const uint64_t streams = sample_len / ((uint64_t)run.rows * 128);
            const uint64_t items = (streams + t - 1) / t;
            score = ms * (double)std::min<uint64_t>(items, (uint64_t)c->num_sms);
        }
        if (score < best_score) {
            best_score = score;
            best = cand;
        }
    }
    c->force_mode = saved_force;
    c->as_batch = false;
    c->cfg = best;
    c->cfg_tuned = true;
    reset_scan(c);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (s == FFBF_OK) {
        CUDA_TRY(c, cudaMemcpyAsync(c->d_ff, saved, c->filter_bytes, cudaMemcpyDeviceToDevice, c->st));
        s = sync(c);
    }
    dfree(c, saved);
    if (s == FFBF_OK) s = prepare_fast(c);
    if (threads) *threads = ffbf::config_threads(best);
    if (mode) *mode = best.mode;
    return s;
}

}  // namespace

extern "C" {

ffbf_status ffbf_autotune(ffbf_ctx* c, const uint8_t* d_text, size_t sample_len, int* threads, int* mode) {
    return autotune_impl(c, d_text, sample_len, false, threads, mode);
}

}  // extern "C"
