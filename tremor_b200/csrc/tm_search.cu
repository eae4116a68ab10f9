// The device pipeline of a prepared group: window statistics (per length, or the
// resident prefix sums), the contraction kernel or the FFT branch with its bounded
// epilogue, the kNN bound and FP32 re-pass, exact re-scoring, and the answers assembled on
// the device and handed to the result in pinned memory.
#include "tm_core.h"

namespace tmh {

LengthStats &ensure_length(tm_ctx *ctx, Lane &L, int m)
{
    auto it = ctx->lengths.find(m);
    if (it != ctx->lengths.end())
    {
        it->second->last_use = ++ctx->use_clock;
        return *it->second;
    }
    const uint64_t total = ctx->n - static_cast<uint64_t>(m) + 1; // windows of the whole waveform
    const uint64_t w0 = std::min(ctx->range_first, total);
    const uint64_t W = std::min(ctx->range_count, total - w0);
    // keep the resident statistics under half of the free memory: evict least recently used
    size_t free_b = 0, total_b = 0;
    TM_CUDA(cudaMemGetInfo(&free_b, &total_b));
    const size_t need = W * 9 + 4096;
    while (!ctx->lengths.empty() && need * 2 > free_b)
    {
        auto victim = ctx->lengths.begin();
        for (auto jt = ctx->lengths.begin(); jt != ctx->lengths.end(); ++jt)
            if (jt->second->last_use < victim->second->last_use)
                victim = jt;
        free_b += victim->second->bytes();
        victim->second->mean.release();
        victim->second->inv.release();
        victim->second->flags.release();
        ctx->lengths.erase(victim);
    }
    auto ls = std::make_unique<LengthStats>();
    ls->m = m;
    ls->w0 = w0;
    ls->W = W;
    if (W > 0)
    {
        ls->mean.reserve(W * sizeof(float) + 64);
        ls->inv.reserve(W * sizeof(float) + 64);
        ls->flags.reserve(W + 64);
        const uint64_t a_count = (w0 + W - 1) / m - w0 / m + 1;
        ctx->suf.reserve(a_count * static_cast<uint64_t>(m) * sizeof(double2));
        TM_CUDA(tmb::launch_window_stats(ctx->clean.as<float>(), ctx->raw.as<float>(), ctx->odd.as<uint32_t>(), ctx->n, m, w0, W,
                                        ctx->suf.as<double2>(), ls->mean.as<float>(), ls->inv.as<float>(),
                                        ls->flags.as<uint8_t>(), L.stream));
        count_launch(L, 3);
    }
    ls->last_use = ++ctx->use_clock;
    LengthStats &ref = *ls;
    ctx->lengths[m] = std::move(ls);
    return ref;
}

// Resident FP64 prefix sums and constant-run lengths of the waveform (built once).
void ensure_prefix(tm_ctx *ctx, Lane &L)
{
    if (ctx->prefix_ready)
        return;
    cudaStream_t s = L.stream;
    const uint64_t n = ctx->n;
    const uint32_t chunks = tmb::prefix_chunks(n);
    const uint64_t blocks = (n + tmb::kPrefixBlock - 1) / tmb::kPrefixBlock;
    // zero tail: the contraction kernels read window-end sums in fixed-size chunks that may
    // run past n (values there belong to no window and are never used)
    ctx->prefix.reserve(sizeof(double2) * (n + 1 + tmb::kStagePad));
    TM_CUDA(cudaMemsetAsync(ctx->prefix.p, 0, sizeof(double2) * (n + 1 + tmb::kStagePad), s));
    // one entry past the last block: a window ending at n = blocks x kPrefixBlock reads it
    ctx->ptot.reserve(sizeof(double2) * (blocks + 1));
    ctx->pcen.reserve(sizeof(double) * (blocks + 1));
    TM_CUDA(cudaMemsetAsync(ctx->ptot.p, 0, sizeof(double2) * (blocks + 1), s));
    ctx->run.reserve(sizeof(uint16_t) * n);
    ScopedBuf totals, run_first;
    totals.reserve(sizeof(double2) * chunks);
    run_first.reserve(sizeof(uint32_t) * chunks);
    // centres: the mean of each block, from uncentred chunk sums
    TM_CUDA(tmb::launch_prefix_totals(ctx->clean.as<float>(), n, nullptr, totals.as<double2>(), s));
    std::vector<double2> ct(chunks);
    TM_CUDA(cudaMemcpyAsync(ct.data(), totals.p, sizeof(double2) * chunks, cudaMemcpyDeviceToHost, s));
    TM_CUDA(cudaStreamSynchronize(s));
    const uint64_t per_block = tmb::kPrefixBlock / 8192;
    std::vector<double> centres(blocks + 1, 0.0);
    for (uint64_t b = 0; b < blocks; b++)
    {
        double sum = 0.0;
        for (uint64_t c = b * per_block; c < std::min<uint64_t>(chunks, (b + 1) * per_block); c++)
            sum += ct[c].x;
        const uint64_t count = std::min<uint64_t>(tmb::kPrefixBlock, n - b * tmb::kPrefixBlock);
        centres[b] = sum / static_cast<double>(count);
    }
    centres[blocks] = blocks > 0 ? centres[blocks - 1] : 0.0;
    TM_CUDA(cudaMemcpyAsync(ctx->pcen.p, centres.data(), sizeof(double) * (blocks + 1), cudaMemcpyHostToDevice, s));
    TM_CUDA(tmb::launch_prefix_sums(ctx->clean.as<float>(), n, ctx->pcen.as<double>(), totals.as<double2>(),
                                    ctx->ptot.as<double2>(), ctx->prefix.as<double2>(), s));
    TM_CUDA(tmb::launch_runs(ctx->clean.as<float>(), ctx->raw.as<float>(), n, ctx->run.as<uint16_t>(),
                             run_first.as<uint32_t>(), s));
    TM_CUDA(cudaStreamSynchronize(s));
    count_launch(L, 4 + 2);
    ctx->prefix_ready = true;
}

// A pinned block of at least `need` bytes that no result holds, from the pool or new.
std::shared_ptr<PinnedBlock> acquire_block(Lane &L, size_t need)
{
    auto &pool = L.pool;
    for (auto &b : pool)
        if (b.use_count() == 1 && b->bytes >= need)
            return b;
    pool.erase(std::remove_if(pool.begin(), pool.end(),
                              [](const std::shared_ptr<PinnedBlock> &b) { return b.use_count() == 1; }),
               pool.end());
    pool.push_back(std::make_shared<PinnedBlock>(std::max<size_t>(need + need / 4, 1u << 20)));
    return pool.back();
}

// Largest k whose selection runs on the device (k_select_knn keeps k windows per block in
// shared memory); groups with a larger k select on the host.
constexpr int kMaxDeviceK = 1024;

// What the device left for a group's answers (host pointers into the pinned block,
// device pointers for the runs that stay on the device).
struct AnswerView
{
    uint32_t *win = nullptr; // threshold runs: windows relative to w0, then ED^2
    float *dist = nullptr;
    const uint32_t *start = nullptr, *end = nullptr, *tkey = nullptr;
    bool device_knn = false; // kNN selections made by k_select_knn:
    int kcap = 0;            //   slot s: knn_n[s] answers at s * kcap
    const uint32_t *knn_n = nullptr, *knn_win = nullptr;
    const float *knn_dist = nullptr;
    const uint32_t *d_win = nullptr; // the sorted runs on the device
    const float *d_dist = nullptr;
};

// Canonical answers of each template of a group.
// Threshold: the template's run (position order, no repeats), thinned in place by the
// merge offset. kNN: the device's exclusion selection over the finite distances. When
// that leaves fewer than k answers and the bound was unbounded (too few separated
// windows for the reference's queue to fill), or k is too large for the device, the
// template's run (in (distance, position) order) is fetched and selected here: the
// windows of distance FLT_MAX (constant windows, which the contraction skips, plus any
// re-scored to FLT_MAX) follow the finite ones in position order, as in the reference.
template <class Degenerate>
void finish_answers(Lane &L, const GroupPlan &g, const AnswerView &v, uint64_t w0, tm_result &res,
                    Degenerate degenerate_windows)
{
    int slot = -1;
    for (int t = 0; t < g.T; t++)
    {
        const bool knn = g.mode[t] == TM_MODE_KNN;
        const bool inert = g.inert[t] != 0; // has no run and no slot: only constant windows can be answers
        slot += knn && !inert ? 1 : 0;
        if (g.index[t] < 0)
            continue; // padding row of a mixed-length tile
        Answer &out = res.answers[g.index[t]];
        const uint32_t a = v.start[t], b = v.end[t];
        if (!knn)
        {
            uint32_t count = b - a;
            if (g.merge[t] > 0) // SkipSequential.cpp:358-370: skip pos < last kept + merge + 1
            {
                const uint64_t gap = static_cast<uint64_t>(g.merge[t]) + 1;
                uint32_t w = a;
                for (uint32_t i = a; i < b; i++)
                {
                    if (w > a && static_cast<uint64_t>(v.win[i]) < static_cast<uint64_t>(v.win[w - 1]) + gap)
                        continue;
                    v.win[w] = v.win[i];
                    v.dist[w] = v.dist[i];
                    w++;
                }
                count = w - a;
            }
            out.hits.clear();
            out.run = true;
            out.win = v.win + a;
            out.dist = v.dist + a;
            out.w0 = w0;
            out.count = count;
            continue;
        }
        std::vector<Hit> kept;
        const bool unbounded = inert || v.tkey[t] == tmb::kEmptyKey;
        if (v.device_knn && !inert && (static_cast<int>(v.knn_n[slot]) >= g.k[t] || !unbounded))
        {
            const size_t at = static_cast<size_t>(slot) * v.kcap;
            for (uint32_t i = 0; i < v.knn_n[slot]; i++)
                kept.push_back(Hit{w0 + v.knn_win[at + i], v.knn_dist[at + i]});
        }
        else
        {
            std::vector<uint32_t> rw(b - a);
            std::vector<float> rd(b - a);
            if (b > a)
            {
                TM_CUDA(cudaMemcpyAsync(rw.data(), v.d_win + a, sizeof(uint32_t) * (b - a), cudaMemcpyDeviceToHost,
                                        L.stream));
                TM_CUDA(cudaMemcpyAsync(rd.data(), v.d_dist + a, sizeof(float) * (b - a), cudaMemcpyDeviceToHost,
                                        L.stream));
                TM_CUDA(cudaStreamSynchronize(L.stream));
                L.d2h_bytes += 8ull * (b - a);
            }
            std::vector<Hit> finite, infinite;
            for (uint32_t i = 0; i < b - a; i++)
                (rd[i] < FLT_MAX ? finite : infinite).push_back(Hit{w0 + rw[i], rd[i]});
            tm_host::select_knn(finite, g.k[t], g.merge[t], kept);
            if (static_cast<int>(kept.size()) < g.k[t] && unbounded)
            {
                degenerate_windows(t, infinite);
                std::sort(infinite.begin(), infinite.end(), [](const Hit &x, const Hit &y) { return x.pos < y.pos; });
                infinite.erase(std::unique(infinite.begin(), infinite.end(),
                                           [](const Hit &x, const Hit &y) { return x.pos == y.pos; }),
                               infinite.end());
                tm_host::extend_knn(infinite, g.k[t], g.merge[t], kept);
            }
        }
        while (static_cast<int>(kept.size()) < g.k[t])
            kept.push_back(Hit{0, FLT_MAX});
        out.set_hits(std::move(kept));
    }
}

void add_span(Lane &L, int phase, cudaEvent_t a, cudaEvent_t b)
{
    float ms = 0.0f;
    TM_CUDA(cudaEventElapsedTime(&ms, a, b));
    L.phase_ms[phase] += ms;
}

// Has the group kNN templates without a merge offset?
static bool tight_bounds(const GroupPlan &g)
{
    for (int t = 0; t < g.T; t++)
        if (g.mode[t] == TM_MODE_KNN && g.merge[t] <= 0)
            return true;
    return false;
}

// What k_passb left for the re-scoring of a group's kNN candidates; no certain minima where the
// buckets are larger than the re-pass's 256 windows.
static tmb::Exclusion exclusion(const Lane &L, const GroupPlan &g, uint32_t nb, int blog)
{
    tmb::Exclusion ex{};
    if (g.nk > 0 && blog == 8)
        ex = tmb::Exclusion{L.bmin_l.as<uint32_t>(), L.bmin_u.as<uint32_t>(), L.tkey.as<uint32_t>(), nb};
    if (tight_bounds(g))
    {
        ex.lower = L.lower.as<float>();
        ex.tight = L.tight.as<float>();
    }
    return ex;
}

// Exact re-scoring of a group's ncand candidates (pv: prefix sums of mixed groups, mean: window means of the others), answer order and kNN selection on the
// device, one copy to a pinned block that the result keeps, canonical answers.
template <class Degenerate>
void rescore_and_answer(tm_ctx *ctx, Lane &L, const GroupPlan &g, uint32_t ncand, const tmb::PrefixView &pv,
                        const float *mean, uint64_t w0, const tmb::Exclusion &ex, tm_result &res, Degenerate degenerate_windows)
{
    cudaStream_t s = L.stream;
    const int T = g.T, nk = g.nk;
    int kcap = 1, shortest = INT_MAX;
    for (int t = 0; t < T; t++)
        if (g.index[t] >= 0)
            shortest = std::min(shortest, g.htp[t].m);
    for (int t = 0; t < T; t++)
        if (g.mode[t] == TM_MODE_KNN)
            kcap = std::max(kcap, g.k[t]);
    const bool device_knn = nk > 0 && kcap <= kMaxDeviceK;
    const size_t cn = std::max<uint32_t>(ncand, 1);
    L.dist.reserve(sizeof(float) * cn);
    L.akeys.reserve(2 * sizeof(unsigned long long) * cn);
    L.avals.reserve(2 * sizeof(float) * cn);
    if (nk > 0)
        L.avals64.reserve(2 * sizeof(unsigned long long) * cn);
    L.segs.reserve(sizeof(uint32_t) * (3 * static_cast<size_t>(std::max(T, 1)) +
                                          (device_knn ? static_cast<size_t>(nk) * (1 + 2 * kcap) : 0)));
    uint32_t *d_kept = L.counters.as<uint32_t>() + 3;
    uint32_t *d_start = L.segs.as<uint32_t>(), *d_end = d_start + T, *d_tcount = d_end + T;
    // answers by template, to choose how they are sorted; not counted where there are too many anyway
    const bool counted = ncand <= (1u << 20);
    L.h_counters.reserve(sizeof(uint32_t) * (8 + static_cast<size_t>(T)));
    uint32_t *hc = L.h_counters.as<uint32_t>();
    if (L.profile)
        TM_CUDA(cudaEventRecord(L.ev2, s));
    TM_CUDA(tmb::launch_rescore(L.cand.as<Candidate>(), ncand, g.tp.as<TemplParam>(), g.q.as<float>(),
                                g.order.as<int>(), ctx->raw.as<float>(), pv, mean, w0, L.dist.as<float>(),
                                L.akeys.as<uint32_t>(), L.counters.as<uint32_t>() + 6, ex, shortest, g.m, ctx->sms, s)); // (the keys come later)
    if (ncand > 0)
        count_launch(L, 2);
    if (L.profile)
        TM_CUDA(cudaEventRecord(L.ev3, s));
    unsigned long long *keys[2] = {L.akeys.as<unsigned long long>(), L.akeys.as<unsigned long long>() + cn};
    float *vals32[2] = {L.avals.as<float>(), L.avals.as<float>() + cn};
    unsigned long long *vals64[2] = {L.avals64.as<unsigned long long>(),
                                     L.avals64.as<unsigned long long>() + (nk > 0 ? cn : 0)};
    TM_CUDA(cudaMemsetAsync(d_kept, 0, 2 * sizeof(uint32_t), s));
    if (counted)
        TM_CUDA(cudaMemsetAsync(d_tcount, 0, sizeof(uint32_t) * T, s));
    TM_CUDA(tmb::launch_answer_keys(L.cand.as<Candidate>(), L.dist.as<float>(), ncand, g.tp.as<TemplParam>(),
                                    keys[0], vals32[0], d_kept, counted ? d_tcount : nullptr, s));
    TM_CUDA(cudaMemcpyAsync(hc + 3, d_kept, 2 * sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    if (counted)
        TM_CUDA(cudaMemcpyAsync(hc + 8, d_tcount, sizeof(uint32_t) * T, cudaMemcpyDeviceToHost, s));
    TM_CUDA(cudaStreamSynchronize(s));
    if (ncand > 0)
        count_launch(L);
    const uint32_t kept = hc[3], knn_kept = hc[4], thr_kept = kept - knn_kept;
    uint32_t *d_knn_n = d_tcount + T, *d_knn_win = d_knn_n + nk;
    float *d_knn_dist = reinterpret_cast<float *>(d_knn_win + static_cast<size_t>(nk) * kcap);
    uint32_t *d_win = reinterpret_cast<uint32_t *>(L.cand.p); // the candidates are consumed: reuse
    float *d_dist = L.dist.as<float>();                       // likewise the re-scored distances
    const uint32_t most = counted && T > 0 ? *std::max_element(hc + 8, hc + 8 + T) : 0;
    if (counted && tmb::answer_runs_apply(kept, T, most))
    {
        TM_CUDA(tmb::launch_answer_runs(keys[0], vals32[0], kept, most, g.tp.as<TemplParam>(), T, d_tcount, d_start, d_end,
                                        d_win, d_dist, s));
        count_launch(L);
    }
    else
    {
        const size_t scratch = tmb::answer_sort_scratch(kept, T);
        L.sort_tmp.reserve(scratch);
        TM_CUDA(cudaMemsetAsync(d_start, 0, 2 * sizeof(uint32_t) * T, s));
        TM_CUDA(tmb::launch_answer_order(keys, vals32, vals64, kept, knn_kept, g.tp.as<TemplParam>(), T, L.sort_tmp.p,
                                         scratch, d_start, d_end, d_win, d_dist, s));
        if (kept > 0)
            count_launch(L, knn_kept > 0 ? 4 : 2); // each radix sort counted as one launch
    }
    if (device_knn)
    {
        TM_CUDA(tmb::launch_select_knn(g.slots.as<int>(), nk, g.tp.as<TemplParam>(), d_start, d_end, d_win, d_dist,
                                       kcap, d_knn_n, d_knn_win, d_knn_dist, s));
        count_launch(L);
    }
    if (L.profile)
        TM_CUDA(cudaEventRecord(L.ev4, s));

    // block layout: win[thr_kept] | dist[thr_kept] | start[T] | end[T] | tkey[T] |
    //               knn_n[nk] | knn_win[nk * kcap] | knn_dist[nk * kcap]
    const size_t knn_words = device_knn ? static_cast<size_t>(nk) * (1 + 2 * kcap) : 0;
    std::shared_ptr<PinnedBlock> block = acquire_block(
        L, sizeof(uint32_t) * (2 * static_cast<size_t>(thr_kept) + 3 * static_cast<size_t>(T) + knn_words) + 64);
    AnswerView v;
    v.win = static_cast<uint32_t *>(block->p);
    v.dist = reinterpret_cast<float *>(v.win + thr_kept);
    uint32_t *h_start = reinterpret_cast<uint32_t *>(v.dist + thr_kept);
    uint32_t *h_tkey = h_start + 2 * static_cast<size_t>(T);
    uint32_t *h_knn = h_tkey + T;
    if (thr_kept > 0)
    {
        TM_CUDA(cudaMemcpyAsync(v.win, d_win, sizeof(uint32_t) * thr_kept, cudaMemcpyDeviceToHost, s));
        TM_CUDA(cudaMemcpyAsync(v.dist, d_dist, sizeof(float) * thr_kept, cudaMemcpyDeviceToHost, s));
    }
    TM_CUDA(cudaMemcpyAsync(h_start, d_start, 2 * sizeof(uint32_t) * T, cudaMemcpyDeviceToHost, s));
    if (nk > 0)
        TM_CUDA(cudaMemcpyAsync(h_tkey, L.tkey.p, sizeof(uint32_t) * T, cudaMemcpyDeviceToHost, s));
    else
        std::fill(h_tkey, h_tkey + T, 0u);
    if (device_knn)
        TM_CUDA(cudaMemcpyAsync(h_knn, d_knn_n, sizeof(uint32_t) * knn_words, cudaMemcpyDeviceToHost, s));
    if (L.profile)
        TM_CUDA(cudaEventRecord(L.ev1, s));
    TM_CUDA(cudaStreamSynchronize(s));
    L.last_candidates += ncand;
    L.d2h_bytes += sizeof(uint32_t) * (2 * static_cast<uint64_t>(thr_kept) + 2 * static_cast<uint64_t>(T) +
                                          (nk > 0 ? T : 0) + knn_words) +
                      16;
    const auto t0 = std::chrono::steady_clock::now();
    if (L.profile)
    {
        add_span(L, 2, L.ev2, L.ev3);
        add_span(L, 3, L.ev3, L.ev4);
        add_span(L, 4, L.ev4, L.ev1);
    }
    v.start = h_start;
    v.end = h_start + T;
    v.tkey = h_tkey;
    v.device_knn = device_knn;
    v.kcap = kcap;
    v.knn_n = h_knn;
    v.knn_win = h_knn + nk;
    v.knn_dist = reinterpret_cast<const float *>(h_knn + nk + static_cast<size_t>(nk) * kcap);
    v.d_win = d_win;
    v.d_dist = d_dist;
    res.blocks.push_back(block);
    finish_answers(L, g, v, w0, res, degenerate_windows);
    if (L.profile)
        L.phase_ms[5] += std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
}

// Does a merge offset of the group exceed a bucket?
static bool super_buckets(const GroupPlan &g, int blog)
{
    for (int t = 0; t < g.T; t++)
        if (g.mode[t] == TM_MODE_KNN && g.merge[t] > (1 << blog))
            return true;
    return false;
}

// The contraction kernels of several lengths see samples that are not finite as 0: minima that may be
// those of windows with such a sample must not bound the answers.
static void forget_odd_buckets(Lane &L, const GroupPlan &g, const tmb::ScanArgs &a)
{
    if (a.odd == nullptr || g.nk == 0)
        return;
    TM_CUDA(tmb::launch_odd_buckets(a.bmin_u, a.nb, a.bucket_log, a.tp, g.slots.as<int>(), g.nk, a.odd, a.w0, a.W, L.stream));
    count_launch(L);
}

// kNN bound, bucket list and FP32 re-pass after a group's contraction (a: its arguments), then
// the counters: the group's candidates, whether the contraction gave up waiting, the candidates for
// want of statistics (in L.h_counters [7]). One wait for the device; a list that did not fit is made again, larger.
static uint32_t collect_candidates(tm_ctx *ctx, Lane &L, const GroupPlan &g, const tmb::ScanArgs &a, bool mixed)
{
    cudaStream_t s = L.stream;
    uint32_t *hc = L.h_counters.as<uint32_t>(), *counters = L.counters.as<uint32_t>();
    if (g.nk > 0)
    {
        const bool super = super_buckets(g, a.bucket_log);
        if (super)
            L.bmin_s.reserve(sizeof(uint32_t) * static_cast<size_t>(g.nk) * a.nb);
        forget_odd_buckets(L, g, a);
        TM_CUDA(tmb::launch_bucket_select(a.bmin_u, L.bmin_s.as<uint32_t>(), a.nb, a.bucket_log, a.tp, g.slots.as<int>(), g.nk,
                                          super, L.tkey.as<uint32_t>(), s));
        count_launch(L, super ? 2 : 1);
    }
    for (int attempt = 0; attempt < 3; attempt++)
    {
        if (g.nk > 0)
        {
            L.list.reserve(sizeof(uint2) * static_cast<size_t>(L.list_cap));
            TM_CUDA(tmb::launch_list_buckets(a.bmin_l, a.nb, g.slots.as<int>(), g.nk, L.tkey.as<uint32_t>(), L.list.as<uint2>(),
                                             counters, L.list_cap, s));
            const bool tight = tight_bounds(g);
            if (tight)
            {
                L.lower.reserve(sizeof(float) * static_cast<size_t>(L.cand_cap));
                L.bins.reserve(sizeof(uint32_t) * tmb::kTightBins * static_cast<size_t>(g.T));
                L.tight.reserve(sizeof(float) * static_cast<size_t>(g.T));
            }
            TM_CUDA(tmb::launch_passb(L.list.as<uint2>(), counters, L.list_cap, a, L.tkey.as<uint32_t>(), mixed,
                                      g.slots.as<int>(), g.nk, tight ? L.lower.as<float>() : nullptr,
                                      tight ? L.bins.as<uint32_t>() : nullptr, L.tight.as<float>(), ctx->sms, s));
            count_launch(L, tight ? 3 : 2);
        }
        if (L.profile)
            TM_CUDA(cudaEventRecord(L.ev2, s));
        TM_CUDA(cudaMemcpyAsync(hc, counters, 8 * sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
        TM_CUDA(cudaStreamSynchronize(s));
        if (L.profile)
            add_span(L, 1, L.ev1, L.ev2);
        if (hc[2] != 0)
            throw Failure{TM_ERR_TIMEOUT, "contraction kernel gave up waiting (code " + std::to_string(hc[2]) + ")"};
        if (g.nk == 0 || hc[1] <= L.list_cap)
            return hc[0];
        // back to the contraction's candidates, and a longer list
        L.list_cap = hc[1] + hc[1] / 2;
        TM_CUDA(cudaMemcpyAsync(counters, counters + 5, sizeof(uint32_t), cudaMemcpyDeviceToDevice, s));
        TM_CUDA(cudaMemsetAsync(counters + 1, 0, sizeof(uint32_t), s));
    }
    throw Failure{TM_ERR_NO_MEMORY, "bucket list overflow"};
}

// Room for the bucket minima of T templates on W windows, and the buckets' size: they are larger where
// small ones would take more than a quarter of the memory that is free without them.
static int reserve_minima(Lane &L, uint64_t T, uint64_t W)
{
    const auto bytes = [&](int blog) { return sizeof(uint32_t) * T * tmb::bucket_count(W, blog); };
    int blog = tmb::bucket_log(T, W);
    if (bytes(blog) > std::min(L.bmin_u.bytes, L.bmin_l.bytes))
    {
        size_t free_b = 0, total_b = 0;
        TM_CUDA(cudaMemGetInfo(&free_b, &total_b));
        blog = tmb::bucket_log(T, W, std::min<uint64_t>(tmb::kMinimaBytes, (free_b + L.bmin_u.bytes + L.bmin_l.bytes) / 4));
    }
    L.bmin_u.reserve(bytes(blog));
    L.bmin_l.reserve(bytes(blog));
    return blog;
}

// Device pipeline and selection for one prepared group; writes answers[index].
void execute_group(tm_ctx *ctx, Lane &L, GroupPlan &g, tm_result &res)
{
    const int m = g.m;
    LengthStats &ls = ensure_length(ctx, L, m);
    const int T = g.T, T_pad = g.T_pad, m_pad = g.m_pad, nk = g.nk;
    const uint64_t w0 = ls.w0, W = ls.W;
    if (W == 0)
    {
        for (int t = 0; t < T; t++)
            res.answers[g.index[t]].set_hits(g.mode[t] == TM_MODE_KNN
                                                 ? std::vector<Hit>(static_cast<size_t>(g.k[t]), Hit{0, FLT_MAX})
                                                 : std::vector<Hit>());
        return;
    }
    if (W >= (1ull << 32))
        throw Failure{TM_ERR_ARGUMENT, "more than 2^32 - 1 windows in one range; split the range"};
    cudaStream_t s = L.stream;
    const bool use_umma = ctx->kernel != TM_KERNEL_FP32 && g.t_rows > 0 && tmb::umma_supported(m, T, W);
    if (ctx->kernel == TM_KERNEL_SPLIT_BF16 && !use_umma)
        throw Failure{TM_ERR_STATE, "split-BF16 kernel not available for this request group"};
    if (use_umma != g.umma_constants) // error-bound constants of the kernel that will run
    {
        for (int t = 0; t < T; t++)
            g.htp[t].a1_main = use_umma ? g.a1_umma[t] : g.htp[t].a1_fp32;
        TM_CUDA(cudaMemcpyAsync(g.tp.p, g.htp.data(), sizeof(TemplParam) * T_pad, cudaMemcpyHostToDevice, s));
        g.umma_constants = use_umma;
    }
    L.tkey.reserve(sizeof(uint32_t) * T);

    const int blog = nk > 0 ? reserve_minima(L, static_cast<uint64_t>(T), W) : tmb::bucket_log(static_cast<uint64_t>(T), W);
    const uint32_t nb = tmb::bucket_count(W, blog);
    L.counters.reserve(8 * sizeof(uint32_t));
    L.h_counters.reserve(8 * sizeof(uint32_t));

    uint32_t ncand = 0;
    for (int attempt = 0; attempt < 3; attempt++)
    {
        L.cand.reserve(sizeof(Candidate) * static_cast<size_t>(L.cand_cap));
        if (nk > 0)
        {
            TM_CUDA(cudaMemsetAsync(L.bmin_u.p, 0xff, sizeof(uint32_t) * static_cast<size_t>(T) * nb, s));
            TM_CUDA(cudaMemsetAsync(L.bmin_l.p, 0xff, sizeof(uint32_t) * static_cast<size_t>(T) * nb, s));
        }
        TM_CUDA(cudaMemsetAsync(L.counters.p, 0, 8 * sizeof(uint32_t), s));
        uint32_t *d_cand_count = L.counters.as<uint32_t>();

        tmb::ScanArgs a{};
        a.x = ctx->clean.as<float>();
        a.q = g.q.as<float>();
        a.tp = g.tp.as<TemplParam>();
        a.mean = ls.mean.as<float>();
        a.inv = ls.inv.as<float>();
        a.w0 = w0;
        a.W = static_cast<uint32_t>(W);
        a.m_pad = m_pad;
        a.T = T;
        a.bmin_u = L.bmin_u.as<uint32_t>();
        a.bmin_l = L.bmin_l.as<uint32_t>();
        a.nb = nb;
        a.bucket_log = blog;
        a.cand = L.cand.as<Candidate>();
        a.cand_count = d_cand_count;
        a.cand_cap = L.cand_cap;
        a.q_hi = g.q_hi.p;
        a.q_lo = g.q_lo.p;
        a.t_rows = g.t_rows;
        a.err = reinterpret_cast<int *>(d_cand_count + 2);

        // 2. contraction with fused epilogue
        if (L.profile)
            TM_CUDA(cudaEventRecord(L.ev0, s));
        a.col_tile = g.col_tile;
        if (use_umma)
            TM_CUDA(g.col_tile > 0 ? tmb::launch_scan_wm(a, s) : tmb::launch_scan_umma(a, s));
        else
        {
            L.fp32_qt.reserve(sizeof(float) * static_cast<size_t>(g.T_pad) * g.m_pad);
            a.qt = L.fp32_qt.as<float>();
            TM_CUDA(tmb::launch_scan_fp32(a, ctx->sms, s));
            count_launch(L); // the template-tile transposition
        }
        count_launch(L);
        if (L.profile)
        {
            TM_CUDA(cudaEventRecord(L.ev1, s));
            TM_CUDA(cudaEventSynchronize(L.ev1));
            float ms = 0.0f;
            TM_CUDA(cudaEventElapsedTime(&ms, L.ev0, L.ev1));
            L.kname = use_umma ? (g.col_tile > 0 ? "k_scan_wm" : "k_scan_umma") : "k_scan_fp32";
            L.prof_launches++;
            L.prof_ms += ms;
            L.phase_ms[0] += ms;
            L.prof_flops += 2.0 * m * static_cast<double>(W) * T;
        }

        // 3. kNN bound, bucket list, FP32 re-pass
        ncand = collect_candidates(ctx, L, g, a, false);
        if (ncand <= L.cand_cap)
            break;
        L.cand_cap = ncand + ncand / 2;
        if (attempt == 2)
            throw Failure{TM_ERR_NO_MEMORY, "candidate buffer overflow"};
    }

    std::vector<uint8_t> flags; // fetched only when some kNN bound is unbounded
    rescore_and_answer(ctx, L, g, ncand, tmb::PrefixView{}, ls.mean.as<float>(), w0, exclusion(L, g, nb, blog), res, [&](int, std::vector<Hit> &degenerate) {
        if (flags.empty())
        {
            flags.resize(W);
            TM_CUDA(cudaMemcpy(flags.data(), ls.flags.p, W, cudaMemcpyDeviceToHost));
        }
        for (uint64_t j = 0; j < W; j++)
            if ((flags[j] & tmb::kFlagDegenerate) && !(flags[j] & tmb::kFlagNotSearched))
                degenerate.push_back(Hit{w0 + j, FLT_MAX});
    });
}

// Spectra of the record's pieces for the FFT branch (tm_fftk.cu), their shifts and norms,
// and the twiddle tables: built once per context and class of lengths, under a lock (serving
// workers may ask at once).
static tm_ctx::FftPieces &ensure_fft(tm_ctx *ctx, Lane &L, int cls)
{
    tm_ctx::FftPieces &f = ctx->fft[cls];
    std::lock_guard<std::mutex> lk(ctx->fft_mu);
    if (f.ready)
        return f;
    ensure_prefix(ctx, L);
    cudaStream_t s = L.stream;
    if (ctx->fft_roots.p == nullptr)
    {
        std::vector<double2> roots(tmb::kFftAllRoots);
        tmb::fft_roots(roots.data());
        DevBuf up;
        up.reserve(sizeof(double2) * roots.size());
        TM_CUDA(cudaMemcpy(up.p, roots.data(), sizeof(double2) * roots.size(), cudaMemcpyHostToDevice));
        std::swap(ctx->fft_roots, up);
        TM_CUDA(cudaDeviceGetAttribute(&ctx->sms, cudaDevAttrMultiProcessorCount, ctx->device));
    }
    const uint32_t P = tmb::fft_pieces(ctx->n, cls);
    f.X.reserve(sizeof(double2) * static_cast<size_t>(P) * tmb::fft_pitch(tmb::fft_class(cls).n));
    f.shift.reserve(sizeof(double) * P);
    f.norm.reserve(sizeof(double) * P);
    TM_CUDA(tmb::launch_fft_pieces(ctx->clean.as<float>(), ctx->n, ctx->pcen.as<double>(), cls,
                                   ctx->fft_roots.as<double2>(), f.X.as<double2>(), f.shift.as<double>(),
                                   f.norm.as<double>(), s));
    count_launch(L);
    TM_CUDA(cudaStreamSynchronize(s));
    f.count = P;
    f.ready = true;
    return f;
}

// The chunks' bounds at the bases of rows [first, first + count), in table; false where the memory
// for them is not to be had: the windows are then all evaluated. All that are kept take at most a
// tenth of the memory that is free without them; those used longest ago go first.
static bool ensure_bounds(tm_ctx *ctx, Lane &L, const GroupPlan &g, int first, int count, const float4 **table)
{
    if (L.no_bounds)
        return false;
    std::lock_guard<std::mutex> lk(ctx->fft_mu);
    const size_t each = sizeof(float4) * tmb::fft_chunks(ctx->n);
    bool wanted[tmb::kFftBases] = {};
    size_t asked = 0, resident = 0;
    std::vector<int> fresh;
    for (int i = first; i < first + count; i++)
    {
        const int base = g.fft_rows[static_cast<size_t>(i)].base;
        if (wanted[base])
            continue;
        wanted[base] = true;
        asked += each;
        if (!ctx->fft_bounds[base].buf)
            fresh.push_back(base);
    }
    if (!fresh.empty())
    {
        for (const tm_ctx::FftBounds &b : ctx->fft_bounds)
            resident += b.buf ? each : 0;
        size_t free_b = 0, total_b = 0;
        TM_CUDA(cudaMemGetInfo(&free_b, &total_b));
        const size_t budget = (free_b + resident) / 10, more = each * fresh.size();
        if (asked > budget)
            return false;
        while (resident + more > budget)
        {
            tm_ctx::FftBounds *oldest = nullptr;
            for (int base = 0; base < tmb::kFftBases; base++)
                if (ctx->fft_bounds[base].buf && !wanted[base] &&
                    (oldest == nullptr || ctx->fft_bounds[base].last_use < oldest->last_use))
                    oldest = &ctx->fft_bounds[base];
            oldest->buf.reset(); // there is one: those wanted fit the budget
            resident -= each;
        }
        std::vector<std::shared_ptr<ScopedBuf>> built;
        try
        {
            const tmb::PrefixView pv{ctx->prefix.as<double2>(), ctx->ptot.as<double2>(), ctx->pcen.as<double>()};
            for (const int base : fresh)
            {
                built.push_back(std::make_shared<ScopedBuf>());
                built.back()->reserve(each);
                TM_CUDA(tmb::launch_chunk_bounds(pv, ctx->run.as<uint16_t>(), ctx->n, tmb::fft_base_length(base),
                                                 built.back()->as<float4>(), L.stream));
                count_launch(L);
            }
            TM_CUDA(cudaStreamSynchronize(L.stream)); // other lanes' streams read them
        }
        catch (const Failure &f)
        {
            cudaStreamSynchronize(L.stream);
            if (f.code != TM_ERR_NO_MEMORY)
                throw;
            return false;
        }
        for (size_t i = 0; i < fresh.size(); i++)
            ctx->fft_bounds[fresh[i]].buf = built[i];
    }
    ctx->fft_bounds_clock++;
    for (int base = 0; base < tmb::kFftBases; base++)
        if (wanted[base])
        {
            ctx->fft_bounds[base].last_use = ctx->fft_bounds_clock;
            L.bounds.push_back(ctx->fft_bounds[base].buf);
            table[base] = ctx->fft_bounds[base].buf->as<float4>();
        }
    return true;
}

// Gives the chunks' bounds back; false where there were none.
static bool drop_bounds(tm_ctx *ctx)
{
    std::lock_guard<std::mutex> lk(ctx->fft_mu);
    bool any = false;
    for (tm_ctx::FftBounds &b : ctx->fft_bounds)
    {
        any = any || b.buf != nullptr;
        b.buf.reset();
    }
    return any;
}

// Where a launch of kNN templates over the pieces from p0 on ends. A bound from the minima of the
// first sixteenth of the pieces, then of the first quarter, lets the rest skip almost all of
// its windows (tm_fftk.cu); where a launch would have fewer than four items per block, the
// bound would come too late or too dear, and there is one launch. (A sixty-fourth first: 1 % less
// for 128 to 512 templates on 2^25 samples and more, 1 % more for 8.)
uint32_t fft_stage_end(uint32_t p0, uint32_t pieces, int rows, int cls, int sms)
{
    const uint64_t blocks = static_cast<uint64_t>(sms) * (tmb::fft_class(cls).n == 4096 ? 2 : 1);
    const uint64_t least = (4 * blocks + static_cast<uint64_t>(rows) - 1) / static_cast<uint64_t>(rows);
    const uint64_t first = std::max<uint64_t>((pieces + 15) / 16, least);
    for (uint64_t end = first; 2 * end <= pieces; end *= 4)
        if (end > p0)
            return static_cast<uint32_t>(end);
    return pieces;
}

FftRange fft_range(const tm_ctx *ctx, int cls, uint64_t windows)
{
    if (windows == 0)
        return FftRange{0, 0};
    const uint64_t step = tmb::fft_class(cls).step, first = ctx->range_first / step;
    const uint64_t last = std::min<uint64_t>((ctx->range_first + windows - 1) / step, tmb::fft_pieces(ctx->n, cls) - 1);
    return FftRange{static_cast<uint32_t>(first), static_cast<uint32_t>(last - first + 1)};
}

FftSkips fft_skips(const tm_ctx *ctx, int cls, uint32_t pieces, int rows)
{
    // fewer items than multiprocessors: bounds and cuts would cost more than they save
    FftSkips skips;
    if (!ctx->fft_skip || static_cast<uint64_t>(pieces) * static_cast<uint64_t>(rows) < static_cast<uint64_t>(ctx->sms))
        return skips;
    skips.thresholds = true;
    for (uint32_t p = fft_stage_end(0, pieces, rows, cls, ctx->sms); p < pieces; p = fft_stage_end(p, pieces, rows, cls, ctx->sms))
        if (++skips.cuts == 1)
            skips.knn_first = static_cast<double>(p) / pieces;
    return skips;
}

// The FFT branch of a group: per set of rows (prepare_fft), their spectra, then persistent
// launches over the pieces their windows touch.
void fft_contract(tm_ctx *ctx, Lane &L, const GroupPlan &g, const tmb::ScanArgs &a)
{
    cudaStream_t s = L.stream;
    for (const GroupPlan::FftSet &set : g.fft_sets)
    {
        const tm_ctx::FftPieces &X = ensure_fft(ctx, L, set.cls);
        const uint32_t step = tmb::fft_class(set.cls).step;
        const size_t pitch = tmb::fft_pitch(tmb::fft_class(set.cls).n) * static_cast<size_t>(set.parts);
        const int most = tmb::fft_launch_rows(set.cls, set.parts);
        L.fft_Y.reserve(sizeof(double2) * static_cast<size_t>(std::min(most, set.count)) * pitch);
        L.fft_stats.reserve(sizeof(float4) * static_cast<size_t>(ctx->sms) * tmb::kFftStats);
        for (int r0 = 0; r0 < set.count; r0 += most)
        {
            const int nr = std::min(most, set.count - r0), first = set.first + r0;
            tmb::FftArgs f{};
            f.rows = g.d_fft.as<tmb::FftRow>() + first;
            f.nrows = nr;
            f.parts = set.parts;
            TM_CUDA(tmb::launch_fft_templates(g.q.as<float>(), g.tp.as<TemplParam>(), f.rows, nr, set.cls, set.parts,
                                              ctx->fft_roots.as<double2>(), L.fft_Y.as<double2>(), s));
            uint64_t wmax = 0;
            int knn = 0;
            for (int i = 0; i < nr; i++)
            {
                const tmb::FftRow &r = g.fft_rows[static_cast<size_t>(first + i)];
                wmax = std::max<uint64_t>(wmax, r.wcount);
                knn += r.mode == TM_MODE_KNN ? 1 : 0;
            }
            const FftRange range = fft_range(ctx, set.cls, wmax);
            const uint32_t pa = range.first, pieces = range.count;
            f.X = X.X.as<double2>();
            f.shifts = X.shift.as<double>();
            f.norms = X.norm.as<double>();
            f.pieces = X.count;
            f.Y = L.fft_Y.as<double2>();
            f.w0 = a.w0;
            f.W = a.W;
            f.pv = tmb::PrefixView{a.P, a.PT, a.PC};
            f.run = a.run;
            f.mean = a.mean;
            f.inv = a.inv;
            f.untrusted = a.cand_count + 7;
            f.bmin_u = a.bmin_u;
            f.bmin_l = a.bmin_l;
            f.nb = a.nb;
            f.bucket_log = a.bucket_log;
            f.cand = a.cand;
            f.cand_count = a.cand_count;
            f.cand_cap = a.cand_cap;
            f.dbg_d = a.dbg_d;
            f.dbg_e = a.dbg_e;
            f.stats = L.fft_stats.as<float4>();
            count_launch(L);
            const FftSkips skips = fft_skips(ctx, set.cls, pieces, nr);
            const bool cuts = (skips.cuts > 0 || (skips.thresholds && knn < nr)) && a.dbg_d == nullptr &&
                              ensure_bounds(ctx, L, g, first, nr, f.bounds);
            for (uint32_t p0 = 0; p0 < pieces;)
            {
                const uint32_t p1 = knn > 0 && cuts ? fft_stage_end(p0, pieces, nr, set.cls, ctx->sms) : pieces;
                f.p_first = pa + p0;
                f.p_count = p1 - p0;
                f.prune = cuts && (knn < nr || p0 > 0) ? 1 : 0;
                TM_CUDA(tmb::launch_fft_corr(f, set.cls, ctx->fft_roots.as<double2>(), ctx->sms, s));
                count_launch(L);
                p0 = p1;
                if (p0 == pieces)
                    break;
                const uint64_t seen = static_cast<uint64_t>(pa + p0) * step - a.w0; // windows
                const uint32_t nb_seen =
                    static_cast<uint32_t>(std::min<uint64_t>(a.nb, (seen + (1ull << a.bucket_log) - 1) >> a.bucket_log));
                const bool super = super_buckets(g, a.bucket_log);
                if (super)
                    L.bmin_s.reserve(sizeof(uint32_t) * static_cast<size_t>(g.nk) * a.nb);
                L.fft_cuts.reserve(sizeof(float) * static_cast<size_t>(nr));
                forget_odd_buckets(L, g, a);
                TM_CUDA(tmb::launch_fft_cuts(f.rows, nr, a.bmin_u, L.bmin_s.as<uint32_t>(), a.nb, nb_seen, a.bucket_log, a.tp,
                                             g.slots.as<int>(), g.nk, super, L.fft_cuts.as<float>(), s));
                count_launch(L, super ? 2 : 1);
                f.cuts = L.fft_cuts.as<float>();
            }
        }
    }
}

// Device pipeline for a mixed-length group (tensor-core kernels or the FFT branch).
void execute_group_mixed(tm_ctx *ctx, Lane &L, GroupPlan &g, tm_result &res)
{
    if (ctx->kernel == TM_KERNEL_FP32 && !g.fft)
        throw Failure{TM_ERR_STATE, "batch of several template lengths was prepared for the tensor-core kernel"};
    ensure_prefix(ctx, L);
    refresh_range(ctx, L, g);
    const int T = g.T, nk = g.nk;
    const uint64_t w0 = ctx->range_first, W = g.w_max;
    if (W == 0)
    {
        for (int t = 0; t < T; t++)
            if (g.index[t] >= 0)
                res.answers[g.index[t]].set_hits(g.mode[t] == TM_MODE_KNN
                                                     ? std::vector<Hit>(static_cast<size_t>(g.k[t]), Hit{0, FLT_MAX})
                                                     : std::vector<Hit>());
        return;
    }
    if (W >= (1ull << 32))
        throw Failure{TM_ERR_ARGUMENT, "more than 2^32 - 1 windows in one range; split the range"};
    cudaStream_t s = L.stream;
    L.tkey.reserve(sizeof(uint32_t) * T);
    const int blog = nk > 0 ? reserve_minima(L, static_cast<uint64_t>(T), W) : tmb::bucket_log(static_cast<uint64_t>(T), W);
    const uint32_t nb = tmb::bucket_count(W, blog);
    L.counters.reserve(8 * sizeof(uint32_t));
    L.h_counters.reserve(8 * sizeof(uint32_t));
    // The prefix sums lose the windows of a block that is much louder elsewhere: every template of the
    // group would have all of them re-scored, by their chains. Where a group of one length takes more
    // time so than the statistics of the length and another contraction, it has these (they stay, for the
    // next searches): 130 templates of 1500 on 2^17 samples, 4000 of them 10^5 times the rest: 25 ms
    // with prefix sums alone, 2.3 with both. (The context keeps these statistics for its own lane only.)
    bool one_length = g.fft && &L == &ctx->main && g.htp[0].m == g.htp[T - 1].m;
    LengthStats *ls = one_length && ctx->lengths.count(g.m) > 0 ? &ensure_length(ctx, L, g.m) : nullptr;
    const double chain_ms = 1.8e-9 * g.m; // of a candidate without statistics
    const double again_ms = 0.1 + static_cast<double>(W) / 33554432.0 * (1.0 + 0.15 * T);
    double flops = 0.0;
    for (int t = 0; t < T; t++)
        flops += 2.0 * g.htp[t].m * static_cast<double>(g.htp[t].wcount);

    uint32_t ncand = 0;
    for (int attempt = 0; attempt < 3; attempt++)
    {
        L.cand.reserve(sizeof(Candidate) * static_cast<size_t>(L.cand_cap));
        if (nk > 0)
        {
            TM_CUDA(cudaMemsetAsync(L.bmin_u.p, 0xff, sizeof(uint32_t) * static_cast<size_t>(T) * nb, s));
            TM_CUDA(cudaMemsetAsync(L.bmin_l.p, 0xff, sizeof(uint32_t) * static_cast<size_t>(T) * nb, s));
        }
        TM_CUDA(cudaMemsetAsync(L.counters.p, 0, 8 * sizeof(uint32_t), s));
        uint32_t *d_cand_count = L.counters.as<uint32_t>();
        tmb::ScanArgs a{};
        a.x = ctx->clean.as<float>();
        a.q = g.q.as<float>();
        a.tp = g.tp.as<TemplParam>();
        a.w0 = w0;
        a.W = static_cast<uint32_t>(W);
        a.m_pad = g.k_stride;
        a.T = T;
        a.bmin_u = L.bmin_u.as<uint32_t>();
        a.bmin_l = L.bmin_l.as<uint32_t>();
        a.nb = nb;
        a.bucket_log = blog;
        a.cand = L.cand.as<Candidate>();
        a.cand_count = d_cand_count;
        a.cand_cap = L.cand_cap;
        a.q_hi = g.q_hi.p;
        a.q_lo = g.q_lo.p;
        a.t_rows = g.t_rows;
        a.err = reinterpret_cast<int *>(d_cand_count + 2);
        a.raw = ctx->raw.as<float>();
        a.P = ctx->prefix.as<double2>();
        a.PT = ctx->ptot.as<double2>();
        a.PC = ctx->pcen.as<double>();
        a.mean = ls != nullptr ? ls->mean.as<float>() : nullptr;
        a.inv = ls != nullptr ? ls->inv.as<float>() : nullptr;
        a.run = ctx->run.as<uint16_t>();
        a.odd = ctx->odd.as<uint32_t>();
        a.tiles = g.d_tiles.as<tmb::TileInfo>();
        a.k_stride = g.k_stride;
        a.n = ctx->n;
        if (L.profile)
            TM_CUDA(cudaEventRecord(L.ev0, s));
        a.col_tile = g.col_tile;
        if (g.fft)
            fft_contract(ctx, L, g, a);
        else
        {
            TM_CUDA(g.col_tile > 0 ? tmb::launch_scan_wm(a, s) : tmb::launch_scan_umma(a, s));
            count_launch(L);
        }
        if (L.profile)
        {
            TM_CUDA(cudaEventRecord(L.ev1, s));
            TM_CUDA(cudaEventSynchronize(L.ev1));
            float ms = 0.0f;
            TM_CUDA(cudaEventElapsedTime(&ms, L.ev0, L.ev1));
            L.kname = g.fft ? "fft" : (g.col_tile > 0 ? "k_scan_wm" : "k_scan_umma");
            L.prof_launches++;
            L.prof_ms += ms;
            L.phase_ms[0] += ms;
            L.prof_flops += flops;
        }
        ncand = collect_candidates(ctx, L, g, a, true);
        if (one_length && ls == nullptr && chain_ms * L.h_counters.as<uint32_t>()[7] > again_ms)
        {
            try
            {
                ls = &ensure_length(ctx, L, g.m);
                attempt--;
                continue;
            }
            catch (const Failure &f)
            {
                if (f.code != TM_ERR_NO_MEMORY)
                    throw;
                one_length = false; // as slow as it is, then
            }
        }
        if (ncand <= L.cand_cap)
            break;
        L.cand_cap = ncand + ncand / 2;
        if (attempt == 2)
            throw Failure{TM_ERR_NO_MEMORY, "candidate buffer overflow"};
    }
    std::vector<uint16_t> run;
    std::vector<float> raw;
    std::vector<uint32_t> odd; // stays empty where all samples are finite
    const tmb::PrefixView pv{ctx->prefix.as<double2>(), ctx->ptot.as<double2>(), ctx->pcen.as<double>()};
    rescore_and_answer(ctx, L, g, ncand, pv, nullptr, w0, exclusion(L, g, nb, blog), res, [&](int t, std::vector<Hit> &degenerate) {
        if (run.empty())
        {
            run.resize(W);
            raw.resize(W);
            TM_CUDA(cudaMemcpy(run.data(), ctx->run.as<uint16_t>() + w0, W * sizeof(uint16_t), cudaMemcpyDeviceToHost));
            TM_CUDA(cudaMemcpy(raw.data(), ctx->raw.as<float>() + w0, W * sizeof(float), cudaMemcpyDeviceToHost));
            if (ctx->odd.p != nullptr)
            {
                odd.resize(W);
                TM_CUDA(cudaMemcpy(odd.data(), ctx->odd.as<uint32_t>() + w0, W * sizeof(uint32_t), cudaMemcpyDeviceToHost));
            }
        }
        const TemplParam &p = g.htp[t];
        const uint64_t windows = windows_in_range(ctx, p.m);
        for (uint64_t j = 0; j < windows; j++)
            if (run[j] >= p.m && raw[j] != TM_MISSING_VALUE && (odd.empty() || odd[j] >= static_cast<uint32_t>(p.m)))
                degenerate.push_back(Hit{w0 + j, FLT_MAX});
    });
}

static void run_groups(tm_ctx *ctx, Lane &L, tm_batch &b, tm_result &res)
{
    res.answers.assign(static_cast<size_t>(b.count), Answer());
    res.blocks.clear();
    L.last_candidates = 0;
    for (GroupPlan &g : b.groups)
    {
        if (g.mixed)
            execute_group_mixed(ctx, L, g, res);
        else
            execute_group(ctx, L, g, res);
    }
}

void run_batch(tm_ctx *ctx, Lane &L, tm_batch &b, tm_result &res)
{
    struct Held // the bounds that a search reads, let go when it ends
    {
        Lane &L;
        ~Held()
        {
            L.bounds.clear();
            L.no_bounds = false;
        }
    } held{L};
    try
    {
        run_groups(ctx, L, b, res);
    }
    catch (const Failure &f)
    {
        // the chunks' bounds save time, not more: without them where the memory is needed
        if (f.code != TM_ERR_NO_MEMORY)
            throw;
        cudaStreamSynchronize(L.stream);
        L.bounds.clear();
        if (!drop_bounds(ctx))
            throw;
        L.no_bounds = true;
        run_groups(ctx, L, b, res);
    }
}

int validate_requests(const tm_ctx *ctx, const tm_request *reqs, int count)
{
    if (count < 0 || (count > 0 && reqs == nullptr))
        return TM_ERR_ARGUMENT;
    for (int i = 0; i < count; i++)
    {
        const tm_request &r = reqs[i];
        if (r.templ == nullptr || r.m < 1 || static_cast<uint64_t>(r.m) > ctx->n || r.merge_offset < 0)
            return TM_ERR_ARGUMENT;
        if (r.mode == TM_MODE_KNN)
        {
            if (r.k < 1)
                return TM_ERR_ARGUMENT;
        }
        else if (r.mode != TM_MODE_THRESHOLD)
            return TM_ERR_ARGUMENT;
    }
    return TM_OK;
}

} // namespace tmh
