// Preparation of a batch's groups on the host: bit-identical template z-normalisation
// and block order (tm_host.cpp), the epilogue's error-bound constants, BF16 halves, row
// or column tiles of templates of several lengths, and the planner that splits each group
// between the FFT branch and a tile shape.
#include "tm_core.h"

namespace tmh {

// Epilogue constants of one template (error-bound terms of fast_distance).
void fill_param(TemplParam &p, int m, double q2, double s1, double gamma_main, double gamma_fp32)
{
    const double qn = std::sqrt(q2), qs = qn * std::sqrt(static_cast<double>(m));
    const double md = static_cast<double>(m);
    const double safety = 1.25;
    p.s1 = static_cast<float>(s1);
    p.c_lin = static_cast<float>(q2 + md);
    p.a1_main = static_cast<float>(safety * 2.0 * (gamma_main + 6.0 * kU) * qs);
    p.a1_fp32 = static_cast<float>(safety * 2.0 * (gamma_fp32 + 6.0 * kU) * qs);
    p.a2 = static_cast<float>(safety * (4.02 * kU * qs + 10.11 * kU * md + 4.0 * kU * (q2 + md)) + 1e-6 * md);
    p.a3 = static_cast<float>(safety * (md / 16.0 + 40.0) * kU);
    p.a4 = static_cast<float>(safety * 8.0 * md * md * kE64);
    p.a5 = static_cast<float>(safety * md * kU * kU);
    p.a6 = static_cast<float>(safety * 8.0 * kU * std::fabs(s1));
    p.m = m;
}

// FP32 chain: one FMA per sample and accumulator; split BF16: three products per
// sample plus the tensor-core accumulation (truncating adds, 2^-22 per MMA step).
double gamma_fp32(int m) { return 1.01 * static_cast<double>((m + 63) & ~63) * kU; }
// FFT branch: the transform's error has its own term, and what is left is the rounding of the dot product
// to float, one unit of at most qs sqrt(1 + r^2) standard deviations, twice that here. (With the
// tensor cores' 1.2e-5 in its place, r up to 27 where a record drifts 200 standard deviations per
// block, 128 kNN templates of 4096 on 2^21 samples left 50 million candidates, 161 ms; now 1.9, 8.8.)
double gamma_fft() { return 2.0 * kU; }
double gamma_bf16(int m) { return 1.2e-5 + (3.0 * ((m + 63) & ~63) / 16.0 + 16.0) * 2.384185791015625e-07; }

// A z-normalised template with a value that is not finite has a finite distance to no window, and on
// the device it is 0, with the constants of padding: the kernels bound a window's error for all
// templates of a tile or length at once. finish_answers has what is left of its answer.
static bool make_inert(GroupPlan &g, int t, float *q, TemplParam &p)
{
    std::fill(q, q + p.m, 0.0f);
    fill_param(p, p.m, 0.0, 0.0, 0.0, 0.0);
    p.mode = TM_MODE_THRESHOLD;
    p.thr_ed = g.thr[t] = -FLT_MAX;
    return g.inert[t] = true;
}

// Host preparation of one group (bit-identical template z-normalisation and block
// order, epilogue constants) and its upload.
void prepare_group(tm_ctx *ctx, Lane &L, int m, const std::vector<int> &idx, const tm_request *reqs, GroupPlan &g,
                   uint64_t &h2d, int col_tile)
{
    g.m = m;
    g.mixed = false; // a reused plan may have held another kind of group
    g.fft = false;
    g.col_tile = col_tile; // tensor cores: window-major column tiles (k_scan_wm) when > 0
    g.T = static_cast<int>(idx.size());
    g.T_pad = (g.T + 63) & ~63;
    g.m_pad = (m + 63) & ~63;
    g.nblk = std::max(1, m / tm_host::kZnormBlock);
    g.umma_constants = false;
    g.index = idx;
    const int T = g.T, T_pad = g.T_pad, m_pad = g.m_pad, nblk = g.nblk;
    L.h_q.reserve(sizeof(float) * static_cast<size_t>(T_pad) * m_pad);
    L.h_order.reserve(sizeof(int) * static_cast<size_t>(T) * nblk);
    L.h_slots.reserve(sizeof(int) * T);
    float *hq = L.h_q.as<float>();
    int *ho = L.h_order.as<int>();
    int *hslots = L.h_slots.as<int>();
    std::memset(hq, 0, sizeof(float) * static_cast<size_t>(T_pad) * m_pad);
    std::memset(ho, 0, sizeof(int) * static_cast<size_t>(T) * nblk);
    g.htp.assign(T_pad, TemplParam{});
    g.mode.assign(T, 0);
    g.k.assign(T, 0);
    g.merge.assign(T, 0);
    g.thr.assign(T, 0.0f);
    g.a1_umma.assign(T, 0.0f);
    g.inert.assign(T, 0);
    g.nk = 0;
    for (int t = 0; t < T; t++)
    {
        const tm_request *r = &reqs[idx[t]];
        float *q = hq + static_cast<size_t>(t) * m_pad;
        std::memcpy(q, r->templ, sizeof(float) * m);
        if (!(r->flags & TM_FLAG_ZNORMALIZED))
            tm_host::znormalize(q, m);
        tm_host::block_order(q, m, ho + static_cast<size_t>(t) * nblk);
        double q2 = 0.0, s1 = 0.0;
        for (int i = 0; i < m; i++)
        {
            q2 += static_cast<double>(q[i]) * q[i];
            s1 += q[i];
        }
        TemplParam &p = g.htp[t];
        fill_param(p, m, q2, s1, gamma_bf16(m), gamma_fp32(m));
        g.a1_umma[t] = p.a1_main;
        p.a1_main = p.a1_fp32;
        p.mode = g.mode[t] = r->mode;
        p.k = g.k[t] = r->k;
        p.merge = g.merge[t] = r->merge_offset;
        p.q_offset = static_cast<int64_t>(t) * m_pad;
        p.order_offset = static_cast<int64_t>(t) * nblk;
        if (!std::isfinite(q2) && make_inert(g, t, q, p))
            g.a1_umma[t] = 0.0f;
        else if (r->mode == TM_MODE_KNN)
            hslots[g.nk++] = t;
        else
            p.thr_ed = g.thr[t] = tm_host::cc_to_ed(r->correlation, m);
    }
    for (int t = T; t < T_pad; t++)
    {
        g.htp[t].mode = TM_MODE_THRESHOLD;
        g.htp[t].thr_ed = -FLT_MAX;
        g.htp[t].m = m;
    }
    cudaStream_t s = L.stream;
    g.q.reserve_on(sizeof(float) * static_cast<size_t>(T_pad) * m_pad, s, ctx->pool);
    g.order.reserve_on(sizeof(int) * static_cast<size_t>(T) * nblk, s, ctx->pool);
    g.tp.reserve_on(sizeof(TemplParam) * T_pad, s, ctx->pool);
    g.slots.reserve_on(sizeof(int) * std::max(g.nk, 1), s, ctx->pool);
    TM_CUDA(cudaMemcpyAsync(g.q.p, hq, sizeof(float) * static_cast<size_t>(T_pad) * m_pad, cudaMemcpyHostToDevice, s));
    TM_CUDA(cudaMemcpyAsync(g.order.p, ho, sizeof(int) * static_cast<size_t>(T) * nblk, cudaMemcpyHostToDevice, s));
    TM_CUDA(cudaMemcpyAsync(g.tp.p, g.htp.data(), sizeof(TemplParam) * T_pad, cudaMemcpyHostToDevice, s));
    if (g.nk > 0)
        TM_CUDA(cudaMemcpyAsync(g.slots.p, hslots, sizeof(int) * g.nk, cudaMemcpyHostToDevice, s));
    if (ctx->kernel != TM_KERNEL_FP32)
    {
        // BF16 halves for the tensor-core kernel: q = hi + lo (round to nearest even)
        g.t_rows = (T + 127) & ~127;
        const size_t elems = static_cast<size_t>(g.t_rows) * m_pad;
        L.h_split.reserve(2 * sizeof(uint16_t) * elems);
        uint16_t *hh = L.h_split.as<uint16_t>(), *hl = hh + elems;
        std::memset(hh, 0, 2 * sizeof(uint16_t) * elems);
        for (int t = 0; t < T; t++)
            for (int i = 0; i < m; i++)
            {
                const size_t at = static_cast<size_t>(t) * m_pad + i;
                const float v = hq[at];
                hh[at] = bf16_bits(v);
                hl[at] = bf16_bits(v - bf16_value(hh[at]));
            }
        g.q_hi.reserve_on(sizeof(uint16_t) * elems, s, ctx->pool);
        g.q_lo.reserve_on(sizeof(uint16_t) * elems, s, ctx->pool);
        TM_CUDA(cudaMemcpyAsync(g.q_hi.p, hh, sizeof(uint16_t) * elems, cudaMemcpyHostToDevice, s));
        TM_CUDA(cudaMemcpyAsync(g.q_lo.p, hl, sizeof(uint16_t) * elems, cudaMemcpyHostToDevice, s));
        h2d += 2 * sizeof(uint16_t) * static_cast<uint64_t>(T) * m;
    }
    // the staging buffers are reused by the next group: finish the copies first
    TM_CUDA(cudaStreamSynchronize(s));
    h2d += sizeof(float) * static_cast<uint64_t>(T) * m + sizeof(int) * static_cast<uint64_t>(T) * nblk +
           sizeof(TemplParam) * T_pad;
}

// Host preparation of a mixed-length group: templates sorted by length (longest first),
// in tiles of 128 rows (col_tile 0, k_scan_umma) or col_tile rows (k_scan_wm), any
// lengths. Padding rows are inert; a tile's K extent is its longest template (shorter rows are
// zero-padded, which leaves their dot products unchanged). Rows are the template slots of
// the group: g.index[row] is the request (-1 for padding rows). A group for the FFT branch
// (fft; prepare_fft completes it and waits for the copies) has no tiles: one row per template,
// as long as that needs, and no BF16 halves. Padded like the tiles, 8 templates of 16384 samples
// took 16 MB of copies and 128 rows of bucket minima.
void prepare_group_mixed(tm_ctx *ctx, Lane &L, const std::vector<int> &idx_in, const tm_request *reqs, GroupPlan &g,
                         uint64_t &h2d, int col_tile, bool fft)
{
    std::vector<int> idx = idx_in;
    std::stable_sort(idx.begin(), idx.end(), [&](int a, int b) { return reqs[a].m > reqs[b].m; });
    const size_t tile_rows = fft ? 1 : col_tile > 0 ? static_cast<size_t>(col_tile) : 128;
    // rows: request per row (-1 = padding)
    std::vector<int> rows;
    std::vector<tmb::TileInfo> tiles;
    std::vector<int> tile_len; // the longest template of each tile
    for (size_t i = 0; i < idx.size();)
    {
        const size_t start = rows.size();
        const int longest = reqs[idx[i]].m;
        while (i < idx.size() && rows.size() - start < tile_rows)
            rows.push_back(idx[i++]);
        while (rows.size() - start < tile_rows)
            rows.push_back(-1);
        tiles.push_back(tmb::TileInfo{(longest + 63) / 64});
        tile_len.push_back(longest);
    }
    const int R = static_cast<int>(rows.size()); // multiple of the tile rows
    const int m_max = reqs[idx[0]].m;
    g.mixed = true;
    g.col_tile = col_tile;
    g.fft = false;
    g.m = m_max;
    g.T = R;
    g.T_pad = R;
    g.t_rows = R;
    g.k_stride = (m_max + 63) & ~63;
    g.m_pad = g.k_stride;
    g.nblk = std::max(1, g.k_stride / tm_host::kZnormBlock);
    g.umma_constants = true;
    g.index = rows;
    const int stride = g.k_stride;
    // where each row's samples and block order begin
    std::vector<size_t> q_at(static_cast<size_t>(R) + 1, 0), o_at(static_cast<size_t>(R) + 1, 0);
    for (int t = 0; t < R; t++)
    {
        const int len = fft ? (reqs[rows[t]].m + 63) & ~63 : stride;
        q_at[t + 1] = q_at[t] + static_cast<size_t>(len);
        o_at[t + 1] = o_at[t] + static_cast<size_t>(std::max(1, len / tm_host::kZnormBlock));
    }
    const size_t elems = q_at[R], orders = o_at[R];
    L.h_q.reserve(sizeof(float) * elems);
    L.h_order.reserve(sizeof(int) * orders);
    L.h_slots.reserve(sizeof(int) * R);
    float *hq = L.h_q.as<float>();
    int *ho = L.h_order.as<int>();
    int *hslots = L.h_slots.as<int>();
    uint16_t *hh = nullptr, *hl = nullptr;
    std::memset(hq, 0, sizeof(float) * elems);
    std::memset(ho, 0, sizeof(int) * orders);
    if (!fft)
    {
        L.h_split.reserve(2 * sizeof(uint16_t) * elems);
        hh = L.h_split.as<uint16_t>();
        hl = hh + elems;
        std::memset(hh, 0, 2 * sizeof(uint16_t) * elems);
    }
    g.htp.assign(R, TemplParam{});
    g.mode.assign(R, TM_MODE_THRESHOLD);
    g.k.assign(R, 0);
    g.merge.assign(R, 0);
    g.thr.assign(R, -FLT_MAX);
    g.a1_umma.assign(R, 0.0f);
    g.inert.assign(R, 0);
    g.range_first = ctx->range_first;
    g.range_count = ctx->range_count;
    g.nk = 0;
    g.w_max = 0;
    uint64_t samples = 0;
    for (int t = 0; t < R; t++)
    {
        TemplParam &p = g.htp[t];
        if (rows[t] < 0)
        {
            p.mode = TM_MODE_THRESHOLD;
            p.thr_ed = -FLT_MAX;
            p.m = tile_len[static_cast<size_t>(t) / tile_rows];
            p.inv_m = 1.0 / p.m;
            p.wcount = 0;
            continue;
        }
        const tm_request *r = &reqs[rows[t]];
        const int m = r->m;
        samples += static_cast<uint64_t>(m);
        float *q = hq + q_at[t];
        std::memcpy(q, r->templ, sizeof(float) * m);
        if (!(r->flags & TM_FLAG_ZNORMALIZED))
            tm_host::znormalize(q, m);
        tm_host::block_order(q, m, ho + o_at[t]);
        double q2 = 0.0, s1 = 0.0;
        for (int i = 0; i < m; i++)
        {
            q2 += static_cast<double>(q[i]) * q[i];
            s1 += q[i];
        }
        fill_param(p, m, q2, s1, fft ? gamma_fft() : gamma_bf16(m), gamma_fp32(m));
        g.a1_umma[t] = p.a1_main;
        p.inv_m = 1.0 / static_cast<double>(m);
        p.qs = static_cast<float>(std::sqrt(q2 * m));
        p.wcount = static_cast<uint32_t>(windows_in_range(ctx, m));
        g.w_max = std::max(g.w_max, p.wcount);
        p.mode = g.mode[t] = r->mode;
        p.k = g.k[t] = r->k;
        p.merge = g.merge[t] = r->merge_offset;
        p.q_offset = static_cast<int64_t>(q_at[t]);
        p.order_offset = static_cast<int64_t>(o_at[t]);
        if (!std::isfinite(q2) && make_inert(g, t, q, p))
        {
            g.a1_umma[t] = p.qs = 0.0f;
            p.wcount = 0;
        }
        else if (r->mode == TM_MODE_KNN)
            hslots[g.nk++] = t;
        else
            p.thr_ed = g.thr[t] = tm_host::cc_to_ed(r->correlation, m);
        for (int i = 0; i < m && !fft; i++)
        {
            const size_t at = q_at[t] + static_cast<size_t>(i);
            hh[at] = bf16_bits(q[i]);
            hl[at] = bf16_bits(q[i] - bf16_value(hh[at]));
        }
    }
    g.tiles = tiles;
    cudaStream_t s = L.stream;
    g.q.reserve_on(sizeof(float) * elems, s, ctx->pool);
    g.order.reserve_on(sizeof(int) * orders, s, ctx->pool);
    g.tp.reserve_on(sizeof(TemplParam) * R, s, ctx->pool);
    g.slots.reserve_on(sizeof(int) * std::max(g.nk, 1), s, ctx->pool);
    TM_CUDA(cudaMemcpyAsync(g.q.p, hq, sizeof(float) * elems, cudaMemcpyHostToDevice, s));
    TM_CUDA(cudaMemcpyAsync(g.order.p, ho, sizeof(int) * orders, cudaMemcpyHostToDevice, s));
    TM_CUDA(cudaMemcpyAsync(g.tp.p, g.htp.data(), sizeof(TemplParam) * R, cudaMemcpyHostToDevice, s));
    if (g.nk > 0)
        TM_CUDA(cudaMemcpyAsync(g.slots.p, hslots, sizeof(int) * g.nk, cudaMemcpyHostToDevice, s));
    h2d += samples * sizeof(float) + sizeof(int) * orders + sizeof(TemplParam) * R;
    if (fft)
        return;
    g.q_hi.reserve_on(sizeof(uint16_t) * elems, s, ctx->pool);
    g.q_lo.reserve_on(sizeof(uint16_t) * elems, s, ctx->pool);
    g.d_tiles.reserve_on(sizeof(tmb::TileInfo) * tiles.size(), s, ctx->pool);
    TM_CUDA(cudaMemcpyAsync(g.q_hi.p, hh, sizeof(uint16_t) * elems, cudaMemcpyHostToDevice, s));
    TM_CUDA(cudaMemcpyAsync(g.q_lo.p, hl, sizeof(uint16_t) * elems, cudaMemcpyHostToDevice, s));
    TM_CUDA(cudaMemcpyAsync(g.d_tiles.p, g.tiles.data(), sizeof(tmb::TileInfo) * tiles.size(), cudaMemcpyHostToDevice,
                            s));
    TM_CUDA(cudaStreamSynchronize(s));
    h2d += samples * 2 * sizeof(uint16_t) + sizeof(tmb::TileInfo) * tiles.size();
}

// Makes a prepared mixed-length group one of the FFT branch: its rows, sorted by length as they
// are, in sets of one class and number of parts, and what the correlation
// kernel needs per row.
void prepare_fft(tm_ctx *ctx, Lane &L, GroupPlan &g, const FftClasses &classes)
{
    g.fft = true;
    g.fft_sets.clear();
    g.fft_rows.clear();
    const float *hq = L.h_q.as<float>(); // the templates as prepare_group_mixed left them
    size_t run = 0;                      // first row of the current length
    for (int t = 0; t < g.T; t++)
    {
        const TemplParam &p = g.htp[static_cast<size_t>(t)];
        if (g.index[t] < 0 || g.inert[t])
            continue;
        const int cls = classes.of(p.m), parts = tmb::fft_parts(p.m, cls);
        const int step = static_cast<int>(tmb::fft_class(cls).step);
        if (g.fft_sets.empty() || g.fft_sets.back().cls != cls || g.fft_sets.back().parts != parts)
            g.fft_sets.push_back(GroupPlan::FftSet{cls, parts, static_cast<int>(g.fft_rows.size()), 0});
        g.fft_sets.back().count++;
        tmb::FftRow r{};
        r.inv_m = p.inv_m;
        if (parts > 1)
            for (int i = step; i < p.m; i++)
                r.sum[i / step - 1] += hq[p.q_offset + i];
        r.s1 = p.s1;
        r.c_lin = p.c_lin;
        r.a3 = p.a3;
        r.thr = p.mode == TM_MODE_KNN ? HUGE_VALF : p.thr_ed;
        r.c0 = make_float4(p.a1_main, p.a2, p.a5, p.a6);
        r.qs = p.qs;
        r.s1_max = std::fabs(p.s1);
        r.row = t;
        r.m = p.m;
        r.mode = p.mode;
        r.wcount = p.wcount;
        r.base = tmb::fft_base(p.m);
        if (g.fft_rows.empty() || g.fft_rows[run].m != p.m)
            run = g.fft_rows.size();
        g.fft_rows.push_back(r);
        // the largest coefficients of a length so far, in its first row
        tmb::FftRow &f = g.fft_rows[run];
        f.c0 = make_float4(std::max(f.c0.x, r.c0.x), std::max(f.c0.y, r.c0.y), std::max(f.c0.z, r.c0.z),
                           std::max(f.c0.w, r.c0.w));
        f.qs = std::max(f.qs, r.qs);
        f.s1_max = std::max(f.s1_max, r.s1_max);
    }
    for (size_t i = 1; i < g.fft_rows.size(); i++) // then in all of them
        if (g.fft_rows[i].m == g.fft_rows[i - 1].m)
        {
            g.fft_rows[i].c0 = g.fft_rows[i - 1].c0;
            g.fft_rows[i].qs = g.fft_rows[i - 1].qs;
            g.fft_rows[i].s1_max = g.fft_rows[i - 1].s1_max;
        }
    for (tmb::FftRow &r : g.fft_rows)
    {
        r.e_norm = tmb::fft_e_norm(r.qs, r.m, classes.of(r.m));
        r.inv_a3 = r.a3 < 0.5f ? (1.0f / (1.0f - r.a3)) * 1.000001f : HUGE_VALF;
    }
    if (!g.fft_rows.empty())
    {
        const size_t bytes = sizeof(tmb::FftRow) * g.fft_rows.size();
        g.d_fft.reserve_on(bytes, L.stream, ctx->pool);
        TM_CUDA(cudaMemcpyAsync(g.d_fft.p, g.fft_rows.data(), bytes, cudaMemcpyHostToDevice, L.stream));
    }
    TM_CUDA(cudaStreamSynchronize(L.stream));
}

// A batch is prepared once and run on whatever range the context has then: windows past the record
// would be read with those of another.
void refresh_range(tm_ctx *ctx, Lane &L, GroupPlan &g)
{
    if (g.range_first == ctx->range_first && g.range_count == ctx->range_count)
        return;
    g.w_max = 0;
    for (int t = 0; t < g.T; t++)
        if (g.index[t] >= 0)
        {
            const uint32_t windows = static_cast<uint32_t>(windows_in_range(ctx, g.htp[t].m));
            g.w_max = std::max(g.w_max, windows);
            g.htp[t].wcount = g.inert[t] ? 0 : windows;
        }
    TM_CUDA(cudaMemcpyAsync(g.tp.p, g.htp.data(), sizeof(TemplParam) * g.htp.size(), cudaMemcpyHostToDevice, L.stream));
    if (g.fft && !g.fft_rows.empty())
    {
        for (tmb::FftRow &r : g.fft_rows)
            r.wcount = g.htp[r.row].wcount;
        TM_CUDA(cudaMemcpyAsync(g.d_fft.p, g.fft_rows.data(), sizeof(tmb::FftRow) * g.fft_rows.size(), cudaMemcpyHostToDevice,
                                L.stream));
    }
    g.range_first = ctx->range_first;
    g.range_count = ctx->range_count;
}

// Modelled milliseconds of 128 template rows x 2^25 windows of shape v at K samples:
// linear between the measured K, proportional to K above the largest, flat below the
// smallest (epilogue-bound there).
double tile_time(const tm_ctx *ctx, bool mixed, int v, double k)
{
    static const double ks[4] = {256.0, 1024.0, 4096.0, 16384.0};
    const double *t = ctx->tile_ms[mixed ? 1 : 0][v];
    if (k <= ks[0])
        return t[0];
    if (k >= ks[3])
        return t[3] * k / ks[3];
    int i = 0;
    while (k > ks[i + 1])
        i++;
    return t[i] + (t[i + 1] - t[i]) * (k - ks[i]) / (ks[i + 1] - ks[i]);
}

// Tile shape of a group: 0 (row tiles of 128 templates, k_scan_umma) or the column-tile
// size (k_scan_wm). Each shape's modelled time sums its tiles (consecutive in length
// order; a tile costs its rows at its longest template's K); the least wins. *cost gets
// the winner's modelled milliseconds per 2^25 windows.
int plan_col_tile(const tm_ctx *ctx, const tm_request *reqs, const std::vector<int> &idx, double *cost)
{
    std::vector<int> m(idx.size());
    for (size_t i = 0; i < idx.size(); i++)
        m[i] = reqs[idx[i]].m;
    std::sort(m.begin(), m.end(), std::greater<int>());
    const bool mixed = !m.empty() && m.front() != m.back();
    const int shapes[4] = {128, 128, 64, 32};
    double costs[4];
    for (int v = 0; v < 4; v++)
    {
        const size_t rows = static_cast<size_t>(shapes[v]);
        costs[v] = 0.0;
        for (size_t i = 0; i < m.size(); i += rows) // row tiles may close early (65 lengths): ignored
            costs[v] += static_cast<double>(rows) / 128.0 *
                        tile_time(ctx, mixed, v, static_cast<double>((m[i] + 63) & ~63));
    }
    int v = 0;
    switch (ctx->tiles)
    {
    case TM_TILES_ROWS:
        v = 0;
        break;
    case TM_TILES_COLS_128:
        v = 1;
        break;
    case TM_TILES_COLS_64:
        v = 2;
        break;
    case TM_TILES_COLS_32:
        v = 3;
        break;
    default:
        for (int u = 1; u < 4; u++)
            if (costs[u] < costs[v])
                v = u;
    }
    if (cost)
        *cost = costs[v];
    return v == 0 ? 0 : shapes[v];
}

// Modelled milliseconds per 2^25 windows of templates with lengths m[0..n) (sorted,
// longest first) in the tile shape TM_TILES_AUTO would pick (or the forced one).
double tensor_cost_sorted(const tm_ctx *ctx, const int *m, size_t n)
{
    if (n == 0)
        return 0.0;
    const bool mixed = m[0] != m[n - 1];
    const int shapes[4] = {128, 128, 64, 32};
    double best = 0.0;
    for (int v = 0; v < 4; v++)
    {
        if ((ctx->tiles == TM_TILES_ROWS && v != 0) || (ctx->tiles == TM_TILES_COLS_128 && v != 1) ||
            (ctx->tiles == TM_TILES_COLS_64 && v != 2) || (ctx->tiles == TM_TILES_COLS_32 && v != 3))
            continue;
        double c = 0.0;
        for (size_t i = 0; i < n; i += static_cast<size_t>(shapes[v]))
            c += shapes[v] / 128.0 * tile_time(ctx, mixed, v, static_cast<double>((m[i] + 63) & ~63));
        if (best == 0.0 || c < best)
            best = c;
    }
    return best;
}

// Modelled milliseconds of the FFT branch per template of length m, in pieces of class cls, per 2^25
// samples. shared: a
// template of the same length precedes it, whose window statistics it takes; skips: it has a
// cut, so that it need not evaluate most windows (tm_fftk.cu). The time depends on the length
// through the pieces' step alone, and within a class little on it; the factors are the classes'
// times over that of a template that evaluates all its windows at 4096 (0.307 ms) or 16000
// (0.63 ms): 0.247, 0.275, 0.307, 0.43 ms at 1000, 2000, 4096, 8192; shared 0.171, 0.168, 0.208,
// 0.326, and 0.43 at 16384; skipping 0.109, 0.127, 0.153, 0.231, and 0.33 at 16000.
double fft_time(const tm_ctx *ctx, int m, int cls, bool shared, bool skips, double evaluated)
{
    static const double all[tmb::kFftClasses] = {0.81, 0.90, 1.0, 1.41};
    static const double same[tmb::kFftClasses] = {0.55, 0.55, 0.66, 1.04};
    static const double skip[tmb::kFftClasses] = {0.36, 0.42, 0.50, 0.75};
    if (tmb::fft_parts(m, cls) > 1)
        return ctx->fft_long_ms * (skips ? 0.53 + 0.47 * evaluated : shared ? 0.69 : 1.0);
    return ctx->fft_ms * (skips ? skip[cls] + (all[cls] - skip[cls]) * evaluated : shared ? same[cls] : all[cls]);
}

// The part of a skipping template's windows that is evaluated all the same, in whole chunks of 128: a
// kNN bound leaves few; a threshold lets the chunks through where noise reaches it, which depends on
// c sqrt(m). Time per template and 2^25 samples of AR(2) noise, chirps of 512 samples at c = 0.1 to
// 0.5 (c sqrt(m) = 2.3 to 11): 0.31, 0.24, 0.17, 0.13, 0.112 ms, with nothing to evaluate 0.111, all
// 0.25; of 1024 at 0.1 to 0.4: 0.25, 0.155, 0.115, 0.111; white noise 0.17 and 0.111 at 0.1 and 0.2. The
// row tiles take 0.137 for 1024 samples, which is passed at c sqrt(m) of 7 and 4: the line, where
// noise is unknown, lies between.
double fft_evaluated(int mode, float correlation, int m)
{
    if (mode == TM_MODE_KNN)
        return 0.0;
    const double reach = (7.0 - static_cast<double>(correlation) * std::sqrt(static_cast<double>(m))) / 6.0;
    return reach > 0.0 ? std::min(reach, 1.0) : 0.0;
}

// Classes for templates of these lengths: each its own (9 to 16 bytes of spectra per sample and class,
// and the prefix sums) where what is not resident yet takes at most 0.8 of the free memory; else
// those that are not resident share a longer one, resident or the longest of them, whose pieces
// serve every shorter template. False where that is too much as well.
static bool fft_classes(tm_ctx *ctx, const std::vector<int> &m, FftClasses &classes)
{
    std::lock_guard<std::mutex> lk(ctx->fft_mu);
    bool wanted[tmb::kFftClasses] = {};
    for (int len : m)
        wanted[tmb::fft_class_of(len)] = true;
    const auto missing = [&](const FftClasses &c) {
        size_t need = ctx->prefix_ready ? 0 : 18 * static_cast<size_t>(ctx->n);
        bool counted[tmb::kFftClasses] = {};
        for (int i = 0; i < tmb::kFftClasses; i++)
        {
            const int cls = c.use[i];
            if (wanted[i] && !ctx->fft[cls].ready && !counted[cls])
                need += sizeof(double2) * static_cast<size_t>(tmb::fft_pieces(ctx->n, cls)) *
                        tmb::fft_pitch(tmb::fft_class(cls).n);
            counted[cls] = counted[cls] || wanted[i];
        }
        return need;
    };
    classes = FftClasses();
    const size_t need = missing(classes);
    if (need == 0)
        return true;
    size_t free_b = 0, total_b = 0;
    TM_CUDA(cudaMemGetInfo(&free_b, &total_b));
    const size_t room = free_b / 10 * 8;
    if (need <= room)
        return true;
    FftClasses fewer;
    int shared = -1; // from the longest down
    for (int i = tmb::kFftClasses - 1; i >= 0; i--)
        if (ctx->fft[i].ready)
            shared = i;
        else if (wanted[i])
            shared = fewer.use[i] = shared < 0 ? i : shared;
    if (missing(fewer) > room)
        return false;
    classes = fewer;
    return true;
}

// Will the chunks' bounds of these lengths fit the memory? (ensure_bounds; asked only where they are
// many times what a device with little memory left would refuse.)
static bool bounds_fit(tm_ctx *ctx, const std::vector<int> &m)
{
    const size_t each = sizeof(float4) * tmb::fft_chunks(ctx->n), little = 64ull << 20;
    if (each * std::min<size_t>(m.size(), tmb::kFftBases) < little)
        return true;
    std::lock_guard<std::mutex> lk(ctx->fft_mu);
    size_t asked = 0, fresh = 0, resident = 0;
    int last = -1; // base of the length before
    for (size_t i = 0; i < m.size(); i++)
        if (i == 0 || m[i] != m[i - 1])
        {
            const int base = tmb::fft_base(m[i]);
            asked += base != last ? each : 0;
            fresh += base != last && !ctx->fft_bounds[base].buf ? each : 0;
            last = base;
        }
    if (fresh < little)
        return true;
    for (const tm_ctx::FftBounds &b : ctx->fft_bounds)
        resident += b.buf ? each : 0;
    size_t free_b = 0, total_b = 0;
    TM_CUDA(cudaMemGetInfo(&free_b, &total_b));
    return asked <= (free_b + resident) / 10;
}

// Milliseconds of a cut on the way through a launch's pieces: the selection, and two launches whose last
// blocks end alone in place of one (128 templates of 1024 on 400000 windows: 0.30 ms with one cut,
// 0.19 by the times above; the row tiles take 0.24).
constexpr double kCutMs = 0.06;
// And of a second group: a re-scoring, sort and copy of its own, a dozen launches and two waits of the
// host (200 thresholds of 700 on 2^21 samples, in one group and in two).
constexpr double kGroupMs = 0.07;

// The f of the least modelled time (plan_fft_split), pieces by these classes; m: the lengths. Which
// templates skip windows is decided as fft_contract does, per class and number of parts, from the
// pieces of the window range and the rows of a launch.
static size_t cheapest_split(tm_ctx *ctx, const tm_request *reqs, const std::vector<int> &sorted_idx,
                             const std::vector<int> &m, const FftClasses &classes)
{
    const size_t n = m.size();
    const bool fit = bounds_fit(ctx, m);
    size_t best_f = 0;
    double best = tensor_cost_sorted(ctx, m.data(), n), done = 0.0; // done: the sets before this one
    double thr[2] = {}, knn[2] = {}, cuts = 0.0; // this set's, evaluating all and skipping, and its cuts
    int cls = -1, parts = 0, rows = 0;
    FftSkips skips;
    const auto set_cost = [&] {
        return thr[skips.thresholds ? 1 : 0] + (knn[0] > 0.0 ? skips.knn_first * knn[0] + (1.0 - skips.knn_first) * knn[1] + cuts : 0.0);
    };
    for (size_t f = 1; f <= n; f++)
    {
        const tm_request &r = reqs[sorted_idx[f - 1]];
        const int c = classes.of(r.m), p = tmb::fft_parts(r.m, c);
        if (c != cls || p != parts)
        {
            done += set_cost();
            cls = c;
            parts = p;
            rows = 0;
            thr[0] = thr[1] = knn[0] = knn[1] = 0.0;
        }
        rows++;
        const uint64_t windows = windows_in_range(ctx, r.m); // the set's shortest so far has the most
        if (fit)
            skips = fft_skips(ctx, cls, fft_range(ctx, cls, windows).count, std::min(rows, tmb::fft_launch_rows(cls, parts)));
        const double scale = windows > 0 ? 33554432.0 / static_cast<double>(windows) : 0.0;
        cuts = kCutMs * skips.cuts * scale;
        double *sum = r.mode == TM_MODE_KNN ? knn : thr;
        sum[0] += fft_time(ctx, r.m, cls, f > 1 && m[f - 2] == r.m, false, 0.0);
        sum[1] += fft_time(ctx, r.m, cls, false, true, fft_evaluated(r.mode, r.correlation, r.m));
        const double cost = done + set_cost() +
                            (f < n ? tensor_cost_sorted(ctx, m.data() + f, n - f) + kGroupMs * scale : 0.0);
        if (cost < best)
        {
            best = cost;
            best_f = f;
        }
    }
    return best_f;
}

// How many of a group's templates (ordered longest first) go to the FFT branch: all of
// them when it is forced (TM_TILES_FFT); under TM_TILES_AUTO with the automatic kernel,
// the f minimising the FFT's time of f templates + the tensor cost of the other
// templates: the longest templates set a tile's K extent, so moving a few of them to the
// FFT (whose cost grows little with the length) can shorten every tile they would have
// padded. Lengths up to 16384 (kFftMaxM); otherwise none. classes: those of their pieces.
size_t plan_fft_split(tm_ctx *ctx, const tm_request *reqs, const std::vector<int> &sorted_idx, FftClasses &classes)
{
    const size_t n = sorted_idx.size();
    if (n == 0 || ctx->kernel == TM_KERNEL_FP32 || !tmb::umma_supported(0, 0, 0))
        return 0;
    for (int i : sorted_idx)
        if (reqs[i].m > tmb::kFftMaxM)
            return 0;
    std::vector<int> m(n);
    for (size_t i = 0; i < n; i++)
        m[i] = reqs[sorted_idx[i]].m;
    if (ctx->tiles == TM_TILES_FFT)
    {
        fft_classes(ctx, m, classes);
        return n;
    }
    if (ctx->tiles != TM_TILES_AUTO || ctx->kernel != TM_KERNEL_AUTO)
        return 0;
    // pieces of other classes where memory is short, at another time; a record too large for the
    // branch's arrays beside its other ones is left to the tiles
    size_t f = 0;
    for (int attempt = 0; attempt < 3; attempt++)
    {
        const FftClasses priced = classes;
        f = cheapest_split(ctx, reqs, sorted_idx, m, priced);
        if (f == 0 || !fft_classes(ctx, std::vector<int>(m.begin(), m.begin() + f), classes))
            return 0;
        if (std::equal(priced.use, priced.use + tmb::kFftClasses, classes.use))
            break;
    }
    return f;
}

// Groups of a batch. Lengths with a full 128-template tile (or any length, on the FP32
// kernel) get their own group with per-length statistics; the remaining templates of
// several lengths share one mixed-length group on the tensor cores.
void create_batch(tm_ctx *ctx, Lane &L, const tm_request *requests, int count, tm_batch &b, bool serving)
{
    b.count = count;
    const bool tensor = ctx->kernel != TM_KERNEL_FP32 && tmb::umma_supported(0, 0, 0);
    // candidate groups (lists of requests); each is then split between the FFT branch and
    // the contraction (plan_fft_split)
    std::vector<std::vector<int>> lists;
    if (serving) // one list over the resident prefix sums, whatever the lengths
    {
        lists.emplace_back(static_cast<size_t>(count));
        for (int i = 0; i < count; i++)
            lists[0][i] = i;
    }
    else
    {
        std::map<int, std::vector<int>> by_m;
        for (int i = 0; i < count; i++)
            by_m[requests[i].m].push_back(i);
        std::vector<int> rest;
        for (auto &kv : by_m)
        {
            if (!tensor || kv.second.size() >= 128 || kv.first > 16384)
                lists.push_back(kv.second);
            else
                rest.insert(rest.end(), kv.second.begin(), kv.second.end());
        }
        if (!rest.empty())
            lists.push_back(rest);
    }
    struct Spec
    {
        std::vector<int> idx;
        int kind; // 0: one length, per-length statistics; 1: prefix statistics, tiles; 2: FFT branch
        FftClasses classes{};
    };
    std::vector<Spec> specs;
    for (std::vector<int> &list : lists)
    {
        std::stable_sort(list.begin(), list.end(), [&](int a, int c) { return requests[a].m > requests[c].m; });
        FftClasses classes;
        const size_t f = tensor ? plan_fft_split(ctx, requests, list, classes) : 0;
        if (f > 0)
            specs.push_back(Spec{std::vector<int>(list.begin(), list.begin() + f), 2, classes});
        if (f < list.size())
        {
            std::vector<int> part(list.begin() + f, list.end());
            const bool one_length = requests[part.front()].m == requests[part.back()].m;
            specs.push_back(Spec{part, one_length && !serving ? 0 : 1});
        }
    }
    for (size_t gi = specs.size(); gi < b.groups.size(); gi++) // a reused batch with fewer groups
        b.groups[gi].release();
    b.groups.resize(specs.size());
    for (size_t gi = 0; gi < specs.size(); gi++)
    {
        GroupPlan &g = b.groups[gi];
        const std::vector<int> &idx = specs[gi].idx;
        const int m = requests[idx.front()].m;
        if (specs[gi].kind == 2)
        {
            prepare_group_mixed(ctx, L, idx, requests, g, b.h2d_bytes, 0, true);
            prepare_fft(ctx, L, g, specs[gi].classes);
        }
        else if (specs[gi].kind == 0)
            prepare_group(ctx, L, m, idx, requests, g, b.h2d_bytes,
                          tensor && m <= 16384 ? plan_col_tile(ctx, requests, idx) : 0);
        else
            prepare_group_mixed(ctx, L, idx, requests, g, b.h2d_bytes, plan_col_tile(ctx, requests, idx), false);
    }
}

} // namespace tmh
