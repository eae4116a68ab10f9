// kNN bound selection, bucket re-pass and exact re-scoring.
//
// Why a bound from bucket minima is valid. The reference's kNN answer is the
// canonical exclusion selection (ZnormSearch.hpp:170-189) over every searched window
// ordered by (FP32 distance, position); its bound queue (2k-1 pairwise separated
// entries with a merge offset, k without, SkipSequential.cpp:378-379) only prunes.
// If 2k-1 windows pairwise at least merge_offset apart all have distance <= T, every
// one of the k answers has distance <= T: each kept answer excludes at most two of
// them (one on each side), so after fewer than k picks one of them is still free.
// Minima over buckets of >= merge_offset windows taken from every other bucket are
// pairwise separated, so with u = d + E >= reference distance,
//     T = min over the two parities of the (2k-1)-th smallest bucket minimum of u
// is such a bound (for merge_offset 0: the k-th smallest over all buckets). Every
// window with reference distance <= T has d - E <= T, so re-scoring the windows of
// the buckets whose minimum of d - E is <= T, and keeping those with d - E <= T,
// yields a candidate set that contains every window the canonical selection can
// pick before it has k answers.
#include <algorithm>

#include "tm_epilogue.cuh"
#include "tm_exact.cuh"
#include "tm_internal.cuh"
#include "tm_prefix.cuh"

namespace tmb {

// The r-th smallest (1-based) of `count` keys, stride apart, by 8-bit radix select over the
// whole block; kEmptyKey when count < r. The keys of one template share their leading bits, so
// a warp counts equal digits with one vote and one atomic per digit (32 conflicting atomics
// otherwise), and a warp scans the 256 bins (one thread alone took half of the 32 us that 32
// keys needed).
__device__ uint32_t block_select(const uint32_t *__restrict__ keys, uint32_t count, uint32_t stride, uint32_t r)
{
    __shared__ uint32_t hist[256];
    __shared__ uint32_t s_prefix, s_r;
    if (count < r)
        return kEmptyKey;
    const int lane = threadIdx.x & 31;
    uint32_t prefix = 0, mask = 0, rr = r;
    for (int shift = 24; shift >= 0; shift -= 8)
    {
        for (int i = threadIdx.x; i < 256; i += blockDim.x)
            hist[i] = 0;
        __syncthreads();
        constexpr int U = 4; // loads in flight
        for (uint32_t i0 = threadIdx.x - lane; i0 < count; i0 += U * blockDim.x)
        {
            uint32_t key[U];
            bool in[U];
#pragma unroll
            for (int u = 0; u < U; u++)
            {
                const uint32_t i = i0 + u * blockDim.x + lane;
                in[u] = i < count;
                key[u] = in[u] ? keys[(size_t)i * stride] : 0u;
            }
#pragma unroll
            for (int u = 0; u < U; u++)
            {
                const bool mine = in[u] && (key[u] & mask) == prefix;
                if (!__any_sync(0xffffffffu, mine))
                    continue;
                const uint32_t digit = mine ? (key[u] >> shift) & 255u : 256u;
                const uint32_t same = __match_any_sync(0xffffffffu, digit);
                if (mine && lane == __ffs(same) - 1)
                    atomicAdd(&hist[digit], (uint32_t)__popc(same));
            }
        }
        __syncthreads();
        if (threadIdx.x < 32)
        {
            uint32_t bins[8], sum = 0;
#pragma unroll
            for (int k = 0; k < 8; k++)
                sum += bins[k] = hist[8 * lane + k];
            uint32_t incl = sum;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1)
            {
                const uint32_t v = __shfl_up_sync(0xffffffffu, incl, off);
                if (lane >= off)
                    incl += v;
            }
            const unsigned reach = __ballot_sync(0xffffffffu, incl >= rr); // count >= r: some lane does
            if (lane == __ffs(reach) - 1)
            {
                uint32_t left = rr - (incl - sum);
                int k = 0;
                while (k < 7 && bins[k] < left)
                    left -= bins[k++];
                s_r = left;
                s_prefix = prefix | ((uint32_t)(8 * lane + k) << shift);
            }
        }
        __syncthreads();
        prefix = s_prefix;
        rr = s_r;
        mask |= 255u << shift;
    }
    __syncthreads(); // s_prefix and s_r may be written again
    return prefix;
}

// Minima over super-buckets of ceil(merge / bucket) buckets, for the templates whose merge
// offset exceeds a bucket: sup[slot][i], i < ceil(nb / buckets per super-bucket).
__global__ void k_super_buckets(const uint32_t *__restrict__ bmin_u, uint32_t nb, int blog, const TemplParam *__restrict__ tp,
                                const int *__restrict__ knn_slots, uint32_t *__restrict__ sup)
{
    const int t = knn_slots[blockIdx.y], merge = tp[t].merge;
    const uint32_t sb = (uint32_t)(((int64_t)merge + (1 << blog) - 1) >> blog);
    if (sb < 2)
        return;
    const uint32_t *u = bmin_u + (size_t)t * nb;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < (nb + sb - 1) / sb; i += gridDim.x * blockDim.x)
    {
        uint32_t best = kEmptyKey;
        for (uint32_t b = i * sb; b < min((i + 1) * sb, nb); b++)
            best = min(best, u[b]);
        sup[(size_t)blockIdx.y * nb + i] = best;
    }
}

// One block per kNN template slot: tkey[t] = key of the bound T (kEmptyKey: +inf).
__global__ void __launch_bounds__(1024) k_bucket_select(const uint32_t *__restrict__ bmin_u, const uint32_t *__restrict__ sup,
                                                        uint32_t nb, int blog, const TemplParam *__restrict__ tp,
                                                        const int *__restrict__ knn_slots, uint32_t *__restrict__ tkey)
{
    const int t = knn_slots[blockIdx.x];
    const int k = tp[t].k, merge = tp[t].merge;
    const uint32_t *u = bmin_u + (size_t)t * nb;
    uint32_t result;
    if (merge <= 0)
        result = block_select(u, nb, 1, (uint32_t)k);
    else
    {
        const uint32_t sb = (uint32_t)(((int64_t)merge + (1 << blog) - 1) >> blog); // buckets per super-bucket
        const uint32_t nsb = (nb + sb - 1) / sb;
        if (sb > 1)
            u = sup + (size_t)blockIdx.x * nb;
        result = kEmptyKey;
        for (uint32_t parity = 0; parity < 2; parity++)
        {
            const uint32_t cnt = nsb > parity ? (nsb - parity + 1) / 2 : 0;
            result = min(result, block_select(u + parity, cnt, 2, (uint32_t)(2 * k - 1)));
        }
    }
    if (threadIdx.x == 0)
        tkey[t] = result;
}

// (template slot, bucket) pairs whose minimum of d - E is within the bound. counters: [0]
// candidates so far, kept in [5] for a list that has to be made again; [1] the list's length.
__global__ void k_list_buckets(const uint32_t *__restrict__ bmin_l, uint32_t nb, const int *__restrict__ knn_slots,
                               const uint32_t *__restrict__ tkey, uint2 *__restrict__ list, uint32_t *__restrict__ counters,
                               uint32_t cap)
{
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0)
        counters[5] = counters[0];
    const int t = knn_slots[blockIdx.y];
    const uint32_t bound = tkey[t];
    const uint4 *row = reinterpret_cast<const uint4 *>(bmin_l + (size_t)t * nb); // nb is a multiple of 4
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nb / 4; i += gridDim.x * blockDim.x)
    {
        const uint4 v = row[i];
        const uint32_t l[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (l[k] != kEmptyKey && l[k] <= bound)
            {
                const uint32_t at = atomicAdd(&counters[1], 1u);
                if (at < cap)
                    list[at] = make_uint2((uint32_t)t, 4 * i + k);
            }
    }
}

// FP32 re-pass over the listed buckets: every window with d - E <= T becomes a candidate. A
// block takes 256 windows of one template at a time; its eight warps split each stage of 512
// samples, a lane holds 8 windows, and the eight partial sums of a window are added at the
// end (shorter chains than the one that a1_fp32 bounds). Shared memory is read 16 bytes at a
// time, one load of samples and one of the template per 32 FMAs, the samples padded by 4
// floats per 32 against bank conflicts. The list's length is read on the device, so the host
// need not wait for it. Measured, bound, list and re-pass together on 2^25 samples, 128
// templates of 4096, k = 100: 1.06 ms; 11.7 ms with buckets of 2048 windows, each re-read by
// one block with three conflicting loads per 32 FMAs, and a host wait between list and re-pass.
constexpr int B_THREADS = 256, B_KC = 512, B_WIN = 256;
__device__ __forceinline__ int bpos(int i) { return i + ((i >> 5) << 2); }
constexpr int B_XS = B_WIN + B_KC + 16;

struct PassB
{
    const uint2 *list;
    const uint32_t *counters; // [1]: the list's length
    uint32_t cap;
    int bucket_log;
    const float *x, *q;
    const TemplParam *tp;
    const uint32_t *tkey;
    uint64_t w0;
    uint32_t W;
    const float *mean, *inv; // one length: its windows' statistics
    const float *raw;        // several lengths: statistics from the prefix sums
    PrefixView pv;
    const uint16_t *run;
    Candidate *cand;
    uint32_t *cand_count, cand_cap;
};

template <bool MIXED> __global__ void __launch_bounds__(B_THREADS) k_passb(const PassB a)
{
    __shared__ __align__(16) float xs[B_XS + ((B_XS + 31) >> 5) * 4];
    __shared__ __align__(16) float qs[B_KC];
    __shared__ float part[B_THREADS / 32][B_WIN];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ulog = a.bucket_log - 8; // 256-window units of a bucket
    const uint64_t units = (uint64_t)min(a.counters[1], a.cap) << ulog;
    for (uint64_t unit = blockIdx.x; unit < units; unit += gridDim.x)
    {
        const uint2 item = a.list[unit >> ulog];
        const uint32_t t = item.x;
        const TemplParam &p = a.tp[t];
        const int m = p.m, m_pad = (m + 63) & ~63;
        const uint32_t windows = MIXED ? p.wcount : a.W;
        const uint32_t jb = (item.y << a.bucket_log) + (((uint32_t)unit & ((1u << ulog) - 1u)) << 8);
        if (jb >= windows)
            continue; // past the template's range (uniform)
        const uint32_t jm = min(jb + B_WIN / 2, windows - 1);
        const float shift = MIXED ? a.x[a.w0 + jm] : a.mean[jm];
        const float *xg = a.x + a.w0 + jb;
        const float *qg = a.q + p.q_offset;
        float acc[8];
#pragma unroll
        for (int w = 0; w < 8; w++)
            acc[w] = 0.0f;
        for (int k0 = 0; k0 < m_pad; k0 += B_KC)
        {
            const int kc = min(B_KC, m_pad - k0), slice = kc / 8; // multiples of 64 and 8
            for (int i = tid; i < B_WIN + kc; i += B_THREADS)
                xs[bpos(i)] = xg[k0 + i] - shift;
            for (int i = tid; i < kc; i += B_THREADS)
                qs[i] = qg[k0 + i];
            __syncthreads();
            const int kb = warp * slice, x0 = 8 * lane + kb;
            float4 xa = *reinterpret_cast<const float4 *>(xs + bpos(x0));
            float4 xb = *reinterpret_cast<const float4 *>(xs + bpos(x0 + 4));
#pragma unroll 4
            for (int kk = 0; kk < slice; kk += 4)
            {
                const float4 xc = *reinterpret_cast<const float4 *>(xs + bpos(x0 + kk + 8));
                const float4 qv = *reinterpret_cast<const float4 *>(qs + kb + kk);
                const float xr[12] = {xa.x, xa.y, xa.z, xa.w, xb.x, xb.y, xb.z, xb.w, xc.x, xc.y, xc.z, xc.w};
#pragma unroll
                for (int w = 0; w < 8; w++)
                {
                    acc[w] = fmaf(xr[w + 0], qv.x, acc[w]);
                    acc[w] = fmaf(xr[w + 1], qv.y, acc[w]);
                    acc[w] = fmaf(xr[w + 2], qv.z, acc[w]);
                    acc[w] = fmaf(xr[w + 3], qv.w, acc[w]);
                }
                xa = xb;
                xb = xc;
            }
            __syncthreads();
        }
#pragma unroll
        for (int w = 0; w < 8; w += 4)
            *reinterpret_cast<float4 *>(&part[warp][8 * lane + w]) = make_float4(acc[w], acc[w + 1], acc[w + 2], acc[w + 3]);
        __syncthreads();
        float dot = 0.0f;
#pragma unroll
        for (int s = 0; s < B_THREADS / 32; s++)
            dot += part[s][tid];
        const uint32_t tk = a.tkey[t], j = jb + tid;
        const float T = tk == kEmptyKey ? inf_f() : key_float(tk);
        bool hit = false;
        if (MIXED)
        {
            if (j < windows && a.raw[a.w0 + j] != kMissing && a.run[a.w0 + j] < m)
            {
                WindowStats ws;
                if (window_prefix_stats(a.pv, a.pv.Q[a.w0 + j], a.pv.Q[a.w0 + j + m], a.w0 + j, m, p.inv_m, ws) != 0)
                    hit = true; // statistics not trustworthy: always re-scored
                else
                {
                    float d, e;
                    fast_distance_mixed(p, p.a1_fp32, dot, ws.mu, ws.iv, shift, stats_error(ws, m, p.qs, p.s1), d, e);
                    hit = d - e <= T;
                }
            }
        }
        else if (j < windows && a.inv[j] != 0.0f)
        {
            float d, e;
            fast_distance(p, p.a1_fp32, dot, a.mean[j], a.inv[j], shift, d, e);
            hit = d - e <= T;
        }
        const unsigned ballot = __ballot_sync(0xffffffffu, hit);
        if (ballot != 0u)
        {
            uint32_t base = 0;
            if (lane == 0)
                base = atomicAdd(a.cand_count, (uint32_t)__popc(ballot));
            base = __shfl_sync(0xffffffffu, base, 0) + (uint32_t)__popc(ballot & ((1u << lane) - 1u));
            if (hit && base < a.cand_cap)
                a.cand[base] = Candidate{t, j};
        }
    }
}

// Exact (reference-arithmetic) distance of every candidate.
__global__ void k_rescore(const Candidate *__restrict__ cand, uint32_t count, const TemplParam *__restrict__ tp,
                          const float *__restrict__ q, const int *__restrict__ order, const float *__restrict__ raw,
                          uint64_t w0, float *__restrict__ dist)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count)
        return;
    const Candidate c = cand[i];
    const TemplParam p = tp[c.templ];
    const uint64_t g = w0 + c.window;
    float mean_f, std_f;
    exact_stats(raw, g, p.m, mean_f, std_f);
    dist[i] = replica_distance(q + p.q_offset, order + p.order_offset, raw, g, p.m, mean_f, std_f);
}

// ---- launchers --------------------------------------------------------------------

// sup: scratch of nk x nb keys (used by templates whose merge offset exceeds a bucket).
cudaError_t launch_bucket_select(const uint32_t *bmin_u, uint32_t *sup, uint32_t nb, int blog, const TemplParam *tp,
                                 const int *knn_slots, int nk, bool super, uint32_t *tkey, cudaStream_t s)
{
    if (super)
        k_super_buckets<<<dim3(std::min(nb / 256 + 1, 64u), (unsigned)nk), 256, 0, s>>>(bmin_u, nb, blog, tp, knn_slots, sup);
    k_bucket_select<<<nk, 1024, 0, s>>>(bmin_u, sup, nb, blog, tp, knn_slots, tkey);
    return cudaGetLastError();
}

cudaError_t launch_list_buckets(const uint32_t *bmin_l, uint32_t nb, const int *knn_slots, int nk,
                                const uint32_t *tkey, uint2 *list, uint32_t *counters, uint32_t cap, cudaStream_t s)
{
    k_list_buckets<<<dim3(std::min(nb / 1024 + 1, 64u), (unsigned)nk), 256, 0, s>>>(bmin_l, nb, knn_slots, tkey, list, counters,
                                                                                   cap);
    return cudaGetLastError();
}

cudaError_t launch_passb(const uint2 *list, const uint32_t *counters, uint32_t cap, const ScanArgs &c, const uint32_t *tkey,
                         bool mixed, int sms, cudaStream_t s)
{
    PassB a{};
    a.list = list;
    a.counters = counters;
    a.cap = cap;
    a.bucket_log = c.bucket_log;
    a.x = c.x;
    a.q = c.q;
    a.tp = c.tp;
    a.tkey = tkey;
    a.w0 = c.w0;
    a.W = c.W;
    a.mean = c.mean;
    a.inv = c.inv;
    a.raw = c.raw;
    a.pv = PrefixView{c.P, c.PT, c.PC};
    a.run = c.run;
    a.cand = c.cand;
    a.cand_count = c.cand_count;
    a.cand_cap = c.cand_cap;
    const unsigned grid = 8u * (unsigned)sms; // resident blocks; the list's length is known on the device only
    if (mixed)
        k_passb<true><<<grid, B_THREADS, 0, s>>>(a);
    else
        k_passb<false><<<grid, B_THREADS, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_rescore(const Candidate *cand, uint32_t count, const TemplParam *tp, const float *q,
                           const int *order, const float *raw, uint64_t w0, float *dist, cudaStream_t s)
{
    if (count > 0)
        k_rescore<<<(count + 127) / 128, 128, 0, s>>>(cand, count, tp, q, order, raw, w0, dist);
    return cudaGetLastError();
}

} // namespace tmb
