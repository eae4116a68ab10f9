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

#include "../../include/tremor_b200.h"
#include "tm_epilogue.cuh"
#include "tm_exact.cuh"
#include "tm_fft.cuh"
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

// Template of a selection's block i: that of a kNN slot, or of a row of the FFT branch.
__device__ __forceinline__ int select_template(const int *slots, const FftRow *rows, int i)
{
    return rows != nullptr ? rows[i].row : slots[i];
}
// Its place in the scratch of super-buckets.
__device__ __forceinline__ int select_slot(const int *slots, int nk, const FftRow *rows, int i)
{
    if (rows == nullptr)
        return i;
    int lo = 0, hi = nk - 1; // the slots' templates ascend
    while (lo < hi)
    {
        const int mid = (lo + hi) / 2;
        if (slots[mid] < rows[i].row)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

// Minima over super-buckets of ceil(merge / bucket) buckets, for the templates whose merge
// offset exceeds a bucket: sup[slot][i], i < ceil(nb_seen / buckets per super-bucket); nb buckets
// per template, of which the first nb_seen are looked at. count: the rows, or the nk slots.
__global__ void k_super_buckets(const uint32_t *__restrict__ bmin_u, uint32_t nb, uint32_t nb_seen, int blog,
                                const TemplParam *__restrict__ tp, const int *__restrict__ knn_slots, int nk,
                                const FftRow *__restrict__ rows, int count, uint32_t *__restrict__ sup)
{
    for (int r = blockIdx.y; r < count; r += gridDim.y)
    {
        const int t = select_template(knn_slots, rows, r), merge = tp[t].merge;
        const uint32_t sb = (uint32_t)(((int64_t)merge + (1 << blog) - 1) >> blog);
        if (sb < 2 || tp[t].mode != TM_MODE_KNN)
            continue;
        const uint32_t *u = bmin_u + (size_t)t * nb;
        uint32_t *s = sup + (size_t)select_slot(knn_slots, nk, rows, r) * nb_seen;
        for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < (nb_seen + sb - 1) / sb; i += gridDim.x * blockDim.x)
        {
            uint32_t best = kEmptyKey;
            for (uint32_t b = i * sb; b < min((i + 1) * sb, nb_seen); b++)
                best = min(best, u[b]);
            s[i] = best;
        }
    }
}

// One block per kNN template slot: tkey[t] = key of the bound T (kEmptyKey: +inf). With rows, one
// per row of the FFT branch: cuts[row] = its threshold, or the bound from the buckets seen.
__global__ void __launch_bounds__(1024) k_bucket_select(const uint32_t *__restrict__ bmin_u, const uint32_t *__restrict__ sup,
                                                        uint32_t nb, uint32_t nb_seen, int blog,
                                                        const TemplParam *__restrict__ tp, const int *__restrict__ knn_slots,
                                                        int nk, const FftRow *__restrict__ rows, uint32_t *__restrict__ tkey,
                                                        float *__restrict__ cuts)
{
    const int t = select_template(knn_slots, rows, blockIdx.x);
    if (rows != nullptr && tp[t].mode != TM_MODE_KNN)
    {
        if (threadIdx.x == 0)
            cuts[blockIdx.x] = rows[blockIdx.x].thr;
        return;
    }
    const int k = tp[t].k, merge = tp[t].merge;
    const uint32_t *u = bmin_u + (size_t)t * nb;
    uint32_t result;
    if (merge <= 0)
        result = block_select(u, nb_seen, 1, (uint32_t)k);
    else
    {
        const uint32_t sb = (uint32_t)(((int64_t)merge + (1 << blog) - 1) >> blog); // buckets per super-bucket
        const uint32_t nsb = (nb_seen + sb - 1) / sb;
        if (sb > 1)
            u = sup + (size_t)select_slot(knn_slots, nk, rows, blockIdx.x) * nb_seen;
        result = kEmptyKey;
        for (uint32_t parity = 0; parity < 2; parity++)
        {
            const uint32_t cnt = nsb > parity ? (nsb - parity + 1) / 2 : 0;
            result = min(result, block_select(u + parity, cnt, 2, (uint32_t)(2 * k - 1)));
        }
    }
    if (threadIdx.x == 0)
    {
        if (rows != nullptr)
            cuts[blockIdx.x] = result == kEmptyKey ? inf_f() : key_float(result);
        else
            tkey[t] = result;
    }
}

// The minima of d + E of buckets with a window that has a sample that is not finite (odd:
// launch_odd_next) are taken out: one such window may have given them.
__global__ void k_odd_buckets(uint32_t *__restrict__ bmin_u, uint32_t nb, int blog, const TemplParam *__restrict__ tp,
                              const int *__restrict__ knn_slots, int nk, const uint32_t *__restrict__ odd, uint64_t w0,
                              uint32_t W)
{
    const uint32_t used = (W - 1 >> blog) + 1; // the rest of a row is padding
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < (uint64_t)nk * used;
         i += (uint64_t)gridDim.x * blockDim.x)
    {
        const int t = knn_slots[i / used];
        const uint32_t b = (uint32_t)(i % used);
        if (odd[w0 + ((uint64_t)b << blog)] < (uint32_t)tp[t].m + (1u << blog) - 1u)
            bmin_u[(size_t)t * nb + b] = kEmptyKey;
    }
}

// (template slot, bucket) pairs whose minimum of d - E is within the bound. counters: [0]
// candidates so far, kept in [5] for a list that has to be made again; [1] the list's length.
__global__ void k_list_buckets(const uint32_t *__restrict__ bmin_l, uint32_t nb, const int *__restrict__ knn_slots, int nk,
                               const uint32_t *__restrict__ tkey, uint2 *__restrict__ list, uint32_t *__restrict__ counters,
                               uint32_t cap)
{
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0)
        counters[5] = counters[0];
    for (int s = blockIdx.y; s < nk; s += gridDim.y)
    {
        const int t = knn_slots[s];
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
    const float *mean, *inv; // one length: its windows' statistics (FFT branch: null where it has none)
    const float *raw;        // several lengths: statistics from the prefix sums
    PrefixView pv;
    const uint16_t *run;
    const uint32_t *odd; // several lengths, a record with samples that are not finite; else null
    Candidate *cand;
    uint32_t *cand_count, cand_cap;
    uint32_t *untrusted; // candidates for want of statistics are counted here
    uint32_t nb;
    const uint32_t *bmin_l;
    uint32_t *certain; // the certain minima (below), over the minima of d + E; null: none
    float *lower;      // for templates without a merge offset, each candidate's d - E,
    uint32_t *bins;    //   and counts of d + E (k_tight_bound); null: none has no offset
};

// Certain minima. The window v of a 256-window bucket with the smallest d + E is certain to be kept
// before any window within its template's merge offset when all of those have d - E above it:
// the bucket's own by the re-pass, the others by their buckets' minima of d - E (those that no
// list holds are above the bound). Then those windows are in no answer, whatever their
// exact distances: k_rescore leaves them out (8 templates of 16384, k = 10, merge 8192: 1.03 ->
// 0.48 ms for the re-scoring, most of it the undecided candidates' chains).
template <bool MIXED> __global__ void __launch_bounds__(B_THREADS) k_passb(const PassB a)
{
    __shared__ uint32_t s_least;
    __shared__ uint32_t s_where;
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
        {
            if (a.certain != nullptr && tid == 0)
                a.certain[(size_t)t * a.nb + item.y] = kNoWindow;
            continue; // past the template's range (uniform)
        }
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
        float lower = inf_f(), upper = inf_f(); // windows that are not searched
        if (MIXED)
        {
            if (j < windows && a.raw[a.w0 + j] != kMissing && a.run[a.w0 + j] < m &&
                (a.odd == nullptr || a.odd[a.w0 + j] >= (uint32_t)m))
            {
                WindowStats ws;
                const int code = window_prefix_stats(a.pv, a.pv.Q[a.w0 + j], a.pv.Q[a.w0 + j + m], a.w0 + j, m, p.inv_m, ws);
                if (code != 0 && (a.inv == nullptr || a.inv[j] == 0.0f))
                {
                    hit = true; // statistics not trustworthy: always re-scored
                    lower = -inf_f();
                }
                else
                {
                    float d, e;
                    if (code == 0)
                        fast_distance_mixed(p, p.a1_fp32, dot, ws.mu, ws.iv, shift, stats_error(ws, m, p.qs, p.s1), d, e);
                    else
                        fast_distance(p, p.a1_fp32, dot, a.mean[j], a.inv[j], shift, d, e);
                    lower = d - e;
                    upper = d + e;
                    hit = lower <= T;
                }
            }
        }
        else if (j < windows && a.inv[j] != 0.0f)
        {
            float d, e;
            fast_distance(p, p.a1_fp32, dot, a.mean[j], a.inv[j], shift, d, e);
            lower = d - e;
            upper = d + e;
            hit = lower <= T;
        }
        if (a.certain != nullptr && p.merge > 0) // uniform
        {
            if (tid == 0)
                s_least = kEmptyKey;
            __syncthreads();
            const uint32_t key = upper < inf_f() ? float_key(upper) : kEmptyKey;
            const uint32_t least_w = __reduce_min_sync(0xffffffffu, key);
            if (lane == 0)
                atomicMin(&s_least, least_w);
            __syncthreads();
            const uint32_t least = s_least;
            if (key == least)
                s_where = j; // one of them; where two are that low, there is no certain one
            const int near = __syncthreads_count(!(lower > key_float(least))); // a NaN is not above
            int bad = least == kEmptyKey || least > tk || near != 1 ? 1 : 0;
            const uint32_t v = s_where;
            if (bad == 0)
            {
                const uint32_t far = (uint32_t)p.merge - 1u;
                const uint32_t b0 = (v > far ? v - far : 0u) >> 8;
                const uint32_t b1 = min((uint32_t)(((uint64_t)v + far) >> 8), a.nb - 1);
                for (uint32_t b = b0 + tid; b <= b1; b += B_THREADS)
                    bad |= b != item.y && a.bmin_l[(size_t)t * a.nb + b] <= least ? 1 : 0;
            }
            bad = __syncthreads_or(bad);
            if (tid == 0)
                a.certain[(size_t)t * a.nb + item.y] = bad != 0 ? kNoWindow : v;
        }
        if (a.bins != nullptr && p.merge <= 0 && upper <= T && T < inf_f() && T > 0.0f)
            atomicAdd(&a.bins[(size_t)t * kTightBins + min((int)(fmaxf(upper, 0.0f) * ((float)kTightBins / T)), kTightBins - 1)],
                      1u);
        const unsigned ballot = __ballot_sync(0xffffffffu, hit);
        if (ballot != 0u)
        {
            const unsigned lost = MIXED ? __ballot_sync(0xffffffffu, hit && lower == -inf_f()) : 0u;
            if (lost != 0u && lane == 0)
                atomicAdd(a.untrusted, (uint32_t)__popc(lost));
            uint32_t base = 0;
            if (lane == 0)
                base = atomicAdd(a.cand_count, (uint32_t)__popc(ballot));
            base = __shfl_sync(0xffffffffu, base, 0) + (uint32_t)__popc(ballot & ((1u << lane) - 1u));
            if (hit && base < a.cand_cap)
            {
                a.cand[base] = Candidate{t, j};
                if (a.lower != nullptr)
                    a.lower[base] = lower;
            }
        }
    }
}

// Without a merge offset the answers are the k nearest windows, wherever they lie: those of a few
// events often fill the k that the bound took from as many buckets. tight[t]: a bound that at
// least k windows of the re-pass have d + E below, from their counts (infinite where there are
// fewer): no window with d - E above it can be an answer. 128 templates of 4096, k = 100, 2^25
// samples, 0.7 M candidates: 2.9 -> 0.26 ms for the re-scoring, 0.35 -> 0.07 for the sort.
__global__ void __launch_bounds__(kTightBins) k_tight_bound(const uint32_t *__restrict__ bins, const TemplParam *__restrict__ tp,
                                                            const int *__restrict__ knn_slots,
                                                            const uint32_t *__restrict__ tkey, float *__restrict__ tight)
{
    __shared__ uint32_t sums[kTightBins / 32];
    const int t = knn_slots[blockIdx.x], tid = threadIdx.x, lane = tid & 31;
    const uint32_t tk = tkey[t];
    if (tid == 0)
        tight[t] = inf_f();
    if (tk == kEmptyKey || tp[t].merge > 0)
        return; // whole block
    const uint32_t k = (uint32_t)tp[t].k, mine = bins[(size_t)t * kTightBins + tid];
    uint32_t incl = mine;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1)
    {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off)
            incl += v;
    }
    if (lane == 31)
        sums[tid >> 5] = incl;
    __syncthreads();
    for (int w = 0; w < tid >> 5; w++)
        incl += sums[w];
    if (incl >= k && incl - mine < k) // one thread at most
        tight[t] = key_float(tk) * (float)(tid + 1) / (float)kTightBins * (1.0f + 1e-6f);
}

// ---- exact (reference-arithmetic) distance of every candidate -------------------------
//
// The reference's window mean and std are floats rounded from FP64 sums taken sample by
// sample. Their rounding is almost always certain without those chains: with S the true sum,
// a chain of m additions is within m u sum |x| of S (u = 2^-53), and the chain of squared
// differences within (m + 4) u of its value plus m (mean error)^2; whatever FP64 estimate of
// mean and variance is at hand, with its own error bound, gives an interval that holds the
// reference's FP64 value, and when both ends round to the same float that is the reference's
// float. certain_stats decides so; the estimate comes from the prefix sums where the group has
// them, else from 16 lanes' sums. A candidate it cannot decide (about one in 10^4; every one
// near a level step or a loud stretch) goes to a list that k_rescore_serial takes one thread
// per candidate, with the chains themselves.
//
// k_rescore gives a candidate 16 lanes (replica_distance16): loads are 64 bytes wide instead
// of one sample per lane and window, and the chains 16 times shorter. Measured with its serial part (before: one
// thread per candidate running both chains, 32 cache lines per load, never less than one
// candidate's latency): 17000 candidates of 8192 samples 0.24 ms (0.63), 68000 of 16384 1.03
// (1.56), 0.7 M of 4096 1.64 (2.73; without prefix sums 2.5-3.0, 3.3), 3.4 M of 256-8192 8.2
// (10.3-12.9). Bound by L1: 8 bytes of sample and template per candidate and sample.
__device__ __forceinline__ bool certain_stats(double mean, double mean_err, double var, double var_rel, int m, float &mean_f,
                                              float &std_f)
{
    constexpr double u = 1.1102230246251565e-16;
    const double md = (double)m;
    // the chain's sum over m, and the division's rounding
    const double chain = (md + 2.0) * u * 1.01 * sqrt(fma(mean, mean, var)) + 2.0 * u * fabs(mean);
    const double em = (mean_err + chain) * 1.01;
    mean_f = __double2float_rn(mean - em);
    if (!(var > 1e-20 && var < 1e36 && var_rel < 1e-3) || mean_f != __double2float_rn(mean + em))
        return false;
    const double es = (0.5 * var_rel + (md + 8.0) * u + chain * chain / var) * 1.01;
    const double sd = sqrt(var);
    std_f = __double2float_rn(sd - sd * es);
    return std_f == __double2float_rn(sd + sd * es);
}

// Statistics of window [g, g + m) from the prefix sums (prefix_stats_tail's quantities, kept in
// FP64): false when their bound does not apply or does not decide.
__device__ __forceinline__ bool prefix_exact_stats(const PrefixView &pv, uint64_t g, int m, double inv_m, float &mean_f,
                                                   float &std_f)
{
    const double2 qa = pv.Q[g], qb = pv.Q[g + (uint64_t)m];
    const uint64_t e = g + (uint64_t)m, b1 = g >> kPrefixBlockLog;
    PrefixSums ps;
    if (e >> kPrefixBlockLog == b1)
        ps = prefix_sums_one_block(qa, qb, (float)(g - (b1 << kPrefixBlockLog)), (float)(e - (b1 << kPrefixBlockLog)),
                                   (float)qa.y);
    else
        ps = prefix_sums_two_blocks(pv, qa, qb, g, m);
    const double c = pv.C[b1], mu = ps.s1 * inv_m, var = fma(-mu, mu, ps.s2 * inv_m);
    // e_var as prefix_stats_tail bounds it; the additional roundings of mu, c + mu and var here
    const double e1 = (double)ps.e_s1 * inv_m, e2 = (double)ps.e_s2 * inv_m;
    const double e_var = e2 + 2.0 * fabs(mu) * e1 + e1 * e1 + 16.0 * kEps64 * (fabs(var) + 2.0 * mu * mu);
    return certain_stats(c + mu, e1 + 4.0 * kEps64 * (fabs(mu) + fabs(c)), var, e_var / var * 1.01, m, mean_f, std_f);
}

// The same from the sums of x - a and (x - a)^2 over the window by 16 lanes, a near the mean (the
// per-length statistics' float; conversions to FP64, 16 per clock and SM, bound this: one each).
__device__ __forceinline__ bool sums_exact_stats(const float *__restrict__ x, int m, double a, int lane, unsigned half,
                                                 float &mean_f, float &std_f)
{
    double s1 = 0.0, s2 = 0.0, t1 = 0.0, t2 = 0.0;
    int i = lane;
    for (; i + 16 < m; i += 32)
    {
        const double c = (double)clean32(x[i]) - a, d = (double)clean32(x[i + 16]) - a;
        s1 += c;
        t1 += d;
        s2 = fma(c, c, s2);
        t2 = fma(d, d, t2);
    }
    if (i < m)
    {
        const double c = (double)clean32(x[i]) - a;
        s1 += c;
        s2 = fma(c, c, s2);
    }
    s1 += t1;
    s2 += t2;
#pragma unroll
    for (int off = 8; off > 0; off >>= 1)
    {
        s1 += __shfl_xor_sync(half, s1, off);
        s2 += __shfl_xor_sync(half, s2, off);
    }
    // additions in any order: within m u of the sum of magnitudes, at most sqrt(m s2); each term's
    // own roundings and the divisions' within the margins
    const double md = (double)m, u = kEps64, del = s1 / md, ms = s2 / md, var = fma(-del, del, ms);
    const double em = (md + 8.0) * u * 1.01 * sqrt(ms) + 2.0 * u * fabs(a + del);
    const double ev = (md + 8.0) * u * 1.01 * ms + 2.0 * fabs(del) * em + em * em + 4.0 * u * del * del;
    return certain_stats(a + del, em, var, ev / var * 1.01, m, mean_f, std_f);
}

// Is window w within the merge offset of a certain minimum of a listed bucket (k_passb)? Lane
// `lane` of `lanes` looks at its share of the buckets up to 16384 windows away: larger merge offsets
// exclude less than they could.
__device__ __forceinline__ bool excluded_window(const Exclusion &x, uint32_t t, uint32_t w, int merge, int lane, int lanes)
{
    const uint32_t far = (uint32_t)min(merge, 16384) - 1u, bound = x.tkey[t];
    const uint32_t b0 = (w > far ? w - far : 0u) >> 8, b1 = min((uint32_t)(((uint64_t)w + far) >> 8), x.nb - 1);
    const uint32_t *l = x.bmin_l + (size_t)t * x.nb, *c = x.certain + (size_t)t * x.nb;
    bool out = false;
    for (uint32_t b = b0 + lane; b <= b1; b += lanes)
    {
        const uint32_t key = l[b];
        if (key != kEmptyKey && key <= bound) // listed
        {
            const uint32_t v = c[b];
            out = out || (v != kNoWindow && v != w && __usad(v, w, 0u) <= far);
        }
    }
    return out;
}

// Up to which length k_rescore_threads takes all candidates, where there are many: T_SHORT samples,
// T_MIDDLE if the prefix sums leave more than a quarter of those sampled undecided.
constexpr int T_SAMPLES = 4096, T_SHORT = 192, T_MIDDLE = 1024;
__device__ __forceinline__ int thread_limit(const uint32_t *sampled)
{
    return *sampled > T_SAMPLES / 4 ? T_MIDDLE : T_SHORT;
}

__global__ void k_rescore_sample(const Candidate *__restrict__ cand, uint32_t count, const TemplParam *__restrict__ tp,
                                 const PrefixView pv, uint64_t w0, uint32_t *__restrict__ sampled)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x; // < T_SAMPLES
    const Candidate c = cand[(uint64_t)k * count / T_SAMPLES];
    const TemplParam &p = tp[c.templ];
    float mean_f, std_f;
    if (p.m <= T_MIDDLE && !prefix_exact_stats(pv, w0 + c.window, p.m, p.inv_m, mean_f, std_f))
        atomicAdd(sampled, 1u);
}

constexpr int R_THREADS = 256;

// PREFIX: statistics from the prefix sums (windows of at most kPrefixBlock samples), else from
// the samples, centred by the means. todo: the undecided candidates' indices, their number in
// *todo_count. What thread_limit leaves to k_rescore_threads is skipped.
template <bool PREFIX>
__global__ void __launch_bounds__(R_THREADS) k_rescore(const Candidate *__restrict__ cand, uint32_t count,
                                                       const TemplParam *__restrict__ tp, const float *__restrict__ q,
                                                       const int *__restrict__ order, const float *__restrict__ raw,
                                                       const PrefixView pv, const float *__restrict__ mean, uint64_t w0,
                                                       float *__restrict__ dist, uint32_t *__restrict__ todo,
                                                       uint32_t *__restrict__ todo_count, const Exclusion ex, const uint32_t *__restrict__ sampled)
{
    const uint32_t i = blockIdx.x * (R_THREADS / 16) + (threadIdx.x >> 4);
    if (i >= count)
        return; // a whole half warp
    const int lane = threadIdx.x & 15;
    const unsigned half = 0xffffu << (threadIdx.x & 16);
    const Candidate c = cand[i];
    const TemplParam &p = tp[c.templ];
    const uint64_t g = w0 + c.window;
    const int m = p.m;
    if (sampled != nullptr && m <= thread_limit(sampled))
        return;
    if (ex.nb > 0 && p.mode == TM_MODE_KNN && p.merge > 0 &&
        __any_sync(half, excluded_window(ex, c.templ, c.window, p.merge, lane, 16)))
    {
        if (lane == 0)
            dist[i] = kExcluded;
        return;
    }
    if (ex.tight != nullptr && p.mode == TM_MODE_KNN && p.merge <= 0 && ex.lower[i] > ex.tight[c.templ])
    {
        if (lane == 0)
            dist[i] = kExcluded;
        return;
    }
    float mean_f, std_f;
    if (!(PREFIX ? prefix_exact_stats(pv, g, m, p.inv_m, mean_f, std_f)
                 : sums_exact_stats(raw + g, m, (double)mean[c.window], lane, half, mean_f, std_f)))
    {
        if (lane == 0)
            todo[atomicAdd(todo_count, 1u)] = i;
        return;
    }
    const float d = replica_distance16(q + p.q_offset, order + p.order_offset, raw, g, m, mean_f, std_f, lane, half);
    if (lane == 0)
        dist[i] = d;
}

// Many candidates of short templates, and many undecided ones (TODO): a thread each, with both chains.
// Where there are many, neighbours in the list are neighbours in the record, whose loads fall in the
// same lines, and the chains of one hide behind another's. ns per candidate, by this kernel and by 16
// lanes (most of them decided; on a record that drifts, half of them not): 100 samples, dense in the
// record 0.13, 0.31 (0.97), one window in 30 0.25, 0.36; 400 samples 0.49, 0.45 (1.65), 0.75, 0.46;
// 1500 samples 1.66, 1.03 (1.15).
constexpr uint32_t T_COUNT = 1u << 16; // this many fill the multiprocessors
constexpr int T_THREADS = 128;

template <bool TODO>
__global__ void __launch_bounds__(T_THREADS) k_rescore_threads(const Candidate *__restrict__ cand, uint32_t count,
                                                               const TemplParam *__restrict__ tp, const float *__restrict__ q,
                                                               const int *__restrict__ order, const float *__restrict__ raw,
                                                               uint64_t w0, float *__restrict__ dist,
                                                               const uint32_t *__restrict__ todo,
                                                               const uint32_t *__restrict__ todo_count,
                                                               const uint32_t *__restrict__ sampled, const Exclusion ex)
{
    const uint32_t n = TODO ? *todo_count : count;
    if (TODO && n < T_COUNT)
        return; // k_rescore_serial's
    const int limit = TODO ? 0 : thread_limit(sampled);
    for (uint64_t k = blockIdx.x * (uint64_t)T_THREADS + threadIdx.x; k < n; k += (uint64_t)gridDim.x * T_THREADS)
    {
        const uint32_t i = TODO ? todo[k] : (uint32_t)k;
        const Candidate c = cand[i];
        const TemplParam &p = tp[c.templ];
        const int m = p.m;
        if (!TODO)
        {
            if (m > limit)
                continue;
            const bool knn = p.mode == TM_MODE_KNN;
            if ((ex.nb > 0 && knn && p.merge > 0 && excluded_window(ex, c.templ, c.window, p.merge, 0, 1)) ||
                (ex.tight != nullptr && knn && p.merge <= 0 && ex.lower[i] > ex.tight[c.templ]))
            {
                dist[i] = kExcluded;
                continue;
            }
        }
        const uint64_t g = w0 + c.window;
        float mean_f, std_f;
        exact_stats(raw, g, m, mean_f, std_f);
        dist[i] = replica_distance(q + p.q_offset, order + p.order_offset, raw, g, m, mean_f, std_f);
    }
}

// The undecided candidates, where they are few (below `most`): four warps per SM quarter, each taking up to 16 at a time. It stages
// 1024 samples in shared memory as doubles, split evenly between its candidates, by coalesced
// loads one stage ahead; then lane c runs candidate c's chain over its share. (One thread per
// candidate loading for itself costs 32 cache lines per load, and converting in the chain is
// bound by the conversions, 16 per clock and SM: 8 windows of 8192 samples took 940 us.)
constexpr int S_WARPS = 4, S_CANDS = 16, S_LOADS = 32; // 32 S_LOADS samples per stage

__global__ void __launch_bounds__(S_WARPS * 32) k_rescore_serial(const Candidate *__restrict__ cand,
                                                                const TemplParam *__restrict__ tp, const float *__restrict__ q,
                                                                const int *__restrict__ order, const float *__restrict__ raw,
                                                                uint64_t w0, float *__restrict__ dist,
                                                                const uint32_t *__restrict__ todo,
                                                                const uint32_t *__restrict__ todo_count, uint32_t most)
{
    __shared__ double tile[S_WARPS][32 * S_LOADS + S_CANDS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t count = *todo_count, warps = gridDim.x * S_WARPS;
    if (count >= most)
        return; // k_rescore_threads'
    const uint32_t per = min((count + warps - 1) / warps, (uint32_t)S_CANDS);
    // samples of a candidate per stage: 64 for 16 candidates .. 1024 for one
    const int slog = 10 - (per > 1 ? 32 - __clz(per - 1) : 0), stage = 1 << slog;
    for (uint32_t n0 = (blockIdx.x * S_WARPS + warp) * per; n0 < count; n0 += warps * per)
    {
        const int nc = (int)min(per, count - n0);
        // lane c: candidate n0 + c
        uint32_t idx = 0, row = 0;
        uint64_t g = 0;
        int m = 0;
        if (lane < nc)
        {
            idx = todo[n0 + lane];
            const Candidate c = cand[idx];
            row = c.templ;
            m = tp[row].m;
            g = w0 + c.window;
        }
        const int longest = (int)__reduce_max_sync(0xffffffffu, (uint32_t)m);
        // each(v): the lane's samples in order, missing ones as 0
        auto chain = [&](auto each) {
            float next[S_LOADS];
            auto load = [&](int s) {
#pragma unroll
                for (int k = 0; k < S_LOADS; k++)
                {
                    const int c = 32 * k >> slog, at = s + (32 * k & (stage - 1)) + lane;
                    const uint64_t gc = __shfl_sync(0xffffffffu, g, c);
                    next[k] = at < __shfl_sync(0xffffffffu, m, c) ? clean32(raw[gc + (uint64_t)at]) : 0.0f;
                }
            };
            load(0);
            for (int s = 0; s < longest; s += stage)
            {
                __syncwarp(); // the last stage has been read
#pragma unroll
                for (int k = 0; k < S_LOADS; k++)
                    tile[warp][(32 * k >> slog) * (stage + 1) + (32 * k & (stage - 1)) + lane] = (double)next[k];
                __syncwarp();
                if (s + stage < longest)
                    load(s + stage);
                const double *v = tile[warp] + (lane & ((32 * S_LOADS >> slog) - 1)) * (stage + 1);
                const int n = min(stage, m - s); // none for lanes without a candidate
                int k = 0;
                for (; k + 32 <= n; k += 32)
                {
#pragma unroll
                    for (int i = 0; i < 32; i++)
                        each(v[k + i]);
                }
                for (; k < n; k++)
                    each(v[k]);
            }
        };
        // exact_stats' operations
        double sum = 0.0, squares = 0.0;
        chain([&](double v) { sum = __dadd_rn(sum, v); });
        const double md = (double)max(m, 1), mean = __ddiv_rn(sum, md);
        chain([&](double v) {
            const double c = __dsub_rn(v, mean);
            squares = __fma_rn(c, c, squares);
        });
        const double sd = __dsqrt_rn(__ddiv_rn(squares, md));
        const float mean_f = __double2float_rn(mean), std_f = sd <= 1e-12 ? 0.0f : __double2float_rn(sd);
        for (int c = 0; c < nc; c += 2) // the distances, one per half warp
        {
            const int src = c + (lane >> 4);
            const uint32_t r = __shfl_sync(0xffffffffu, row, src);
            const uint64_t gc = __shfl_sync(0xffffffffu, g, src);
            const float mc = __shfl_sync(0xffffffffu, mean_f, src), sc = __shfl_sync(0xffffffffu, std_f, src);
            const uint32_t at = __shfl_sync(0xffffffffu, idx, src);
            if (src < nc)
            {
                const TemplParam &p = tp[r];
                const float d = replica_distance16(q + p.q_offset, order + p.order_offset, raw, gc, p.m, mc, sc, lane & 15,
                                                   0xffffu << (lane & 16));
                if ((lane & 15) == 0)
                    dist[at] = d;
            }
            __syncwarp();
        }
    }
}

// ---- launchers --------------------------------------------------------------------

// Templates side by side in a grid, whose y extent is limited; the kernels take the rest in turn.
static unsigned grid_rows(int count) { return (unsigned)std::min(count, 32768); }

// sup: scratch of nk x nb keys (used by templates whose merge offset exceeds a bucket).
cudaError_t launch_bucket_select(const uint32_t *bmin_u, uint32_t *sup, uint32_t nb, int blog, const TemplParam *tp,
                                 const int *knn_slots, int nk, bool super, uint32_t *tkey, cudaStream_t s)
{
    const FftRow *rows = nullptr;
    float *cuts = nullptr;
    if (super)
        k_super_buckets<<<dim3(std::min(nb / 256 + 1, 64u), grid_rows(nk)), 256, 0, s>>>(bmin_u, nb, nb, blog, tp, knn_slots, nk,
                                                                                         rows, nk, sup);
    k_bucket_select<<<nk, 1024, 0, s>>>(bmin_u, sup, nb, nb, blog, tp, knn_slots, nk, rows, tkey, cuts);
    return cudaGetLastError();
}

cudaError_t launch_fft_cuts(const FftRow *rows, int nrows, const uint32_t *bmin_u, uint32_t *sup, uint32_t nb, uint32_t nb_seen,
                            int blog, const TemplParam *tp, const int *slots, int nk, bool super, float *cuts, cudaStream_t s)
{
    uint32_t *tkey = nullptr;
    if (super)
        k_super_buckets<<<dim3(std::min(nb_seen / 256 + 1, 64u), grid_rows(nrows)), 256, 0, s>>>(bmin_u, nb, nb_seen, blog, tp,
                                                                                                 slots, nk, rows, nrows, sup);
    k_bucket_select<<<nrows, 1024, 0, s>>>(bmin_u, sup, nb, nb_seen, blog, tp, slots, nk, rows, tkey, cuts);
    return cudaGetLastError();
}

cudaError_t launch_odd_buckets(uint32_t *bmin_u, uint32_t nb, int blog, const TemplParam *tp, const int *knn_slots, int nk,
                               const uint32_t *odd, uint64_t w0, uint32_t W, cudaStream_t s)
{
    k_odd_buckets<<<1184, 256, 0, s>>>(bmin_u, nb, blog, tp, knn_slots, nk, odd, w0, W);
    return cudaGetLastError();
}

cudaError_t launch_list_buckets(const uint32_t *bmin_l, uint32_t nb, const int *knn_slots, int nk,
                                const uint32_t *tkey, uint2 *list, uint32_t *counters, uint32_t cap, cudaStream_t s)
{
    k_list_buckets<<<dim3(std::min(nb / 1024 + 1, 64u), grid_rows(nk)), 256, 0, s>>>(bmin_l, nb, knn_slots, nk, tkey, list,
                                                                                    counters, cap);
    return cudaGetLastError();
}

cudaError_t launch_passb(const uint2 *list, const uint32_t *counters, uint32_t cap, const ScanArgs &c, const uint32_t *tkey,
                         bool mixed, const int *knn_slots, int nk, float *lower, uint32_t *bins, float *tight, int sms,
                         cudaStream_t s)
{
    PassB a{};
    if (bins != nullptr)
        if (const cudaError_t e = cudaMemsetAsync(bins, 0, sizeof(uint32_t) * kTightBins * (size_t)c.T, s); e != cudaSuccess)
            return e;
    a.lower = lower;
    a.bins = bins;
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
    a.odd = c.odd;
    a.cand = c.cand;
    a.cand_count = c.cand_count;
    a.cand_cap = c.cand_cap;
    a.untrusted = c.cand_count + 7;
    a.nb = c.nb;
    a.bmin_l = c.bmin_l;
    a.certain = c.bucket_log == 8 ? c.bmin_u : nullptr; // the bound has been selected
    const unsigned grid = 8u * (unsigned)sms; // resident blocks; the list's length is known on the device only
    if (mixed)
        k_passb<true><<<grid, B_THREADS, 0, s>>>(a);
    else
        k_passb<false><<<grid, B_THREADS, 0, s>>>(a);
    if (bins != nullptr)
        k_tight_bound<<<nk, kTightBins, 0, s>>>(bins, c.tp, knn_slots, tkey, tight);
    return cudaGetLastError();
}

// pv: the prefix sums, when the group's windows have them (Q not null); else mean: the
// windows' means, near enough to centre their sums. shortest, longest: of the templates. todo: scratch
// of `count` indices; todo_count: its counter and one more, zeroed here.
cudaError_t launch_rescore(const Candidate *cand, uint32_t count, const TemplParam *tp, const float *q,
                           const int *order, const float *raw, const PrefixView &pv, const float *mean, uint64_t w0, float *dist,
                           uint32_t *todo, uint32_t *todo_count, const Exclusion &ex, int shortest, int longest, int sms,
                           cudaStream_t s)
{
    if (count == 0)
        return cudaSuccess;
    if (const cudaError_t e = cudaMemsetAsync(todo_count, 0, 2 * sizeof(uint32_t), s); e != cudaSuccess)
        return e;
    const bool many = count >= T_COUNT, prefix = pv.Q != nullptr;
    uint32_t *sampled = many ? todo_count + 1 : nullptr;
    const unsigned threads = std::min((count - 1) / T_THREADS + 1, 64u * (unsigned)sms);
    if (many && shortest <= T_MIDDLE)
    {
        if (prefix && longest > T_SHORT)
            k_rescore_sample<<<T_SAMPLES / 256, 256, 0, s>>>(cand, count, tp, pv, w0, sampled);
        k_rescore_threads<false><<<threads, T_THREADS, 0, s>>>(cand, count, tp, q, order, raw, w0, dist, todo, todo_count, sampled,
                                                               ex);
        if (longest <= T_SHORT)
            return cudaGetLastError();
    }
    const unsigned grid = (count - 1) / (R_THREADS / 16) + 1;
    auto *kernel = prefix ? k_rescore<true> : k_rescore<false>;
    kernel<<<grid, R_THREADS, 0, s>>>(cand, count, tp, q, order, raw, pv, mean, w0, dist, todo, todo_count, ex, sampled);
    // how many are undecided the device knows
    if (many)
        k_rescore_threads<true><<<threads, T_THREADS, 0, s>>>(cand, count, tp, q, order, raw, w0, dist, todo, todo_count, sampled,
                                                              ex);
    const unsigned serial = std::min((count - 1) / S_WARPS + 1, 4u * (unsigned)sms);
    k_rescore_serial<<<serial, S_WARPS * 32, 0, s>>>(cand, tp, q, order, raw, w0, dist, todo, todo_count,
                                                     many ? T_COUNT : 0xffffffffu);
    return cudaGetLastError();
}

} // namespace tmb
