// Answer assembly on the device, after the exact re-scoring (tm_select.cu k_rescore).
//
// The reference collects, per template, every verified window: threshold hits whose
// ED^2 <= threshold (Tremor.cpp:2008, SkipSequential.cpp:279-290) and the kNN
// candidates offered to the bound queue. Threshold post-processing sorts a template's
// hits by position (Tremor.cpp:2760-2795); the kNN answer is the canonical exclusion
// selection over the candidates in (ED^2, position) order (ZnormSearch.hpp:170-189).
// Here both happen on the device, so the host receives finished runs:
//   k_answer_keys      keeps the candidates that can be answers (threshold templates:
//                      exact ED^2 <= threshold; kNN templates: all that are not excluded) as
//                      (template << 32 | window, ED^2) pairs
//   radix sort 1       by that key: template-major, position order within a template
//   k_answer_rekey     (only when the group has kNN templates) kNN entries get the key
//                      (flag, template, ED^2 bits) and threshold entries keep
//                      (template, window); the flag, above the template bits, moves
//                      every kNN run after all threshold runs
//   radix sort 2       by the new key; the sort is stable, so equal distances stay in
//                      position order: (distance, position) order within a kNN run
//   k_answer_segments  each template's run [start, end), its windows and distances
// Few answers (launch_answer_runs has the rule) take k_answer_runs in place of the sorts, the rekeying
// and the segments: one block per template gathers its entries and sorts them in shared memory.
//   k_select_knn       one block per kNN template: the greedy exclusion selection over
//                      its run (finite distances only), up to k answers
// The sorts are CUB's device radix sort from the CUDA toolkit, over 32 + ceil(log2 T)
// (+1) key bits. Within a template no window appears twice: every (template, window)
// pair is visited by exactly one contraction tile, and the kNN re-pass lists each
// bucket once.
#include <cub/device/device_radix_sort.cuh>

#include "../../include/tremor_b200.h"
#include "tm_internal.cuh"

namespace tmb {

constexpr int kAnswerThreads = 256;
constexpr int kSelectThreads = 256, kRunThreads = 512;

__device__ __forceinline__ void warp_slot(bool keep, uint32_t *counter, uint32_t &slot)
{
    const unsigned ballot = __ballot_sync(0xffffffffu, keep);
    const int lane = threadIdx.x & 31;
    uint32_t base = 0;
    if (ballot != 0u)
    {
        const int leader = __ffs(ballot) - 1;
        if (lane == leader)
            base = atomicAdd(counter, (uint32_t)__popc(ballot));
        base = __shfl_sync(0xffffffffu, base, leader);
    }
    slot = base + (uint32_t)__popc(ballot & ((1u << lane) - 1u));
}

// kept[0]: answers kept, kept[1]: of which belong to kNN templates; tcount: by template (or null).
__global__ void __launch_bounds__(kAnswerThreads)
    k_answer_keys(const Candidate *__restrict__ cand, const float *__restrict__ dist, uint32_t count,
                  const TemplParam *__restrict__ tp, unsigned long long *__restrict__ keys, float *__restrict__ vals,
                  uint32_t *__restrict__ kept, uint32_t *__restrict__ tcount)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    bool keep = false, knn = false;
    Candidate c{0u, 0u};
    float d = 0.0f;
    if (i < count)
    {
        c = cand[i];
        d = dist[i];
        knn = tp[c.templ].mode == TM_MODE_KNN;
        keep = knn ? d != kExcluded : d <= tp[c.templ].thr_ed;
    }
    uint32_t slot, unused;
    warp_slot(keep, kept, slot);
    warp_slot(keep && knn, kept + 1, unused);
    if (tcount != nullptr)
    {
        const uint32_t same = __match_any_sync(0xffffffffu, keep ? c.templ : 0xffffffffu);
        if (keep && (int)(threadIdx.x & 31) == __ffs(same) - 1)
            atomicAdd(&tcount[c.templ], (uint32_t)__popc(same));
    }
    if (keep)
    {
        keys[slot] = ((unsigned long long)c.templ << 32) | (unsigned long long)c.window;
        vals[slot] = d;
    }
}

__global__ void __launch_bounds__(kAnswerThreads)
    k_answer_rekey(const unsigned long long *__restrict__ keys, const float *__restrict__ vals, uint32_t count,
                   const TemplParam *__restrict__ tp, int tbits, unsigned long long *__restrict__ keys2,
                   unsigned long long *__restrict__ vals2)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count)
        return;
    const unsigned long long k = keys[i];
    const uint32_t t = (uint32_t)(k >> 32), w = (uint32_t)k;
    const float d = vals[i];
    const bool knn = tp[t].mode == TM_MODE_KNN;
    keys2[i] = knn ? (1ull << (32 + tbits)) | ((unsigned long long)t << 32) | float_key(d) : k;
    vals2[i] = ((unsigned long long)w << 32) | __float_as_uint(d);
}

// start[t], end[t] (zeroed before: templates without answers keep the empty run [0, 0)),
// and the run's windows and distances. PACKED: values are (window << 32 | ED^2 bits);
// otherwise the window is the key's low half and the values are the distances.
template <bool PACKED>
__global__ void __launch_bounds__(kAnswerThreads)
    k_answer_segments(const unsigned long long *__restrict__ keys, const void *__restrict__ vals, uint32_t count,
                      uint32_t tmask, uint32_t *__restrict__ start, uint32_t *__restrict__ end,
                      uint32_t *__restrict__ window, float *__restrict__ dist)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count)
        return;
    const uint32_t t = (uint32_t)(keys[i] >> 32) & tmask;
    if (PACKED)
    {
        const unsigned long long v = static_cast<const unsigned long long *>(vals)[i];
        window[i] = (uint32_t)(v >> 32);
        dist[i] = __uint_as_float((uint32_t)v);
    }
    else
    {
        window[i] = (uint32_t)keys[i];
        dist[i] = static_cast<const float *>(vals)[i];
    }
    if (i == 0 || ((uint32_t)(keys[i - 1] >> 32) & tmask) != t)
        start[t] = i;
    if (i + 1 == count || ((uint32_t)(keys[i + 1] >> 32) & tmask) != t)
        end[t] = i + 1;
}

// The run of template blockIdx.x: its entries among all that are kept, in (distance, position) order
// for kNN, by position for a threshold, after the runs of the templates before it, thresholds
// first. Bound by latency, of the walk over the answers and of the 66 to 78 steps of the bitonic
// sort: 3300 answers of 16 templates in 15 us, where two radix sorts of five passes, of one
// block each, and what lay between took 110.
__global__ void __launch_bounds__(kRunThreads)
    k_answer_runs(const unsigned long long *__restrict__ keys, const float *__restrict__ vals, uint32_t kept,
                  const TemplParam *__restrict__ tp, int T, const uint32_t *__restrict__ tcount, uint32_t *__restrict__ start,
                  uint32_t *__restrict__ end, uint32_t *__restrict__ window, float *__restrict__ dist)
{
    extern __shared__ unsigned long long run[];
    __shared__ uint32_t offset, filled;
    const int t = blockIdx.x, tid = threadIdx.x;
    const bool knn = tp[t].mode == TM_MODE_KNN;
    const uint32_t n = tcount[t];
    if (tid == 0)
        offset = filled = 0u;
    __syncthreads();
    uint32_t before = 0;
    for (int i = tid; i < T; i += kRunThreads)
    {
        const bool other = tp[i].mode == TM_MODE_KNN;
        if (other == knn ? i < t : knn)
            before += tcount[i];
    }
    before = __reduce_add_sync(0xffffffffu, before);
    if ((tid & 31) == 0 && before > 0)
        atomicAdd(&offset, before);
    for (uint32_t i = tid; i < kept && n > 0; i += kRunThreads)
    {
        const unsigned long long key = keys[i];
        if ((int)(key >> 32) == t)
        {
            const unsigned long long w = (uint32_t)key, d = float_key(vals[i]);
            run[atomicAdd(&filled, 1u)] = knn ? d << 32 | w : w << 32 | d;
        }
    }
    uint32_t size = 2;
    while (size < n)
        size *= 2;
    for (uint32_t i = n + tid; i < size; i += kRunThreads)
        run[i] = ~0ull;
    __syncthreads();
    for (uint32_t k = 2; k <= size && n > 1; k *= 2)
        for (uint32_t j = k / 2; j > 0; j /= 2)
        {
            for (uint32_t p = tid; p < size / 2; p += kRunThreads)
            {
                const uint32_t i = 2 * p - (p & (j - 1)), o = i + j; // bit j of i is clear
                const unsigned long long a = run[i], b = run[o];
                if ((a > b) == ((i & k) == 0u))
                {
                    run[i] = b;
                    run[o] = a;
                }
            }
            __syncthreads();
        }
    const uint32_t at = offset;
    for (uint32_t i = tid; i < n; i += kRunThreads)
    {
        const uint32_t hi = (uint32_t)(run[i] >> 32), lo = (uint32_t)run[i];
        window[at + i] = knn ? lo : hi;
        dist[at + i] = key_float(knn ? hi : lo);
    }
    if (tid == 0)
    {
        start[t] = n > 0 ? at : 0u;
        end[t] = n > 0 ? at + n : 0u;
    }
}

// Greedy exclusion selection of one kNN template per block over its run in (distance,
// position) order: a candidate is kept when no kept window lies closer than merge
// (|gap| < merge), until k are kept (ZnormSearch.hpp:170-189). Only finite distances
// take part; the run's FLT_MAX entries, at its end, are left to the host, which needs
// them only when the reference's queue would not have filled. out_n[slot] = answers kept.
//
// A run is long when its nearest windows crowd around few events (tens of thousands of
// candidates for 100 answers), and almost all of it falls to the check against the kept
// windows: the block takes one candidate per thread, with the next ones on their way from
// memory, and only the survivors, in order, go to one warp, which accepts them in turn,
// each one removing the later ones within merge of it. Bound by the chain of chunks, one
// after another, of the longest run: 3.4 million candidates of 512 templates in 0.41 ms,
// where a warp per template, 32 candidates at a time, took 4.8.
__global__ void __launch_bounds__(kSelectThreads)
    k_select_knn(const int *__restrict__ slots, const TemplParam *__restrict__ tp, const uint32_t *__restrict__ start,
                 const uint32_t *__restrict__ end, const uint32_t *__restrict__ window,
                 const float *__restrict__ dist, int kcap, uint32_t *__restrict__ out_n,
                 uint32_t *__restrict__ out_win, float *__restrict__ out_dist)
{
    extern __shared__ uint4 kept_smem[]; // the kept windows: kcap, rounded up to fours
    __shared__ uint32_t left_win[kSelectThreads], warp_left[kSelectThreads / 32];
    __shared__ float left_dist[kSelectThreads];
    __shared__ int kept_count;
    uint32_t *kw = reinterpret_cast<uint32_t *>(kept_smem);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, slot = blockIdx.x;
    const int t = slots[slot];
    const int k = min(tp[t].k, kcap);
    const uint32_t merge = (uint32_t)max(tp[t].merge, 0);
    const uint32_t a = start[t], b = end[t];
    uint32_t *ow = out_win + (size_t)slot * kcap;
    float *od = out_dist + (size_t)slot * kcap;
    int n = 0;
    uint32_t w = 0u;
    float d = kFltMax;
    if (a + tid < b)
    {
        w = window[a + tid];
        d = dist[a + tid];
    }
    for (uint32_t base = a; base < b && n < k; base += kSelectThreads)
    {
        const uint32_t cw = w, next = base + kSelectThreads + tid;
        const float cd = d;
        w = 0u;
        d = kFltMax;
        if (next < b)
        {
            w = window[next];
            d = dist[next];
        }
        bool pass = cd < kFltMax; // false past the run's end too
        const bool last = !pass;
        if (merge > 0 && pass)
        {
            int j = 0;
            for (; j + 4 <= n && pass; j += 4)
            {
                const uint4 q = kept_smem[j / 4];
                pass = __usad(cw, q.x, 0u) >= merge && __usad(cw, q.y, 0u) >= merge && __usad(cw, q.z, 0u) >= merge &&
                       __usad(cw, q.w, 0u) >= merge;
            }
            for (; j < n && pass; j++)
                pass = __usad(cw, kw[j], 0u) >= merge;
        }
        // the survivors, in order
        const unsigned ballot = __ballot_sync(0xffffffffu, pass);
        if (lane == 0)
            warp_left[warp] = (uint32_t)__popc(ballot);
        const bool stop = __syncthreads_or(last);
        uint32_t pos = (uint32_t)__popc(ballot & ((1u << lane) - 1u)), total = 0;
#pragma unroll
        for (int i = 0; i < kSelectThreads / 32; i++)
        {
            const uint32_t c = warp_left[i];
            pos += i < warp ? c : 0u;
            total += c;
        }
        if (total > 0) // the same in every thread
        {
            if (pass)
            {
                left_win[pos] = cw;
                left_dist[pos] = cd;
            }
            __syncthreads();
            if (warp == 0)
            {
                const int n0 = n;
                for (uint32_t i0 = 0; i0 < total && n < k; i0 += 32)
                {
                    const bool valid = i0 + lane < total;
                    const uint32_t lw = valid ? left_win[i0 + lane] : 0u;
                    const float ld = valid ? left_dist[i0 + lane] : 0.0f;
                    bool open = valid;
                    for (int j = n0; j < n && merge > 0; j++) // kept since the check
                        open = open && __usad(lw, kw[j], 0u) >= merge;
                    unsigned ob = __ballot_sync(0xffffffffu, open);
                    if (merge == 0)
                    {
                        const int at = n + __popc(ob & ((1u << lane) - 1u));
                        if (open && at < k)
                        {
                            ow[at] = lw;
                            od[at] = ld;
                        }
                        n = min(k, n + __popc(ob));
                        continue;
                    }
                    while (ob != 0u && n < k)
                    {
                        const int leader = __ffs(ob) - 1;
                        const uint32_t aw = __shfl_sync(0xffffffffu, lw, leader);
                        if (lane == leader)
                        {
                            kw[n] = lw;
                            ow[n] = lw;
                            od[n] = ld;
                        }
                        n++;
                        open = open && lane != leader && __usad(lw, aw, 0u) >= merge;
                        ob = __ballot_sync(0xffffffffu, open);
                    }
                    __syncwarp();
                }
                if (lane == 0)
                    kept_count = n;
            }
            __syncthreads();
            n = kept_count;
        }
        else
            __syncthreads(); // warp_left is written again
        if (stop)
            break;
    }
    if (tid == 0)
        out_n[slot] = (uint32_t)n;
}

// Key bits for T templates: the window's 32 and enough for the template index.
int answer_template_bits(int T)
{
    int b = 0;
    while (b < 30 && (1u << b) < (uint32_t)T)
        b++;
    return b;
}

cudaError_t launch_answer_keys(const Candidate *cand, const float *dist, uint32_t count, const TemplParam *tp,
                               unsigned long long *keys, float *vals, uint32_t *kept, uint32_t *tcount, cudaStream_t s)
{
    if (count > 0)
        k_answer_keys<<<(count + kAnswerThreads - 1) / kAnswerThreads, kAnswerThreads, 0, s>>>(cand, dist, count, tp,
                                                                                              keys, vals, kept, tcount);
    return cudaGetLastError();
}

// When few answers are few: at most 4096 of one template, which fit in shared memory (45 us; 58 by
// radix for thresholds, twice that for kNN), and at most 32768 in all, since each template's block
// walks over all of them (50000 took 62 us, by radix 66), 2^24 looks by all blocks.
constexpr uint32_t kRunMost = 4096, kRunAnswers = 32768;
constexpr uint64_t kRunLooks = 1ull << 24;
bool answer_runs_apply(uint32_t count, int T, uint32_t most)
{
    return most <= kRunMost && count <= kRunAnswers && (uint64_t)count * (uint64_t)T <= kRunLooks;
}

cudaError_t launch_answer_runs(const unsigned long long *keys, const float *vals, uint32_t count, uint32_t most,
                               const TemplParam *tp, int T, const uint32_t *tcount, uint32_t *start, uint32_t *end,
                               uint32_t *window, float *dist, cudaStream_t s)
{
    uint32_t size = 2;
    while (size < most)
        size *= 2;
    if (T > 0)
        k_answer_runs<<<T, kRunThreads, sizeof(unsigned long long) * size, s>>>(keys, vals, count, tp, T, tcount, start, end,
                                                                               window, dist);
    return cudaGetLastError();
}

// Scratch bytes both sorts need for `count` pairs (a size query: nothing is launched).
size_t answer_sort_scratch(uint32_t count, int T)
{
    const int tb = answer_template_bits(T);
    size_t b1 = 0, b2 = 0;
    cub::DoubleBuffer<unsigned long long> k(nullptr, nullptr), v64(nullptr, nullptr);
    cub::DoubleBuffer<float> v32(nullptr, nullptr);
    cub::DeviceRadixSort::SortPairs(nullptr, b1, k, v32, count, 0, 32 + tb);
    cub::DeviceRadixSort::SortPairs(nullptr, b2, k, v64, count, 0, 33 + tb);
    return b1 > b2 ? b1 : b2;
}

// The answer order of the `count` kept pairs in (keys[0], vals32[0]); knn_count of them
// belong to kNN templates. Leaves each template's run in start/end, its windows in
// `window` and distances in `dist` (count entries each; threshold runs first).
cudaError_t launch_answer_order(unsigned long long *const keys[2], float *const vals32[2],
                                unsigned long long *const vals64[2], uint32_t count, uint32_t knn_count,
                                const TemplParam *tp, int T, void *scratch, size_t scratch_bytes, uint32_t *start,
                                uint32_t *end, uint32_t *window, float *dist, cudaStream_t s)
{
    if (count == 0)
        return cudaSuccess;
    const int tb = answer_template_bits(T);
    const uint32_t tmask = (1u << tb) - 1u;
    const unsigned grid = (count + kAnswerThreads - 1) / kAnswerThreads;
    cub::DoubleBuffer<unsigned long long> k(keys[0], keys[1]);
    cub::DoubleBuffer<float> v(vals32[0], vals32[1]);
    cudaError_t e = cub::DeviceRadixSort::SortPairs(scratch, scratch_bytes, k, v, count, 0, 32 + tb, s);
    if (e != cudaSuccess)
        return e;
    if (k.selector != v.selector)
        return cudaErrorUnknown;
    if (knn_count == 0)
    {
        k_answer_segments<false><<<grid, kAnswerThreads, 0, s>>>(k.Current(), v.Current(), count, ~0u, start,
                                                                 end, window, dist);
        return cudaGetLastError();
    }
    unsigned long long *k2a = k.Alternate(), *k2b = k.Current();
    k_answer_rekey<<<grid, kAnswerThreads, 0, s>>>(k.Current(), v.Current(), count, tp, tb, k2a, vals64[0]);
    cub::DoubleBuffer<unsigned long long> k2(k2a, k2b), v2(vals64[0], vals64[1]);
    e = cub::DeviceRadixSort::SortPairs(scratch, scratch_bytes, k2, v2, count, 0, 33 + tb, s);
    if (e != cudaSuccess)
        return e;
    if (k2.selector != v2.selector)
        return cudaErrorUnknown;
    k_answer_segments<true><<<grid, kAnswerThreads, 0, s>>>(k2.Current(), v2.Current(), count, tmask, start, end,
                                                            window, dist);
    return cudaGetLastError();
}

cudaError_t launch_select_knn(const int *slots, int nk, const TemplParam *tp, const uint32_t *start,
                              const uint32_t *end, const uint32_t *window, const float *dist, int kcap,
                              uint32_t *out_n, uint32_t *out_win, float *out_dist, cudaStream_t s)
{
    if (nk > 0)
        k_select_knn<<<nk, kSelectThreads, sizeof(uint4) * ((kcap + 3) / 4), s>>>(slots, tp, start, end, window, dist,
                                                                                  kcap, out_n, out_win, out_dist);
    return cudaGetLastError();
}

} // namespace tmb
