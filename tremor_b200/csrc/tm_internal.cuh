// Internal declarations shared by the tremor_b200 CUDA sources.
#pragma once

#include <cuda_runtime.h>
#include <cstdint>

namespace tmb {

constexpr float kMissing = -100000.0f; // ZnormSearch.hpp:21
constexpr float kFltMax = 3.402823466e+38f;
constexpr int kZnormBlock = 32;      // ZnormSearch.hpp:65
// Windows per kNN bound bucket: 2^8, or as many (up to 2^11) as keep a group's minima, 8 bytes
// per template and bucket, within `most` bytes: 2 GiB, or less where memory is short. Small buckets bound the k-th distance more tightly and
// leave the re-pass fewer windows; each contraction kernel's tile or chunk is at most 2^8
// windows, so none of them does more work for a smaller bucket.
constexpr int kBucketLogMin = 8, kBucketLogMax = 11;
constexpr uint64_t kMinimaBytes = 2ull << 30;
inline int bucket_log(uint64_t templates, uint64_t windows, uint64_t most = kMinimaBytes)
{
    int b = kBucketLogMin;
    while (b < kBucketLogMax && 8 * templates * ((windows >> b) + 4) > most)
        b++;
    return b;
}
// Buckets of a row of minima, rounded up so that rows start at 16-byte boundaries (the padding
// stays empty).
inline uint32_t bucket_count(uint64_t windows, int log)
{
    return (uint32_t)(((windows + (1ull << log) - 1) >> log) + 3) & ~3u;
}
// Distance given to a kNN candidate that is excluded without one (k_rescore): no candidate has it.
constexpr float kExcluded = -1.0f;
// What excludes kNN candidates. With a merge offset: the buckets' minima of d - E, the certain minima
// that k_passb left where those of d + E were, the bounds; nb = 0: nothing does (or the buckets are
// too large). Without: the candidates' d - E and the templates' tight bounds (k_tight_bound), or
// null.
struct Exclusion
{
    const uint32_t *bmin_l, *certain, *tkey;
    uint32_t nb;
    const float *lower, *tight;
};
constexpr int kTightBins = 256; // counts of a template's d + E between 0 and its bound
constexpr uint32_t kNoWindow = 0xffffffffu;
constexpr uint32_t kNoOdd = 0xffffffffu; // no sample that is not finite follows (launch_odd_next)
constexpr int kStagePad = 16384 + 512; // zero samples after the waveform (template padding)

// per-window flags (one byte per window and length)
constexpr uint8_t kFlagNotSearched = 1;  // first sample missing, or a sample that is not finite
constexpr uint8_t kFlagDegenerate = 2;   // reference std <= 1e-12: distance FLT_MAX
constexpr uint8_t kFlagNeedsExact = 4;   // prefix-sum statistics not trusted: two-pass fix-up
constexpr uint8_t kFlagExact = 8;        // statistics are the reference's two-pass values

// Per-template constants of the fused epilogue (one per template in a batch).
struct TemplParam
{
    double inv_m;  // 1 / m (statistics from prefix sums)
    float s1;      // sum of z-normalised template samples
    float c_lin;   // sum q^2 + m
    float thr_ed;  // threshold mode: cc_to_ed(correlation, m); kNN: unused
    float a1_main; // error-bound coefficients, see fast_distance (tm_epilogue.cuh);
    float a1_fp32; //   a1 for the main contraction kernel and for the FP32 re-pass
    float a2, a3, a4, a5, a6;
    int mode;         // TM_MODE_KNN (1) / TM_MODE_THRESHOLD (0)
    int m;            // template length
    int k;            // kNN answers
    int merge;        // merge offset
    int64_t q_offset; // float offset of the template in the packed template array
    int64_t order_offset; // int offset of its block order
    uint32_t wcount;  // windows of this template in the searched range (mixed-length tiles)
    float qs;         // |q| sqrt(m)
};

// A tile of a mixed-length group (128 template rows, or a column tile): its K extent.
struct TileInfo
{
    int kb; // K blocks of 64 samples (the longest template of the tile)
};

// A candidate window for exact re-scoring: template slot and window index relative
// to the window range start, plus (after re-scoring) the reference FP32 distance.
struct Candidate
{
    uint32_t templ;
    uint32_t window;
};

// Monotone map float -> uint32 so that unsigned min equals float min.
__host__ __device__ inline uint32_t float_key(float f)
{
    uint32_t b;
#ifdef __CUDA_ARCH__
    b = __float_as_uint(f);
#else
    __builtin_memcpy(&b, &f, 4);
#endif
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__host__ __device__ inline float key_float(uint32_t k)
{
    uint32_t b = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
    float f;
#ifdef __CUDA_ARCH__
    f = __uint_as_float(b);
#else
    __builtin_memcpy(&f, &b, 4);
#endif
    return f;
}
constexpr uint32_t kEmptyKey = 0xffffffffu; // above every finite float's key
__host__ __device__ inline float inf_f()
{
#ifdef __CUDA_ARCH__
    return __int_as_float(0x7f800000);
#else
    return __builtin_huge_valf();
#endif
}

} // namespace tmb
