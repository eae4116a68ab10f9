// The FFT branch's constants, launch arguments and launchers (tm_fftk.cu).
#pragma once

#include <cmath>

#include "tm_internal.cuh"
#include "tm_prefix.cuh"

namespace tmb {

// Pieces of 2 n samples, one every `step` (tm_fftk.cu). A template of up to 2 n - step + 1
// samples has every window of a piece in one transform; a longer one is cut in parts of
// `step` samples.
struct FftClass
{
    int n;
    uint32_t step;
};
constexpr int kFftClasses = 4;
__host__ __device__ constexpr FftClass fft_class(int cls)
{
    return cls == 0   ? FftClass{4096, 7168}
           : cls == 1 ? FftClass{4096, 6144}
           : cls == 2 ? FftClass{8192, 12288}
                      : FftClass{8192, 8192};
}
// entries of a spectrum: its n + 1 bins in whole 128-byte lines
__host__ __device__ constexpr int fft_pitch(int n) { return n + 8; }
constexpr int kFftMaxM = 16384; // longest template of the FFT branch
constexpr int kFftMaxParts = 2;
inline int fft_class_of(int m) { return m <= 1025 ? 0 : m <= 2049 ? 1 : m <= 4097 ? 2 : 3; }
inline int fft_parts(int m, int cls)
{
    const int single = 2 * fft_class(cls).n - (int)fft_class(cls).step + 1, step = (int)fft_class(cls).step;
    return m <= single ? 1 : (m + step - 1) / step;
}

// Templates of one correlation launch: 25 MB of spectra, well within L2, where every block reads them
// once per piece.
inline int fft_launch_rows(int cls, int parts) { return 192 * 8200 / (fft_pitch(fft_class(cls).n) * parts); }

// Lengths that the bounds of the record's chunks of 128 windows are kept at (k_chunk_bounds): a
// template takes those of the largest of them that it reaches, at most a tenth shorter.
constexpr int kFftBases = 100;
__host__ __device__ constexpr int fft_base_next(int m) { return m + 1 > m * 11 / 10 ? m + 1 : m * 11 / 10; }
inline int fft_base(int m) // its index
{
    int i = 0;
    for (int b = 1; fft_base_next(b) <= m; b = fft_base_next(b))
        i++;
    return i;
}
inline int fft_base_length(int index)
{
    int b = 1;
    for (int i = 0; i < index; i++)
        b = fft_base_next(b);
    return b;
}
// Chunks of a record, those of its last pieces' windows past the end included.
inline size_t fft_chunks(uint64_t n) { return (size_t)((n + 16384) / 128); }

// One template of a correlation launch. The bound coefficients (a1_main, a2, a5, a6), qs and
// |s1| are the largest of the launch's templates of its length.
struct FftRow
{
    double inv_m;
    double sum[kFftMaxParts - 1]; // the sums of its parts after the first
    float s1, c_lin, a3, thr; // thr: infinite for kNN
    float4 c0;
    float qs, s1_max;
    int row; // its row in tp
    int m, mode;
    uint32_t wcount;
    float e_norm; // fft_e_norm
    float inv_a3; // 1 / (1 - a3), rounded up
    int base;     // fft_base(m)
    int pad[3];
};

// An FFT dot product's error: norms of the template and of the piece's samples times this; the
// largest norm of a template of length m is qs / sqrt(m). 1 % is left for FP32 rounding.
constexpr double kFftKappa = 10.0 * 16.0 * 111.0 * 1.1102230246251565e-16;
inline float fft_e_norm(float qs, int m, int cls)
{
    const double sm = sqrt((double)m);
    return (float)(1.01 * kFftKappa * (double)qs / sm * (2.0 * sm + sqrt(2.0 * fft_class(cls).n)));
}

struct FftArgs
{
    const double2 *X;             // piece spectra, fft_pitch(n) entries per piece
    const double *shifts, *norms; // per piece: its shift s_p and ||x - s_p||_2
    uint32_t pieces, step;        // pieces of the record, samples between their starts
    uint32_t p_first, p_count;    // pieces of this launch
    const double2 *Y;             // template spectra, one per part and entry of rows
    const FftRow *rows;           // the launch's templates, equal lengths adjacent
    int nrows, parts;
    const double2 *tabs;          // twiddle tables of the correlation kernel
    uint64_t w0;                  // window range start (windows are relative to it)
    uint32_t W;
    PrefixView pv;
    const uint16_t *run;
    const float *mean, *inv; // one length, where the prefix sums lose windows: its own statistics; else null
    uint32_t *untrusted;     // candidates for want of statistics are counted here
    uint32_t *bmin_u, *bmin_l;
    uint32_t nb;
    int bucket_log;
    Candidate *cand;
    uint32_t *cand_count, cand_cap;
    float *dbg_d, *dbg_e; // diagnostics: d and e of every window, [t][W]; null in searches
    int prune;            // some template has a cut: no window with d - e above it is wanted
    const float *cuts;    // the cuts of rows' templates; null: their thr
    const float4 *bounds[kFftBases]; // with prune, the chunks' bounds at the rows' bases
    float4 *stats;        // per block, the folded statistics of a piece's windows (a lane's scratch, kFftStats)
};

// float4s of the statistics scratch per SM: 3 floats per output, two blocks of the shorter
// transform or one of the longer
constexpr int kFftStats = 3 * (16384 / 4);

constexpr int kFftRoots = 384; // entries of the forward kernel's twiddle tables; the correlation kernels' follow
constexpr int kFftAllRoots = kFftRoots + (513 + 16 + 128) + (257 + 8 + 64);

uint32_t fft_pieces(uint64_t n, int cls);
void fft_roots(double2 *host); // kFftAllRoots entries
cudaError_t launch_fft_pieces(const float *clean, uint64_t n, const double *centres, int cls, const double2 *roots,
                              double2 *X, double *shifts, double *norms, cudaStream_t s);
cudaError_t launch_fft_templates(const float *q, const TemplParam *tp, const FftRow *rows, int nrows, int cls, int parts,
                                 const double2 *roots, double2 *Y, cudaStream_t s);
// Cuts of the templates of rows from the minima of the first nb_seen buckets (tm_select.cu): a
// threshold, a kNN bound or infinity. sup: nk x nb_seen keys of scratch, where super is set.
cudaError_t launch_fft_cuts(const FftRow *rows, int nrows, const uint32_t *bmin_u, uint32_t *sup, uint32_t nb, uint32_t nb_seen,
                            int blog, const TemplParam *tp, const int *slots, int nk, bool super, float *cuts, cudaStream_t s);
cudaError_t launch_chunk_bounds(const PrefixView &pv, const uint16_t *run, uint64_t n, int m, float4 *bounds, cudaStream_t s);
cudaError_t launch_fft_corr(FftArgs a, int cls, const double2 *roots, int sms, cudaStream_t s);

} // namespace tmb
