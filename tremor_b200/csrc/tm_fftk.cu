// In-tree FP64 FFT kernels of the FFT branch: the spectra of the record's pieces, the
// templates' spectra, and one fused kernel that correlates every template of a group with
// every piece and evaluates the distance bound, bucket minima and threshold candidates
// straight from shared memory. TREMOR's FFT branch (fft_fallback.hpp:67-117: per piece,
// the product with the template spectrum, an inverse real FFT, the dot product of each
// window and the distance filter with an error bound) has this structure; here neither the
// product spectrum nor the correlation leaves the SM.
//
// Pieces of L samples, one every S; the window j = p S + o, 0 <= o < S, of piece p has its dot
// product at output o + m - 1 of the circular correlation, which does not wrap for m <= L - S
// + 1. The work per piece does not depend on S, so the step is as large as the template's
// length allows (fft_class_of): L = 8192 and S = 7168 or 6144 for templates of up to 1025 or
// 2049 samples, L = 16384 and S = 12288 up to 4097 samples and 8192 above. Two blocks of the
// shorter pieces share an SM and overlap; at 2049 samples and above the shorter pieces' wasted
// outputs cost more than that gains (an item takes 3.44 us per SM with L = 8192 and 8.3 with
// 16384, windows skipped: m = 4096 0.19 ms per template and 2^25 samples with L = 8192, 0.153
// with 16384; m = 1024 0.109 against 0.123). A template longer than 8192 samples
// is cut in two parts whose products are added before the one inverse transform (part 1 meets
// the next piece, whose start is 8192 samples later):
//     V[k] = X_p[k] Y_0[k] + X_{p+1}[k] Y_1[k],
// so its cost per window is that of a short template plus a second product. Each piece is
// shifted by s_p, the centre of the prefix block holding its start, rounded to float (the
// second part's other shift is corrected by (s_{p+1} - s_p) sum q_1 on the dot product).
//
// Real transforms of length L go through complex ones of N = L / 2 points:
//   forward: z[n] = x[2n] + i x[2n+1], Z = FFT_N(z),
//            X[k] = (Z[k] + conj Z[N-k]) / 2 - i e^{-2 pi i k / L} (Z[k] - conj Z[N-k]) / 2;
//   inverse: for a Hermitian spectrum V,
//            C[k] = (V[k] + conj V[N-k]) + i e^{2 pi i k / L} (V[k] - conj V[N-k]),
//            c = IFFT_N(C) (unnormalised), out[2n] = Re c[n], out[2n+1] = Im c[n],
//            and out / L is the circular correlation of x with the reversed template (the
//            templates' spectra carry the exact factor 1 / L).
//
// Twiddles of the forward transforms: e^{2 pi i e / 32768} = R2[e >> 7] R1[e & 127] from
// tables of 128 and 256 entries computed on the host in extended precision and rounded
// (error <= 4u with u = 2^-53, the product included); a pass's powers w^r (r = 1..15) by
// repeated multiplication (error <= 7 r u <= 105u). Those of the inverse come from tables of
// the same precision, their powers and products with 16th roots of unity by at most four
// multiplications (error <= 40u). Error of an output (Higham, Accuracy and Stability of
// Numerical Algorithms, Thm 24.2, ||fl(FFT x) - FFT x||_2 <= t eta / (1 - t eta)
// ||FFT x||_2, eta = mu + gamma_4 (sqrt 2 + mu), mu the twiddle error): with mu = 105u,
// t = 16 = log2 16384 + 2 (the complex stages plus the real-transform packing) and a factor 10 for
// the higher-radix and packing arithmetic, kappa = 10 t 111u. With X = FFT(x - s_p), Y =
// FFT(reversed q), ||X||_2 = sqrt(L) ||x - s_p||_2, ||Y||_inf <= ||q||_1 <= sqrt(m)
// ||q||_2: ||fl(X) fl(Y) - X Y||_2 <= kappa sqrt(L) ||x - s_p|| ||q|| (sqrt m + sqrt L)
// (+ rounding), and the inverse adds kappa ||X Y||_2 <= kappa sqrt(L) ||x - s_p|| sqrt(m)
// ||q||, so every correlation output is within kappa ||x - s_p||_2 ||q||_2 (2 sqrt m +
// sqrt L) of the exact one; two parts add their bounds.
#include <cmath>

#include "../../include/tremor_b200.h"
#include "tm_epilogue.cuh"
#include "tm_fft.cuh"

namespace tmb {

// The forward transform's block of N / 16 threads: its work buffer, padded complex entries,
// and the twiddle tables (R1 then R2).
template <int N> constexpr int kFBuf = N + N / 16 + 16;
template <int N> constexpr size_t kFSmem = sizeof(double2) * (size_t)(kFBuf<N> + kFftRoots);

__device__ __forceinline__ int pidx(int i) { return i + (i >> 4); }

__device__ __forceinline__ double2 cmul(double2 a, double2 b)
{
    return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 cscale(double2 a, double s) { return make_double2(a.x * s, a.y * s); }
__device__ __forceinline__ double2 conj2(double2 a) { return make_double2(a.x, -a.y); }
// a * (s i): s = +1 or -1
template <int S> __device__ __forceinline__ double2 mul_si(double2 a)
{
    return S > 0 ? make_double2(-a.y, a.x) : make_double2(a.y, -a.x);
}

// Position of R1[a] in shared memory: the low three bits XOR-ed with bits 3-5, so that the
// lookups of a quarter warp at strides 1, 2, 4 or 8 (the passes' and epilogue's patterns)
// fall in distinct banks.
__device__ __forceinline__ int r1_slot(int a) { return a ^ ((a >> 3) & 7); }

// e^{S 2 pi i e / 32768}, 0 <= e < 32768, from the shared tables R (R1 then R2).
template <int S> __device__ __forceinline__ double2 root(const double2 *R, int e)
{
    const double2 w = cmul(R[128 + (e >> 7)], R[r1_slot(e & 127)]);
    return S > 0 ? w : conj2(w);
}

// 4-point DFT with e^{S 2 pi i / 4} = S i, in place on x0..x3.
template <int S> __device__ __forceinline__ void dft4(double2 &x0, double2 &x1, double2 &x2, double2 &x3)
{
    const double2 a = cadd(x0, x2), b = csub(x0, x2), c = cadd(x1, x3), d = mul_si<S>(csub(x1, x3));
    x0 = cadd(a, c);
    x2 = csub(a, c);
    x1 = cadd(b, d);
    x3 = csub(b, d);
}

// 16-point DFT in natural order, as 4 x 4: t[b][c] = DFT4_a(v[4a + b])[c], times
// W16^{bc}, then X[c + 4d] = DFT4_b(t[b][c])[d].
template <int S> __device__ __forceinline__ void dft16(double2 (&v)[16])
{
    constexpr double c1 = 0.92387953251128675613, s1 = 0.38268343236508977173, h = 0.70710678118654752440;
#pragma unroll
    for (int b = 0; b < 4; b++)
        dft4<S>(v[b], v[4 + b], v[8 + b], v[12 + b]); // v[4c + b] now holds t[b][c]
    // twiddles W16^{bc} (b, c = 1..3): exponents 1, 2, 3, 2, 4, 6, 3, 6, 9
    const double2 w1 = make_double2(c1, S * s1), w2 = make_double2(h, S * h), w3 = make_double2(s1, S * c1);
    const double2 w6 = make_double2(-h, S * h), w9 = make_double2(-c1, -S * s1);
    v[4 + 1] = cmul(v[4 + 1], w1);
    v[8 + 1] = cmul(v[8 + 1], w2);
    v[12 + 1] = cmul(v[12 + 1], w3);
    v[4 + 2] = cmul(v[4 + 2], w2);
    v[8 + 2] = mul_si<S>(v[8 + 2]); // W16^4 = S i
    v[12 + 2] = cmul(v[12 + 2], w6);
    v[4 + 3] = cmul(v[4 + 3], w3);
    v[8 + 3] = cmul(v[8 + 3], w6);
    v[12 + 3] = cmul(v[12 + 3], w9);
#pragma unroll
    for (int c = 0; c < 4; c++)
        dft4<S>(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]); // X[c + 4d] in v[4c + d]
    // natural order: X[c + 4d] from v[4c + d] (a 4 x 4 transpose of registers)
#pragma unroll
    for (int c = 0; c < 4; c++)
#pragma unroll
        for (int d = c + 1; d < 4; d++)
        {
            const double2 t = v[4 * c + d];
            v[4 * c + d] = v[4 * d + c];
            v[4 * d + c] = t;
        }
}

// One Stockham radix-16 pass over the padded buffer of N points (N / 16 threads, in place: every
// thread reads its 16 points, the block synchronises, then every thread writes).
template <int N, int S> __device__ __forceinline__ void pass16(double2 *buf, const double2 *R, int Ns)
{
    const int j = threadIdx.x;
    double2 v[16];
#pragma unroll
    for (int r = 0; r < 16; r++)
        v[r] = buf[pidx(j + N / 16 * r)];
    __syncthreads();
    const int k = j & (Ns - 1);
    if (Ns > 1)
    {
        const double2 w1 = root<S>(R, k * (2048 / Ns)); // W^k, W = e^{S 2 pi i / (16 Ns)}
        double2 w = w1;
#pragma unroll
        for (int r = 1; r < 16; r++)
        {
            v[r] = cmul(v[r], w);
            if (r < 15)
                w = cmul(w, w1);
        }
    }
    dft16<S>(v);
    const int d0 = (j - k) * 16 + k;
#pragma unroll
    for (int r = 0; r < 16; r++)
        buf[pidx(d0 + r * Ns)] = v[r];
    __syncthreads();
}

__device__ __forceinline__ void load_roots(double2 *R, const double2 *roots)
{
    for (int i = threadIdx.x; i < kFftRoots; i += blockDim.x)
        R[i < 128 ? r1_slot(i) : i] = roots[i];
}

// Where a spectrum holds bin k (0 <= k <= N). The correlation kernel reads the bins in pairs
// k, N - k (32 bytes), with Q = N / 8 thread t of Q / 2 the pairs of bins t + Q r, r < 8 (thread
// 0: Q r, r < 4, and Q / 2 + Q (r - 4), r >= 4): pair (r, t) is at 2 (r Q / 2 + t), bin N / 2
// after them.
template <int N> __device__ __forceinline__ int spectrum_slot(int k)
{
    constexpr int Q = N / 8, T = Q / 2;
    if (k == N / 2)
        return N;
    const int res = k & (Q - 1);
    const bool second = res == 0 || res == T ? k > N / 2 : res > T; // the pair's first bin is N - k
    const int f = second ? N - k : k, t = f & (Q - 1);
    const int r = t == T ? 4 + f / Q : f / Q;
    return 2 * (T * r + (t == T ? 0 : t)) + (second ? 1 : 0);
}

// Forward real FFT of one piece of the record (block b: the piece at (p0 + b) step), or of one
// part of a template (block b: part b % parts of rows[b / parts], reversed, zero-padded
// and scaled by 1 / L), into out[b fft_pitch(N) ..] in the order of spectrum_slot. The whole of a template in one part is
// reversed end to end; a part of a longer one (of `step` samples each) as if it had `step`, so that the
// outputs of all its parts meet at the same index.
template <int N>
__global__ void __launch_bounds__(N / 16) k_fft_forward(const float *__restrict__ clean, uint64_t n,
                                       const double *__restrict__ centres, uint32_t p0, uint32_t step,
                                       const float *__restrict__ q, const TemplParam *__restrict__ tp,
                                       const FftRow *__restrict__ rows, int parts, const double2 *__restrict__ roots,
                                       double2 *__restrict__ out, double *__restrict__ shifts,
                                       double *__restrict__ norms)
{
    constexpr int T = N / 16, L = 2 * N;
    extern __shared__ double2 sm2[];
    double2 *buf = sm2, *R = sm2 + kFBuf<N>;
    __shared__ double part[T / 32];
    load_roots(R, roots);
    const bool templ = q != nullptr;
    double s = 0.0, sq = 0.0;
    uint64_t start = 0;
    const float *qt = nullptr;
    int m = 0, top = 0; // the part's samples; its last one's index before the reversal
    if (templ)
    {
        const TemplParam &p = tp[rows[blockIdx.x / parts].row];
        const int first = (int)(blockIdx.x % parts) * (int)step;
        qt = q + p.q_offset + first;
        m = parts > 1 ? min(p.m - first, (int)step) : p.m;
        top = parts > 1 ? (int)step - 1 : m - 1;
    }
    else
    {
        start = (uint64_t)(p0 + blockIdx.x) * step;
        s = (double)(float)centres[start >> kPrefixBlockLog];
    }
    for (int i = threadIdx.x; i < N; i += T)
    {
        double a, b;
        if (templ)
        {
            const int i0 = top - 2 * i, i1 = i0 - 1; // y[i] = q[top - i]
            a = i0 >= 0 && i0 < m ? (double)qt[i0] : 0.0;
            b = i1 >= 0 && i1 < m ? (double)qt[i1] : 0.0;
        }
        else
        {
            const uint64_t g = start + 2 * (uint64_t)i;
            a = g < n ? (double)clean[g] - s : 0.0;
            b = g + 1 < n ? (double)clean[g + 1] - s : 0.0;
            sq = fma(a, a, sq);
            sq = fma(b, b, sq);
        }
        buf[pidx(i)] = make_double2(a, b);
    }
    __syncthreads();
    // radix 16 three times; for N = 8192 then a radix-2 pass, in place (each thread owns the
    // pairs (i, i + 4096) it touches)
    pass16<N, -1>(buf, R, 1);
    pass16<N, -1>(buf, R, 16);
    pass16<N, -1>(buf, R, 256);
    if (N == 8192)
    {
        for (int i = threadIdx.x; i < 4096; i += T)
        {
            const double2 a = buf[pidx(i)], b = cmul(buf[pidx(i + 4096)], root<-1>(R, 4 * i));
            buf[pidx(i)] = cadd(a, b);
            buf[pidx(i + 4096)] = csub(a, b);
        }
        __syncthreads();
    }
    double2 *o = out + (size_t)blockIdx.x * fft_pitch(N);
    const double scale = templ ? 1.0 / (double)L : 1.0; // a power of two: exact
    for (int k = threadIdx.x; k <= N / 2; k += T)
    {
        // X[k] and X[N - k] from Z[k] and Z[N - k] (Z[N] = Z[0])
        const double2 A = buf[pidx(k)], Bc = conj2(buf[pidx(k == 0 ? 0 : N - k)]);
        const double2 E = make_double2(0.5 * (A.x + Bc.x), 0.5 * (A.y + Bc.y));
        const double2 D = csub(A, Bc);
        const double2 O = make_double2(0.5 * D.y, -0.5 * D.x); // -i (A - B) / 2
        const double2 w = root<-1>(R, 32768 / L * k);           // e^{-2 pi i k / L}
        o[spectrum_slot<N>(k)] = cscale(cadd(E, cmul(O, w)), scale);
        if (k == 0)
            o[spectrum_slot<N>(N)] = cscale(csub(E, O), scale); // twiddle e^{-i pi} = -1
        else if (k < N / 2)
        {
            const double2 A2 = conj2(Bc), B2c = conj2(A); // Z[N - k], conj Z[k]
            const double2 E2 = make_double2(0.5 * (A2.x + B2c.x), 0.5 * (A2.y + B2c.y));
            const double2 D2 = csub(A2, B2c);
            const double2 O2 = make_double2(0.5 * D2.y, -0.5 * D2.x);
            o[spectrum_slot<N>(N - k)] = cscale(csub(E2, cmul(O2, conj2(w))), scale); // e^{-2 pi i (N - k) / L} = -e^{2 pi i k / L}
        }
    }
    if (!templ)
    {
        for (int off = 16; off > 0; off >>= 1)
            sq += __shfl_down_sync(0xffffffffu, sq, off);
        if ((threadIdx.x & 31) == 0)
            part[threadIdx.x >> 5] = sq;
        __syncthreads();
        if (threadIdx.x == 0)
        {
            double t = 0.0;
            for (int w = 0; w < T / 32; w++)
                t += part[w];
            shifts[p0 + blockIdx.x] = s;
            norms[p0 + blockIdx.x] = sqrt(t) * (1.0 + 1e-12); // rounding of the norm itself, generously
        }
    }
}

// ---- the fused correlation ----------------------------------------------------------
//
// N / 16 threads hold the N complex points of one inverse transform in registers, 16 each.
// Pass 1 is radix 8 over the bins b + Q r, Q = N / 8, decimated in frequency (Govindaraju et
// al., "High Performance Discrete Fourier Transforms on Graphics Processors", SC 2008, for the
// passes in shared memory): thread t takes the butterflies t and Q - t, whose bins t + Q r and
// N - t - Q r are each other's partners in the real-transform packing, so the product, the
// packing and the pass need no exchange (thread 0: butterflies 0 and Q / 2, each its own
// partner). It leaves eight independent Q-point transforms, outputs n = 8 n1 + g of transform
// g, and each of those is the work of one warp (N = 4096: passes of radix 8, 8, 8) or two (N =
// 8192: 16, 8, 8), so that there are two block-wide barriers per transform. The planes are
// padded by 2 doubles per 16, which puts the quarter warps' accesses in distinct banks. The
// twiddles are folded into the butterflies, a + w b by four FMAs and a - w b = 2 a - (a + w b)
// by two.
//
// Skipped windows. Once a template has a cut (its threshold; a kNN bound from the first pieces),
// almost no window can be an answer, and a chunk of 128 windows needs its statistics only where
// some dot product exceeds what 1 / sd of that chunk allows. The bounds of 1 / sd and of the mean
// are kept for the record, at lengths a tenth apart (k_chunk_bounds); those at the next
// shorter length bound them at the template's (chunk_limit has the argument). Each thread
// compares the outputs that it holds in registers; where none of the block's is above its limit,
// the item ends there: no float outputs in shared memory, no prefix sums.
//
// What bounds it: the load/store unit's data pipe (50 to 70 % busy: three exchanges of 16 bytes a
// point and the spectra), the FP64 pipe 40 %, and with N = 8192 one block per multiprocessor,
// whose phases hardly overlap; an item that evaluates all its windows also reads 34 bytes of
// prefix sums and runs per window (or 12 bytes of a shared length's kept statistics) and issues
// 70 instructions for it. Per template and 2^25 samples, in ms, skipping / kept statistics / all
// its own (FP64 passes of radix 16, 16, 16, 2 with block-wide barriers, steps of 8192 for up to
// 8192 samples, longer pieces above and no skipping took 0.49 with kept statistics and 0.71
// without, 0.62 and 1.07 above 8192): m = 1024 0.109 / 0.171 / 0.25, 2048 0.127 / 0.169 / 0.28,
// 4096 0.153 / 0.214 / 0.32, 8192 0.231 / 0.331 / 0.44, 16000 0.33 / 0.44 / 0.63. With the outputs
// compared after they went through shared memory, and four roots per radix-8 pass loaded instead
// of one, skipping took 0.128, 0.149, 0.167, 0.248 and 0.38; with the chunks' bounds from the last
// template of the piece that evaluated every window, if at most a tenth shorter, one item in
// ten to one in two evaluated them all. 32 points per thread and two exchanges (radix 16,
// 16, 16; 8 warps per multiprocessor) took 0.177 at m = 2048 and 0.409 with distinct lengths at
// 4096 before windows were skipped, also with the epilogue on warps of its own: too few warps to
// hide the latencies.
struct FftItem // what an item needs of its piece, and its row's cut
{
    double shift[kFftMaxParts], norm[kFftMaxParts];
    float cut, pad[3];
};
template <int N> struct FftShape
{
    static constexpr int T = N / 16;             // threads
    static constexpr int GT = N / 128;           // of them, those of one transform of N / 8 points
    static constexpr int Group = N / 8 + N / 64; // doubles of that transform's plane, padding included
    static constexpr int Ex = 8 * Group;         // doubles of one exchange plane
    static constexpr int Pitch = fft_pitch(N);   // entries of a spectrum
    static constexpr int Dot = N / 4 + 4;        // floats of that transform's outputs (the pad: see the epilogue)
    // the twiddle tables: the packing's roots, then those of the two last radix-8 passes, even
    // entries before odd ones: a thread takes an even one and the next, and a quarter warp's 16-byte
    // loads fall in distinct banks (side by side, two to a bank, 1 to 2.5 % of the kernel's time)
    static constexpr int TabB = T + 1, TabC = TabB + (N == 4096 ? 8 : 16), Tabs = TabC + N / 64;
    static constexpr int Chunks = N == 4096 ? 56 : 96; // 128-window chunks of the longest step
    static constexpr size_t Smem = 2 * sizeof(double) * Ex + 8 * sizeof(float) * Dot + sizeof(double2) * Tabs +
                                   3 * sizeof(FftRow) + 2 * sizeof(FftItem) + sizeof(float4) * Chunks +
                                   sizeof(int) * (N / 64 + 2 * (N / 2048));
};
static_assert(FftShape<8192>::Smem <= 227 * 1024, "shared memory of k_fft_corr");
static_assert(2 * (FftShape<4096>::Smem + 1024) <= 228 * 1024, "two blocks of k_fft_corr<4096> per SM");
static_assert(FftShape<8192>::Tabs + FftShape<4096>::Tabs == kFftAllRoots - kFftRoots, "twiddle tables");
static_assert(sizeof(FftRow) % 16 == 0 && sizeof(FftRow) / 16 <= 8 && sizeof(FftItem) % 16 == 0, "one warp copies them");

// (a, b) -> (a + w b, a - w b), and with i w in place of w
__device__ __forceinline__ void bfly(double2 &a, double2 &b, double2 w)
{
    const double2 s = make_double2(fma(-w.y, b.y, fma(w.x, b.x, a.x)), fma(w.y, b.x, fma(w.x, b.y, a.y)));
    b = make_double2(fma(2.0, a.x, -s.x), fma(2.0, a.y, -s.y));
    a = s;
}
__device__ __forceinline__ void bfly_i(double2 &a, double2 &b, double2 w)
{
    const double2 s = make_double2(fma(-w.y, b.x, fma(-w.x, b.y, a.x)), fma(-w.y, b.y, fma(w.x, b.x, a.y)));
    b = make_double2(fma(2.0, a.x, -s.x), fma(2.0, a.y, -s.y));
    a = s;
}
__device__ __forceinline__ void bfly1(double2 &a, double2 &b)
{
    const double2 s = cadd(a, b);
    b = csub(a, b);
    a = s;
}
__device__ __forceinline__ void bfly1_i(double2 &a, double2 &b)
{
    const double2 s = make_double2(a.x - b.y, a.y + b.x);
    b = make_double2(a.x + b.y, a.y - b.x);
    a = s;
}

constexpr double kH = 0.70710678118654752440, kC16 = 0.92387953251128675613, kS16 = 0.38268343236508977173;
__device__ __forceinline__ double2 mul_w8(double2 a) // a e^{2 pi i / 8}
{
    return make_double2(kH * (a.x - a.y), kH * (a.x + a.y));
}

// v[a] +- w8 v[b], w8 = e^{2 pi i / 8}, and with i w8
__device__ __forceinline__ void bfly_w8(double2 &a, double2 &b)
{
    const double2 p = make_double2(b.x - b.y, b.x + b.y), s = a;
    a = make_double2(fma(kH, p.x, s.x), fma(kH, p.y, s.y));
    b = make_double2(fma(-kH, p.x, s.x), fma(-kH, p.y, s.y));
}
__device__ __forceinline__ void bfly_iw8(double2 &a, double2 &b)
{
    const double2 p = make_double2(b.x - b.y, b.x + b.y), s = a;
    a = make_double2(fma(-kH, p.y, s.x), fma(kH, p.x, s.y));
    b = make_double2(fma(kH, p.y, s.x), fma(-kH, p.x, s.y));
}

// X[k] = sum_r v[r] e^{2 pi i r k / 8}: X[0..7] left in v[0], v[4], v[2], v[6], v[1], v[5], v[3], v[7]
__device__ __forceinline__ void radix8_first(double2 (&v)[8])
{
#pragma unroll
    for (int r = 0; r < 4; r++)
        bfly1(v[r], v[r + 4]);
    bfly1(v[0], v[2]);
    bfly1_i(v[4], v[6]);
    bfly1(v[1], v[3]);
    bfly1_i(v[5], v[7]);
    bfly1(v[0], v[1]);
    bfly1_i(v[2], v[3]);
    bfly_w8(v[4], v[5]);
    bfly_iw8(v[6], v[7]);
}
// register of output k of a radix-8 butterfly
__device__ constexpr int out8(int k) { return (k & 3) == 0 ? (k >> 2) : (k & 3) == 2 ? 2 + (k >> 2) : (k & 3) == 1 ? 4 + (k >> 2) : 6 + (k >> 2); }

// the same of v[r] w^r, with w, w^2, w^4 and w e^{2 pi i / 8}
__device__ __forceinline__ void radix8(double2 (&v)[8], double2 w, double2 w2, double2 w4, double2 w8)
{
#pragma unroll
    for (int r = 0; r < 4; r++)
        bfly(v[r], v[r + 4], w4);
    bfly(v[0], v[2], w2);
    bfly_i(v[4], v[6], w2);
    bfly(v[1], v[3], w2);
    bfly_i(v[5], v[7], w2);
    bfly(v[0], v[1], w);
    bfly_i(v[2], v[3], w);
    bfly(v[4], v[5], w8);
    bfly_i(v[6], v[7], w8);
}

__device__ __forceinline__ double2 csqr(double2 w) { return make_double2(fma(w.x, w.x, -w.y * w.y), 2.0 * w.x * w.y); }

// X[k] = sum_r v[r] e^{2 pi i r k / 16}: X[k] left in v[out16(k)]
__device__ __forceinline__ void radix16_first(double2 (&v)[16])
{
#pragma unroll
    for (int r = 0; r < 8; r++)
        bfly1(v[r], v[r + 8]);
#pragma unroll
    for (int r = 0; r < 4; r++)
    {
        bfly1(v[r], v[r + 4]);
        bfly1_i(v[r + 8], v[r + 12]);
    }
#pragma unroll
    for (int r = 0; r < 2; r++)
    {
        bfly1(v[r], v[r + 2]);
        bfly1_i(v[r + 4], v[r + 6]);
        bfly_w8(v[r + 8], v[r + 10]);
        bfly_iw8(v[r + 12], v[r + 14]);
    }
    bfly1(v[0], v[1]);
    bfly1_i(v[2], v[3]);
    bfly_w8(v[4], v[5]);
    bfly_iw8(v[6], v[7]);
    const double2 wa = make_double2(kC16, kS16), wc = make_double2(kS16, kC16);
    bfly(v[8], v[9], wa);
    bfly_i(v[10], v[11], wa);
    bfly(v[12], v[13], wc);
    bfly_i(v[14], v[15], wc);
}
// register of output k of the radix-16 butterfly: the pair of k mod 8, then k / 8
__device__ constexpr int out16(int k)
{
    constexpr int pair[8] = {0, 4, 2, 6, 1, 5, 3, 7};
    return 2 * pair[k & 7] + (k >> 3);
}

// A window's folded statistics for the templates of one length in one piece: 1 / std, mean -
// shift, and every term of the distance bound that does not depend on the dot product
// (fast_distance_mixed's bound without a3 max(d, 0), with the largest coefficients c0 = (a1,
// a2, a5, a6), qs and |s1| of the launch's templates of this length, so it bounds each of
// them; sqrt(1 + r^2) <= 1 + |r|), plus the transform's error 2 e_dot / std. A window that is
// not searched has (0, 0, NaN): no comparison accepts its bounds and fminf ignores them; one
// whose statistics are not trusted has (0, 0, +inf): d - e = -inf, it is re-scored exactly.
__device__ __forceinline__ void fold_window(float mu, float iv, float rel_sd, float e_mu, float4 c0, float qs, float s1,
                                            int m, float shift, float e_dot, float &ms, float &ew)
{
    ms = mu - shift;
    const float r = ms * iv, r0 = mu * iv;
    WindowStats ws;
    ws.mu = mu;
    ws.iv = iv;
    ws.rel_sd = rel_sd;
    ws.e_mu = e_mu;
    ew = c0.x * (1.0f + fabsf(r)) + c0.y + c0.z * r0 * r0 + c0.w * (fabsf(mu) + fabsf(shift)) * iv +
         stats_error(ws, m, qs, s1) + 2.0f * e_dot * iv * 1.01f;
}

// The same from the statistics of the one length (fast_distance's bound, its a4 a function of m).
__device__ __forceinline__ void fold_length_window(float mu, float iv, float4 c0, int m, float shift, float e_dot, float &ms,
                                                   float &ew)
{
    ms = mu - shift;
    const float r = ms * iv, r0 = mu * iv, a4 = 1.25f * 8.0f * (float)m * (float)m * (float)kEps64;
    ew = c0.x * (1.0f + fabsf(r)) + c0.y + a4 * (1.0f + 2.0f * r0 * r0) + c0.z * r0 * r0 +
         c0.w * (fabsf(mu) + fabsf(shift)) * iv + 2.0f * e_dot * iv * 1.01f;
}

// The terms of ew = k0 + kr |r| + kq (mu / sd)^2 + (ki + s1m kb + km |mu|) / sd, the fast path's
// statistics, that an item's windows share; kb is of the window's prefix block.
struct FoldItem
{
    float k0, kr, kq, km, ki, s1m, e_dot, shift;
};
__device__ __forceinline__ FoldItem fold_item(const FftRow &P, const FftItem &I, int parts)
{
    FoldItem f;
    f.s1m = 2.5f * P.s1_max;
    f.kr = P.c0.x;
    f.kq = P.c0.z;
    f.km = P.c0.w + f.s1m * 1.3e-7f;
    f.k0 = P.c0.x + P.c0.y + 1.25f * (4.0f * (float)P.m + 2.0f * P.qs) * kFastRelSd;
    float norm = (float)I.norm[0], moved = 0.0f; // moved: the rounding of the other parts' shift corrections
    for (int i = 1; i < parts; i++)
    {
        norm += (float)I.norm[i];
        moved += fabsf((float)(I.shift[i] - I.shift[0]));
    }
    f.e_dot = fmaf(P.e_norm, norm, (float)(8.1 * kEps64) * P.qs * moved);
    f.shift = (float)I.shift[0];
    f.ki = P.c0.w * fabsf(f.shift) + 2.02f * f.e_dot;
    return f;
}

// The dot product below which no window has d - e <= cut, among windows whose 1 / sd is at most
// iv at a length m0 <= m, |mu - shift| / sd at most r and |mu| / sd at most r0. For the windows
// of m samples that begin at the same places the sum of squared deviations is no smaller (it
// splits into that of the first m0 samples and two terms >= 0), so 1 / sd is at most g = sqrt(m /
// m0) times larger; and the means differ by at most h sd, h = sqrt((m - m0) / m0): with D between
// the means of the first m0 and of the other samples, m var >= (m0 (m - m0) / m) D^2, and mu moves
// by D (m - m0) / m. d - e > cut where d > (cut + ew) / (1 - a3) for every window, and d = c_lin - 2
// (dot / sd - s1 (mu - shift) / sd). 1e-5 of c_lin is left for the FP32 rounding of all of this. A
// NaN or a value <= 0: no dot product is below it.
__device__ __forceinline__ float sqrt_approx(float x)
{
    float y;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float max_nan(float a, float b) { return a > b || a != a ? a : b; } // NaN if one is
__device__ __forceinline__ float chunk_limit(const FftRow &P, float iv, float r, float r0, float inv_m0, float cut,
                                             const FoldItem &f)
{
    const float q = (float)P.m * inv_m0;
    const float g = sqrt_approx(q), h = sqrt_approx(fmaxf(q - 1.0f, 0.0f) + 1e-6f);
    iv *= g;
    r = fmaf(r, g, h);
    r0 = fmaf(r0, g, h);
    const float ew = f.k0 + f.kr * r + f.kq * r0 * r0 + f.km * r0 + f.ki * iv;
    const float cross = 0.5f * (P.c_lin * (1.0f - 2e-5f) - (fmaxf(cut, 0.0f) + ew) * P.inv_a3) - r * fabsf(P.s1);
    return __fdividef(cross, iv); // below 0, NaN or infinite where no window is searched: any will do
}

// The bounds of each chunk of 128 windows of m samples, a warp per chunk: the largest 1 / sd and |mu
// - c| / sd, c the centre of the first window's prefix block, then c and 1 / m. Infinite where the
// statistics of a window are not trusted, or it is part of a constant run that a window of the lengths
// up to the next base may leave. Bound by the loads of the prefix sums, and read only once per
// record and length: 0.14 ms per 2^25 samples.
__global__ void __launch_bounds__(256) k_chunk_bounds(PrefixView pv, const uint16_t *__restrict__ run, uint64_t n, int m,
                                                      double inv_m, uint32_t chunks, float4 *__restrict__ bounds)
{
    const int lane = threadIdx.x & 31;
    const uint32_t c = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (c >= chunks)
        return; // whole warp
    const uint64_t first = 128ull * c;
    const float centre = first < n ? (float)pv.C[first >> kPrefixBlockLog] : 0.0f;
    float iv_max = 0.0f, r_max = 0.0f;
#pragma unroll
    for (int j = 0; j < 4; j++)
    {
        const uint64_t w = first + 32 * j + lane;
        if (w + (uint64_t)m > n)
            continue;
        const uint32_t rn = run[w];
        if (rn + 1u >= (uint32_t)fft_base_next(m))
            continue; // missing, or constant for every length that takes these bounds: not searched
        WindowStats ws;
        const bool ok = rn < (uint32_t)m && window_prefix_stats(pv, pv.Q[w], pv.Q[w + m], w, m, inv_m, ws) == 0;
        const float iv = ok ? ws.iv * (1.0f + 2.0f * ws.rel_sd) : inf_f();
        iv_max = fmaxf(iv_max, iv);
        if (ok)
            r_max = fmaxf(r_max, (fabsf(ws.mu - centre) + ws.e_mu + 2e-7f * (fabsf(ws.mu) + fabsf(centre))) * iv);
    }
    // as whole numbers: not negative, and a NaN above all
    const uint32_t mi = __reduce_max_sync(0xffffffffu, __float_as_uint(iv_max));
    const uint32_t mr = __reduce_max_sync(0xffffffffu, __float_as_uint(r_max));
    if (lane == 0)
        bounds[c] = make_float4(__uint_as_float(mi), __uint_as_float(mr), centre, (float)inv_m * 1.000001f);
}

// Statistics by the full bound (two prefix blocks, or ill-conditioned): false when they are
// not trusted.
__device__ __forceinline__ bool window_stats_full(const PrefixView &pv, double2 qa, double2 qb, uint64_t g, int m,
                                                  double inv_m, float4 &out)
{
    WindowStats ws;
    if (window_prefix_stats(pv, qa, qb, g, m, inv_m, ws) != 0)
        return false;
    out = make_float4(ws.mu, ws.iv, ws.rel_sd, ws.e_mu);
    return true;
}

// The threads that share one of the eight transforms of N / 8 points: a warp (N = 4096) or two
// (N = 8192, a named barrier).
template <int N> __device__ __forceinline__ void group_sync(int g)
{
    if (N == 4096)
        __syncwarp();
    else
        asm volatile("bar.sync %0, 64;" ::"r"(g + 1) : "memory");
}

// Candidates: bit j of mask is window j0 + 32 j of template t. Every lane of the warp calls it.
__device__ __forceinline__ void emit_strided(uint32_t mask, int lane, uint32_t t, uint32_t j0, Candidate *cand,
                                             uint32_t *count, uint32_t cap)
{
    const int c = __popc(mask);
    int incl = c;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1)
    {
        const int v = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off)
            incl += v;
    }
    uint32_t base = 0;
    if (lane == 31)
        base = atomicAdd(count, (uint32_t)incl);
    uint32_t pos = __shfl_sync(0xffffffffu, base, 31) + (uint32_t)(incl - c);
    for (; mask != 0u; mask &= mask - 1, pos++)
        if (pos < cap)
            cand[pos] = Candidate{t, j0 + 32u * (uint32_t)(__ffs(mask) - 1)};
}

// kNN bucket minima of a warp's windows (key values of d + e and d - e): one atomic per bucket
// and key, none for a bucket without searched windows. Every lane of the warp calls it.
__device__ __forceinline__ void bucket_min(const FftArgs &a, int row, uint32_t bucket, float umin, float lmin, int lane)
{
    const uint32_t ku = __reduce_min_sync(0xffffffffu, float_key(umin));
    const uint32_t kl = __reduce_min_sync(0xffffffffu, float_key(lmin));
    const uint32_t none = float_key(inf_f());
    if (lane == 0 && (ku != none || kl != none))
    {
        atomicMin(&a.bmin_u[(size_t)row * a.nb + bucket], ku);
        atomicMin(&a.bmin_l[(size_t)row * a.nb + bucket], kl);
    }
}

// A copy from global to shared memory in the background (16, 8 or 4 bytes), and the wait for
// all of this thread's.
template <int BYTES> __device__ __forceinline__ void copy_async(void *dst, const void *src)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    if (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(d), "l"(src), "n"(BYTES) : "memory");
}
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Two adjacent bins of a spectrum (32 bytes), X[k] and its partner X[N - k] (spectrum_slot). A
// block reads them once per item, so they are not kept in L1 (4 % of the kernel's time).
__device__ __forceinline__ void load_pair(const double2 *p, double2 &x, double2 &xn)
{
    asm("ld.global.nc.L1::no_allocate.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(x.x), "=d"(x.y), "=d"(xn.x), "=d"(xn.y) : "l"(p));
}

// Persistent blocks over contiguous ranges of the (piece, template) items, template fastest,
// so that the blocks end together whatever the numbers of pieces and templates are; a block
// meets a piece's templates in length order, and keeps the folded statistics of the last
// length in its slice of a global scratch (L2-resident).
//
// Per item: product, packing and pass 1; the eight transforms, whose outputs go to shared
// memory as floats; the epilogue over the item's windows (those it cannot skip), 128 per warp at a
// time. A warp goes
// on to the next item's product while others are in the epilogue.
template <int N, bool PARTS> __global__ void __launch_bounds__(N / 16, N == 4096 ? 2 : 1) k_fft_corr(const FftArgs a)
{
    using C = FftShape<N>;
    constexpr int T = C::T, L = 2 * N, H = C::Pitch, Q = N / 8;
    extern __shared__ __align__(16) double csm[];
    double *re = csm, *im = csm + C::Ex;
    float *dots = reinterpret_cast<float *>(csm + 2 * C::Ex);
    double2 *tab = reinterpret_cast<double2 *>(dots + 8 * C::Dot);
    FftRow *srow = reinterpret_cast<FftRow *>(tab + C::Tabs); // the rows of this item and the next two
    FftItem *sitem = reinterpret_cast<FftItem *>(srow + 3);   // of this item and the next
    float4 *bounds = reinterpret_cast<float4 *>(sitem + 2);   // the next item's chunks (this item's until pass 1)
    int *limits = reinterpret_cast<int *>(bounds + C::Chunks); // of the 128 outputs from 128 k on
    uint32_t *above = reinterpret_cast<uint32_t *>(limits + N / 64); // those with an output above, a bit each: two items
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const uint64_t total = (uint64_t)a.p_count * (uint32_t)a.nrows;
    const uint64_t item0 = total * blockIdx.x / gridDim.x;
    const uint32_t items = (uint32_t)(total * (blockIdx.x + 1) / gridDim.x - item0);
    uint32_t pi = (uint32_t)(item0 / (uint32_t)a.nrows);
    int ti = (int)(item0 % (uint32_t)a.nrows), cached_m = -1;
    // by warp 0, in the background: an item's row, and, once that is here, what else it needs
    auto fetch_row = [&](uint32_t item, int i) {
        if (t < (int)(sizeof(FftRow) / 16))
            copy_async<16>(reinterpret_cast<char *>(&srow[item % 3]) + 16 * t, reinterpret_cast<const char *>(a.rows + i) + 16 * t);
    };
    auto fetch_item = [&](uint32_t item, int i, uint32_t p) {
        const int parts = PARTS ? (int)min((uint32_t)a.parts, a.pieces - p) : 1;
        FftItem &I = sitem[item & 1];
        if (t == 8 && a.cuts != nullptr)
            copy_async<4>(&I.cut, a.cuts + i);
        else if (t >= 16 && t < 16 + parts)
            copy_async<8>(&I.shift[t - 16], a.shifts + p + (t - 16));
        else if (t >= 24 && t < 24 + parts)
            copy_async<8>(&I.norm[t - 24], a.norms + p + (t - 24));
        if (a.prune != 0)
        {
            const float4 *b = a.bounds[srow[item % 3].base] + (size_t)p * (a.step / 128);
            for (int c = t; c < (int)a.step / 128; c += 32)
                copy_async<16>(bounds + c, b + c);
        }
    };
    auto after = [&](int i) { return i + 1 < a.nrows ? i + 1 : 0; };
    for (int i = t; i < C::Tabs; i += T)
        tab[i] = a.tabs[i];
    if (warp == 0)
    {
        fetch_row(0, ti);
        fetch_row(1, after(ti));
        copies_wait();
        __syncwarp();
        fetch_item(0, ti, a.p_first + pi);
        copies_wait();
    }
    __syncthreads();
    float4 *cache = a.stats + (size_t)blockIdx.x * (3 * (L / 4));
    const int g = t / C::GT, s = t % C::GT; // this thread's transform of N / 8 points and its place there
    double *gre = re + g * C::Group, *gim = im + g * C::Group;
    for (uint32_t item = 0; item < items; item++)
    {
        const FftRow &P = srow[item % 3];
        const FftItem &I = sitem[item & 1];
        const uint32_t p = a.p_first + pi;
        const int m = P.m, base = (PARTS ? (int)a.step : m) - 1;
        const uint64_t piece_w = (uint64_t)p * a.step;
        // parts of the template that meet samples of the record
        const int parts = PARTS ? (int)min((uint32_t)a.parts, a.pieces - p) : 1;
        double add = 0.0;
        if (PARTS)
            for (int i = 1; i < parts; i++)
                add = fma(I.shift[i] - I.shift[0], P.sum[i - 1], add);

        // ---- may the item skip chunks of its windows? limits of the outputs 128 k to 128 k + 127, whose
        // windows lie in two chunks, as the high words of doubles ----
        const int chunks = (int)a.step / 128; // a multiple of the warps
        const float cut = a.cuts != nullptr ? I.cut : P.thr;
        const bool skip = a.prune != 0 && cut < inf_f();
        if (skip && t < N / 64)
        {
            const int c = t - ((base + 127) >> 7);
            const float shift = (float)I.shift[0];
            float iv = 0.0f, r = 0.0f, r0 = 0.0f, inv_m0 = 1.0f;
            for (int i = max(c, 0); i <= min(c + 1, chunks - 1); i++)
            {
                const float4 x = bounds[i];
                iv = max_nan(iv, x.x);
                r = max_nan(r, fmaf(fabsf(x.z - shift), x.x, x.y));
                r0 = max_nan(r0, fmaf(fabsf(x.z), x.x, x.y));
                inv_m0 = x.w;
            }
            const float limit = chunk_limit(P, iv, r, r0, inv_m0, cut, fold_item(P, I, parts));
            limits[t] = c + 1 < 0 || c >= chunks ? 0x7fffffff : limit > 0.0f ? __double2hiint((double)limit) : (int)0x80000000;
            if (t < N / 2048)
                above[(item & 1) * (N / 2048) + t] = 0u;
        }

        // ---- product, real-transform packing: C[k] for this thread's bins ----
        double2 A[8], B[8];
        {
            const double2 *X = a.X + (size_t)p * H, *Y = a.Y + (size_t)ti * (PARTS ? a.parts : 1) * H;
            const double2 wA = tab[t], wB = t != 0 ? make_double2(-wA.y, wA.x) : tab[T];
#pragma unroll
            for (int r = 0; r < 8; r++)
            {
                double2 x, xn, y, yn;
                load_pair(X + 2 * (r * T + t), x, xn);
                load_pair(Y + 2 * (r * T + t), y, yn);
                double2 V = cmul(x, y), Vn = cmul(xn, yn);
                if (PARTS)
                    for (int i = 1; i < parts; i++)
                    {
                        load_pair(X + i * H + 2 * (r * T + t), x, xn);
                        load_pair(Y + i * H + 2 * (r * T + t), y, yn);
                        V = make_double2(fma(x.x, y.x, fma(-x.y, y.y, V.x)), fma(x.x, y.y, fma(x.y, y.x, V.y)));
                        Vn = make_double2(fma(xn.x, yn.x, fma(-xn.y, yn.y, Vn.x)), fma(xn.x, yn.y, fma(xn.y, yn.x, Vn.y)));
                    }
                // w = e^{2 pi i k / L} of the bin k = t + Q r from the thread's root and a 16th root of unity
                const double2 w0 = r < 4 ? wA : wB;
                double2 w = w0;
                if ((r & 3) == 1)
                    w = make_double2(fma(w0.x, kC16, -w0.y * kS16), fma(w0.x, kS16, w0.y * kC16));
                if ((r & 3) == 2)
                    w = mul_w8(w0);
                if ((r & 3) == 3)
                    w = make_double2(fma(w0.x, kS16, -w0.y * kC16), fma(w0.x, kC16, w0.y * kS16));
                // E = V + conj Vn, D = V - conj Vn, C[k] = E + i w D, C[N-k] = conj E + i conj(w D)
                const double2 E = make_double2(V.x + Vn.x, V.y - Vn.y), D = make_double2(V.x - Vn.x, V.y + Vn.y);
                const double2 c = make_double2(fma(-w.y, D.x, fma(-w.x, D.y, E.x)), fma(-w.y, D.y, fma(w.x, D.x, E.y)));
                A[r] = c;
                B[(8 - r) & 7] = make_double2(fma(2.0, E.x, -c.x), fma(-2.0, E.y, c.y)); // bin -t + Q ((8 - r) & 7)
            }
            if (t == 0)
            {
                // butterflies 0 (bins Q r, partners within) and Q / 2 (bins Q / 2 + Q r, likewise)
                double2 V = cmul(X[N], Y[N]); // the slot of bin N / 2
                if (PARTS)
                    for (int i = 1; i < parts; i++)
                        V = cadd(V, cmul(X[i * H + N], Y[i * H + N]));
                const double2 s4 = A[4], s5 = A[5], s6 = A[6], s7 = A[7];
                const double2 n1 = B[7], n2 = B[6], n3 = B[5], n4 = B[4], n5 = B[3], n6 = B[2], n7 = B[1];
                A[4] = make_double2(2.0 * V.x, -2.0 * V.y); // C[N/2] = 2 conj V[N/2]
                A[5] = n3;
                A[6] = n2;
                A[7] = n1;
                B[0] = s4;
                B[1] = s5;
                B[2] = s6;
                B[3] = s7;
                B[4] = n7;
                B[5] = n6;
                B[6] = n5;
                B[7] = n4;
            }
        }

        // ---- pass 1: output g of butterfly b, times e^{2 pi i b g / N}, is point b of transform g ----
        radix8_first(A);
        radix8_first(B);
        {
            const int bB = t != 0 ? Q - t : Q / 2;
            const int eA = t + 2 * (t >> 4), eB = bB + 2 * (bB >> 4);
            const double2 w1 = csqr(tab[t]), w2 = csqr(w1), w3 = cmul(w2, w1), w4 = csqr(w2);
            const double2 w[8] = {make_double2(1.0, 0.0), w1, w2, w3, w4, cmul(w4, w1), csqr(w3), cmul(w4, w3)};
#pragma unroll
            for (int i = 0; i < 8; i++)
            {
                double2 va = A[out8(i)], vb = B[out8(i)];
                if (i > 0)
                {
                    va = cmul(va, w[i]);
                    vb = cmul(vb, conj2(w[i])); // butterfly -t
                    if (t == 0)                 // butterfly Q / 2: e^{2 pi i g / 16}
                    {
                        constexpr double c[8] = {1.0, kC16, kH, kS16, 0.0, -kS16, -kH, -kC16};
                        constexpr double n[8] = {0.0, kS16, kH, kC16, 1.0, kC16, kH, kS16};
                        vb = cmul(vb, make_double2(c[i], n[i]));
                    }
                }
                re[i * C::Group + eA] = va.x;
                im[i * C::Group + eA] = va.y;
                re[i * C::Group + eB] = vb.x;
                im[i * C::Group + eB] = vb.y;
            }
        }
        __syncthreads();
        if (warp == 0 && item + 1 < items) // the last item's epilogue is over: its slots are free
        {
            const int next = after(ti);
            fetch_item(item + 1, next, next > 0 ? p : p + 1);
            fetch_row(item + 2, after(next));
        }

        // ---- transform g: radix 16 (N = 8192) or 8 (N = 4096) with Ns = 1, then 8 and 8 ----
        constexpr int Ns2 = N == 4096 ? 8 : 16, R8 = Q / 8 + Q / 64; // R8: elements Q / 8 apart, padded
        const int rd = 2 * s + 2 * (s >> 3); // element r of the butterflies 2 s and 2 s + 1 at rd + R8 r
        auto read_pairs = [&]() {
#pragma unroll
            for (int r = 0; r < 8; r++)
            {
                const double2 x = *reinterpret_cast<const double2 *>(gre + rd + R8 * r);
                const double2 y = *reinterpret_cast<const double2 *>(gim + rd + R8 * r);
                A[r] = make_double2(x.x, y.x);
                B[r] = make_double2(x.y, y.y);
            }
        };
        if (N == 8192)
        {
            double2 v[16];
            const int e = s + 2 * (s >> 4);
#pragma unroll
            for (int r = 0; r < 16; r++)
                v[r] = make_double2(gre[e + 72 * r], gim[e + 72 * r]);
            radix16_first(v);
            group_sync<N>(g); // the group has read its points
#pragma unroll
            for (int r = 0; r < 16; r += 2)
            {
                *reinterpret_cast<double2 *>(gre + 18 * s + r) = make_double2(v[out16(r)].x, v[out16(r + 1)].x);
                *reinterpret_cast<double2 *>(gim + 18 * s + r) = make_double2(v[out16(r)].y, v[out16(r + 1)].y);
            }
        }
        else
        {
            read_pairs();
            radix8_first(A);
            radix8_first(B);
            group_sync<N>(g);
#pragma unroll
            for (int r = 0; r < 8; r += 2)
            {
                *reinterpret_cast<double2 *>(gre + 18 * s + r) = make_double2(A[out8(r)].x, A[out8(r + 1)].x);
                *reinterpret_cast<double2 *>(gim + 18 * s + r) = make_double2(A[out8(r)].y, A[out8(r + 1)].y);
                *reinterpret_cast<double2 *>(gre + 18 * s + 8 + r) = make_double2(B[out8(r)].x, B[out8(r + 1)].x);
                *reinterpret_cast<double2 *>(gim + 18 * s + 8 + r) = make_double2(B[out8(r)].y, B[out8(r + 1)].y);
            }
        }
        group_sync<N>(g);
        read_pairs();
        {
            const int k = (2 * s) & (Ns2 - 1);
            const double2 *w = tab + C::TabB + k / 2; // of k, then of k + 1
            {
                const double2 w1 = w[0], w2 = csqr(w1);
                radix8(A, w1, w2, csqr(w2), mul_w8(w1));
            }
            {
                const double2 w1 = w[Ns2 / 2], w2 = csqr(w1);
                radix8(B, w1, w2, csqr(w2), mul_w8(w1));
            }
            group_sync<N>(g);
            const int b = 9 * (2 * s - k) + k;
#pragma unroll
            for (int r = 0; r < 8; r++)
            {
                const int e = b + Ns2 * r + 2 * (Ns2 * r >> 4);
                *reinterpret_cast<double2 *>(gre + e) = make_double2(A[out8(r)].x, B[out8(r)].x);
                *reinterpret_cast<double2 *>(gim + e) = make_double2(A[out8(r)].y, B[out8(r)].y);
            }
        }
        group_sync<N>(g);
        read_pairs();
        {
            const double2 *w = tab + C::TabC + s; // of 2 s, then of 2 s + 1
            {
                const double2 w1 = w[0], w2 = csqr(w1);
                radix8(A, w1, w2, csqr(w2), mul_w8(w1));
            }
            {
                const double2 w1 = w[C::GT], w2 = csqr(w1);
                radix8(B, w1, w2, csqr(w2), mul_w8(w1));
            }
        }
        // outputs n1 = 2 s + (Q / 8) r and the next of transform g: correlation outputs 16 n1 + 2 g (+ 1)
        if (PARTS)
        {
#pragma unroll
            for (int r = 0; r < 8; r++)
            {
                A[r] = make_double2(A[r].x + add, A[r].y + add);
                B[r] = make_double2(B[r].x + add, B[r].y + add);
            }
        }
        copies_wait();
        bool any = true; // has a chunk to be evaluated?
        if (skip)
        {
            const int *limit = limits + (s >> 2);
            uint32_t high = 0;
#pragma unroll
            for (int r = 0; r < 8; r++)
            {
                const double2 x = A[out8(r)], y = B[out8(r)];
                const int most = max(max(__double2hiint(x.x), __double2hiint(x.y)), max(__double2hiint(y.x), __double2hiint(y.y)));
                high |= (most >= limit[(Q / 64) * r] ? 1u : 0u) << r;
            }
            any = __syncthreads_or(high != 0u) != 0;
            uint32_t *mine = above + (item & 1) * (N / 2048);
            for (; high != 0u; high &= high - 1)
            {
                const int k = (s >> 2) + (Q / 64) * (__ffs(high) - 1);
                atomicOr(&mine[k >> 5], 1u << (k & 31));
            }
        }
        if (any)
        {
            float *d = dots + g * C::Dot + 4 * s;
#pragma unroll
            for (int r = 0; r < 8; r++)
            {
                const double2 x = A[out8(r)], y = B[out8(r)];
                *reinterpret_cast<float4 *>(d + (Q / 4) * r) = make_float4((float)x.x, (float)x.y, (float)y.x, (float)y.y);
            }
            __syncthreads();
        }

        // ---- epilogue: window o of the piece is output i = o + base; a lane's windows are 128 c +
        // 32 j + lane, j < 4. Output i = 16 n1 + 2 g + h is at dots[g Dot + 2 n1 + h]: the pad puts a
        // warp's 32 consecutive outputs in distinct banks but for a few. What a chunk needs from
        // global memory is loaded while the one before is evaluated ----
        constexpr int kWarps = T / 32;
        const int per = chunks / kWarps;
        const bool knn = P.mode == TM_MODE_KNN;
        const int64_t rel = (int64_t)piece_w - (int64_t)a.w0; // window o of the piece is rel + o of the range
        const float s1 = P.s1, c_lin = P.c_lin, a3 = P.a3, thr = P.thr;
        const int i0 = base + lane;
        const float *dl = dots + ((i0 >> 1) & 7) * C::Dot + 2 * (i0 >> 4) + (i0 & 1);
        auto evaluate = [&](int c, const float (&iv)[4], const float (&ms)[4], const float (&ew)[4]) {
            const int64_t first = rel + 128 * c; // the warp's first window
            float d[4], lo[4], umin = inf_f(), lmin = inf_f();
#pragma unroll
            for (int j = 0; j < 4; j++)
            {
                const float cross = (dl[16 * c + 4 * j] - ms[j] * s1) * iv[j];
                // at most FLT_MAX, not NaN: d - e is -inf where ew is inf, whatever the dot product
                d[j] = fminf(c_lin - 2.0f * cross, kFltMax);
                const float e = ew[j] + a3 * fmaxf(d[j], 0.0f);
                lo[j] = d[j] - e;
                lmin = fminf(lmin, lo[j]);
                if (a.dbg_d != nullptr && iv[j] > 0.0f)
                {
                    a.dbg_d[(size_t)P.row * a.W + (size_t)(first + 32 * j + lane)] = d[j];
                    a.dbg_e[(size_t)P.row * a.W + (size_t)(first + 32 * j + lane)] = e;
                }
                d[j] += e;
                umin = fminf(umin, d[j]);
            }
            if (knn)
            {
                // the warp's 128 windows lie in one bucket or in two
                const uint32_t bk_lo = (uint32_t)((first > 0 ? first : 0) >> a.bucket_log);
                const uint32_t bk_hi = (uint32_t)((first + 127 > 0 ? first + 127 : 0) >> a.bucket_log);
                if (bk_lo == bk_hi)
                    bucket_min(a, P.row, bk_lo, umin, lmin, lane);
                else
                    for (uint32_t bk = bk_lo; bk <= bk_hi; bk++)
                    {
                        umin = lmin = inf_f();
#pragma unroll
                        for (int j = 0; j < 4; j++)
                            if ((uint32_t)((uint64_t)(first + 32 * j + lane) >> a.bucket_log) == bk)
                            {
                                umin = fminf(umin, d[j]);
                                lmin = fminf(lmin, lo[j]);
                            }
                        bucket_min(a, P.row, bk, umin, lmin, lane);
                    }
            }
            else if (__any_sync(0xffffffffu, lmin <= thr))
            {
                uint32_t mask = 0, lost = 0;
#pragma unroll
                for (int j = 0; j < 4; j++)
                {
                    mask |= (lo[j] <= thr ? 1u : 0u) << j;
                    lost += lo[j] == -inf_f() ? 1u : 0u;
                }
                if (lost > 0)
                    atomicAdd(a.untrusted, lost);
                emit_strided(mask, lane, (uint32_t)P.row, (uint32_t)(first + lane), a.cand, a.cand_count, a.cand_cap);
            }
        };
        uint32_t todo = any ? (1u << per) - 1u : 0u; // this warp's chunks warp + kWarps i
        if (skip && any)
            for (int i = 0; i < per; i++)
            {
                // its outputs are among 128 and the next (none past the last)
                const int k = (128 * (warp + kWarps * i) + base) >> 7, n = min(k + 1, N / 64 - 1);
                const uint32_t *set = above + (item & 1) * (N / 2048);
                if (((set[k >> 5] >> (k & 31) | set[n >> 5] >> (n & 31)) & 1u) == 0u)
                    todo &= ~(1u << i);
            }
        int c = warp + kWarps * (__ffs(todo) - 1);
        auto next_chunk = [&]() { // after c, or c again at the end
            todo &= todo - 1;
            return todo != 0u ? warp + kWarps * (__ffs(todo) - 1) : c;
        };
        if (todo == 0u)
        {
        }
        else if (m == cached_m)
        {
            const float4 *cc = cache + lane;
            float4 x = cc[32 * c], y = cc[L / 4 + 32 * c], z = cc[L / 2 + 32 * c];
            while (todo != 0u)
            {
                const float iv[4] = {x.x, x.y, x.z, x.w}, ms[4] = {y.x, y.y, y.z, y.w}, ew[4] = {z.x, z.y, z.z, z.w};
                const int n = next_chunk();
                x = cc[32 * n];
                y = cc[L / 4 + 32 * n];
                z = cc[L / 2 + 32 * n];
                evaluate(c, iv, ms, ew);
                c = n;
            }
        }
        else
        {
            // the next item's template has the same length and meets the same piece
            const bool keep = !skip && item + 1 < items && ti + 1 < a.nrows && srow[(item + 1) % 3].m == m;
            const FoldItem F = fold_item(P, I, parts);
            const float shift = F.shift;
            const float s1m = F.s1m, k0 = F.k0, kr = F.kr, kq = F.kq, km = F.km;
            // the piece's windows in the template's range; loads for windows outside take the
            // nearest one inside (an empty range takes the piece's first sample, which exists)
            const int64_t left = (int64_t)P.wcount - rel;
            const int o_lo = rel < 0 ? (int)min(-rel, (int64_t)a.step) : 0;
            const int o_hi = left < (int64_t)a.step ? (int)max(left, (int64_t)0) : (int)a.step;
            const bool any = o_lo < o_hi;
            const int w_lo = any ? o_lo : 0, w_hi = any ? o_hi - 1 : 0, len = any ? m : 0;
            const double2 *Qp = a.pv.Q + piece_w;
            const uint16_t *rp = a.run + piece_w;
            const double inv_m = P.inv_m;
            const float fim = (float)inv_m * (1.0f + 1.1920929e-07f);
            double2 qa[4], qb[4];
            uint32_t rn[4];
            auto load = [&](int n) {
                const int f = 128 * n; // the warp's first window
                if (f >= w_lo && f + 127 <= w_hi)
                {
                    const double2 *x = Qp + (f + lane);
                    const double2 *y = x + len;
                    const uint16_t *z = rp + (f + lane);
#pragma unroll
                    for (int j = 0; j < 4; j++)
                    {
                        qa[j] = x[32 * j];
                        qb[j] = y[32 * j];
                        rn[j] = z[32 * j];
                    }
                }
                else
                {
#pragma unroll
                    for (int j = 0; j < 4; j++)
                    {
                        const int w = min(max(f + 32 * j + lane, w_lo), w_hi);
                        qa[j] = Qp[w];
                        qb[j] = Qp[w + len];
                        rn[j] = rp[w];
                    }
                }
            };
            uint64_t b0 = ~0ull; // the prefix block whose constants follow
            float cen = 0.0f, kib = 0.0f, va = 0.0f, vb = 0.0f;
            load(c);
            while (todo != 0u)
            {
                const int f = 128 * c, o = f + lane;
                // the block of the warp's first window; almost always that of every window's samples too
                const uint64_t b = (piece_w + (uint64_t)min(max(f, w_lo), w_hi)) >> kPrefixBlockLog;
                const uint64_t be = (piece_w + (uint64_t)(min(max(f + 127, w_lo), w_hi) + len)) >> kPrefixBlockLog;
                if (b != b0)
                {
                    // prefix_stats_fast's condition is fvar >= va + vb |mu_c| and its e_mu is
                    // bb.b / m + 1.3e-7 |mu| + 1.9e-7 |c|, all of it folded in kib and km
                    b0 = b;
                    cen = (float)a.pv.C[b];
                    const BlockBounds bb = block_bounds(a.pv.T[b].y);
                    kib = F.ki + s1m * (bb.b * fim + 1.9e-7f * fabsf(cen));
                    va = bb.a * fim * (1.00001f / 0.9e-7f);
                    vb = 2.0f * bb.b * fim * (1.00001f / 0.9e-7f);
                }
                float iv[4], ms[4], ew[4];
                uint32_t slow = 0;
#pragma unroll
                for (int j = 0; j < 4; j++)
                {
                    const double mu_c = (qb[j].x - qa[j].x) * inv_m;
                    const double var = fma(-mu_c, mu_c, (qb[j].y - qa[j].y) * inv_m);
                    const float fvar = (float)var, fmu = (float)mu_c;
                    const float mu = fmu + cen;
                    // vb is NaN where the block's squares pass FLT_MAX: a comparison of its own, false then
                    const bool ok = fvar >= fmaf(vb, fabsf(fmu), va) && fvar > fmaxf(1e-6f * fmu * fmu, 2e-22f) && fvar < 1e36f;
                    const bool srch = o + 32 * j >= o_lo && o + 32 * j < o_hi && rn[j] < (uint32_t)m;
                    const float v = rsqrtf(fvar), x = mu - shift, r0 = mu * v;
                    const float e = fmaf(kr, fabsf(x * v), k0) + fmaf(kq * r0, r0, fmaf(km, fabsf(mu), kib) * v);
                    iv[j] = srch ? v : 0.0f;
                    ms[j] = srch ? x : 0.0f;
                    ew[j] = srch ? e : __int_as_float(0x7fc00000);
                    slow |= (srch && (!ok || be != b) ? 1u : 0u) << j;
                }
                // two prefix blocks, or ill-conditioned: the full bound, one window at a time
                for (; slow != 0u; slow &= slow - 1)
                {
                    const int jj = __ffs(slow) - 1, w = o + 32 * jj;
                    float4 st;
                    const bool ok = window_stats_full(a.pv, Qp[w], Qp[w + m], piece_w + (uint64_t)w, m, inv_m, st);
                    float v = ok ? st.y : 0.0f;
                    float x = 0.0f, e = inf_f();
                    if (ok)
                        fold_window(st.x, v, st.z, st.w, P.c0, P.qs, P.s1_max, m, shift, F.e_dot, x, e);
                    else if (a.inv != nullptr && a.inv[rel + w] != 0.0f)
                    {
                        v = a.inv[rel + w];
                        fold_length_window(a.mean[rel + w], v, P.c0, m, shift, F.e_dot, x, e);
                    }
#pragma unroll
                    for (int j = 0; j < 4; j++)
                        if (j == jj)
                        {
                            iv[j] = v;
                            ms[j] = x;
                            ew[j] = e;
                        }
                }
                const int n = next_chunk();
                load(n);
                if (keep)
                {
                    float4 *cc = cache + 32 * c + lane;
                    cc[0] = make_float4(iv[0], iv[1], iv[2], iv[3]);
                    cc[L / 4] = make_float4(ms[0], ms[1], ms[2], ms[3]);
                    cc[L / 2] = make_float4(ew[0], ew[1], ew[2], ew[3]);
                }
                evaluate(c, iv, ms, ew);
                c = n;
            }
        }
        if (!skip)
            cached_m = m;
        if (++ti == a.nrows)
        {
            ti = 0;
            pi++;
            cached_m = -1; // the cache holds the last piece's statistics
        }
    }
}

// The twiddle tables, in extended precision rounded to double: the forward kernel's R1[a] =
// e^{2 pi i a / 32768} (a < 128) and R2[b] = e^{2 pi i 128 b / 32768} (b < 256), then the
// correlation kernel's, for N = 8192: e^{2 pi i t / L} (t <= 512), e^{2 pi i k / 128} (k < 16) and
// e^{2 pi i b / 1024} (b < 128).
static double2 root_of(long double num, long double den)
{
    const long double a = 6.283185307179586476925286766559005768L * num / den;
    return make_double2((double)cosl(a), (double)sinl(a));
}

template <int N> static void corr_tables(double2 *tab)
{
    using C = FftShape<N>;
    constexpr int Ns = N == 4096 ? 8 : 16;
    for (int i = 0; i <= C::T; i++)
        tab[i] = root_of(i, 2 * N);
    for (int k = 0; k < Ns; k++)
    {
        tab[C::TabB + (k & 1) * (Ns / 2) + k / 2] = root_of(k, 8 * Ns);
    }
    for (int b = 0; b < N / 64; b++)
        tab[C::TabC + (b & 1) * C::GT + b / 2] = root_of(b, N / 8);
}

void fft_roots(double2 *host)
{
    for (int a = 0; a < 128; a++)
        host[a] = root_of(a, 32768);
    for (int b = 0; b < 256; b++)
        host[128 + b] = root_of(128 * b, 32768);
    corr_tables<8192>(host + kFftRoots);
    corr_tables<4096>(host + kFftRoots + FftShape<8192>::Tabs);
}

uint32_t fft_pieces(uint64_t n, int cls) { return (uint32_t)((n + fft_class(cls).step - 1) / fft_class(cls).step); }

template <int N, class... Args> static cudaError_t launch_forward(unsigned blocks, cudaStream_t s, Args... args)
{
    const cudaError_t e =
        cudaFuncSetAttribute(k_fft_forward<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFSmem<N>);
    if (e != cudaSuccess)
        return e;
    k_fft_forward<N><<<blocks, N / 16, kFSmem<N>, s>>>(args...);
    return cudaGetLastError();
}

cudaError_t launch_fft_pieces(const float *clean, uint64_t n, const double *centres, int cls, const double2 *roots,
                              double2 *X, double *shifts, double *norms, cudaStream_t s)
{
    const FftClass c = fft_class(cls);
    const float *q = nullptr;
    const TemplParam *tp = nullptr;
    const FftRow *rows = nullptr;
    return c.n == 4096 ? launch_forward<4096>(fft_pieces(n, cls), s, clean, n, centres, 0u, c.step, q, tp, rows, 1, roots, X,
                                              shifts, norms)
                       : launch_forward<8192>(fft_pieces(n, cls), s, clean, n, centres, 0u, c.step, q, tp, rows, 1, roots, X,
                                              shifts, norms);
}

cudaError_t launch_fft_templates(const float *q, const TemplParam *tp, const FftRow *rows, int nrows, int cls, int parts,
                                 const double2 *roots, double2 *Y, cudaStream_t s)
{
    const FftClass c = fft_class(cls);
    const float *clean = nullptr;
    const double *centres = nullptr;
    double *none = nullptr;
    const unsigned blocks = (unsigned)(nrows * parts);
    return c.n == 4096 ? launch_forward<4096>(blocks, s, clean, (uint64_t)0, centres, 0u, c.step, q, tp, rows, parts, roots, Y,
                                              none, none)
                       : launch_forward<8192>(blocks, s, clean, (uint64_t)0, centres, 0u, c.step, q, tp, rows, parts, roots, Y,
                                              none, none);
}

template <int N, bool PARTS> static cudaError_t launch_corr(FftArgs a, int sms, cudaStream_t s)
{
    constexpr size_t smem = FftShape<N>::Smem;
    auto *kernel = k_fft_corr<N, PARTS>;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess)
        return e;
    const uint64_t items = (uint64_t)a.p_count * (uint32_t)a.nrows;
    const uint64_t most = (uint64_t)sms * (N == 4096 ? 2 : 1);
    if (items > 0)
        kernel<<<(unsigned)std::min(items, most), N / 16, smem, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_chunk_bounds(const PrefixView &pv, const uint16_t *run, uint64_t n, int m, float4 *bounds, cudaStream_t s)
{
    const uint32_t chunks = (uint32_t)fft_chunks(n);
    k_chunk_bounds<<<(chunks + 7) / 8, 256, 0, s>>>(pv, run, n, m, 1.0 / m, chunks, bounds);
    return cudaGetLastError();
}

// roots: the tables of fft_roots; a.step and a.tabs are filled in here.
cudaError_t launch_fft_corr(FftArgs a, int cls, const double2 *roots, int sms, cudaStream_t s)
{
    const FftClass c = fft_class(cls);
    a.step = c.step;
    a.tabs = roots + kFftRoots + (c.n == 4096 ? FftShape<8192>::Tabs : 0);
    if (c.n == 4096)
        return a.parts > 1 ? launch_corr<4096, true>(a, sms, s) : launch_corr<4096, false>(a, sms, s);
    return a.parts > 1 ? launch_corr<8192, true>(a, sms, s) : launch_corr<8192, false>(a, sms, s);
}

} // namespace tmb
