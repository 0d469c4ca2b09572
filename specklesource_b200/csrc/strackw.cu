// strackw.cu -- corrTrackFast (Strackw/corrTrackFast.c:89-231) on the GPU.
//
// Grid points go through the kernels below in chunks; every kernel spreads the
// lines (or rows) of all points of the chunk over the chip.  Per point
// (W = wRa = waa, N = 2W, e = edgePad + NFAST/4, chip c2 = N - 4e, lags
// L = 4e + 1):
//  1. estDopCarrier1 on the raw windows (:340; window_batch.cuh);
//  2. upsampling by two (:718-761).  The 2W x 2W zero-padded inverse is
//     separable, its even samples are the window's own samples (times a phase
//     in azimuth that the detection removes) and its odd samples the window
//     shifted by half a sample: sw_cols makes the azimuth-shifted window
//     (forward line, roll, half-sample phase, inverse line), sw_rows the range
//     shift of the raw and of the shifted rows.  Six line passes instead of
//     the eight that four parity transforms of a 2-D spectrum take, and only
//     the intensities |z|^2 * scale leave the chip;
//  3. detectPatch (:765-839): optional (2 navg + 1)^2 box sums in float in the
//     reference's order and clamps (the chip's azimuth clamp uses edgePadR),
//     range sums in sw_rows, azimuth sums and sqrt in sw_amps; the chip of
//     image 2 is embedded in zeros, image 1 is the full search area;
//  4. computeMeanSigma (:407-477): chip mean and variance from sw_amps' sums;
//     the search window's at every one of the L^2 placements in sw_stats, in
//     double: running column windows started from 16-row sums, then prefix
//     sums along the row;
//  5. ampMatchEdge (:903-947): one packed forward transform of
//     (search + i chip), the Hermitian cross spectrum and the real inverse on
//     half the columns (sw_fwd, sw_corr, sw_ncc); with both images' means
//     removed first, the result is the covariance term of getPeakCorr directly
//     (an exact identity that avoids the float cancellation of
//     c*scaleW - meanR*meanS);
//  6. getPeakCorr (:862-899): normalised correlation on the lags, argmax
//     inside the user radius (row-major first maximum) in sw_ncc / sw_peak;
//  7. overSampleC (:951-990): the 21 x 21 block's symmetric zero pad to
//     336 x 336 evaluated on the searched 64 x 64 window only, as B X B^T with
//     the real kernel B[n][t] = 1 + 2 sum_{f=1..10} cos(2 pi f (n - 16 t)/336),
//     in double; cMax = sqrt(max |.|^2)/441, shifts in 1/32 px.
// Windows whose far edge leaves the image (the reference checks only the
// near corner, :170-171, then reads stale buffer rows) read zeros here.
#include <cuda_runtime.h>

#include <vector>

#include "capi_internal.h"
#include "strack_device.cuh"
#include "window_batch.cuh"

namespace sbk {

constexpr int W_NOVER = 16;  // corrTrackFast.c:11
constexpr int W_NFAST = 20;  // corrTrackFast.c:12
constexpr int W_N1 = W_NFAST + 1;
constexpr int W_OSW = 64;    // searched window [168-32, 168+32)
constexpr int W_SEG = 16;    // rows per partial column sum

// What sw_reduce makes of sw_amps' sums.
struct SwMoments {
    double meanR, sigmaR, meanS;
};

struct SwArgs {
    WinArgs win;      // the chunk's windows
    const int* list;  // grid index of each point of the chunk
    const int* az;    // Doppler roll of each point
    int e;            // edge pad including the internal +5
    int navgR, navgA;
    int taps;         // box half width when both axes share it (2, 3), -1: no box, 0: any
    float scale;
    const float2* twW;
    const float2* twN;
    const float2* tau;
    // planes, one per point of the chunk
    float2* xv;       // 2 x W x W: azimuth half-sample shift of both windows
    float* H;         // 2 x N x N: intensities, range box sums
    float2* Z;        // N x N row transforms (over H, which is spent by then)
    float* A1;        // N x N search amplitudes
    float* A2;        // c2 x c2 chip amplitudes
    double* seg;      // N/16 x 2 x N: sums of A1 and A1^2 over 16 rows
    double* part;     // N/16 x 3 partial sums of the moments
    SwMoments* mom;
    double* norm;     // L x L: scaleW / sqrt(sigmaR sigmaS)
    float2* T;        // L x corr_ts(N)
    double* ncc;      // L x L
    double* bestV;    // per row-pair tile
    int* bestE;
    const double* B;  // 64 x 21 oversampling kernel
    float* offR;
    float* offA;
    float* corr;
    uint8_t* type;
    unsigned long long* stats;  // [0] matched, [1] failed
};

struct DArg {
    double v;
    int rank;
};
__device__ __forceinline__ bool darg_better(double v, int r, double bv, int br)
{
    return v > bv || (v == bv && r < br);
}
template <int NT>
__device__ __forceinline__ DArg block_argmax_d(DArg a, double* dsc, int* isc)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double v = __shfl_xor_sync(0xffffffffu, a.v, o);
        const int r = __shfl_xor_sync(0xffffffffu, a.rank, o);
        if (darg_better(v, r, a.v, a.rank)) {
            a.v = v;
            a.rank = r;
        }
    }
    if (lane == 0) {
        dsc[warp] = a.v;
        isc[warp] = a.rank;
    }
    __syncthreads();
    DArg b;
    b.v = dsc[0];
    b.rank = isc[0];
    for (int w = 1; w < NT / 32; ++w)
        if (darg_better(dsc[w], isc[w], b.v, b.rank)) {
            b.v = dsc[w];
            b.rank = isc[w];
        }
    __syncthreads();
    return b;
}

template <int W>
struct SwCfg {
    static constexpr int N = 2 * W;
    static constexpr int G = 8;                    // lines per CTA of sw_cols, sw_rows, sw_fwd, sw_ncc
    static constexpr int NTW = 128;                // threads for lines of W points
    static constexpr int NTN = 128;                // threads for lines of N points
    using CW = sbfft::LineTile<W, G, false>;
    using RW = sbfft::LineTile<W, G, true>;
    using RN = sbfft::LineTile<N, G, true>;
    static_assert(G * 16 <= NTW, "lines of W points: one item a thread and step");
    static constexpr size_t smCols = sizeof(float2) * CW::elems;
    static constexpr size_t smRows = sizeof(float2) * RW::elems;  // and the intensities
    static constexpr size_t smFwd = sizeof(float2) * RN::elems;
    static constexpr size_t smNcc = smFwd + sizeof(double) * (NTN / 32) + sizeof(int) * (NTN / 32);
    static constexpr int NTS = N <= 256 ? N : N / 2;  // sw_stats: one or two columns a thread
    static constexpr int CL = N / 32;              // columns per lane of its prefix sums
    static constexpr int PS = N + 32;              // padded prefix row
    static constexpr size_t smStats = sizeof(double) * 8 * PS;
};

// Azimuth half-sample shift of columns c0 .. c0+7 of one window: forward line,
// X'[k] = F[(k + roll) mod W] tau[k], inverse line.
template <int W, bool F32>
__global__ void __launch_bounds__(128) sw_cols_kernel(SwArgs a)
{
    chain_begin();
    using C = SwCfg<W>;
    constexpr int G = C::G, NT = C::NTW, TILES = W / G;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2* s = reinterpret_cast<float2*>(smem_raw);
    const int tile = blockIdx.x % TILES, q = blockIdx.x / TILES % 2, pt = blockIdx.x / (2 * TILES);
    const Window<F32> win(a.win, q, a.win.win[pt], W);
    const int c0 = tile * G;
    int da = a.az[pt];
    if (da < 0 || da >= W) da = 0;
    sbfft::line_fft<W, -1, G, NT, false, false, true>(
        s, a.twW, [&](int l, int k) { return win(k, c0 + l); },
        [&](int l, int k, float2 v) {
            const int r = k - da < 0 ? k - da + W : k - da;
            s[r * G + l] = sbfft::cmul(v, __ldg(a.tau + r));
        });
    __syncthreads();
    float2* out = a.xv + ((size_t)pt * 2 + q) * W * W + c0;
    sbfft::line_fft<W, 1, G, NT, false, true, false>(
        s, a.twW, [&](int l, int k) { return s[k * G + l]; },
        [&](int l, int k, float2 v) { out[k * W + l] = v; });
}

// Rows j of the doubled window (even: the raw window's, odd: the shifted
// one's): range half-sample shift, intensities of the N samples, range box
// sums.  Rows [0, N) of image 1; of image 2 those whose box sums the chip
// reads.  The intensity rows carry `pad` copies of their end values on both
// sides, so that the sums need no clamps (the chip's own clamps, kmax and lmax
// of detectPatch, never bind inside the N x N area).
template <int W, bool F32>
__global__ void __launch_bounds__(128) sw_rows_kernel(SwArgs a, int hr0, int hr1, int pad)
{
    chain_begin();
    using C = SwCfg<W>;
    constexpr int N = C::N, G = C::G, NT = C::NTW, TILES = N / G;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2* s = reinterpret_cast<float2*>(smem_raw);
    float* in = reinterpret_cast<float*>(s + C::RW::elems) + pad;
    const int PR = N + 2 * pad;  // intensity row
    const int tiles2 = (hr1 - hr0 + G) / G, per = TILES + tiles2;
    const int pt = blockIdx.x / per, b = blockIdx.x % per;
    const int q = b >= TILES;
    const int j0 = q ? hr0 + (b - TILES) * G : b * G;
    const Window<F32> win(a.win, q, a.win.win[pt], W);
    const float2* xv = a.xv + ((size_t)pt * 2 + q) * W * W;
    // every line pass is unnormalised (a factor W an axis, W^4 in intensity)
    const float s0 = a.scale * ((float)W * W * W * W), s1 = a.scale * ((float)W * W);
    // lines 0 .. 3 are the raw rows of the tile and 4 .. 7 the shifted ones
    // (j0 is even), so that a warp loads from one of the two
    auto row = [](int l) { return l < G / 2 ? 2 * l : 2 * l - G + 1; };
    sbfft::line_fft<W, -1, G, NT, true, false, true>(
        s, a.twW,
        [&](int l, int k) {
            const int i = min((j0 >> 1) + (l & (G / 2 - 1)), W - 1);
            return l < G / 2 ? win(i, k) : xv[i * W + k];
        },
        [&](int l, int k, float2 v) { s[l * C::RW::L + k] = sbfft::cmul(v, __ldg(a.tau + k)); },
        [&](int l, int k, float2 v) {
            in[row(l) * PR + 2 * k] = (v.x * v.x + v.y * v.y) * (l < G / 2 ? s0 : s1);
        });
    __syncthreads();
    sbfft::line_fft<W, 1, G, NT, true, true, false>(
        s, a.twW, [&](int l, int k) { return s[l * C::RW::L + k]; },
        [&](int l, int k, float2 v) {
            in[row(l) * PR + 2 * k + 1] = (v.x * v.x + v.y * v.y) * (l < G / 2 ? s1 : a.scale);
        });
    __syncthreads();
    if (pad) {
        for (int e = threadIdx.x; e < 2 * G * pad; e += NT) {
            const int l = e % G, m = e / G;
            if (m < pad) in[l * PR - 1 - m] = in[l * PR];
            else in[l * PR + N + m - pad] = in[l * PR + N - 1];
        }
        __syncthreads();
    }
    float* H = a.H + ((size_t)pt * 2 + q) * N * N;
    const int c0 = q ? 2 * a.e : 0, c1 = q ? N - 2 * a.e : N;  // image 2: the chip's columns
    const int rows = q ? min(G, hr1 - j0 + 1) : G;
    // Half width 2, the 5 x 5 box that fast-flow pairs are run with, has its own
    // loop: 2.87 ms for 3.05 in the general one at W = 64 (7,018 points), 1.96
    // for 2.13 at 128 (1,566), 3.57 for 3.81 at 224 (836).  The other widths take
    // the general one; half width 3 would gain as much (3.17 -> 2.92, 2.23 ->
    // 2.00, 3.94 -> 3.61) and has no loop of its own here.
    const int lane = threadIdx.x & 31;
    for (int l = threadIdx.x >> 5; l < rows; l += NT / 32) {
        const float* p = in + l * PR;
        float* h = H + (size_t)(j0 + l) * N;
        if (a.taps == 2) {
            for (int j = c0 + lane; j < c1; j += 32) h[j] = p[j - 2] + p[j - 1] + p[j] + p[j + 1] + p[j + 2];
        } else if (a.taps < 0) {
            for (int j = c0 + lane; j < c1; j += 32) h[j] = p[j];
        } else {
            for (int j = c0 + lane; j < c1; j += 32) {
                float t = 0.f;
                for (int m = -a.navgR; m <= a.navgR; m++) t += p[min(max(j + m, -pad), N - 1 + pad)];
                h[j] = t;
            }
        }
    }
}

// Azimuth box sums and amplitudes, a thread per column and 16 rows a CTA; the
// sums that the moments and sw_stats start from.  TAPS: the half width of the
// box (-1: none), so that a thread loads each row once and adds from
// registers; 0: any, as separate loads.
template <int W, int TAPS>
__global__ void __launch_bounds__(2 * W) sw_amps_kernel(SwArgs a)
{
    chain_begin();
    constexpr int N = 2 * W, NT = N;
    __shared__ double red[(NT / 32 + 1) * 3];
    const int pt = blockIdx.x / (N / W_SEG), sg = blockIdx.x % (N / W_SEG), j = threadIdx.x;
    const int e2 = 2 * a.e, c2 = N - 2 * e2;
    const float* H1 = a.H + (size_t)pt * 2 * N * N + j;
    const float* H2 = H1 + (size_t)N * N;
    float* A1 = a.A1 + (size_t)pt * N * N + j;
    float* A2 = a.A2 + (size_t)pt * c2 * c2 + (j - e2);
    double cs[3] = {0, 0, 0}, q1 = 0, q2 = 0;
    const bool col = j >= e2 && j < e2 + c2;
    const int i0 = sg * W_SEG;
    // amplitudes of 16 rows of one plane
    auto rows = [&](const float* H, float (&v)[W_SEG]) {
        if constexpr (TAPS < 0) {
#pragma unroll
            for (int r = 0; r < W_SEG; ++r) v[r] = H[(i0 + r) * N];
        } else if constexpr (TAPS > 0) {
            float h[W_SEG + 2 * TAPS];
#pragma unroll
            for (int r = 0; r < W_SEG + 2 * TAPS; ++r) h[r] = H[min(max(i0 + r - TAPS, 0), N - 1) * N];
#pragma unroll
            for (int r = 0; r < W_SEG; ++r) {
                v[r] = h[r];
#pragma unroll
                for (int m = 1; m <= 2 * TAPS; ++m) v[r] += h[r + m];
            }
        } else {
            for (int r = 0; r < W_SEG; ++r) {
                v[r] = 0.f;
                for (int m = -a.navgA; m <= a.navgA; m++) v[r] += H[min(max(i0 + r + m, 0), N - 1) * N];
            }
        }
    };
    float v[W_SEG];
    rows(H1, v);
#pragma unroll
    for (int r = 0; r < W_SEG; ++r) {
        const float x = sqrtf(v[r]);
        A1[(i0 + r) * N] = x;
        q1 += x;
        q2 += (double)(x * x);
    }
    if (col && i0 + W_SEG > e2 && i0 < e2 + c2) {
        rows(H2, v);
#pragma unroll
        for (int r = 0; r < W_SEG; ++r) {
            const int ci = i0 + r - e2;
            if (ci >= 0 && ci < c2) {
                const float x = sqrtf(v[r]);
                A2[ci * c2] = x;
                cs[0] += x;
                cs[1] += (double)(x * x);
            }
        }
    }
    double* seg = a.seg + ((size_t)pt * (N / W_SEG) + sg) * 2 * N;
    seg[j] = q1;
    seg[N + j] = q2;
    cs[2] = q1;
    block_allsum<3, NT>(cs, red);
    if (j == 0)
#pragma unroll
        for (int k = 0; k < 3; ++k) a.part[(size_t)blockIdx.x * 3 + k] = cs[k];
}

// Moments of a point (a warp each).
template <int W>
__global__ void sw_reduce_kernel(SwArgs a)
{
    chain_begin();
    constexpr int N = 2 * W, NS = N / W_SEG;
    const int pt = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (pt >= a.win.n) return;
    double cs[3] = {0, 0, 0};
    if (lane < NS)
        for (int k = 0; k < 3; ++k) cs[k] = a.part[((size_t)pt * NS + lane) * 3 + k];
    for (int k = 0; k < 3; ++k) cs[k] = warp_allsum(cs[k]);
    if (lane == 0) {
        const int c2 = N - 4 * a.e;
        const double nchip = (double)(c2 * c2);
        SwMoments m;
        m.meanR = cs[0] / nchip;
        m.sigmaR = cs[1] / (nchip - 1.) - m.meanR * m.meanR;
        m.meanS = cs[2] / ((double)N * N);
        a.mom[pt] = m;
    }
}

// scaleW / sqrt(sigmaR sigmaS) of 16 lag rows a CTA.  A thread keeps the c2-row
// window sums of its columns of A1 and A1^2, started from the 16-row sums and
// moved down a row at a time; four rows of both go to shared memory, where a
// warp each turns them into prefix sums, and the L windows along the row are
// differences of two prefixes.
template <int W>
__global__ void __launch_bounds__(SwCfg<W>::NTS) sw_stats_kernel(SwArgs a)
{
    chain_begin();
    using C = SwCfg<W>;
    constexpr int N = C::N, NT = C::NTS, CPT = N / NT, CL = C::CL, PS = C::PS, NW = NT / 32;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* P = reinterpret_cast<double*>(smem_raw);  // 4 rows x 2 sums, PS each; column s at s + s / CL
    const int L = 4 * a.e + 1, c2 = N - 4 * a.e, tiles = (L + W_SEG - 1) / W_SEG;
    const int pt = blockIdx.x / tiles, tile = blockIdx.x % tiles;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float* A1 = a.A1 + (size_t)pt * N * N;
    const SwMoments mom = a.mom[pt];
    const double nchip = (double)(c2 * c2);
    const double inv0 = 1.0 / nchip, inv1 = 1.0 / (nchip - 1);
    const double wp = W - 2 * a.e;
    const double scaleW = 1.0 / ((OS * OS * OS * OS) * W * wp * W * wp);
    const int l0 = tile * W_SEG, lEnd = min(L, l0 + W_SEG);
    double v1[CPT], v2[CPT];
#pragma unroll
    for (int u = 0; u < CPT; ++u) {
        const int s = tid + u * NT;
        const double* seg = a.seg + ((size_t)pt * (N / W_SEG) + tile) * 2 * N;
        double t1 = 0, t2 = 0;
        for (int g = 0; g < c2 / W_SEG; ++g) {
            t1 += seg[(size_t)g * 2 * N + s];
            t2 += seg[(size_t)g * 2 * N + N + s];
        }
        for (int r = l0 + c2 / W_SEG * W_SEG; r < l0 + c2; ++r) {
            const float x = A1[(size_t)r * N + s];
            t1 += x;
            t2 += (double)(x * x);
        }
        v1[u] = t1;
        v2[u] = t2;
    }
    for (int lb = l0; lb < lEnd; lb += 4) {
        const int nr = min(4, lEnd - lb);
        float in[CPT][4], out[CPT][4];
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int u = 0; u < CPT; ++u) {
                const bool more = lb + r + 1 < lEnd;
                in[u][r] = more ? A1[(size_t)(lb + r + c2) * N + tid + u * NT] : 0.f;
                out[u][r] = more ? A1[(size_t)(lb + r) * N + tid + u * NT] : 0.f;
            }
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int u = 0; u < CPT; ++u) {
                const int s = tid + u * NT;
                P[(2 * r) * PS + s + s / CL] = v1[u];
                P[(2 * r + 1) * PS + s + s / CL] = v2[u];
                v1[u] += (double)in[u][r] - (double)out[u][r];
                v2[u] += (double)(in[u][r] * in[u][r]) - (double)(out[u][r] * out[u][r]);
            }
        __syncthreads();
        for (int row = warp; row < 2 * nr; row += NW) {  // inclusive prefix sums
            double* p = P + row * PS + lane * (CL + 1);
            double t = 0, x[CL];
#pragma unroll
            for (int c = 0; c < CL; ++c) {
                t += p[c];
                x[c] = t;
            }
            double sc = t;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const double y = __shfl_up_sync(0xffffffffu, sc, o);
                if (lane >= o) sc += y;
            }
            sc -= t;
#pragma unroll
            for (int c = 0; c < CL; ++c) p[c] = x[c] + sc;
        }
        __syncthreads();
        for (int r = 0; r < nr; ++r)
        for (int s1 = tid; s1 < L; s1 += NT) {
            const int hi = s1 + c2 - 1;
            const double* p = P + 2 * r * PS;
            double a1 = p[hi + hi / CL], a2 = p[PS + hi + hi / CL];
            if (s1 > 0) {
                a1 -= p[s1 - 1 + (s1 - 1) / CL];
                a2 -= p[PS + s1 - 1 + (s1 - 1) / CL];
            }
            const double ms = a1 * inv0;
            const double sg = a2 * inv1 - ms * ms;
            a.norm[((size_t)pt * L + lb + r) * L + s1] = scaleW * rsqrt(mom.sigmaR * sg);
        }
        __syncthreads();
    }
}

// Row transforms of (search - mean) + i (chip - mean, zeros around it).
// getPeakCorr forms c*scaleW - meanR*meanS with c the correlation of the raw
// amplitudes; both terms are ~mean^2 and their difference is the covariance.
// Correlating the chip minus its mean (on its support) with the search image
// minus any constant gives that difference directly, because
// sum(chip - meanR) = 0 over the support.
template <int W>
__global__ void __launch_bounds__(SwCfg<W>::NTN) sw_fwd_kernel(SwArgs a)
{
    chain_begin();
    using C = SwCfg<W>;
    constexpr int N = C::N, G = C::G, NT = C::NTN, TILES = N / G;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2* s = reinterpret_cast<float2*>(smem_raw);
    const int pt = blockIdx.x / TILES, r0 = blockIdx.x % TILES * G;
    const int e2 = 2 * a.e, c2 = N - 2 * e2;
    const float* A1 = a.A1 + (size_t)pt * N * N;
    const float* A2 = a.A2 + (size_t)pt * c2 * c2;
    const float mS = (float)a.mom[pt].meanS, mR = (float)a.mom[pt].meanR;
    float2* Z = a.Z + (size_t)pt * N * N;
    sbfft::line_fft<N, -1, G, NT, true, false, false>(
        s, a.twN,
        [&](int l, int k) {
            const int ci = r0 + l - e2, cj = k - e2;
            float2 v = make_float2(A1[(size_t)(r0 + l) * N + k] - mS, 0.f);
            if (ci >= 0 && ci < c2 && cj >= 0 && cj < c2) v.y = A2[(size_t)ci * c2 + cj] - mR;
            return v;
        },
        [&](int l, int k, float2 v) { Z[(size_t)(r0 + l) * N + k] = v; });
}

// Forward columns, cross spectrum, inverse columns of the lag rows.
template <int W>
__global__ void __launch_bounds__(ColCfg<2 * W>::NT) sw_corr_kernel(SwArgs a)
{
    chain_begin();
    constexpr int N = 2 * W;
    using C = ColCfg<N>;
    const int pt = blockIdx.x / C::TILES, tile = blockIdx.x % C::TILES;
    const int L = 4 * a.e + 1, e2 = 2 * a.e;
    corr_columns<N>(a.Z + (size_t)pt * N * N, a.T + (size_t)pt * L * corr_ts(N), tile, a.twN,
                    [e2](int m) { return m <= e2 ? m + e2 : m >= N - e2 ? m - (N - e2) : -1; });
}

// Inverse rows of pairs of lag rows, normalised correlation, the best
// position inside the user radius of each CTA's 16 rows.
template <int W>
__global__ void __launch_bounds__(SwCfg<W>::NTN) sw_ncc_kernel(SwArgs a)
{
    chain_begin();
    using C = SwCfg<W>;
    constexpr int N = C::N, G = C::G, NT = C::NTN, TS = corr_ts(N);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2* s = reinterpret_cast<float2*>(smem_raw);
    double* dsc = reinterpret_cast<double*>(s + C::RN::elems);
    int* isc = reinterpret_cast<int*>(dsc + NT / 32);
    const int L = 4 * a.e + 1, e2 = 2 * a.e, tiles = (L + 2 * G - 1) / (2 * G);
    const int pt = blockIdx.x / tiles, i0 = blockIdx.x % tiles * 2 * G;
    const float2* T = a.T + (size_t)pt * L * TS;
    const double* norm = a.norm + (size_t)pt * L * L;
    double* ncc = a.ncc + (size_t)pt * L * L;
    const int lim = e2 - OS * (W_NFAST / 4);
    float* c = reinterpret_cast<float*>(s);  // 2 G rows of covariances, over the spent line slots
    sbfft::line_fft<N, 1, G, NT, true, false, true>(
        s, a.twN,
        [&](int l, int k) {
            const int ra = min(i0 + 2 * l, L - 1), rb = min(i0 + 2 * l + 1, L - 1);
            return pair_row_input<N>(T + (size_t)ra * TS, T + (size_t)rb * TS, k);
        },
        [&](int l, int k, float2 v) {
            const int j = k <= e2 ? k + e2 : k >= N - e2 ? k - (N - e2) : -1;
            if (j < 0) return;
            c[2 * l * N + j] = v.x;
            c[(2 * l + 1) * N + j] = v.y;
        });
    __syncthreads();
    DArg best;
    best.v = -1e30;
    best.rank = 0x7fffffff;
    const int lane = threadIdx.x & 31;
    for (int h = threadIdx.x >> 5; h < 2 * G; h += NT / 32) {
        const int i = i0 + h;
        if (i >= L) break;
        const bool in = abs(i - e2) <= lim;
#pragma unroll 4
        for (int j = lane; j < L; j += 32) {
            const double x = (double)c[h * N + j] * __ldg(norm + i * L + j);
            ncc[i * L + j] = x;
            if (in && abs(j - e2) <= lim && darg_better(x, i * L + j, best.v, best.rank)) {
                best.v = x;
                best.rank = i * L + j;
            }
        }
    }
    best = block_argmax_d<NT>(best, dsc, isc);
    if (threadIdx.x == 0) {
        a.bestV[blockIdx.x] = best.v;
        a.bestE[blockIdx.x] = best.rank;
    }
}

// The peak of a point, oversampled; its outputs.
__global__ void __launch_bounds__(512) sw_peak_kernel(SwArgs a, int tiles)
{
    chain_begin();
    constexpr int NT = 512;
    __shared__ double Bm[W_OSW * W_N1], X[W_N1 * W_N1], T[W_N1 * W_OSW], dsc[NT / 32];
    __shared__ int isc[NT / 32];
    const int pt = blockIdx.x, tid = threadIdx.x, L = 4 * a.e + 1;
    DArg best;
    best.v = -1e30;
    best.rank = 0x7fffffff;
    for (int t = tid; t < tiles; t += NT) {
        const double v = a.bestV[(size_t)pt * tiles + t];
        const int r = a.bestE[(size_t)pt * tiles + t];
        if (darg_better(v, r, best.v, best.rank)) {
            best.v = v;
            best.rank = r;
        }
    }
    best = block_argmax_d<NT>(best, dsc, isc);
    const int gidx = a.list[pt];
    if (!(best.v >= 0.0) || best.rank == 0x7fffffff) {  // maxCorr < 0: no match (:511-512)
        if (tid == 0) {
            a.offR[gidx] = -2.0e9f;
            a.offA[gidx] = -2.0e9f;
            a.corr[gidx] = 0.0f;
            a.type[gidx] = SB_AMPMATCH;
            atomicAdd(&a.stats[1], 1ull);
        }
        return;
    }
    const int iMax = best.rank / L, jMax = best.rank % L;
    const double* ncc = a.ncc + (size_t)pt * L * L;
    for (int e = tid; e < W_OSW * W_N1; e += NT) Bm[e] = __ldg(a.B + e);
    for (int e = tid; e < W_N1 * W_N1; e += NT)
        X[e] = ncc[(size_t)(iMax - W_NFAST / 2 + e / W_N1) * L + (jMax - W_NFAST / 2 + e % W_N1)];
    __syncthreads();
    // T[t1][n2] = sum_t2 X[t1][t2] B[n2][t2]
    for (int e = tid; e < W_N1 * W_OSW; e += NT) {
        const int t1 = e / W_OSW, n2 = e % W_OSW;
        double acc = 0.0;
        for (int t2 = 0; t2 < W_N1; ++t2) acc += X[t1 * W_N1 + t2] * Bm[n2 * W_N1 + t2];
        T[e] = acc;
    }
    __syncthreads();
    DArg ob;
    ob.v = -1.0e30;
    ob.rank = 0x7fffffff;
    for (int e = tid; e < W_OSW * W_OSW; e += NT) {
        const int n1 = e / W_OSW, n2 = e % W_OSW;
        double acc = 0.0;
        for (int t1 = 0; t1 < W_N1; ++t1) acc += Bm[n1 * W_N1 + t1] * T[t1 * W_OSW + n2];
        const double v = acc * acc;
        if (darg_better(v, e, ob.v, ob.rank)) {
            ob.v = v;
            ob.rank = e;
        }
    }
    ob = block_argmax_d<NT>(ob, dsc, isc);
    if (tid == 0) {
        const int4 pl = a.win.win[pt];
        const int c0 = (W_N1 * W_NOVER) / 2 - W_NOVER * 2;  // 136
        const int iMax1 = ob.rank / W_OSW + c0, jMax1 = ob.rank % W_OSW + c0;
        const float cMax = (float)(sqrt(ob.v) / (W_N1 * W_N1));
        const int iMo = iMax * W_NOVER + iMax1 - (W_NOVER * W_NFAST) / 2;
        const int jMo = jMax * W_NOVER + jMax1 - (W_NOVER * W_NFAST) / 2;
        const float rShift1 = ((float)jMo - a.e * OS * W_NOVER) / (W_NOVER * OS);
        const float aShift1 = ((float)iMo - a.e * OS * W_NOVER) / (W_NOVER * OS);
        const float rShift = (float)(pl.z - pl.x), aShift = (float)(pl.w - pl.y);
        if (cMax > 0.0f) {
            a.offR[gidx] = rShift - rShift1;
            a.offA[gidx] = aShift - aShift1;
            atomicAdd(&a.stats[0], 1ull);
        } else {
            a.offR[gidx] = -2.0e9f;
            a.offA[gidx] = -2.0e9f;
            atomicAdd(&a.stats[1], 1ull);
        }
        a.corr[gidx] = cMax;
        a.type[gidx] = SB_AMPMATCH;
    }
}

__global__ void strackw_init_kernel(float* offR, float* offA, float* corr, uint8_t* type, int n)
{
    chain_begin();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    offR[k] = -2.0e9f;
    offA[k] = -2.0e9f;
    corr[k] = 0.0f;
    type[k] = SB_BAD;
}

// Planes in flight at a margin of e samples: two points' per SM of the working
// set of one (window pair, upsampled pair, correlation), the figure serve.py
// admits jobs by.  Large launches matter more than L2 (126 MB): the kernels are
// short of instruction issue and shared-memory bandwidth, not of DRAM (10 to
// 45 % of its rate).  With plain launches the 2000 x 4000 pair at W = 224 takes
// 27.7 ms with these 2 GB, 28.5 with half, 27.0 with four times that; the 1024 x
// 2048 pair at W = 64 1.58 ms with 220 MB (840 points), 1.76 with half, 1.38
// with four times that, where jobs that a server's budget admits would no
// longer fit.
static size_t sw_chunk_bytes(int numSM, int W, int e)
{
    const size_t N = 2 * W, L = 4 * e + 1;
    return (size_t)2 * numSM * sizeof(float2) * (3 * W * W + 3 * N * N + 2 * N * L + 3 * L * L);
}

// Workspace of a chunk, carved from one buffer; base null: returns its size.
struct SwSpace {
    char* base;
    size_t used = 0;
    template <typename T>
    T* take(size_t n)
    {
        T* p = base ? reinterpret_cast<T*>(base + used) : nullptr;
        used += (n * sizeof(T) + 255) / 256 * 256;
        return p;
    }
};

template <int W>
struct SwRun {
    using C = SwCfg<W>;
    static constexpr int N = 2 * W;

    static size_t layout(SwArgs& a, int n, char* base, double** dop, int** az)
    {
        const size_t L = 4 * a.e + 1, c2 = N - 4 * a.e, NN = (size_t)N * N;
        SwSpace s{base};
        // what a step is done with makes room for a later one: xv, then A1, then
        // T; H, then Z, then ncc (L <= N)
        const size_t xt = (size_t)L * corr_ts(N) > 2 * W * W ? (size_t)L * corr_ts(N) : 2 * W * W;
        a.xv = s.take<float2>(n * xt);
        a.A1 = reinterpret_cast<float*>(a.xv);
        a.T = a.xv;
        a.H = s.take<float>((size_t)n * 2 * NN);
        a.Z = reinterpret_cast<float2*>(a.H);
        a.ncc = reinterpret_cast<double*>(a.H);
        a.A2 = s.take<float>((size_t)n * c2 * c2);
        a.seg = s.take<double>((size_t)n * (N / W_SEG) * 2 * N);
        a.part = s.take<double>((size_t)n * (N / W_SEG) * 3);
        a.mom = s.take<SwMoments>(n);
        a.norm = s.take<double>((size_t)n * L * L);
        a.bestV = s.take<double>((size_t)n * (L + 15) / 16 + n);
        a.bestE = s.take<int>((size_t)n * (L + 15) / 16 + n);
        *dop = s.take<double>(dop_scratch_doubles<W>(n));
        *az = s.take<int>(n);
        return s.used;
    }

    // Copies of the end values beside an intensity row: the box half width,
    // as far as shared memory goes (a wider box clamps its reads).
    static int row_pad(const SwArgs& a) { return a.taps < 0 ? 0 : a.navgR < 0 ? 0 : a.navgR < 32 ? a.navgR : 32; }

    template <bool F32>
    static cudaError_t attributes()
    {
        struct { const void* f; size_t sm; } k[] = {
            {(const void*)sw_cols_kernel<W, F32>, C::smCols},
            {(const void*)sw_rows_kernel<W, F32>, C::smRows + sizeof(float) * C::G * (N + 64)},
            {(const void*)sw_stats_kernel<W>, C::smStats}, {(const void*)sw_fwd_kernel<W>, C::smFwd},
            {(const void*)sw_corr_kernel<W>, ColCfg<N>::smem}, {(const void*)sw_ncc_kernel<W>, C::smNcc}};
        for (auto& x : k) {
            const cudaError_t e = cudaFuncSetAttribute(x.f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)x.sm);
            if (e != cudaSuccess) return e;
        }
        return cudaSuccess;
    }

    // One chunk of a.win.n points.
    template <bool F32>
    static cudaError_t chunk(const SwArgs& a, double* dop, int* az, cudaStream_t st, int64_t* launches)
    {
        const int n = a.win.n, e2 = 2 * a.e, c2 = N - 2 * e2, L = 2 * e2 + 1;
        // rows of image 2 whose range sums the chip's azimuth sums read
        const int g = a.taps >= 0 && a.navgA > 0 ? a.navgA : 0;
        const int hr0 = e2 - g < 0 ? 0 : (e2 - g) & ~1, hr1 = e2 + c2 - 1 + g < N - 1 ? e2 + c2 - 1 + g : N - 1;
        const int tiles2 = (hr1 - hr0 + C::G) / C::G, tilesL = (L + 15) / 16, pad = row_pad(a);
        cudaError_t e = launch_dop<W>(a.win, W, dop, az, st);
        if (e != cudaSuccess) return e;
        chain(sw_cols_kernel<W, F32>, n * 2 * (W / C::G), C::NTW, C::smCols, st, a);
        chain(sw_rows_kernel<W, F32>, n * (N / C::G + tiles2), C::NTW,
              C::smRows + sizeof(float) * C::G * (N + 2 * pad), st, a, hr0, hr1, pad);
        const int ga = n * (N / W_SEG);
        switch (a.taps) {
        case -1: chain(sw_amps_kernel<W, -1>, ga, N, 0, st, a); break;
        case 2: chain(sw_amps_kernel<W, 2>, ga, N, 0, st, a); break;
        case 3: chain(sw_amps_kernel<W, 3>, ga, N, 0, st, a); break;
        default: chain(sw_amps_kernel<W, 0>, ga, N, 0, st, a); break;
        }
        chain(sw_reduce_kernel<W>, (n + 3) / 4, 128, 0, st, a);
        chain(sw_stats_kernel<W>, n * tilesL, C::NTS, C::smStats, st, a);
        chain(sw_fwd_kernel<W>, n * (N / C::G), C::NTN, C::smFwd, st, a);
        chain(sw_corr_kernel<W>, n * ColCfg<N>::TILES, ColCfg<N>::NT, ColCfg<N>::smem, st, a);
        chain(sw_ncc_kernel<W>, n * tilesL, C::NTN, C::smNcc, st, a);
        chain(sw_peak_kernel, n, 512, 0, st, a, tilesL);
        *launches += 12;
        return cudaGetLastError();
    }
};

static bool sw_supported(int W)
{
    return W == 32 || W == 48 || W == 64 || W == 96 || W == 128 || W == 192 || W == 224 || W == 256;
}

// Matches nl planned points (win, list: device) in chunks.
template <int W>
static int run_sw(sb_context* c, SwArgs a, int nl)
{
    const bool f32 = a.win.sampleType == SB_CFLOAT32;
    cudaError_t e = f32 ? SwRun<W>::template attributes<true>() : SwRun<W>::template attributes<false>();
    if (e != cudaSuccess) return sb_ctx_cuda(c, e, "strackw attributes");
    a.twW = batch_tw_table<W>(c);
    a.twN = batch_tw_table<2 * W>(c);
    a.tau = tau_table(c, W);
    if (!a.twW || !a.twN || !a.tau) return sb_ctx_fail(c, SB_ERR_NOMEM, "table allocation failed");
    double* dop;
    int* az;
    SwArgs probe = a;
    const size_t one = SwRun<W>::layout(probe, 16, nullptr, &dop, &az) / 16 + 1;
    int B = (int)(sw_chunk_bytes(c->numSM, W, a.e) / one);
    B = B < 16 ? 16 : B;
    char* base = sb_chunk_buf(c, "w_scratch", nl, &B,
                              [&](int b) { return SwRun<W>::layout(a, b, nullptr, &dop, &az); });
    if (!base) return sb_ctx_fail(c, SB_ERR_NOMEM, "strackw workspace allocation failed");
    SwRun<W>::layout(a, B, base, &dop, &az);
    a.az = az;
    const int4* win = a.win.win;
    const int* list = a.list;
    for (int off = 0; off < nl; off += B) {
        a.win.win = win + off;
        a.list = list + off;
        a.win.n = nl - off < B ? nl - off : B;
        e = f32 ? SwRun<W>::template chunk<true>(a, dop, az, c->stream, &c->launches)
                : SwRun<W>::template chunk<false>(a, dop, az, c->stream, &c->launches);
        if (e != cudaSuccess) return sb_ctx_cuda(c, e, "strackw");
    }
    return SB_OK;
}

static int run_sw_any(int W, sb_context* c, const SwArgs& a, int nl)
{
    switch (W) {
    case 32: return run_sw<32>(c, a, nl);
    case 48: return run_sw<48>(c, a, nl);
    case 64: return run_sw<64>(c, a, nl);
    case 96: return run_sw<96>(c, a, nl);
    case 128: return run_sw<128>(c, a, nl);
    case 192: return run_sw<192>(c, a, nl);
    case 224: return run_sw<224>(c, a, nl);
    default: return run_sw<256>(c, a, nl);
    }
}

}  // namespace sbk

using namespace sbk;

namespace {

// bilinear interpolation with sentinels, the stand-in for mosaicSource's
// bilinearInterp (absent from the reference tree) shared with the oracle.
float bilinearW(const float* img, double x, double y, int nx, int ny, float minvalue, float noData)
{
    if (x < 0 || y < 0 || x > (double)(nx - 1) || y > (double)(ny - 1)) return noData;
    if (nx < 2 || ny < 2) return noData;
    int j = (int)x, i = (int)y;
    if (j >= nx - 1) j = nx - 2;
    if (i >= ny - 1) i = ny - 2;
    const double t = x - j, u = y - i;
    const float p1 = img[(size_t)i * nx + j], p2 = img[(size_t)i * nx + j + 1];
    const float p3 = img[(size_t)(i + 1) * nx + j + 1], p4 = img[(size_t)(i + 1) * nx + j];
    if (p1 <= minvalue || p2 <= minvalue || p3 <= minvalue || p4 <= minvalue) return noData;
    return (float)((1.0 - t) * (1.0 - u) * p1 + t * (1.0 - u) * p2 + t * u * p3 + (1.0 - t) * u * p4);
}

// findImage2Pos (corrTrackFast.c:257-292)
void findImage2PosW(const sb_track_params* p, int r1, int a1, int* r2, int* a2)
{
    double aShift, rShift;
    const double sc = (double)p->scaleFactor;
    if (p->polyShift) {
        rShift = p->rShiftPoly[0] + (double)(r1 * sc) * p->rShiftPoly[1] + (double)(a1 * sc) * p->rShiftPoly[2];
        aShift = p->aShiftPoly[0] + (double)(r1 * sc) * p->aShiftPoly[1] + (double)(a1 * sc) * p->aShiftPoly[2];
    } else {
        const sb_offset_grid* o = p->initOffsets;
        const float minvalue = (float)((float)-SB_LARGEINT * 0.9);
        const double range = (r1 - o->r0) / o->deltaR, azimuth = (a1 - o->a0) / o->deltaA;
        rShift = bilinearW(o->dr, range, azimuth, o->nr, o->na, minvalue, (float)-SB_LARGEINT);
        aShift = bilinearW(o->da, range, azimuth, o->nr, o->na, minvalue, (float)-SB_LARGEINT);
        if (rShift <= minvalue || aShift <= minvalue) {
            rShift = minvalue;
            aShift = minvalue;
        }
        if (rShift < (-SB_LARGEINT + 1)) {
            rShift = p->rShiftPoly[0] + (double)(r1 * sc) * p->rShiftPoly[1] + (double)(a1 * sc) * p->rShiftPoly[2];
            aShift = p->aShiftPoly[0] + (double)(r1 * sc) * p->aShiftPoly[1] + (double)(a1 * sc) * p->aShiftPoly[2];
        }
    }
    rShift /= sc;
    aShift /= sc;
    *r2 = (rShift >= 0) ? r1 + (int)(rShift + 0.5) : r1 + (int)(rShift - 0.5);
    *a2 = (aShift >= 0) ? a1 + (int)(aShift + 0.5) : a1 + (int)(aShift - 0.5);
}

// maskValue (corrTrackFast.c:1135-1154)
int maskValueW(const sb_track_params* p, int r1, int a1)
{
    const sb_mask* m = p->mask;
    if (!m) return 1;
    const int dr = (p->wRa / 2 - m->r0) * p->scaleFactor;
    const int da = (p->wAa / 2 - m->a0) * p->scaleFactor;
    const int ia1 = (a1 + da) / m->nal, ir1 = (r1 + dr) / m->nrl;
    if (ia1 < 0 || ia1 >= m->na || ir1 < 0 || ir1 >= m->nr) return 0;
    return (int)(signed char)m->mask[(size_t)ia1 * m->nr + ir1];
}

#define CKW(call, what)                                              \
    do {                                                             \
        cudaError_t _e = (call);                                     \
        if (_e != cudaSuccess) return sb_ctx_cuda(c, _e, what);      \
    } while (0)

}  // namespace

extern "C" int sb_strackw(sb_context* c, const sb_track_params* p, const sb_image* img1, const sb_image* img2,
                          sb_track_result* out)
{
    if (!c) return SB_ERR_ARG;
    c->err.clear();
    c->launches = 0;
    if (!p || !out || !img1 || !img2 || !img1->data || !img2->data)
        return sb_ctx_fail(c, SB_ERR_ARG, "null params, image or result");
    if (img1->sampleType != img2->sampleType || img1->byteOrder != img2->byteOrder)
        return sb_ctx_fail(c, SB_ERR_ARG, "images differ in sample type or byte order");
    if (p->nR <= 0 || p->nA <= 0) return sb_ctx_fail(c, SB_ERR_ARG, "empty grid");
    if (p->scaleFactor <= 0) return sb_ctx_fail(c, SB_ERR_ARG, "scaleFactor must be positive");
    if (p->polyShift == 0 && !p->initOffsets) return sb_ctx_fail(c, SB_ERR_ARG, "polyShift=0 needs initOffsets");
    if (!out->offR || !out->offA || !out->corr || !out->type) return sb_ctx_fail(c, SB_ERR_ARG, "null output grid");
    const int W = p->wRa;
    if (p->wRa != p->wAa) return sb_ctx_fail(c, SB_ERR_UNSUPPORTED, "search window must be square (wra == waa)");
    if (!sw_supported(W)) return sb_ctx_fail(c, SB_ERR_UNSUPPORTED, "search window %d not supported", W);
    const int eR = p->edgePadR + W_NFAST / 4, eA = p->edgePadA + W_NFAST / 4;
    if (eR != eA) return sb_ctx_fail(c, SB_ERR_UNSUPPORTED, "edgeR != edgeA not supported");
    if ((W - 2 * eR) <= 0 || p->edgePadR < W_NFAST / 4)
        return sb_ctx_fail(c, SB_ERR_ARG, "edge pad leaves no chip (wra=%d, edgepad=%d)", W, p->edgePadR);
    CKW(cudaSetDevice(c->device), "cudaSetDevice");
    cudaEventRecord(c->ev[0], c->stream);
    // ---- plan (host, raster order; corrTrackFast.c:144-172)
    const int n = p->nR * p->nA;
    std::vector<int4> plan;
    std::vector<int> list;
    std::vector<int> masked0;  // maskVal != 1: outputs stay -2e9 / 0 / type 0
    for (int i = 0; i < p->nA; i++) {
        const int a1 = p->aStart + i * p->deltaA - p->wAa / 2;
        for (int j = 0; j < p->nR; j++) {
            const int r1 = p->rStart + j * p->deltaR - p->wRa / 2;
            int r2, a2;
            findImage2PosW(p, r1, a1, &r2, &a2);
            const int mv = maskValueW(p, r1 * p->scaleFactor, a1 * p->scaleFactor);
            if (mv == 1 && r1 > 0 && r1 < img1->nr && a1 > 0 && a1 < img1->na && r2 > 0 && r2 < img2->nr && a2 > 0 &&
                a2 < img2->na) {
                plan.push_back(make_int4(r1, a1, r2, a2));
                list.push_back(i * p->nR + j);
            }
        }
    }
    const void *d1, *d2;
    int rc;
    if ((rc = sb_image_to_device(c, img1, "img1", &d1)) != SB_OK) return rc;
    if ((rc = sb_image_to_device(c, img2, "img2", &d2)) != SB_OK) return rc;
    cudaError_t e;
    const int nl = (int)list.size();
    int4* dplan = (int4*)sb_ctx_buf(c, "w_plan", sizeof(int4) * (nl + 1), &e);
    int* dlist = (int*)sb_ctx_buf(c, "w_list", sizeof(int) * (nl + 1), &e);
    Packed lay;
    const size_t atR = lay.add(sizeof(float) * n), atA = lay.add(sizeof(float) * n), atC = lay.add(sizeof(float) * n);
    const size_t atT = lay.add(n), atS = lay.add(4 * sizeof(unsigned long long));
    char* dout = (char*)sb_ctx_buf(c, "out", lay.bytes(), &e);
    if (!dout) return sb_ctx_fail(c, SB_ERR_NOMEM, "device allocation failed");
    float* dR = (float*)(dout + atR);
    float* dA = (float*)(dout + atA);
    float* dC = (float*)(dout + atC);
    uint8_t* dT = (uint8_t*)(dout + atT);
    unsigned long long* dst = (unsigned long long*)(dout + atS);
    // the real oversampling kernel of the 21 -> 336 symmetric zero pad
    const double* dB = (const double*)sb_table(c, "w_B", [] {
        std::vector<double> B(W_OSW * W_N1);
        for (int nn = 0; nn < W_OSW; ++nn)
            for (int t = 0; t < W_N1; ++t) {
                const int d = (nn + (W_N1 * W_NOVER) / 2 - W_NOVER * 2) - W_NOVER * t;
                double v = 1.0;
                for (int f = 1; f <= W_NFAST / 2; ++f)
                    v += 2.0 * cos(2.0 * 3.14159265358979323846 * f * d / (W_N1 * W_NOVER));
                B[nn * W_N1 + t] = v;
            }
        return B;
    });
    if (!dplan || !dlist || !dB)
        return sb_ctx_fail(c, SB_ERR_NOMEM, "device allocation failed");
    if (nl) {
        CKW(cudaMemcpyAsync(dplan, plan.data(), sizeof(int4) * nl, cudaMemcpyHostToDevice, c->stream), "plan");
        CKW(cudaMemcpyAsync(dlist, list.data(), sizeof(int) * nl, cudaMemcpyHostToDevice, c->stream), "list");
    }
    CKW(cudaMemsetAsync(dst, 0, 4 * sizeof(unsigned long long), c->stream), "memset");
    cudaEventRecord(c->ev[1], c->stream);
    strackw_init_kernel<<<(n + 255) / 256, 256, 0, c->stream>>>(dR, dA, dC, dT, n);
    CKW(cudaGetLastError(), "strackw_init");
    c->launches++;
    if (nl) {
        SwArgs a = {};
        a.win.img1 = d1;
        a.win.img2 = d2;
        a.win.nr1 = img1->nr; a.win.na1 = img1->na; a.win.nr2 = img2->nr; a.win.na2 = img2->na;
        a.win.sampleType = img1->sampleType;
        a.win.byteOrder = img1->byteOrder;
        a.win.win = dplan;
        a.list = dlist;
        a.e = eR;
        a.navgR = p->navgR;
        a.navgA = p->navgA;
        a.taps = p->navgA <= 1 && p->navgR <= 1 ? -1
                 : p->navgA == p->navgR && (p->navgR == 2 || p->navgR == 3) ? p->navgR : 0;
        a.scale = 1.f / ((float)W * (float)W * (float)W * (float)W * (float)(OS * OS * OS * OS) *
                         (float)(OS * OS * (p->navgA + 1) * (p->navgR + 1)));
        a.B = dB;
        a.offR = dR; a.offA = dA; a.corr = dC; a.type = dT;
        a.stats = dst;
        cudaEventRecord(c->sev[0], c->stream);
        if ((rc = run_sw_any(W, c, a, nl)) != SB_OK) return rc;
        cudaEventRecord(c->sev[1], c->stream);
    }
    cudaEventRecord(c->ev[2], c->stream);
    const bool od = out->onDevice != 0;
    OutCopies oc(c);
    if ((rc = oc.add(out->offR, dR, sizeof(float) * n, od)) != SB_OK) return rc;
    if ((rc = oc.add(out->offA, dA, sizeof(float) * n, od)) != SB_OK) return rc;
    if ((rc = oc.add(out->corr, dC, sizeof(float) * n, od)) != SB_OK) return rc;
    if ((rc = oc.add(out->type, dT, n, od)) != SB_OK) return rc;
    unsigned long long st[4];
    if ((rc = oc.add(st, dst, sizeof(st))) != SB_OK) return rc;
    if ((rc = oc.finish("strackw")) != SB_OK) return rc;
    out->nComplex = 0;
    out->nAmp = (int64_t)st[0];
    out->nAmpL = 0;
    out->nFail = (int64_t)st[1];
    out->nAttempted = nl;
    cudaEventElapsedTime(&c->timing[0], c->ev[0], c->ev[3]);
    cudaEventElapsedTime(&c->timing[1], c->ev[0], c->ev[1]);
    cudaEventElapsedTime(&c->timing[2], c->ev[1], c->ev[2]);
    cudaEventElapsedTime(&c->timing[3], c->ev[2], c->ev[3]);
    for (int q = 0; q < 8; ++q) c->stage[q] = 0.f;
    if (nl) cudaEventElapsedTime(&c->stage[0], c->sev[0], c->sev[1]);
    c->stage[5] = (float)nl;
    return SB_OK;
}
