// strack_amp.cu -- amplitude tries of strack with windows from 48 up (small
// window s = 1, large window s = LA = 2); strack_amps.cu keeps the smaller ones
// in one CTA's shared memory.
//
// Follows getAmpPatches (Strack/speckleTrack.c:1006-1189), ampMatch
// (:398-484) and ampTrackFast (:489-597).  List entries go through the kernels
// below in chunks, each spreading the lines of every entry of the chunk over
// the chip.  With Ws = wa*s and N = 2*Ws:
//  1. am_prep, dop: window corners, Doppler roll (estDopCarrier1 on the windows
//     when -noComplex and s = 1);
//  2. am_rows, am_cols, am_detect: detected images
//     |IDFT_N(zeroPadFFT(F, azShift))|^2 * scale of both windows: forward rows;
//     forward columns, roll and the two azimuth parities of the padded inverse
//     (plain and half-sample phase) in one kernel; the two range parities,
//     the zero-count / empty-patch sums and the square roots in the third;
//  3. am_moments: sums of a point's tiles, the tests, the means;
//  4. am_fwd: mean removal, powers p1, p2, forward rows of z = a1 + i a2;
//  5. am_corr: forward columns, the cross spectrum from the packed pair
//     (Hermitian, half the columns), inverse columns;
//  6. am_mag: inverse rows, two real rows at a time, |c| at its fftshifted
//     position and the best (value, scan rank) of each 16 rows;
//  7. am_peak: findCPeak's maximum, Gaussian-width samples, 8x8 -> 96x96
//     oversampling of the peak, normalisation by N^4 * 64 * sqrt(p1 p2).
#include <cuda_runtime.h>

#include "capi_internal.h"
#include "strack_device.cuh"
#include "strack_kernels.h"
#include "window_batch.cuh"

namespace sbk {

// What am_moments makes of a point's partial sums.
struct AmMoments {
    double avg1, avg2;
    int hd;  // 1: the patch holds data
};

struct AmChunk {
    AmpArgs a;        // the try
    WinArgs win;      // the chunk's windows
    const int* list;  // the chunk's list entries
    FitJob* fit;
    float scale, thr;
    const float2* twW;  // step-order tables of Ws and N points
    const float2* twN;
    int4* corner;     // window corners
    int* az;          // azShift in effect
    // planes, one per list entry of the chunk
    float2* F;        // 2 x Ws x Ws row spectra
    float2* R;        // 2 x N x Ws, azimuth doubled
    float2* z;        // N x N (a1, a2), then row spectra
    float2* T;        // N x corr_ts(N)
    float* mag;       // N x N |c|
    double* part;     // N/4 x 5 sums of am_detect
    double* pw;       // N/8 x 2 powers of am_fwd
    AmMoments* mom;
    unsigned long long* best;  // N/16
};

template <int WS>
struct AmCfg {
    static constexpr int N = 2 * WS;
    static constexpr int G = 8, NT = 128;  // lines and threads of every line kernel
    using RW = sbfft::LineTile<WS, G, true>;
    using CW = sbfft::LineTile<WS, G, false>;
    using RN = sbfft::LineTile<N, G, true>;
    static constexpr size_t smRows = sizeof(float2) * RW::elems;
    static constexpr size_t smCols = sizeof(float2) * (CW::elems + G * WS);
    static constexpr size_t smDetect = smRows + sizeof(float) * G * N + sizeof(double) * (NT / 32 + 1) * 5;
    static constexpr size_t smFwd = sizeof(float2) * RN::elems;
};

__global__ void am_prep_kernel(AmChunk c)
{
    chain_begin();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= c.win.n) return;
    const AmpArgs& a = c.a;
    const int p = c.list[k];
    const PointPlan pl = a.plan[p];
    // window corners (computeAmpImageLocations, speckleTrack.c:147-156):
    // a1a = aStart + i deltaA - (wA/2) s = a1 + wA/2 - (wA/2) s, from the plan
    const int a1a = pl.a1 + a.wA / 2 - a.wA / 2 * a.s;
    const int r1a = pl.r1 + a.wR / 2 - a.wR / 2 * a.s;
    c.corner[k] = make_int4(r1a, a1a, r1a + (pl.r2 - pl.r1), a1a + (pl.a2 - pl.a1));
    const int az = a.azEff ? a.azEff[p] : a.rec[p].azset;
    c.az[k] = az < 0 ? 0 : az;
}

// Forward rows of both windows.
template <int WS, bool F32>
__global__ void __launch_bounds__(128) am_rows_kernel(AmChunk c)
{
    chain_begin();
    using C = AmCfg<WS>;
    constexpr int G = C::G, NT = C::NT, TILES = WS / G;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2* s = reinterpret_cast<float2*>(smem_raw);
    const int tile = blockIdx.x % TILES, q = blockIdx.x / TILES % 2, pt = blockIdx.x / (2 * TILES);
    const Window<F32> win(c.win, q, c.corner[pt], WS);
    float2* F = c.F + (((size_t)pt * 2 + q) * WS + tile * G) * WS;
    sbfft::line_fft<WS, -1, G, NT, true, false, false>(
        s, c.twW, [&](int l, int k) { return win(tile * G + l, k); },
        [&](int l, int k, float2 v) { F[l * WS + k] = v; });
}

// Forward columns, Doppler roll, both azimuth parities of the padded inverse.
template <int WS>
__global__ void __launch_bounds__(128) am_cols_kernel(AmChunk c)
{
    chain_begin();
    using C = AmCfg<WS>;
    constexpr int G = C::G, NT = C::NT, TILES = WS / G;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2* s = reinterpret_cast<float2*>(smem_raw);
    float2* spec = s + C::CW::elems;
    const int tile = blockIdx.x % TILES, pq = blockIdx.x / TILES, pt = pq / 2;
    const int az = (int)((float)c.az[pt] * (float)WS / (float)c.a.wA);
    const float2* F = c.F + (size_t)pq * WS * WS + tile * G;
    float2* R = c.R + (size_t)pq * C::N * WS + tile * G;
    const float2* tau = c.a.tau;
    sbfft::line_fft<WS, -1, G, NT, false, false, false>(
        s, c.twW, [&](int l, int k) { return F[k * WS + l]; },
        [&](int l, int k, float2 v) { spec[(k - az < 0 ? k - az + WS : k - az) * G + l] = v; });
    __syncthreads();
    sbfft::line_fft<WS, 1, G, NT, false, false, false>(
        s, c.twW, [&](int l, int k) { return spec[k * G + l]; },
        [&](int l, int k, float2 v) { R[2 * k * WS + l] = v; });
    __syncthreads();
    sbfft::line_fft<WS, 1, G, NT, false, false, false>(
        s, c.twW, [&](int l, int k) { return sbfft::cmul(spec[k * G + l], __ldg(tau + k)); },
        [&](int l, int k, float2 v) { R[(2 * k + 1) * WS + l] = v; });
}

// Both range parities of four rows of both images (lines 0 .. 3: image 1),
// intensities, the sums getAmpPatches tests, amplitudes.
template <int WS>
__global__ void __launch_bounds__(128) am_detect_kernel(AmChunk c)
{
    chain_begin();
    using C = AmCfg<WS>;
    constexpr int N = C::N, G = C::G, H = G / 2, NT = C::NT, TILES = N / H;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2* s = reinterpret_cast<float2*>(smem_raw);
    float* in = reinterpret_cast<float*>(s + C::RW::elems);  // G x N intensities
    double* red = reinterpret_cast<double*>(in + G * N);
    const int tile = blockIdx.x % TILES, pt = blockIdx.x / TILES;
    const float2* R = c.R + (size_t)pt * 2 * N * WS + tile * H * WS;
    const float2* tau = c.a.tau;
    auto src = [&](int l, int k) { return R[(l < H ? l : l - H + N) * WS + k]; };
    sbfft::line_fft<WS, 1, G, NT, true, false, false>(
        s, c.twW, src,
        [&](int l, int k, float2 v) { in[l * N + 2 * k] = (v.x * v.x + v.y * v.y) * c.scale; });
    __syncthreads();
    sbfft::line_fft<WS, 1, G, NT, true, false, false>(
        s, c.twW, [&](int l, int k) { return sbfft::cmul(src(l, k), __ldg(tau + k)); },
        [&](int l, int k, float2 v) { in[l * N + 2 * k + 1] = (v.x * v.x + v.y * v.y) * c.scale; });
    __syncthreads();
    float2* z = c.z + (size_t)pt * N * N + tile * H * N;
    double m[5] = {0, 0, 0, 0, 0};  // samples under the threshold, intensities, amplitudes
    for (int e = threadIdx.x; e < H * N; e += NT) {
        const float i1 = in[e], i2 = in[H * N + e];
        const float a1 = sqrtf(i1), a2 = sqrtf(i2);
        z[e] = make_float2(a1, a2);
        m[0] += (i1 < c.thr || i2 < c.thr) ? 1.0 : 0.0;
        m[1] += i1;
        m[2] += i2;
        m[3] += a1;
        m[4] += a2;
    }
    block_allsum<5, NT>(m, red);
    if (threadIdx.x == 0)
#pragma unroll
        for (int k = 0; k < 5; ++k) c.part[(size_t)blockIdx.x * 5 + k] = m[k];
}

// A warp per point.
template <int WS>
__global__ void am_moments_kernel(AmChunk c)
{
    chain_begin();
    constexpr int N = 2 * WS, TILES = N / 4;
    const int pt = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (pt >= c.win.n) return;
    double m[5] = {0, 0, 0, 0, 0};
    for (int t = lane; t < TILES; t += 32)
#pragma unroll
        for (int k = 0; k < 5; ++k) m[k] += c.part[((size_t)pt * TILES + t) * 5 + k];
#pragma unroll
    for (int k = 0; k < 5; ++k) m[k] = warp_allsum(m[k]);
    if (lane == 0) {
        AmMoments r;
        r.avg1 = m[3] / ((double)N * N);
        r.avg2 = m[4] / ((double)N * N);
        r.hd = !(m[0] > 20.0) && !(m[1] < 1.0e-6 || m[2] < 1.0e-6);
        c.mom[pt] = r;
    }
}

// Mean removal, powers, forward rows (in place).
template <int WS>
__global__ void __launch_bounds__(128) am_fwd_kernel(AmChunk c)
{
    chain_begin();
    using C = AmCfg<WS>;
    constexpr int N = C::N, G = C::G, NT = C::NT, TILES = N / G;
    __shared__ double red[(NT / 32 + 1) * 2];
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2* s = reinterpret_cast<float2*>(smem_raw);
    const int tile = blockIdx.x % TILES, pt = blockIdx.x / TILES;
    const AmMoments mom = c.mom[pt];
    if (!mom.hd) return;  // uniform
    float2* z = c.z + (size_t)pt * N * N + tile * G * N;
    double pw[2] = {0, 0};
    sbfft::line_fft<N, -1, G, NT, true, false, false>(
        s, c.twN,
        [&](int l, int k) {
            float2 v = z[l * N + k];
            if (v.x > 1.0e-20f) v.x = (float)((double)v.x - mom.avg1);
            v.y = (float)((double)v.y - mom.avg2);
            return v;
        },
        [&](int l, int k, float2 v) { z[l * N + k] = v; },
        [&](int, int, float2 v) {
            pw[0] += (double)(v.x * v.x);
            pw[1] += (double)(v.y * v.y);
        });
    block_allsum<2, NT>(pw, red);
    if (threadIdx.x == 0) {
        c.pw[(size_t)blockIdx.x * 2] = pw[0];
        c.pw[(size_t)blockIdx.x * 2 + 1] = pw[1];
    }
}

template <int WS>
__global__ void __launch_bounds__(ColCfg<2 * WS>::NT) am_corr_kernel(AmChunk c)
{
    chain_begin();
    constexpr int N = 2 * WS;
    using C = ColCfg<N>;
    const int pt = blockIdx.x / C::TILES, tile = blockIdx.x % C::TILES;
    if (!c.mom[pt].hd) return;  // uniform
    corr_columns<N>(c.z + (size_t)pt * N * N, c.T + (size_t)pt * N * corr_ts(N), tile, c.twN,
                    [](int m) { return m; });
}

// The correlation surface is real: |c| = |re|.
template <int WS>
__global__ void __launch_bounds__(128) am_mag_kernel(AmChunk c)
{
    chain_begin();
    using C = AmCfg<WS>;
    constexpr int N = C::N, G = C::G, NT = C::NT, TS = corr_ts(N), TILES = N / (2 * G);
    __shared__ unsigned long long sc[NT / 32];
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2* s = reinterpret_cast<float2*>(smem_raw);
    const int tile = blockIdx.x % TILES, pt = blockIdx.x / TILES;
    if (!c.mom[pt].hd) return;  // uniform
    const float2* T = c.T + ((size_t)pt * N + tile * 2 * G) * TS;
    float* mag = c.mag + (size_t)pt * N * N;
    unsigned long long best = 0ull;
    sbfft::line_fft<N, 1, G, NT, true, false, false>(
        s, c.twN,
        [&](int l, int k) { return pair_row_input<N>(T + 2 * l * TS, T + (2 * l + 1) * TS, k); },
        [&](int l, int k, float2 v) {
            const int x = k < WS ? k + WS : k - WS;  // fftshift
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int cy = tile * 2 * G + 2 * l + h, y = cy < WS ? cy + WS : cy - WS;
                const float m = fabsf(h ? v.y : v.x);
                mag[y * N + x] = m;
                const unsigned long long key = am_key(m, (unsigned)cpeak_rank(y, x, WS));
                best = key > best ? key : best;
            }
        });
    best = block_max_u64(best, sc);
    if (threadIdx.x == 0) c.best[blockIdx.x] = best;
}

template <int WS, bool GAUSS>
__global__ void __launch_bounds__(128) am_peak_kernel(AmChunk c)
{
    chain_begin();
    constexpr int N = 2 * WS, NT = 128;
    __shared__ __align__(16) float2 osd[OSW * NFAST / 2 + 16];
    __shared__ float2 Yb[NFAST * NFAST], T[NFAST * OSW];
    __shared__ float blk[NFAST * NFAST];
    __shared__ double red[(NT / 32 + 1) * 2];
    const AmpArgs& a = c.a;
    const int tid = threadIdx.x, pt = blockIdx.x, st = a.stage, p = c.list[pt];
    const bool ownDop = a.noComplex != 0 && st == 1;
    FitJob* fj = &c.fit[pt];
    if (!c.mom[pt].hd) {
        if (tid == 0) {
            a.rec[p].flags |= (st == 1 ? RF_DONE_S : RF_DONE_L);
            if (ownDop) a.rec[p].azset = c.az[pt];
            fj->point = p;
            fj->gate = -1;  // no data: nothing for the fit kernel to decide
        }
        return;
    }
    for (int e = tid; e < OSW * NFAST / 2 + 16; e += NT) osd[e] = a.osD[e];
    double pw[2] = {0, 0};
    if (tid < N / 8) {
        pw[0] = c.pw[((size_t)pt * (N / 8) + tid) * 2];
        pw[1] = c.pw[((size_t)pt * (N / 8) + tid) * 2 + 1];
    }
    block_allsum<2, NT>(pw, red);
    const double nn = (double)N * N;
    const double p1 = pw[0] / nn, p2 = pw[1] / nn;
    const float* mag = c.mag + (size_t)pt * N * N;
    unsigned long long* sc = reinterpret_cast<unsigned long long*>(red);
    __syncthreads();
    const unsigned long long top =
        block_max_u64(tid < N / 16 ? c.best[(size_t)pt * (N / 16) + tid] : 0ull, sc);
    int iMax = 0, jMax = 0;  // nothing above 0: findCPeak keeps (0, 0)
    double cMax = 0.0;
    if (top >> 32) {
        const unsigned rank = 0xffffffffu - (unsigned)top;
        const int q = rank & 3, ij = rank >> 2;
        iMax = ij / WS + ((q == 1 || q == 2) ? WS : 0);
        jMax = ij % WS + ((q == 1 || q == 3) ? WS : 0);
        cMax = (double)__uint_as_float((unsigned)(top >> 32));
    }
    if (iMax < NFAST / 2 || iMax > N - NFAST / 2 || jMax < NFAST / 2 || jMax > N - NFAST / 2) {
        cMax = -1.0;
        iMax = -1000;
        jMax = -1000;
    }
    // samples for the Gaussian widths (gate: speckleTrack.c:538-539, strict)
    const int gate = iMax > NGAUSS / 2 && iMax < N - NGAUSS / 2 && jMax > NGAUSS / 2 && jMax < N - NGAUSS / 2;
    if (gate && tid < 2 * NGAUSS) {
        const int f = tid / NGAUSS, k = tid % NGAUSS;
        if (f == 0)
            fj->samp[0][k] = mag[iMax * N + (jMax - NGAUSS / 2 + k)];
        else
            fj->samp[1][k] = mag[(iMax - NGAUSS / 2 + k) * N + jMax];
        if (k == 0) fj->x0[f] = (f == 0 ? jMax : iMax) - NGAUSS / 2;
    }
    const double cRaw = cMax;
    const int iC = iMax, jC = jMax;
    if (GAUSS && iMax >= -999) {
        // -gauss: cmpTrackGauss on the amplitude plane (:553-557; pScale
        // 16, no hanning correction), unless the fit kernel takes the
        // early return of ampTrackFast
        const double hw = (double)(N / 2) * (double)(N / 2);
        const double scale = 1.0 / (sqrt((p1 * 16.0) * (p2 * 16.0)) * pow(hw, 2));
        gauss2d_peak<NT>([=](int i, int j) { return mag[i * N + j]; }, N, scale, reinterpret_cast<float*>(T), blk,
                         iMax, jMax, cMax);
    } else if (iMax >= -999) {
        // 8x8 -> 96x96 oversampling (used unless the fit kernel takes the
        // early return of ampTrackFast, :551-553)
        if (tid < NFAST * NFAST)
            blk[tid] = mag[(iMax - NFAST / 2 + tid / NFAST) * N + (jMax - NFAST / 2 + tid % NFAST)];
        __syncthreads();
        const ArgMax ob = oversample_peak_real<NT>(blk, reinterpret_cast<const float*>(osd), Yb, T, sc);
        const int iMax1 = ob.pos / OSW + (NFAST * NOVER) / 2 - 2 * NOVER;
        const int jMax1 = ob.pos % OSW + (NFAST * NOVER) / 2 - 2 * NOVER;
        cMax = (double)ob.v;
        cMax = cMax / ((double)N * N * N * N * NFAST * NFAST);  // exact
        cMax = cMax / sqrt(p1 * p2);
        iMax = (iMax * NOVER) + iMax1 - (NOVER * NFAST) / 2;
        jMax = (jMax * NOVER) + jMax1 - (NOVER * NFAST) / 2;
    }
    if (tid == 0) {
        PointRec* r = &a.rec[p];
        r->cMax[st] = cMax;
        r->iMax[st] = iMax;
        r->jMax[st] = jMax;
        r->cRaw = cRaw;
        r->iC = iC;
        r->jC = jC;
        if (ownDop) r->azset = c.az[pt];
        r->azUsed = c.az[pt];
        r->flags |= (st == 1 ? (RF_DONE_S | RF_HD_S) : (RF_DONE_L | RF_HD_L));
        fj->point = p;
        fj->gate = gate;
    }
}

// Planes in flight: nine planes of Ws x Ws complex values for two points per SM
// (87 MB at window 64, 349 MB at 128), the figure serve.py admits jobs by, in
// which the 64 Ws^2 bytes of a point leave room for 330 points.  The tries of a
// 1024 x 2048 pair at windows 64 and 128 take 5.8 ms (plain launches), 6.6 with
// half, 5.1 with four times that, where jobs that a server's budget admits
// would no longer fit.
static size_t am_chunk_bytes(int numSM, int Ws) { return (size_t)2 * numSM * sizeof(float2) * 9 * Ws * Ws; }

template <int WS>
struct AmRun {
    using C = AmCfg<WS>;
    static constexpr int N = 2 * WS;

    // Carves the planes of n entries from base (null: counts); returns the size.
    static size_t layout(AmChunk& c, int n, char* base, double** dop)
    {
        size_t used = 0;
        auto take = [&](size_t bytes) {
            char* p = base ? base + used : nullptr;
            used += (bytes + 255) / 256 * 256;
            return p;
        };
        const size_t nn = (size_t)N * N;
        // what a step is done with makes room for a later one: F, then z, then
        // mag; R, then T
        c.z = (float2*)take(sizeof(float2) * n * nn);
        c.F = c.z;
        c.mag = (float*)c.z;
        c.R = (float2*)take(sizeof(float2) * n * 2 * N * WS);
        c.T = c.R;
        static_assert(corr_ts(N) <= 2 * WS, "T fits over R");
        c.part = (double*)take(sizeof(double) * n * (N / 4) * 5);
        c.pw = (double*)take(sizeof(double) * n * (N / 8) * 2);
        c.best = (unsigned long long*)take(sizeof(unsigned long long) * n * (N / 16));
        c.mom = (AmMoments*)take(sizeof(AmMoments) * n);
        c.corner = (int4*)take(sizeof(int4) * n);
        c.az = (int*)take(sizeof(int) * n);
        *dop = (double*)take(sizeof(double) * dop_scratch_doubles<WS>(n));
        return used;
    }

    static cudaError_t attributes()
    {
        struct { const void* f; size_t sm; } k[] = {
            {(const void*)am_rows_kernel<WS, true>, C::smRows}, {(const void*)am_rows_kernel<WS, false>, C::smRows},
            {(const void*)am_cols_kernel<WS>, C::smCols},       {(const void*)am_detect_kernel<WS>, C::smDetect},
            {(const void*)am_fwd_kernel<WS>, C::smFwd},         {(const void*)am_corr_kernel<WS>, ColCfg<N>::smem},
            {(const void*)am_mag_kernel<WS>, C::smFwd}};
        for (auto& x : k) {
            const cudaError_t e = cudaFuncSetAttribute(x.f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)x.sm);
            if (e != cudaSuccess) return e;
        }
        return cudaSuccess;
    }

    static cudaError_t chunk(const AmChunk& c, double* dop, cudaStream_t st, int64_t* launches)
    {
        const int n = c.win.n;
        chain(am_prep_kernel, (n + 127) / 128, 128, 0, st, c);
        *launches += 9;
        if (c.a.noComplex != 0 && c.a.stage == 1) {
            const cudaError_t e = launch_dop<WS>(c.win, c.a.wA, dop, c.az, st);
            if (e != cudaSuccess) return e;
            *launches += 3;
        }
        const int g = n * 2 * (WS / C::G);
        if (c.win.sampleType == SB_CFLOAT32)
            chain(am_rows_kernel<WS, true>, g, C::NT, C::smRows, st, c);
        else
            chain(am_rows_kernel<WS, false>, g, C::NT, C::smRows, st, c);
        chain(am_cols_kernel<WS>, g, C::NT, C::smCols, st, c);
        chain(am_detect_kernel<WS>, n * (N / 4), C::NT, C::smDetect, st, c);
        chain(am_moments_kernel<WS>, (n + 3) / 4, 128, 0, st, c);
        chain(am_fwd_kernel<WS>, n * (N / C::G), C::NT, C::smFwd, st, c);
        chain(am_corr_kernel<WS>, n * ColCfg<N>::TILES, ColCfg<N>::NT, ColCfg<N>::smem, st, c);
        chain(am_mag_kernel<WS>, n * (N / (2 * C::G)), C::NT, C::smFwd, st, c);
        if (c.a.gauss)
            chain(am_peak_kernel<WS, true>, n, 128, 0, st, c);
        else
            chain(am_peak_kernel<WS, false>, n, 128, 0, st, c);
        return cudaGetLastError();
    }

    static int run(sb_context* ctx, const AmpArgs& a, int cnt)
    {
        cudaError_t e = attributes();
        if (e != cudaSuccess) return sb_ctx_cuda(ctx, e, "strack_amp attributes");
        AmChunk c = {};
        c.a = a;
        c.win.img1 = a.img1;
        c.win.img2 = a.img2;
        c.win.nr1 = a.nr1; c.win.na1 = a.na1; c.win.nr2 = a.nr2; c.win.na2 = a.na2;
        c.win.sampleType = a.sampleType;
        c.win.byteOrder = a.byteOrder;
        c.scale = (float)(1. / ((size_t)WS * WS * WS * WS * OS * OS * OS));
        c.thr = a.sampleType == SB_CFLOAT32 ? 1.0e-15f : 1.0e-6f;
        c.twW = batch_tw_table<WS>(ctx);
        c.twN = batch_tw_table<N>(ctx);
        if (!c.twW || !c.twN) return sb_ctx_fail(ctx, SB_ERR_NOMEM, "table allocation failed");
        double* dop;
        const size_t one = layout(c, 16, nullptr, &dop) / 16 + 1;
        int B = (int)(am_chunk_bytes(ctx->numSM, WS) / one);
        B = B < 16 ? 16 : B;
        char* base = sb_chunk_buf(ctx, "ampScratch", cnt, &B, [&](int b) { return layout(c, b, nullptr, &dop); });
        if (!base) return sb_ctx_fail(ctx, SB_ERR_NOMEM, "amplitude workspace allocation failed");
        layout(c, B, base, &dop);
        c.win.win = c.corner;
        for (int off = 0; off < cnt; off += B) {
            c.list = a.list + off;
            c.fit = a.fit + off;
            c.win.n = cnt - off < B ? cnt - off : B;
            e = chunk(c, dop, ctx->stream, &ctx->launches);
            if (e != cudaSuccess) return sb_ctx_cuda(ctx, e, "strack_amp");
        }
        return SB_OK;
    }
};

bool amp_supported(int Ws) { return amps_supported(Ws) || Ws == 48 || Ws == 64 || Ws == 96 || Ws == 128; }

int run_strack_amp(sb_context* c, int Ws, const AmpArgs& a, int cnt)
{
    switch (Ws) {
    case 48: return AmRun<48>::run(c, a, cnt);
    case 64: return AmRun<64>::run(c, a, cnt);
    case 96: return AmRun<96>::run(c, a, cnt);
    case 128: return AmRun<128>::run(c, a, cnt);
    default: return sb_ctx_fail(c, SB_ERR_UNSUPPORTED, "amplitude window %d not supported", Ws);
    }
}

}  // namespace sbk
