// window_batch.cuh -- kernels shared by strackw and strack's large amplitude
// tries, which both run a chunk of grid points through a sequence of kernels
// over global planes instead of one CTA per point: the Doppler carrier of the
// raw windows, and the column half of the correlation of two real planes.
#pragma once
#include <cuda_runtime.h>

#include <type_traits>

#include "capi_internal.h"
#include "chain.cuh"
#include "fft_batch.cuh"
#include "strack_device.cuh"

namespace sbk {

// Two images and the corners (r1, a1, r2, a2) of a chunk's windows.
struct WinArgs {
    const void* img1;
    const void* img2;
    int nr1, na1, nr2, na2;
    int sampleType, byteOrder;
    const int4* win;
    int n;  // points of the chunk
};

// One image's W x W window: sample (i, j), zero outside the image.  The file
// type is a template parameter and the byte order a predicate, so nothing
// keeps a thread's loads from going out together.
template <bool F32>
struct Window {
    using Raw = typename std::conditional<F32, uint2, uint32_t>::type;
    const Raw* p;  // sample (0, 0)
    int nr, i0, i1, j0, j1;  // pitch; rows and columns inside the image
    bool msb;
    __device__ __forceinline__ Window(const WinArgs& a, int q, int4 w, int W)
    {
        const int r = q ? w.z : w.x, az = q ? w.w : w.y, na = q ? a.na2 : a.na1;
        nr = q ? a.nr2 : a.nr1;
        p = reinterpret_cast<const Raw*>(q ? a.img2 : a.img1) + ((ptrdiff_t)az * nr + r);
        i0 = max(0, -az);
        i1 = min(W, na - az);
        j0 = max(0, -r);
        j1 = min(W, nr - r);
        msb = a.byteOrder == SB_MSB;
    }
    __device__ __forceinline__ float2 operator()(int i, int j) const
    {
        Raw w = {};
        if (i >= i0 && i < i1 && j >= j0 && j < j1) w = __ldg(p + (ptrdiff_t)i * nr + j);
        if constexpr (F32) {
            if (msb) {
                w.x = bswap32(w.x);
                w.y = bswap32(w.y);
            }
            return make_float2(__uint_as_float(w.x), __uint_as_float(w.y));
        } else {
            if (msb) w = bswap16x2(w);
            return make_float2((float)(int16_t)(w & 0xffffu), (float)(int16_t)(w >> 16));
        }
    }
};

// ---------------------------------------------------------------- Doppler carrier
// estDopCarrier1 (Strack/dopplerEstimation.c:25-88) of the chunk's windows: a
// thread walks 16 rows of a column, band sums per CTA, the lag-1 products about
// the mean in a second kernel, the angle in a third (all in double, bands added
// in order).
template <int W>
struct DopCfg {
    static constexpr int NT = 256;
    static constexpr int RUN = 16;
    static constexpr int GR = NT / W < W / RUN ? NT / W : W / RUN;  // runs side by side in a CTA
    static constexpr int NB = (W + GR * RUN - 1) / (GR * RUN);
};

template <int W, bool F32>
__global__ void __launch_bounds__(256) dop_sum_kernel(WinArgs a, double* part)
{
    chain_begin();
    using C = DopCfg<W>;
    __shared__ double red[9 * 4];
    const int pt = blockIdx.x / C::NB, band = blockIdx.x % C::NB;
    const int4 w = a.win[pt];
    const int j = threadIdx.x % W, i0 = (band * C::GR + threadIdx.x / W) * C::RUN;
    double m[4] = {0, 0, 0, 0};
    if (threadIdx.x < W * C::GR && i0 < W)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const Window<F32> win(a, q, w, W);
            float2 z[C::RUN];
#pragma unroll
            for (int r = 0; r < C::RUN; ++r) z[r] = win(i0 + r, j);
#pragma unroll
            for (int r = 0; r < C::RUN; ++r) {
                m[2 * q] += z[r].x;
                m[2 * q + 1] += z[r].y;
            }
        }
    block_allsum<4, C::NT>(m, red);
    if (threadIdx.x == 0)
#pragma unroll
        for (int k = 0; k < 4; ++k) part[(size_t)blockIdx.x * 4 + k] = m[k];
}

template <int W, bool F32>
__global__ void __launch_bounds__(256, 4) dop_lag_kernel(WinArgs a, const double* sums, double* part)
{
    chain_begin();
    using C = DopCfg<W>;
    __shared__ double red[9 * 4];
    const int pt = blockIdx.x / C::NB, band = blockIdx.x % C::NB;
    const int4 w = a.win[pt];
    double m[4] = {0, 0, 0, 0};
    for (int b = 0; b < C::NB; ++b)
#pragma unroll
        for (int k = 0; k < 4; ++k) m[k] += sums[((size_t)pt * C::NB + b) * 4 + k];
    const double n = (double)(W * W);
#pragma unroll
    for (int k = 0; k < 4; ++k) m[k] /= n;
    const int j = threadIdx.x % W, i0 = (band * C::GR + threadIdx.x / W) * C::RUN;
    double d[4] = {0, 0, 0, 0};
    if (threadIdx.x < W * C::GR && i0 < W)
#pragma unroll 1
        for (int q = 0; q < 2; ++q) {
            const Window<F32> win(a, q, w, W);
            float2 z[C::RUN + 1];
#pragma unroll
            for (int r = 0; r <= C::RUN; ++r) z[r] = i0 + r < W ? win(i0 + r, j) : make_float2(0.f, 0.f);
            const double mr = q ? m[2] : m[0], mi = q ? m[3] : m[1];
            double br = (double)z[0].x - mr, bi = (double)z[0].y - mi, dr = 0, di = 0;
#pragma unroll
            for (int r = 1; r <= C::RUN; ++r) {
                const double ar = (double)z[r].x - mr, ai = (double)z[r].y - mi;
                if (i0 + r < W) {
                    dr += ar * br + ai * bi;
                    di += ai * br - ar * bi;
                }
                br = ar;
                bi = ai;
            }
            if (q) {
                d[2] = dr;
                d[3] = di;
            } else {
                d[0] = dr;
                d[1] = di;
            }
        }
    block_allsum<4, C::NT>(d, red);
    if (threadIdx.x == 0)
#pragma unroll
        for (int k = 0; k < 4; ++k) part[(size_t)blockIdx.x * 4 + k] = d[k];
}

// az[pt] = the roll rescaled to wOut rows.
template <int W>
__global__ void dop_angle_kernel(int n, const double* part, int wOut, int* az)
{
    chain_begin();
    const int pt = blockIdx.x * blockDim.x + threadIdx.x;
    if (pt >= n) return;
    double d[4] = {0, 0, 0, 0};
    for (int b = 0; b < DopCfg<W>::NB; ++b)
#pragma unroll
        for (int k = 0; k < 4; ++k) d[k] += part[((size_t)pt * DopCfg<W>::NB + b) * 4 + k];
    az[pt] = dop_shift(d[0], d[1], d[2], d[3], W, wOut);
}

template <int N>
inline const float2* batch_tw_table(sb_context* c)
{
    using S = sbfft::BSplit<N>;
    return ::batch_tw_table(c, S::N1, S::N2);
}

// part: 8 doubles per point and band.
template <int W>
inline size_t dop_scratch_doubles(int n)
{
    return (size_t)8 * n * DopCfg<W>::NB;
}
template <int W>
inline cudaError_t launch_dop(const WinArgs& a, int wOut, double* part, int* az, cudaStream_t st)
{
    using C = DopCfg<W>;
    double* lag = part + (size_t)4 * a.n * C::NB;
    if (a.sampleType == SB_CFLOAT32) {
        chain(dop_sum_kernel<W, true>, a.n * C::NB, C::NT, 0, st, a, part);
        chain(dop_lag_kernel<W, true>, a.n * C::NB, C::NT, 0, st, a, part, lag);
    } else {
        chain(dop_sum_kernel<W, false>, a.n * C::NB, C::NT, 0, st, a, part);
        chain(dop_lag_kernel<W, false>, a.n * C::NB, C::NT, 0, st, a, part, lag);
    }
    chain(dop_angle_kernel<W>, (a.n + 127) / 128, 128, 0, st, a.n, lag, wOut, az);
    return cudaGetLastError();
}

// ---------------------------------------------------------------- correlation, column half
// Z holds the row transforms of the packed real pair u + i v (N x N per
// point).  A CTA takes columns c0 .. c0+7 and their mirrors N - c: forward
// column transforms of both, the two real spectra from the Hermitian parts
// (U[k] = (Z[k] + conj Z[-k]) / 2, V[k] = (Z[k] - conj Z[-k]) / 2i), the cross
// spectrum U conj(V) of columns c0 .. c0+7 only -- the correlation is real, so
// columns past N/2 are conjugates of these -- and its inverse column
// transform, of which rows(m) >= 0 says where row m goes (T: rows x TS per
// point, TS = corr_ts(N)).  One read of Z and one write of half a plane do
// what a forward column pass, a cross-spectrum pass and an inverse pass did.
__host__ __device__ constexpr int corr_ts(int N) { return N / 2 + 8; }

template <int N>
struct ColCfg {
    static constexpr int GP = 8;       // column pairs per CTA
    static constexpr int G = 2 * GP;
    static constexpr int NT = N >= 128 ? 256 : 128;
    static constexpr int TILES = (N / 2 + GP) / GP;  // columns 0 .. N/2
    using LT = sbfft::LineTile<N, G, false>;
    using LI = sbfft::LineTile<N, GP, false>;
    static constexpr int BUF = LT::elems > LI::elems ? LT::elems : LI::elems;
    static constexpr size_t smem = sizeof(float2) * BUF;
};

template <int N, typename Rows>
__device__ __forceinline__ void corr_columns(const float2* __restrict__ Z, float2* __restrict__ T, int tile,
                                             const float2* __restrict__ tw, Rows rows)
{
    using C = ColCfg<N>;
    constexpr int G = C::G, GP = C::GP, TS = corr_ts(N);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2* s = reinterpret_cast<float2*>(smem_raw);
    const int c0 = tile * GP;
    // line l < GP: column c0 + l; line GP + l: its mirror
    auto src = [Z, c0](int l, int k) {
        int c = c0 + (l & (GP - 1));
        c = c > N / 2 ? N / 2 : c;
        if (l >= GP) c = c ? N - c : 0;
        return Z[(size_t)k * N + c];
    };
    auto nat = [s](int l, int k, float2 v) { s[k * G + l] = v; };
    sbfft::line_fft<N, -1, G, C::NT, false, false, true>(s, tw, src, nat);
    __syncthreads();
    auto cross = [s](int l, int k) {
        const float2 a = s[k * G + l], b = s[(k ? N - k : 0) * G + GP + l];
        const float2 f1 = make_float2(0.5f * (a.x + b.x), 0.5f * (a.y - b.y));
        const float2 f2 = make_float2(0.5f * (a.y + b.y), -0.5f * (a.x - b.x));
        return sbfft::cconjmul(f1, f2);
    };
    auto out = [T, c0, rows](int l, int k, float2 v) {
        const int r = rows(k);
        if (r >= 0 && c0 + l <= N / 2) T[(size_t)r * TS + c0 + l] = v;
    };
    sbfft::line_fft<N, 1, GP, C::NT, false, true, false>(s, tw, cross, out);
}

// Input k of the row transform of two Hermitian rows packed as one complex
// line: (row a) + i (row b), rows held for columns 0 .. N/2.  Its inverse
// transform is (real row a) + i (real row b).
template <int N>
__device__ __forceinline__ float2 pair_row_input(const float2* __restrict__ ra, const float2* __restrict__ rb, int k)
{
    const bool up = k > N / 2;
    float2 x = ra[up ? N - k : k], y = rb[up ? N - k : k];
    if (up) {
        x.y = -x.y;
        y.y = -y.y;
    }
    return make_float2(x.x - y.y, x.y + y.x);
}

}  // namespace sbk
