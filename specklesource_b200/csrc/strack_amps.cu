// strack_amps.cu -- amplitude tries of strack for windows up to 32,
// one CTA per grid point with every array resident in shared memory.
//
// Same computation as strack_amp.cu (ampMatch / ampTrackFast,
// Strack/speckleTrack.c:398-597, getAmpPatches :1006-1189), on lines that
// belong to one warp each (warp_lines.cuh), so that the passes are separated
// by one block barrier: both images' spectra (the Doppler roll folded into the
// column pass), row transforms for both range parities, and the column
// transforms of both azimuth parities of both images, a column's inputs kept
// in registers, intensity |c|^2 * scale written as pairs (I1, I2) into the
// 2W x 2W plane z; the no-data test and sqrt in one pass over z; mean removal
// and powers in the forward row pass of z = A1 + i A2; then a warp takes
// columns c and N - c together -- forward transforms, the Hermitian split and
// cross spectrum of column c, its inverse transform -- and finally pairs of
// real rows as one complex inverse line (the correlation is real: half the
// inverse lines of a complex plane).  |c| stays in the rows, findCPeak is the
// maximum with its tie order recovered by a rescan, and the 8x8 -> 96x96
// oversampling uses the real kernel D.
//
// Shared memory (Ws = 32): four Ws x (Ws+4) complex buffers and the
// 2Ws x (2Ws+4) plane, 72 KB: three CTAs per SM.  Block-wide passes over three
// buffers took 1.29 ms for 15,375 tries at Ws = 32, 56,000 instructions a try.
// From Ws = 48 up the arrays leave one CTA per SM, and strack_amp.cu's chunked
// kernels win: 3.58 against 6.07 ms at Ws = 48 (15,004 tries) and 5.25 against
// 7.13 ms at 64 (14,637 tries); at 32 they lost, 1.99 against 1.25 ms.
#include <cuda_runtime.h>

#include <type_traits>

#include "chain.cuh"
#include "strack_device.cuh"
#include "strack_kernels.h"
#include "warp_lines.cuh"

namespace sbk {

template <int WS, int NT>
struct AmpsSmem {
    static constexpr int N = 2 * WS;
    static constexpr int RS = WS + 4, RZ = N + 4;  // row strides, float2
    static constexpr int S = WS * RS;              // one Ws buffer
    static constexpr size_t bytes = sizeof(float2) * (4 * S + N * RZ + WS) + sizeof(double) * (NT / 32 + 1) * 5 + 16;
    // scratch of the oversampling, in the Ws buffers (spent by then)
    static_assert(sizeof(float2) * 4 * S >= sizeof(float2) * (OSW * NFAST / 2 + 16 + NFAST * NFAST + NFAST * OSW) +
                                                sizeof(float) * NFAST * NFAST, "scratch");
};

// Exact findCPeak over the N x N surface |c| (rows of RZ float2, N floats each,
// unshifted), given each thread's maximum: ties of the largest value > 0 go to
// the smallest cpeak_rank of the fftshifted position.  Returns y * N + x
// (fftshifted), or -1 when nothing is above 0.
template <int N, int RZ, int NT>
__device__ __forceinline__ int cpeak_plane(const float* mag, float pmax, unsigned* iscr)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    unsigned u = __reduce_max_sync(0xffffffffu, __float_as_uint(pmax));  // |c| >= 0: bits order as values
    if (lane == 0) iscr[warp] = u;
    __syncthreads();
    u = iscr[0];
#pragma unroll
    for (int w = 1; w < NT / 32; ++w) u = max(u, iscr[w]);
    const float pm = __uint_as_float(u);
    if (!(pm > 0.f)) return -1;  // uniform
    unsigned best = 0xffffffffu;
    for (int e = tid; e < N * N / 4; e += NT) {
        const int row = e / (N / 4), i4 = e % (N / 4);
        const float4 v = reinterpret_cast<const float4*>(mag + row * 2 * RZ)[i4];
        if (fmaxf(fmaxf(v.x, v.y), fmaxf(v.z, v.w)) < pm) continue;  // candidates are rare
        const float vv[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int c = 0; c < 4; ++c)
            if (vv[c] == pm) {
                const int cx = 4 * i4 + c;
                const int y = row < N / 2 ? row + N / 2 : row - N / 2, x = cx < N / 2 ? cx + N / 2 : cx - N / 2;
                best = min(best, (unsigned)cpeak_rank(y, x, N / 2));
            }
    }
    best = __reduce_min_sync(0xffffffffu, best);
    if (lane == 0) iscr[NT / 32 + warp] = best;
    __syncthreads();
    best = iscr[NT / 32];
#pragma unroll
    for (int w = 1; w < NT / 32; ++w) best = min(best, iscr[NT / 32 + w]);
    __syncthreads();
    const int h = N / 2, q = best & 3, ij = best >> 2;
    const int y = ij / h + ((q == 1 || q == 2) ? h : 0);
    const int x = ij % h + ((q == 1 || q == 3) ? h : 0);
    return y * N + x;
}

// Raw sample words are decoded after all of a thread's loads are out.
template <bool F32>
__device__ __forceinline__ float2 amps_decode(typename std::conditional<F32, uint2, uint32_t>::type w, bool msb)
{
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

template <int WS, int NT, bool F32, bool GAUSS>
__global__ void __launch_bounds__(NT, (WS == 32 ? 3 : WS == 24 ? 3 : 8)) strack_amps_kernel(AmpArgs a)
{
    chain_begin();
    using M = AmpsSmem<WS, NT>;
    constexpr int N = M::N, RS = M::RS, RZ = M::RZ, S = M::S, NW = NT / 32;
    using LW = sbfft::WarpLines<WS, 8>;
    using LZ = sbfft::WarpLines<N, WS == 16 ? 8 : 4>;
    constexpr int G = LW::LG, GZ = LZ::LG, RUN = WS * WS / NT;
    static_assert(WS * WS % NT == 0 && NT % WS == 0, "whole rows per thread");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2* F = reinterpret_cast<float2*>(smem_raw);  // image q at F + q S: spectrum, then its e2 = 1 rows
    float2* R = F + 2 * S;                            // the e2 = 0 rows
    float2* z = R + 2 * S;
    float2* tau = z + N * RZ;
    double* red = reinterpret_cast<double*>(tau + WS);
    int* azs = reinterpret_cast<int*>(red + (NW + 1) * 5);  // the try's roll
    float* zf = reinterpret_cast<float*>(z);
    // oversampling scratch over the Ws buffers
    float* osD = reinterpret_cast<float*>(F);
    float2* Yb = F + OSW * NFAST / 2 + 16;
    float2* T = Yb + NFAST * NFAST;
    float* blk = reinterpret_cast<float*>(T + NFAST * OSW);
    const int tid = threadIdx.x, warp = tid >> 5;
    for (int e = tid; e < WS; e += NT) tau[e] = a.tau[e];

    const float thr = F32 ? 1.0e-15f : 1.0e-6f;
    const float scale = (float)(1. / ((size_t)WS * WS * WS * WS * OS * OS * OS));
    const int st = a.stage;
    const bool ownDop = (a.noComplex != 0 && st == 1);
    const bool msb = a.byteOrder == SB_MSB;
    const int jc = tid % WS, i0 = tid / WS;  // load phase: column jc, rows i0, i0 + NT / WS, ...
    __syncthreads();

    const int nList = a.nListDev ? min(a.nList, *a.nListDev) : a.nList;
    for (int it = blockIdx.x; it < nList; it += gridDim.x) {
        const int p = a.list[it];
        const PointPlan pl = a.plan[p];
        // window corners (computeAmpImageLocations, speckleTrack.c:147-156):
        // a1a = aStart + i deltaA - (wA/2) s = a1 + wA/2 - (wA/2) s, from the plan
        const int a1a = pl.a1 + a.wA / 2 - a.wA / 2 * a.s;
        const int r1a = pl.r1 + a.wR / 2 - a.wR / 2 * a.s;
        const int r2a = r1a + (pl.r2 - pl.r1);
        const int a2a = a1a + (pl.a2 - pl.a1);
        double m[4] = {0, 0, 0, 0};
        {
            using Raw = typename std::conditional<F32, uint2, uint32_t>::type;
            Raw w1[RUN], w2[RUN];
#pragma unroll
            for (int u = 0; u < RUN; ++u) {
                const int i = i0 + u * (NT / WS);
                w1[u] = __ldg(reinterpret_cast<const Raw*>(a.img1) + ((size_t)(a1a + i) * a.nr1 + r1a + jc));
                w2[u] = __ldg(reinterpret_cast<const Raw*>(a.img2) + ((size_t)(a2a + i) * a.nr2 + r2a + jc));
            }
#pragma unroll
            for (int u = 0; u < RUN; ++u) {
                const int o = (i0 + u * (NT / WS)) * RS + jc;
                const float2 z1 = amps_decode<F32>(w1[u], msb), z2 = amps_decode<F32>(w2[u], msb);
                F[o] = z1;
                F[S + o] = z2;
                if (ownDop) {
                    m[0] += z1.x; m[1] += z1.y; m[2] += z2.x; m[3] += z2.y;
                }
            }
        }
        // ---------------------------------------------------- Doppler
        int azShift;
        if (ownDop) {
            // estDopCarrier1(im1in, im2in, wAa, wRa) (speckleTrack.c:1141-1144)
            block_allsum<4, NT>(m, red);
            const double n = (double)(WS * WS);
            const double m1r = m[0] / n, m1i = m[1] / n, m2r = m[2] / n, m2i = m[3] / n;
            double d[4] = {0, 0, 0, 0};
#pragma unroll 2
            for (int u = 0; u < RUN; ++u) {
                const int i = i0 + u * (NT / WS), o = i * RS + jc;
                if (i < WS - 1) {
                    const float2 p0 = F[o], p1 = F[o + RS];
                    double ar = (double)p1.x - m1r, ai = (double)p1.y - m1i, br = (double)p0.x - m1r,
                           bi = (double)p0.y - m1i;
                    d[0] += ar * br + ai * bi;
                    d[1] += ai * br - ar * bi;
                    const float2 q0 = F[S + o], q1 = F[S + o + RS];
                    ar = (double)q1.x - m2r; ai = (double)q1.y - m2i; br = (double)q0.x - m2r; bi = (double)q0.y - m2i;
                    d[2] += ar * br + ai * bi;
                    d[3] += ai * br - ar * bi;
                }
            }
            block_allsum<4, NT>(d, red);
            // one thread evaluates the roll (two double atan2); the barrier
            // after the row pass publishes it
            if (tid == 0) *azs = dop_shift(d[0], d[1], d[2], d[3], a.wAa, a.wA);
        } else {
            if (tid == 0) {
                const int az = a.azEff ? a.azEff[p] : a.rec[p].azset;
                *azs = az < 0 ? 0 : az;
            }
            __syncthreads();
        }
        // ---------------------------------------------------- detected images
        {
            const LW lw(a.twWs);
            constexpr int R1 = LW::R1, N1 = LW::N1, R2 = LW::R2, N2 = LW::N2;
#pragma unroll 1
            for (int g = warp; g < 2 * WS / G; g += NW) {
                float2* b = F + (g / (WS / G)) * S + (g % (WS / G)) * G * RS;
                float2 v[R1][N1];
                lw.load(v, [b](int l, int k) { return b[l * RS + k]; });
                __syncwarp();
                lw.template run<-1, 1>(v, [b](int l) { return b + l * RS; },
                                       [b](int l, int k, float2 c, int, int) { b[l * RS + k] = c; });
            }
            __syncthreads();
            azShift = *azs;
            const int az = (int)((float)azShift * (float)WS / (float)a.wA);
#pragma unroll 1
            for (int g = warp; g < 2 * WS / G; g += NW) {
                float2* b = F + (g / (WS / G)) * S + (g % (WS / G)) * G;
                float2 v[R1][N1];
                lw.load(v, [b](int l, int k) { return b[k * RS + l]; });
                __syncwarp();
                lw.template run<-1, RS>(v, [b](int l) { return b + l; }, [b, az](int l, int k, float2 c, int, int) {
                    b[(k < az ? k - az + WS : k - az) * RS + l] = c;
                });
            }
            __syncthreads();
            auto times_tau = [&](float2(&u)[R1][N1]) {
#pragma unroll
                for (int r = 0; r < R1; ++r)
#pragma unroll
                    for (int n = 0; n < N1; ++n) u[r][n] = sbfft::cmul(u[r][n], tau[N2 * n + lw.n2()]);
            };
            // rows: plain into R, times tau[k2] in place
#pragma unroll 1
            for (int g = warp; g < 2 * WS / G; g += NW) {
                float2* b = F + (g / (WS / G)) * S + (g % (WS / G)) * G * RS;
                float2* c = b + 2 * S;
                float2 u[R1][N1], v[R1][N1];
                lw.load(u, [b](int l, int k) { return b[l * RS + k]; });
#pragma unroll
                for (int r = 0; r < R1; ++r)
#pragma unroll
                    for (int n = 0; n < N1; ++n) v[r][n] = u[r][n];
                __syncwarp();
                lw.template run<1, 1>(v, [c](int l) { return c + l * RS; },
                                      [c](int l, int k, float2 x, int, int) { c[l * RS + k] = x; });
                times_tau(u);
                lw.template run<1, 1>(u, [b](int l) { return b + l * RS; },
                                      [b](int l, int k, float2 x, int, int) { b[l * RS + k] = x; });
            }
            __syncthreads();
            // columns: both azimuth parities of both images, pairs into z
#pragma unroll 1
            for (int g = warp; g < 2 * WS / G; g += NW) {
                const int e2 = g / (WS / G), c0 = (g % (WS / G)) * G;
                float p[2][R2][N2];  // image 1: e1 = 0, 1
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    float2* b = (e2 ? F : R) + q * S + c0;
                    auto line = [b](int l) { return b + l; };
                    float2 u[R1][N1], v[R1][N1];
                    lw.load(u, [b](int l, int k) { return b[k * RS + l]; });
#pragma unroll
                    for (int r = 0; r < R1; ++r)
#pragma unroll
                        for (int n = 0; n < N1; ++n) v[r][n] = u[r][n];
                    __syncwarp();
#pragma unroll
                    for (int e1 = 0; e1 < 2; ++e1) {
                        if (e1) times_tau(u);
                        lw.template run<1, RS>(e1 ? u : v, line, [&](int l, int k, float2 x, int r, int k2) {
                            const float I = (x.x * x.x + x.y * x.y) * scale;
                            if (q == 0)
                                p[e1][r][k2] = I;
                            else
                                z[(2 * k + e1) * RZ + 2 * (c0 + l) + e2] = make_float2(p[e1][r][k2], I);
                        });
                    }
                }
            }
        }
        __syncthreads();
        // ---------------------------------------------------- tests, amplitudes
        double r5[5] = {0, 0, 0, 0, 0};  // samples under the threshold, intensities, amplitudes
        {
            int cnt = 0;
#pragma unroll 4
            for (int e = tid; e < N * N; e += NT) {
                const int o = (e / N) * RZ + e % N;
                float2 v = z[o];
                cnt += v.x < thr || v.y < thr;
                r5[1] += v.x;
                r5[2] += v.y;
                v.x = sqrtf(v.x);
                v.y = sqrtf(v.y);
                z[o] = v;
                r5[3] += v.x;
                r5[4] += v.y;
            }
            r5[0] = cnt;
        }
        block_allsum<5, NT>(r5, red);
        const bool hd = !(r5[0] > 20.0) && !(r5[1] < 1.0e-6 || r5[2] < 1.0e-6);
        if (!hd) {
            if (tid == 0) {
                a.rec[p].flags |= (st == 1 ? RF_DONE_S : RF_DONE_L);
                if (ownDop) a.rec[p].azset = azShift;
                a.fit[it].point = p;
                a.fit[it].gate = -1;  // no data: nothing for the fit kernel to decide
            }
            __syncthreads();
            continue;  // uniform across the block
        }
        const double nn = (double)N * N;
        const double avg1 = r5[3] / nn, avg2 = r5[4] / nn;
        // ---------------------------------------------------- correlation
        double pw[2] = {0, 0};
        float pmax = 0.f;
        {
            const LZ lz(a.tw2Ws);
            constexpr int R1 = LZ::R1, N1 = LZ::N1;
#pragma unroll 1
            for (int g = warp; g < N / GZ; g += NW) {
                float2* b = z + g * GZ * RZ;
                float2 v[R1][N1];
                lz.load(v, [&](int l, int k) {
                    float2 x = b[l * RZ + k];
                    if (x.x > 1.0e-20f) x.x = (float)((double)x.x - avg1);
                    x.y = (float)((double)x.y - avg2);
                    pw[0] += (double)(x.x * x.x);
                    pw[1] += (double)(x.y * x.y);
                    return x;
                });
                __syncwarp();
                lz.template run<-1, 1>(v, [b](int l) { return b + l * RZ; },
                                       [b](int l, int k, float2 x, int, int) { b[l * RZ + k] = x; });
            }
            __syncthreads();
            // Columns c0 .. c0+GZ-1 (all below N/2) and their mirrors N - c by
            // one warp; column N/2 takes the place of column 0's mirror.
            // Columns 0 and N/2 of the cross spectrum have real inverses, so
            // they go through as one line, S_0 + i S_{N/2}.
#pragma unroll 1
            for (int g = warp; g < WS / GZ; g += NW) {
                const int c0 = g * GZ;
                auto col = [c0](int l) { return c0 + l; };
                auto mir = [c0](int l) { return c0 + l == 0 ? N / 2 : N - c0 - l; };
                float2 v[R1][N1];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    lz.load(v, [&](int l, int k) { return z[k * RZ + (h ? mir(l) : col(l))]; });
                    __syncwarp();
                    lz.template run<-1, RZ>(v, [&](int l) { return z + (h ? mir(l) : col(l)); },
                                            [&](int l, int k, float2 x, int, int) {
                                                z[k * RZ + (h ? mir(l) : col(l))] = x;
                                            });
                }
                __syncwarp();
                // U[k] = (Z[k] + conj Z[-k]) / 2, V[k] = (Z[k] - conj Z[-k]) / 2i
                auto cross = [](float2 x, float2 y) {
                    const float2 f1 = make_float2(0.5f * (x.x + y.x), 0.5f * (x.y - y.y));
                    const float2 f2 = make_float2(0.5f * (x.y + y.y), -0.5f * (x.x - y.x));
                    return sbfft::cconjmul(f1, f2);
                };
                lz.load(v, [&](int l, int k) {
                    const int km = k ? N - k : 0;
                    const bool self = c0 + l == 0;
                    const float2 s0 = cross(z[k * RZ + col(l)], z[km * RZ + (self ? 0 : mir(l))]);
                    if (!self) return s0;
                    const float2 s1 = cross(z[k * RZ + N / 2], z[km * RZ + N / 2]);
                    return make_float2(s0.x - s1.y, s0.y + s1.x);
                });
                __syncwarp();
                lz.template run<1, RZ>(v, [&](int l) { return z + col(l); }, [&](int l, int k, float2 x, int, int) {
                    if (c0 + l == 0) {
                        z[k * RZ] = make_float2(x.x, 0.f);
                        z[k * RZ + N / 2] = make_float2(x.y, 0.f);
                    } else {
                        z[k * RZ + col(l)] = x;
                    }
                });
            }
            __syncthreads();
            // rows 2i and 2i + 1 as one complex line; |c| = |re| into the rows
#pragma unroll 1
            for (int g = warp; g < WS / GZ; g += NW) {
                float2* b = z + 2 * g * GZ * RZ;
                float2 v[R1][N1];
                lz.load(v, [b](int l, int k) {
                    const bool up = k > N / 2;
                    const float2* q = b + 2 * l * RZ + (up ? N - k : k);
                    float2 x = q[0], y = q[RZ];
                    if (up) {
                        x.y = -x.y;
                        y.y = -y.y;
                    }
                    return make_float2(x.x - y.y, x.y + y.x);
                });
                __syncwarp();
                lz.template run<1, 1>(v, [b](int l) { return b + 2 * l * RZ; }, [&](int l, int k, float2 x, int, int) {
                    float* f = reinterpret_cast<float*>(b + 2 * l * RZ) + k;
                    const float ca = fabsf(x.x), cb = fabsf(x.y);
                    f[0] = ca;
                    f[2 * RZ] = cb;
                    pmax = fmaxf(pmax, fmaxf(ca, cb));
                });
            }
        }
        block_allsum<2, NT>(pw, red);
        const double p1 = pw[0] / nn, p2 = pw[1] / nn;
        // |c| at a fftshifted position
        auto mag = [zf](int y, int x) {
            const int cy = y < WS ? y + WS : y - WS, cx = x < WS ? x + WS : x - WS;
            return zf[cy * 2 * RZ + cx];
        };
        // ---------------------------------------------------- findCPeak, fits, oversampling
        __syncthreads();
        const int pos = cpeak_plane<N, RZ, NT>(zf, pmax, reinterpret_cast<unsigned*>(red));
        int iMax = 0, jMax = 0;
        double cMax = 0.0;
        if (pos >= 0) {
            iMax = pos / N;
            jMax = pos % N;
            cMax = (double)mag(iMax, jMax);
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
            FitJob* fj = &a.fit[it];
            if (f == 0)
                fj->samp[0][k] = mag(iMax, jMax - NGAUSS / 2 + k);
            else
                fj->samp[1][k] = mag(iMax - NGAUSS / 2 + k, jMax);
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
            gauss2d_peak<NT>(mag, N, scale, reinterpret_cast<float*>(T), blk, iMax, jMax, cMax);
        } else if (iMax >= -999) {
            // 8x8 -> 96x96 oversampling (used unless the fit kernel takes the
            // early return of ampTrackFast, :551-553)
            if (tid < NFAST * NFAST) {
                const int t1 = tid / NFAST, t2 = tid % NFAST;
                blk[tid] = mag(iMax - NFAST / 2 + t1, jMax - NFAST / 2 + t2);
            }
            for (int e = tid; e < OSW * NFAST / 2 + 16; e += NT) reinterpret_cast<float2*>(osD)[e] = __ldg(a.osD + e);
            __syncthreads();
            const ArgMax ob = oversample_peak_real<NT>(blk, osD, Yb, T, reinterpret_cast<unsigned long long*>(red));
            const int iMax1 = ob.pos / OSW + (NFAST * NOVER) / 2 - 2 * NOVER;
            const int jMax1 = ob.pos % OSW + (NFAST * NOVER) / 2 - 2 * NOVER;
            if (tid == 0) {
                cMax = (double)ob.v;
                cMax = cMax / ((double)N * N * N * N * NFAST * NFAST);  // exact
                cMax = cMax / sqrt(p1 * p2);
            }
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
            if (ownDop) r->azset = azShift;
            r->azUsed = azShift;
            r->flags |= (st == 1 ? (RF_DONE_S | RF_HD_S) : (RF_DONE_L | RF_HD_L));
            a.fit[it].point = p;
            a.fit[it].gate = gate;
        }
        __syncthreads();
    }
}

template <int WS, int NT, bool F32, bool GAUSS>
static cudaError_t launch_amps_t(const AmpArgs& a, int nCta, cudaStream_t st)
{
    const size_t sm = AmpsSmem<WS, NT>::bytes;
    cudaError_t e = cudaFuncSetAttribute(strack_amps_kernel<WS, NT, F32, GAUSS>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    chain(strack_amps_kernel<WS, NT, F32, GAUSS>, nCta, NT, sm, st, a);
    return cudaGetLastError();
}

template <int WS, int NT>
static cudaError_t launch_amps(const AmpArgs& a, int nCta, cudaStream_t st)
{
    if (a.sampleType == SB_CFLOAT32)
        return a.gauss ? launch_amps_t<WS, NT, true, true>(a, nCta, st) : launch_amps_t<WS, NT, true, false>(a, nCta, st);
    return a.gauss ? launch_amps_t<WS, NT, false, true>(a, nCta, st) : launch_amps_t<WS, NT, false, false>(a, nCta, st);
}

template <int WS, int NT>
static int occupancy_amps()
{
    int nb = 0;
    const size_t sm = AmpsSmem<WS, NT>::bytes;
    cudaFuncSetAttribute(strack_amps_kernel<WS, NT, true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, strack_amps_kernel<WS, NT, true, false>, NT, sm);
    return nb;
}

bool amps_supported(int Ws) { return Ws == 16 || Ws == 24 || Ws == 32; }

int amps_blocks_per_sm(int Ws)
{
    switch (Ws) {
    case 16: return occupancy_amps<16, 64>();
    case 24: return occupancy_amps<24, 192>();
    case 32: return occupancy_amps<32, 256>();
    default: return 0;
    }
}

cudaError_t launch_strack_amps(int Ws, const AmpArgs& a, int nCta, cudaStream_t st)
{
    switch (Ws) {
    case 16: return launch_amps<16, 64>(a, nCta, st);
    case 24: return launch_amps<24, 192>(a, nCta, st);
    case 32: return launch_amps<32, 256>(a, nCta, st);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace sbk
