// fft_engine.cuh -- batched complex DFTs in shared memory for sm_100a.
//
// Conventions match FFTW 2 as used by the reference (fftwnd_one,
// Strack/speckleTrack.c:1507-1550): unnormalised, forward = exp(-2 pi i jk/N)
// (DIR = -1), backward = exp(+2 pi i jk/N) (DIR = +1).
//
// A length-N line (N = N1 * N2) is transformed in place in two steps
// (the "four-step" factorisation, x index n = N2*n1 + n2, X index
// k = k1 + N1*k2):
//   step 1: for every (line, n2): radix-N1 DFT over n1 in registers, times the
//           twiddle W_N^{n2 k1}, stored back to the same slots;
//   step 2: for every (line, k1): radix-N2 DFT over the N2 contiguous slots,
//           held in registers until every thread has loaded, then stored to
//           natural order k1 + N1*k2.
// Threads are mapped line-fastest, so with an odd row stride (N+1 float2) or
// unit line stride (column passes) every access pattern is bank-conflict free.
//
// Register DFTs of composite size R are built at compile time by splitting off
// the smallest prime factor; prime factors use the direct sum.  Twiddles come
// from a table W_TN^e = exp(-2 pi i e/TN), e < TN, read with compile-time
// indices (uniform across the warp, so broadcast) for the inter-step twiddles,
// while the twiddles inside the register DFTs are compile-time constants;
// factors of +-1, +-i are applied without a multiply.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace sbfft {

__device__ __forceinline__ float2 cmul(float2 a, float2 b)
{
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 cconjmul(float2 a, float2 b)  // a * conj(b)
{
    return make_float2(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}

constexpr int smallest_factor(int n)
{
    for (int p = 2; p * p <= n; ++p)
        if (n % p == 0) return p;
    return n;
}

// ---------------------------------------------------------------- compile-time twiddles
// cos and sin of 2 pi e / n for integers, evaluated by the compiler: octant
// reduction with exact integer arithmetic, then the Taylor series of sin and
// cos on [0, pi/4] in double (14 terms: truncation below 1e-20), rounded once
// to float where used.  Compile-time twiddles become immediate operands.
struct CxPair {
    double c, s;
};
constexpr double kQuarterPi = 0.78539816339744830961566084581987572;
__host__ __device__ constexpr double cx_sin(double x)
{
    double term = x, sum = x;
    for (int k = 1; k < 14; ++k) {
        term *= -x * x / ((2.0 * k) * (2.0 * k + 1.0));
        sum += term;
    }
    return sum;
}
__host__ __device__ constexpr double cx_cos(double x)
{
    double term = 1.0, sum = 1.0;
    for (int k = 1; k < 14; ++k) {
        term *= -x * x / ((2.0 * k - 1.0) * (2.0 * k));
        sum += term;
    }
    return sum;
}
__host__ __device__ constexpr CxPair cx_cossin(int e, int n)  // (cos, sin)(2 pi e / n)
{
    const long long r = ((e % n) + n) % n;
    const long long m = 8 * r;                  // theta / (pi/4) = m / n
    const int oct = (int)(m / n);
    const long long fnum = m - (long long)oct * n;  // phi = (pi/4) fnum / n
    const double phi = kQuarterPi * (double)fnum / (double)n;
    const double psi = kQuarterPi * (double)(n - fnum) / (double)n;  // pi/4 - phi
    const double Sp = cx_sin(phi), Cp = cx_cos(phi), Sq = cx_sin(psi), Cq = cx_cos(psi);
    switch (oct) {
    case 0: return {Cp, Sp};
    case 1: return {Sq, Cq};
    case 2: return {-Sp, Cp};
    case 3: return {-Cq, Sq};
    case 4: return {-Cp, -Sp};
    case 5: return {-Sq, -Cq};
    case 6: return {Sp, -Cp};
    default: return {Cq, -Sq};
    }
}

// v * W_TN^{E} for the direction DIR (W = exp(DIR * 2 pi i / TN)); E reduced mod TN.
template <int E, int TN, int DIR>
__device__ __forceinline__ float2 twmul(float2 v, const float2* __restrict__ tw)
{
    constexpr int e = ((E % TN) + TN) % TN;
    if constexpr (e == 0) {
        return v;
    } else if constexpr (4 * e == 2 * TN) {
        return make_float2(-v.x, -v.y);
    } else if constexpr (4 * e == TN) {
        // exp(DIR * i pi/2) = DIR * i
        return DIR > 0 ? make_float2(-v.y, v.x) : make_float2(v.y, -v.x);
    } else if constexpr (4 * e == 3 * TN) {
        return DIR > 0 ? make_float2(v.y, -v.x) : make_float2(-v.y, v.x);
    } else {
        constexpr CxPair w = cx_cossin(e, TN);
        constexpr float wr = (float)w.c;
        constexpr float wi = (float)(DIR > 0 ? w.s : -w.s);
        return cmul(v, make_float2(wr, wi));
    }
}

// Runtime-index twiddle multiply (inter-step twiddles).
template <int DIR>
__device__ __forceinline__ float2 twmul_rt(float2 v, const float2* __restrict__ tw, int e)
{
    float2 w = tw[e];
    if (DIR > 0) w.y = -w.y;
    return cmul(v, w);
}

// ---------------------------------------------------------------- register DFT
// SYM: odd primes through sums and differences of the pairs t[q], t[P - q]
// (real factors only: 60 operations at P = 7 against 140 for the direct sum).
template <int R, int DIR, int TN, bool SYM = false>
struct RegDFT {
    static_assert(TN % R == 0, "twiddle table size must be a multiple of R");
    static constexpr int P = (R % 4 == 0 && R > 4) ? 4 : smallest_factor(R);  // radix 4 first
    static constexpr int M = R / P;

    template <int Q, int K>
    __device__ __forceinline__ static float2 sub_tw(float2 v, const float2* tw)
    {
        return twmul<Q * K * (TN / R), TN, DIR>(v, tw);
    }

    // direct P-point DFT of t[] into out[r] (prime P)
    template <int Pp>
    __device__ __forceinline__ static void small_dft(float2 (&t)[Pp], float2 (&o)[Pp], const float2* tw)
    {
        if constexpr (Pp == 2) {
            o[0] = cadd(t[0], t[1]);
            o[1] = csub(t[0], t[1]);
        } else if constexpr (Pp == 4) {
            float2 a0 = cadd(t[0], t[2]), a1 = csub(t[0], t[2]);
            float2 b0 = cadd(t[1], t[3]), b1 = csub(t[1], t[3]);
            float2 jb1 = DIR > 0 ? make_float2(-b1.y, b1.x) : make_float2(b1.y, -b1.x);
            o[0] = cadd(a0, b0);
            o[2] = csub(a0, b0);
            o[1] = cadd(a1, jb1);
            o[3] = csub(a1, jb1);
        } else if constexpr (SYM) {
            constexpr int H = (Pp - 1) / 2;
            float2 a[H], b[H];
            o[0] = t[0];
#pragma unroll
            for (int q = 0; q < H; ++q) {
                a[q] = cadd(t[q + 1], t[Pp - 1 - q]);
                b[q] = csub(t[q + 1], t[Pp - 1 - q]);
                o[0] = cadd(o[0], a[q]);
            }
            sym_rows<Pp, 1>(t[0], a, b, o);
        } else {
#pragma unroll
            for (int r = 0; r < Pp; ++r) o[r] = t[0];
            small_dft_acc<Pp, 1>(t, o, tw);
        }
    }
    // outputs r and Pp - r of the symmetric form: c -+ i s with
    // c = t0 + sum a_q cos(2 pi q r / P), s = sum b_q sin(2 pi q r / P)
    template <int Pp, int Rr, int H>
    __device__ __forceinline__ static void sym_rows(float2 t0, float2 (&a)[H], float2 (&b)[H], float2 (&o)[Pp])
    {
        if constexpr (Rr <= H) {
            float2 c = t0, s = make_float2(0.f, 0.f);
            sym_terms<Pp, Rr, 1>(a, b, c, s);
            const float2 js = DIR > 0 ? make_float2(-s.y, s.x) : make_float2(s.y, -s.x);
            o[Rr] = cadd(c, js);
            o[Pp - Rr] = csub(c, js);
            sym_rows<Pp, Rr + 1>(t0, a, b, o);
        }
    }
    template <int Pp, int Rr, int Q, int H>
    __device__ __forceinline__ static void sym_terms(float2 (&a)[H], float2 (&b)[H], float2& c, float2& s)
    {
        if constexpr (Q <= H) {
            constexpr CxPair w = cx_cossin(Q * Rr, Pp);
            constexpr float wc = (float)w.c, ws = (float)w.s;
            c = make_float2(fmaf(a[Q - 1].x, wc, c.x), fmaf(a[Q - 1].y, wc, c.y));
            s = Q == 1 ? make_float2(b[0].x * ws, b[0].y * ws)
                       : make_float2(fmaf(b[Q - 1].x, ws, s.x), fmaf(b[Q - 1].y, ws, s.y));
            sym_terms<Pp, Rr, Q + 1>(a, b, c, s);
        }
    }
    template <int Pp, int Q>
    __device__ __forceinline__ static void small_dft_acc(float2 (&t)[Pp], float2 (&o)[Pp], const float2* tw)
    {
        if constexpr (Q < Pp) {
            small_dft_acc_r<Pp, Q, 0>(t, o, tw);
            small_dft_acc<Pp, Q + 1>(t, o, tw);
        }
    }
    template <int Pp, int Q, int Rr>
    __device__ __forceinline__ static void small_dft_acc_r(float2 (&t)[Pp], float2 (&o)[Pp], const float2* tw)
    {
        if constexpr (Rr < Pp) {
            o[Rr] = cadd(o[Rr], twmul<((Q * Rr) % Pp) * (TN / Pp), TN, DIR>(t[Q], tw));
            small_dft_acc_r<Pp, Q, Rr + 1>(t, o, tw);
        }
    }

    template <int K>
    __device__ __forceinline__ static void combine(float2 (&sub)[P][M], float2 (&v)[R], const float2* tw)
    {
        if constexpr (K < M) {
            float2 t[P], o[P];
            t[0] = sub[0][K];
            combine_tw<K, 1>(sub, t, tw);
            small_dft<P>(t, o, tw);
#pragma unroll
            for (int r = 0; r < P; ++r) v[K + M * r] = o[r];
            combine<K + 1>(sub, v, tw);
        }
    }
    template <int K, int Q>
    __device__ __forceinline__ static void combine_tw(float2 (&sub)[P][M], float2 (&t)[P], const float2* tw)
    {
        if constexpr (Q < P) {
            t[Q] = sub_tw<Q, K>(sub[Q][K], tw);
            combine_tw<K, Q + 1>(sub, t, tw);
        }
    }

    __device__ __forceinline__ static void run(float2 (&v)[R], const float2* __restrict__ tw)
    {
        if constexpr (R == 1) {
            return;
        } else if constexpr (R == 4) {
            float2 o[4];
            small_dft<4>(v, o, tw);
#pragma unroll
            for (int r = 0; r < 4; ++r) v[r] = o[r];
        } else if constexpr (P == R) {
            float2 o[R];
            small_dft<R>(v, o, tw);
#pragma unroll
            for (int r = 0; r < R; ++r) v[r] = o[r];
        } else {
            float2 sub[P][M];
#pragma unroll
            for (int q = 0; q < P; ++q)
#pragma unroll
                for (int t = 0; t < M; ++t) sub[q][t] = v[q + P * t];
#pragma unroll
            for (int q = 0; q < P; ++q) RegDFT<M, DIR, TN, SYM>::run(sub[q], tw);
            combine<0>(sub, v, tw);
        }
    }
};

// ---------------------------------------------------------------- line FFTs
// In-place transform of NL lines with NT threads: element k of line l at
// l LS + k ES.  All strides are compile-time constants, so addresses fold to
// immediates.  In the first step a thread stores exactly the slots it read; in
// the second every input is loaded before the first store.  Ends with a barrier.
template <int N1, int N2, int DIR, int NL, int NT, int LS, int ES>
__device__ __forceinline__ void fft_lines(float2* base, const float2* __restrict__ tw)
{
    constexpr int N = N1 * N2;
    constexpr int T1 = NL * N2, T2 = NL * N1;
    constexpr int R1 = (T1 + NT - 1) / NT, R2 = (T2 + NT - 1) / NT;
    const int tid = threadIdx.x;
#pragma unroll
    for (int r = 0; r < R1; ++r) {
        const int t = tid + r * NT;
        if (T1 % NT == 0 || t < T1) {
            const int l = t % NL, n2 = t / NL;
            float2* p = base + l * LS + n2 * ES;
            float2 v[N1];
#pragma unroll
            for (int n1 = 0; n1 < N1; ++n1) v[n1] = p[(N2 * n1) * ES];
            RegDFT<N1, DIR, N>::run(v, tw);
            // k1 * n2 < N1 * N2 = N: the twiddle index needs no reduction
#pragma unroll
            for (int k1 = 1; k1 < N1; ++k1) v[k1] = twmul_rt<DIR>(v[k1], tw, k1 * n2);
#pragma unroll
            for (int k1 = 0; k1 < N1; ++k1) p[(N2 * k1) * ES] = v[k1];
        }
    }
    __syncthreads();
    float2 v[R2][N2];
#pragma unroll
    for (int r = 0; r < R2; ++r) {
        const int t = tid + r * NT;
        if (T2 % NT == 0 || t < T2) {
            const float2* p = base + (t % NL) * LS + (N2 * (t / NL)) * ES;
#pragma unroll
            for (int n2 = 0; n2 < N2; ++n2) v[r][n2] = p[n2 * ES];
            RegDFT<N2, DIR, N>::run(v[r], tw);
        }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < R2; ++r) {
        const int t = tid + r * NT;
        if (T2 % NT == 0 || t < T2) {
            float2* p = base + (t % NL) * LS + (t / NL) * ES;
#pragma unroll
            for (int k2 = 0; k2 < N2; ++k2) p[(N1 * k2) * ES] = v[r][k2];
        }
    }
    __syncthreads();
}

// Factorisation used for each supported transform length.
template <int N>
struct Split;
template <> struct Split<8>   { static constexpr int N1 = 2,  N2 = 4;  };
template <> struct Split<16>  { static constexpr int N1 = 4,  N2 = 4;  };
template <> struct Split<24>  { static constexpr int N1 = 3,  N2 = 8;  };
template <> struct Split<32>  { static constexpr int N1 = 4,  N2 = 8;  };
template <> struct Split<48>  { static constexpr int N1 = 6,  N2 = 8;  };
template <> struct Split<64>  { static constexpr int N1 = 8,  N2 = 8;  };
template <> struct Split<96>  { static constexpr int N1 = 6,  N2 = 16; };
template <> struct Split<128> { static constexpr int N1 = 8,  N2 = 16; };

// ---------------------------------------------------------------- staged planes
// Tile of G lines of an N x N row-major array in a global workspace.
template <int N>
struct StagedTile {
    static constexpr int G = (N % 16 == 0) ? 16 : 8;
    static constexpr int elems = (G * (N + 1) > N * (G + 1)) ? G * (N + 1) : N * (G + 1);
};

// Line transforms of one staged tile (rows: G lines of N at stride N+1;
// columns: lines at stride 1, elements at stride G+1), in place.
template <int N, int DIR, int NT, int LS, int ES>
__device__ __forceinline__ void staged_tile_fft(float2* tile, const float2* __restrict__ tw)
{
    constexpr int G = StagedTile<N>::G;
    fft_lines<Split<N>::N1, Split<N>::N2, DIR, G, NT, LS, ES>(tile, tw);
}

// 2-D transform of an N x N row-major array anywhere in memory (row stride N;
// normally a per-CTA global workspace) staged through shared-memory tiles of G
// lines: rows, then columns, in place.
template <int N, int DIR, int NT>
__device__ __forceinline__ void fft2d_staged(float2* g, float2* tile, const float2* __restrict__ tw)
{
    constexpr int G = StagedTile<N>::G;
    const int tid = threadIdx.x;
    for (int r0 = 0; r0 < N; r0 += G) {
#pragma unroll 4
        for (int e = tid; e < G * N; e += NT) {
            const int l = e / N, k = e % N;
            tile[l * (N + 1) + k] = g[(size_t)(r0 + l) * N + k];
        }
        __syncthreads();
        staged_tile_fft<N, DIR, NT, N + 1, 1>(tile, tw);
#pragma unroll 4
        for (int e = tid; e < G * N; e += NT) {
            const int l = e / N, k = e % N;
            g[(size_t)(r0 + l) * N + k] = tile[l * (N + 1) + k];
        }
        __syncthreads();
    }
    for (int c0 = 0; c0 < N; c0 += G) {
#pragma unroll 4
        for (int e = tid; e < N * G; e += NT) {
            const int k = e / G, l = e % G;
            tile[k * (G + 1) + l] = g[(size_t)k * N + c0 + l];
        }
        __syncthreads();
        staged_tile_fft<N, DIR, NT, 1, G + 1>(tile, tw);
#pragma unroll 4
        for (int e = tid; e < N * G; e += NT) {
            const int k = e / G, l = e % G;
            g[(size_t)k * N + c0 + l] = tile[k * (G + 1) + l];
        }
        __syncthreads();
    }
}

}  // namespace sbfft
