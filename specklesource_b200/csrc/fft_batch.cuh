// fft_batch.cuh -- line DFTs for transforms too large for one CTA: a CTA takes
// G lines of N points straight from where they lie (global memory, an image, a
// shared buffer) and hands the results straight to where they go.
//
// A line of N = N1 N2 points is transformed in two steps of register DFTs (x
// index n = N2 n1 + n2, X index k = k1 + N1 k2).  The first step reads its
// inputs from src(l, n) into registers and the second hands its outputs to
// dst(l, k, value), so a line makes one trip through shared memory.  The tile
// form this replaces (load to shared, three steps, store out of place, copy
// out) made five and ran one CTA-wide barrier chain per 8 lines.  Three steps
// with 448 = 7 x 8 x 8 (two trips) took 42.8 us where 16 x 28 takes 33.3 us
// (sw_fwd, 54 points at W = 224): shared-memory wavefronts, not registers, are
// what such a kernel runs out of.
// Conventions as in fft_engine.cuh (unnormalised, DIR = -1 forward).
//
// Lane order: ROW tiles let neighbouring lanes walk along a line (rows of a
// row-major plane: 128 bytes and more per access), column tiles let them walk
// across lines (G columns of a row-major plane: 8 G bytes).  The paddings keep
// the shared accesses of both steps conflict-free or nearly so: in a ROW tile
// the k1 blocks start an odd number of slots apart, in a column tile of 8
// lines 8 slots apart modulo 16.
#pragma once
#include "fft_engine.cuh"

namespace sbfft {

// The second radix is the larger one where the first step's lanes should read
// 128 contiguous bytes (N2 >= 16).
template <int N> struct BSplit;
template <> struct BSplit<32>  { static constexpr int N1 = 4,  N2 = 8;  };
template <> struct BSplit<48>  { static constexpr int N1 = 6,  N2 = 8;  };
template <> struct BSplit<64>  { static constexpr int N1 = 8,  N2 = 8;  };
template <> struct BSplit<96>  { static constexpr int N1 = 8,  N2 = 12; };
template <> struct BSplit<128> { static constexpr int N1 = 8,  N2 = 16; };
template <> struct BSplit<192> { static constexpr int N1 = 12, N2 = 16; };
template <> struct BSplit<224> { static constexpr int N1 = 14, N2 = 16; };
template <> struct BSplit<256> { static constexpr int N1 = 16, N2 = 16; };
template <> struct BSplit<384> { static constexpr int N1 = 16, N2 = 24; };
template <> struct BSplit<448> { static constexpr int N1 = 16, N2 = 28; };
template <> struct BSplit<512> { static constexpr int N1 = 16, N2 = 32; };

// The twiddle table of a length holds W_N^{k1 n2} at k1 N2 + n2: in step order
// neighbouring lanes read neighbouring entries, where one table of W_N^e
// indexed by k1 n2 costs up to eight-way bank conflicts.

// Shared-memory slots of a tile of G lines: element N2 k1 + n2 of line l is at
// l L + k1 K1 + n2 K2.
template <int N, int G, bool ROW>
struct LineTile {
    using S = BSplit<N>;
    static constexpr int K2 = ROW ? 1 : G;
    static constexpr int K1 = ROW ? S::N2 | 1 : S::N2 * G + (G == 8 ? 8 : 0);
    static constexpr int L = ROW ? S::N1 * K1 : 1;
    static constexpr int elems = ROW ? G * L : S::N1 * K1;
};

struct NoTap {
    __device__ __forceinline__ void operator()(int, int, float2) const {}
};

// Transforms G lines with NT threads.  s: LineTile<N, G, ROW>::elems slots; tw:
// the length's table in global memory (a few KB that stay in L1).  HOLD_IN:
// src reads slots of s (every input is loaded before the first store);
// HOLD_OUT: dst writes slots of s (every slot is read before the first dst);
// both are free where a thread has one item.  tap(l, n, v) sees every input
// once, after a thread's loads are out.  The caller puts barriers before the
// next use of s and after dst's stores.
template <int N, int DIR, int G, int NT, bool ROW, bool HOLD_IN, bool HOLD_OUT, typename Src, typename Dst,
          typename Tap = NoTap>
__device__ __forceinline__ void line_fft(float2* s, const float2* __restrict__ tw, Src src, Dst dst, Tap tap = Tap())
{
    using L = LineTile<N, G, ROW>;
    constexpr int N1 = BSplit<N>::N1, N2 = BSplit<N>::N2;
    const int tid = threadIdx.x;
    {
        constexpr int T = G * N2, IT = (T + NT - 1) / NT;
        float2 v[HOLD_IN ? IT : 1][N1];
        auto load = [&](int t, float2(&u)[N1]) {
            const int l = ROW ? t / N2 : t % G, m = ROW ? t % N2 : t / G;
#pragma unroll
            for (int n1 = 0; n1 < N1; ++n1) u[n1] = src(l, N2 * n1 + m);
#pragma unroll
            for (int n1 = 0; n1 < N1; ++n1) tap(l, N2 * n1 + m, u[n1]);
        };
        auto step = [&](int t, float2(&u)[N1]) {
            const int l = ROW ? t / N2 : t % G, m = ROW ? t % N2 : t / G;
            float2* p = s + l * L::L + m * L::K2;
            RegDFT<N1, DIR, N, true>::run(u, tw);
            p[0] = u[0];
#pragma unroll
            for (int k1 = 1; k1 < N1; ++k1) {
                float2 w = __ldg(tw + k1 * N2 + m);
                if (DIR > 0) w.y = -w.y;
                p[k1 * L::K1] = cmul(u[k1], w);
            }
        };
        if constexpr (HOLD_IN) {
#pragma unroll
            for (int r = 0; r < IT; ++r)
                if (T % NT == 0 || tid + r * NT < T) load(tid + r * NT, v[r]);
            __syncthreads();
#pragma unroll
            for (int r = 0; r < IT; ++r)
                if (T % NT == 0 || tid + r * NT < T) step(tid + r * NT, v[r]);
        } else {
#pragma unroll 1
            for (int t = tid; t < T; t += NT) {
                load(t, v[0]);
                step(t, v[0]);
            }
        }
    }
    __syncthreads();
    {
        constexpr int T = G * N1, IT = (T + NT - 1) / NT;
        float2 v[HOLD_OUT ? IT : 1][N2];
        auto load = [&](int t, float2(&u)[N2]) {
            const int l = ROW ? t / N1 : t % G, k1 = ROW ? t % N1 : t / G;
            const float2* p = s + l * L::L + k1 * L::K1;
#pragma unroll
            for (int n = 0; n < N2; ++n) u[n] = p[n * L::K2];
            RegDFT<N2, DIR, N, true>::run(u, tw);
        };
        auto store = [&](int t, float2(&u)[N2]) {
            const int l = ROW ? t / N1 : t % G, k1 = ROW ? t % N1 : t / G;
#pragma unroll
            for (int k2 = 0; k2 < N2; ++k2) dst(l, k1 + N1 * k2, u[k2]);
        };
        if constexpr (HOLD_OUT) {
#pragma unroll
            for (int r = 0; r < IT; ++r)
                if (T % NT == 0 || tid + r * NT < T) load(tid + r * NT, v[r]);
            __syncthreads();
#pragma unroll
            for (int r = 0; r < IT; ++r)
                if (T % NT == 0 || tid + r * NT < T) store(tid + r * NT, v[r]);
        } else {
#pragma unroll 1
            for (int t = tid; t < T; t += NT) {
                load(t, v[0]);
                store(t, v[0]);
            }
        }
    }
}

}  // namespace sbfft
