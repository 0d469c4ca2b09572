// warp_lines.cuh -- in-place line DFTs in shared memory, each line owned by one
// warp.
//
// A warp takes LG lines of LEN = N1 N2 points (rows or columns alike) at a
// time: four lines side by side times N2 (first step) or N1 (second step)
// threads a line, so the exchange between the two steps needs a warp barrier
// instead of a block barrier, and a thread's n2 -- and with it its inter-step
// twiddles -- never changes.  With a row stride of 4 or 12 modulo 16 slots the
// order n2 ^ k1 inside the k1 blocks makes every access of both passes
// conflict-free: in a row pass four lines start 4 slots apart modulo 16 and
// the lanes of a half warp add four neighbouring slots, in a column pass rows
// are 4 slots apart.
#pragma once
#include "fft_engine.cuh"

namespace sbfft {

template <int LEN, int LG_>
struct WarpLines {
    static constexpr int N1 = Split<LEN>::N1, N2 = Split<LEN>::N2, LG = LG_;
    static constexpr int R1 = LG * N2 / 32;         // rounds of the first step
    static constexpr int R2 = (LG * N1 + 31) / 32;  // rounds of the second step
    static_assert(N2 == 4 || N2 == 8, "power of two: the exchange order is an xor");
    static_assert(LG * N2 % 32 == 0 && LEN % LG == 0, "whole rounds and groups");

    int lane;
    float2 tw[N1];  // W_LEN^{k1 n2}

    // table: exp(-2 pi i e / LEN), e < LEN
    __device__ __forceinline__ WarpLines(const float2* __restrict__ table) : lane(threadIdx.x & 31)
    {
#pragma unroll
        for (int k = 0; k < N1; ++k) tw[k] = __ldg(table + k * n2());
    }
    // line and sub-index of a lane in a round of the first and second step;
    // lanes past the last item of the second step repeat it: the same values
    // into the same slots (a predicate around the step costs 300 to 450 bytes
    // of spills at 80 registers)
    __device__ __forceinline__ int l1(int r) const { return (lane & 3) + 4 * ((r * 32 + lane) / (4 * N2)); }
    __device__ __forceinline__ int n2() const { return (lane >> 2) % N2; }
    __device__ __forceinline__ int item2(int r) const { return min(r * 32 + lane, LG * N1 - 1); }
    __device__ __forceinline__ int l2(int r) const { return (item2(r) & 3) + 4 * (item2(r) / (4 * N1)); }
    __device__ __forceinline__ int k1(int r) const { return (item2(r) >> 2) % N1; }
    // o[k] = (m ^ k) S for k < N, one addition each: flipping bit b of k moves
    // m ^ k by +-2^b
    template <int N, int S>
    __device__ __forceinline__ static void xor_offsets(int (&o)[N], int m)
    {
        const int d[3] = {m & 1 ? -S : S, m & 2 ? -2 * S : 2 * S, m & 4 ? -4 * S : 4 * S};
        o[0] = m * S;
#pragma unroll
        for (int k = 1; k < N; ++k) o[k] = o[k & (k - 1)] + d[k & 1 ? 0 : k & 2 ? 1 : 2];
    }
    // inputs in(l, k, round, n1), l the line within the group
    template <typename In>
    __device__ __forceinline__ void load(float2 (&v)[R1][N1], In in) const
    {
#pragma unroll
        for (int r = 0; r < R1; ++r)
#pragma unroll
            for (int n = 0; n < N1; ++n) v[r][n] = in(l1(r), N2 * n + n2());
    }
    // Transforms the inputs v through the slots line(l) + S k of the group's
    // lines; outputs to out(l, k, value, round, k2) once every lane has read
    // its slots.  Lanes must have finished reading the lines before the call.
    template <int DIR, int S, typename Line, typename Out>
    __device__ __forceinline__ void run(float2 (&v)[R1][N1], Line line, Out out) const
    {
#pragma unroll
        for (int r = 0; r < R1; ++r) {
            RegDFT<N1, DIR, LEN, true>::run(v[r], nullptr);
            int o[N1];
            xor_offsets<N1, S>(o, n2());
            float2* p = line(l1(r));
#pragma unroll
            for (int k = 0; k < N1; ++k) {
                float2 w = tw[k];
                if (DIR > 0) w.y = -w.y;
                p[N2 * k * S + o[k]] = k ? cmul(v[r][k], w) : v[r][0];
            }
        }
        __syncwarp();
        float2 u[R2][N2];
#pragma unroll
        for (int r = 0; r < R2; ++r) {
            const int k = k1(r);
            int o[N2];
            xor_offsets<N2, S>(o, k & (N2 - 1));
            const float2* p = line(l2(r)) + N2 * k * S;
#pragma unroll
            for (int j = 0; j < N2; ++j) u[r][j] = p[o[j]];
            RegDFT<N2, DIR, LEN, true>::run(u[r], nullptr);
        }
        __syncwarp();
#pragma unroll
        for (int r = 0; r < R2; ++r)
#pragma unroll
            for (int k = 0; k < N2; ++k) out(l2(r), k1(r) + N1 * k, u[r][k], r, k);
    }
};

}  // namespace sbfft
