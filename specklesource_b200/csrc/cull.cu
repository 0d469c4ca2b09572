// cull.cu -- the cullst passes on the GPU (Cullst/cullst.c:71-101).
//
//  cullSTData (cullSTData.c:13-125): the median test runs in place in raster
//    order, so a cull changes the neighbourhoods of later points.  The GPU
//    solves that recurrence as a parallel fixpoint (cull_fix_first_kernel and
//    revisit lists, exact when it converges); for boxes of more than 128
//    values, or without convergence, it keeps the order with a row
//    wavefront: one warp per grid row
//    (rows claimed in increasing order from a counter, so the row a warp waits
//    on is always held by a running warp), each warp walks its row left to
//    right and, before deciding column j, waits until the previous row has
//    finished column j + bR/2 (transitively every earlier row in the box is
//    done that far).  Both medians (the 1-based k = ngood/2 smallest of the
//    valid neighbours, what Numerical Recipes' select returns) come from a
//    warp-wide radix select over order-preserving float keys.  Waits are
//    bounded: on time-out the kernel records an error and releases its row.
//  cullStats (cullStats.c:19-144), cullSmooth (cullSmooth.c:29-103): one
//    thread per point.  The plane fit is least squares with singular values
//    below 1e-5 * max dropped (svdfit), via the 3x3 normal matrix's Jacobi
//    eigen-decomposition, in double precision.
//  cullls (Cullls/cullls.c:23-56) runs the same kernels: its median pass
//    (cullLSData.c:13-138) adds the slow-flow limits and the NODATA test to
//    the decision rule (StRule), its stats (cullLSStats.c) the quantisation
//    variance, its smoothing (cullLSSmooth.c) is the unweighted box mean of
//    cullls_smooth_kernel, and its islands pass is cullIslands'.
//  cullIslands (cullIslands.c:13-198): union-find labelling (links to the
//    smaller index, so each root is its component's first pixel in raster
//    order), labels numbered by first appearance, bounding boxes, and the cull
//    of components no wider or taller than islandThresh -- except the one
//    labelled last, which the reference's loops (i < maxLabel) skip.
#include <cuda/atomic>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>

#include "capi_internal.h"
#include "chain.cuh"

namespace sbk {

constexpr float kCulled = -2.0e9f;  // (float)-LARGEINT
constexpr float kValidLim = -2.0e9f; // (float)(1 - LARGEINT): 1 - 2e9 rounds to -2e9 in float

__device__ __forceinline__ bool valid_pt(float r, float a) { return r > kValidLim && a > kValidLim; }

// ---------------------------------------------------------------- pre-pass

// The decision rule of one median pass.  cullst (cullSTData.c:80-123): cull
// unless more than nGood valid neighbours and both deviations from the box
// medians within maxA/maxR.  cullls (cullLSData.c:63-134) adds: the limits
// become slowMaxA/slowMaxR when every valid point of the box carries a
// slowMask bit in slowType, and the point's own offA must exceed selfLim.
struct StRule {
    int nGood;
    double maxR, maxA;
    double slowMaxR, slowMaxA;
    const uint8_t* slowType;  // null: no slow-flow test (cullst)
    unsigned slowMask;
    bool selfTest;            // cullls: the point's offA must exceed selfLim (false for NaN)
    double selfLim;
};

struct CullArgs {
    float* offR;
    float* offA;
    const float* corr;
    uint8_t* type;
    const uint8_t* mask;
    int nR, nA;
    int bR, bA;
    StRule rule;
    float corrThresh;
    int singleMT;
    int* rowCounter;
    int* progress;
    int* errFlag;
    unsigned long long* nCulled;
};

__global__ void cull_prepass_kernel(CullArgs a)
{
    chain_begin();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= a.nR * a.nA) return;
    if (a.corr[k] < a.corrThresh) {  // cullSTData.c:38-43
        a.offR[k] = kCulled;
        a.offA[k] = kCulled;
        a.type[k] = 0;
    }
    if (a.mask) {  // :44-61 (singleMT is only honoured with a mask)
        const unsigned char mv = a.mask[k] & 4;
        if (mv > 0 && (signed char)a.type[k] > 2) {
            a.offR[k] = kCulled;
            a.offA[k] = kCulled;
            a.type[k] = 0;
        }
        if (a.singleMT > 0 && (signed char)a.type[k] != a.singleMT) {
            a.offR[k] = kCulled;
            a.offA[k] = kCulled;
            a.type[k] = 0;
        }
    }
}

// ---------------------------------------------------------------- median pass

__device__ __forceinline__ uint32_t fkey(float f)
{
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float fkey_inv(uint32_t k)
{
    const uint32_t u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
    return __uint_as_float(u);
}

// k-th smallest key (1-based) among the lane's NV keys flagged by vmask.
template <int NV>
__device__ __forceinline__ uint32_t warp_kth(const uint32_t (&key)[NV], uint32_t vmask, int k)
{
    uint32_t prefix = 0;
    int below = 0;
#pragma unroll 1
    for (int bit = 31; bit >= 0; --bit) {
        const uint32_t hi = (bit == 31) ? 0u : (0xffffffffu << (bit + 1));
        int c = 0;
#pragma unroll
        for (int v = 0; v < NV; ++v)
            c += ((vmask >> v) & 1u) && ((key[v] & hi) == prefix) && !((key[v] >> bit) & 1u);
        c = __reduce_add_sync(0xffffffffu, c);
        if (below + c < k)
            below += c, prefix |= (1u << bit);
    }
    return prefix;
}

// One point's decision, by a whole warp (uniform result).  kr/ka: the lanes'
// keys of the valid box points (vm), notSlow: this lane saw a valid point
// without the slow bit; oR/oA: the point's own offsets.
template <int NV>
__device__ __forceinline__ bool st_decide(const StRule& r, const uint32_t (&kr)[NV], const uint32_t (&ka)[NV],
                                          uint32_t vm, int ngood, bool notSlow, float oR, float oA)
{
    const bool slow = r.slowType != nullptr && !__any_sync(0xffffffffu, notSlow);
    if ((unsigned)ngood > (unsigned)r.nGood && (!r.selfTest || (double)oA > r.selfLim)) {
        int mid = ngood / 2;
        if (mid < 1) mid = 1;
        const float medR = fkey_inv(warp_kth<NV>(kr, vm, mid));
        const float medA = fkey_inv(warp_kth<NV>(ka, vm, mid));
        const double dA = (double)(oA - medA), dR = (double)(oR - medR);
        return fabs(dA) > (slow ? r.slowMaxA : r.maxA) || fabs(dR) > (slow ? r.slowMaxR : r.maxR);
    }
    return true;
}

template <int NV>
__global__ void cull_median_kernel(CullArgs a, long long spinLimit)
{
    const int lane = threadIdx.x & 31;
    const int hA = a.bA / 2, hR = a.bR / 2;
    const int boxW = 2 * hR + 1;
    cuda::atomic_ref<int, cuda::thread_scope_device> ctr(*a.rowCounter);
    unsigned long long culledHere = 0;
    while (true) {
        int row = 0;
        if (lane == 0) row = ctr.fetch_add(1, cuda::memory_order_relaxed);
        row = __shfl_sync(0xffffffffu, row, 0);
        if (row >= a.nA) break;
        const int i1 = row - hA > 0 ? row - hA : 0;
        const int i2 = row + hA < a.nA - 1 ? row + hA : a.nA - 1;
        bool timedOut = false;
        for (int j = 0; j < a.nR; ++j) {
            // wait for the previous row to finish column j + hR
            if (row > 0) {
                const int need = (j + hR + 1 < a.nR) ? j + hR + 1 : a.nR;
                cuda::atomic_ref<int, cuda::thread_scope_device> prev(a.progress[row - 1]);
                int ok = 1;
                if (lane == 0) {
                    long long spins = 0;
                    while (prev.load(cuda::memory_order_acquire) < need) {
                        if (++spins > spinLimit) {
                            ok = 0;
                            break;
                        }
                        __nanosleep(64);
                    }
                }
                ok = __shfl_sync(0xffffffffu, ok, 0);
                if (!ok) {
                    timedOut = true;
                    break;
                }
                (void)prev.load(cuda::memory_order_acquire);  // every lane acquires what lane 0 saw
                __syncwarp();
            }
            const int j1 = j - hR > 0 ? j - hR : 0;
            const int j2 = j + hR < a.nR - 1 ? j + hR : a.nR - 1;
            const int rows = i2 - i1 + 1, cols = j2 - j1 + 1;
            const int cnt = rows * cols;
            uint32_t kr[NV], ka[NV];
            uint32_t vm = 0;
            bool notSlow = false;
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                const int e = lane + 32 * v;
                kr[v] = ka[v] = 0;
                if (e < cnt) {
                    const int ii = i1 + e / cols, jj = j1 + e % cols;
                    const size_t q = (size_t)ii * a.nR + jj;
                    const float r = __ldcg(&a.offR[q]), az = __ldcg(&a.offA[q]);
                    if (valid_pt(r, az)) {
                        vm |= 1u << v;
                        kr[v] = fkey(r);
                        ka[v] = fkey(az);
                        if (a.rule.slowType && !(a.rule.slowType[q] & a.rule.slowMask)) notSlow = true;
                    }
                }
            }
            int ngood = 0;
#pragma unroll
            for (int v = 0; v < NV; ++v) ngood += (vm >> v) & 1u;
            ngood = __reduce_add_sync(0xffffffffu, ngood);
            const size_t c = (size_t)row * a.nR + j;
            const bool cull =
                st_decide<NV>(a.rule, kr, ka, vm, ngood, notSlow, __ldcg(&a.offR[c]), __ldcg(&a.offA[c]));
            if (lane == 0) {
                if (cull) {
                    a.offR[c] = kCulled;
                    a.offA[c] = kCulled;
                    culledHere++;
                }
                cuda::atomic_ref<int, cuda::thread_scope_device> mine(a.progress[row]);
                mine.store(j + 1, cuda::memory_order_release);
            }
            __syncwarp();
            (void)boxW;
        }
        if (timedOut) {
            if (lane == 0) {
                atomicExch(a.errFlag, 1);
                cuda::atomic_ref<int, cuda::thread_scope_device> mine(a.progress[row]);
                mine.store(a.nR, cuda::memory_order_release);
            }
        }
    }
    if (lane == 0 && culledHere) atomicAdd(a.nCulled, culledHere);
}

// ---------------------------------------------------------------- median pass, parallel fixpoint
// The sequential pass decides point p from the values at the start of the pass
// and from the decisions of the points before p (raster order) in its box:
// C[p] = decide(p, {C[q] : q < p, q in box(p)}).  This recurrence over a DAG
// has exactly one solution, the sequential result.  Jacobi iteration
// C_{t+1} = decide(., C_t) from C_0 = 0 reaches it, and a step that changes
// nothing proves it was reached (a fixpoint of the recurrence is its solution).
// Step t decides only the points on its revisit list (every point at t = 0;
// after that the later box neighbours of the valid points that flipped in step
// t - 1: a point without a value is in nobody's box, so its flips concern
// nobody); any other point has no predecessor that changed, so its decision
// is already C_t's.  The decisions of a step are read from C_t and the flips
// applied afterwards, so every step is exactly a Jacobi step.  offR/offA are
// not modified until the fixpoint is applied.
//
// A decision needs no median, only which side of the limits the median lies
// on: x - m > t holds for the smallest values m of the box and m's rank decides
// (the float difference is monotone in m), so the k-th smallest satisfies it
// exactly when at least k values do; x - m < -t likewise from the top.  One
// count over the box by one thread replaces two 32-step radix selects by a
// warp: the first step on a 1969 x 993 grid, box 5, took 3.8 ms and takes
// 0.07.  The limits are compared in float: for a float d and a double t,
// d > t is d > t rounded down.
//
// Two steps run over the whole chip; the rest, whose lists are short as a rule,
// in one cluster of CTAs that goes on until a list is empty, so a pass has no
// host round trip.  A list of more than kFixLong points, half a list for the
// cluster's 8,192 threads, stops the cluster once its lists add up to more than
// kFixSum: steps over the whole chip follow, kFixBatch of them per host round
// trip, then the cluster again.  With the cluster alone and with this rule, one
// pass: 2000 x 2000 points, box 5, a tenth of them holes, nGood 20: 28.2 and
// 3.7 ms; box 9, nGood 70: 39.7 and 4.5; culls that eat their way in from the
// edges of 1000 x 1000 points (box 9, nGood 60): 23.6 and 14.6.  Lists that
// only start long are left to the cluster: 1969 x 993 points with 8 % outliers,
// box 5, three passes and the statistics 1.84 and 1.85 ms (2.00 to 2.09 without
// kFixSum).  Chains that do not end in kFixSteps steps (1000 rows of 2000
// points, box 3 x 1) take 24 ms either way, the wavefront after them included.
constexpr int kFixSteps = 512;       // bound on the steps of a pass (then the wavefront)
constexpr int kFixCluster = 8;       // CTAs of the tail kernel
constexpr unsigned kFixLong = 4096, kFixSum = 32768;
constexpr int kFixBatch = 16;
constexpr int kFixPasses = 16;       // passes enqueued together (4 KB of counters each)

struct FixArgs {
    const float* offR;
    const float* offA;
    uint8_t* c;              // C_t
    int* list[2];            // revisit lists of even and odd steps
    int* flipped;            // points whose decision flips in this step; ~p without a value
    int* mark;               // the step that listed a point last
    unsigned* nList;         // per step
    unsigned* nFlipped;      // per step
    int* stop;               // 0, or the pass of the group (from 1) that its tail kernel left unfinished
    int* resume;             // the step that pass goes on from
    int nR, nA, hR, hA;
    int nGood;
    float maxR, maxA, slowMaxR, slowMaxA;  // rounded down to float
    const uint8_t* slowType;
    unsigned slowMask;
    bool selfTest;
    double selfLim;
    int pass;
};

// The decision of point (i, j) by one thread.  FIRST: C_0 = 0.
template <bool FIRST, bool SLOW>
__device__ __forceinline__ bool fix_decide(const FixArgs& a, int i, int j, float oR, float oA)
{
    const int i1 = max(i - a.hA, 0), i2 = min(i + a.hA, a.nA - 1);
    const int j1 = max(j - a.hR, 0), j2 = min(j + a.hR, a.nR - 1);
    int n = 0, r1 = 0, r2 = 0, a1 = 0, a2 = 0;  // valid, and beyond the limits on either side
    int s1 = 0, s2 = 0, t1 = 0, t2 = 0;         // the same for the slow-flow limits
    bool notSlow = false;
    for (int ii = i1; ii <= i2; ++ii) {
        const int q0 = ii * a.nR;
        // no branches: the loads of several neighbours go out together
#pragma unroll 4
        for (int jj = j1; jj <= j2; ++jj) {
            const int q = q0 + jj;
            const float r = a.offR[q], z = a.offA[q];
            const bool gone = !FIRST && (ii < i || (ii == i && jj < j)) && __ldcg(a.c + q);
            const bool v = valid_pt(r, z) && !gone;
            const float dr = oR - r, da = oA - z;
            n += v;
            r1 += v && dr > a.maxR;
            r2 += v && dr < -a.maxR;
            a1 += v && da > a.maxA;
            a2 += v && da < -a.maxA;
            if (SLOW) {
                notSlow = notSlow || (v && !(__ldg(a.slowType + q) & a.slowMask));
                s1 += v && dr > a.slowMaxR;
                s2 += v && dr < -a.slowMaxR;
                t1 += v && da > a.slowMaxA;
                t2 += v && da < -a.slowMaxA;
            }
        }
    }
    if (!((unsigned)n > (unsigned)a.nGood && (!a.selfTest || (double)oA > a.selfLim))) return true;
    const int k = max(n / 2, 1);
    if (SLOW && !notSlow) return s1 >= k || n - s2 < k || t1 >= k || n - t2 < k;
    return r1 >= k || n - r2 < k || a1 >= k || n - a2 < k;
}

// Appends to a list with one atomic per warp; every lane of the warp calls.
__device__ __forceinline__ void warp_append(bool yes, int v, int* list, unsigned* n)
{
    const unsigned m = __ballot_sync(0xffffffffu, yes);
    if (!m) return;
    const int lane = threadIdx.x & 31;
    unsigned base = 0;
    if (lane == 0) base = atomicAdd(n, (unsigned)__popc(m));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (yes) list[base + __popc(m & ((1u << lane) - 1u))] = v;
}

// Launch of a block per tile of 32 x 8 points.  Rows of tiles past 65,535, where
// the second launch dimension ends (grids of 524,281 rows and more), go into
// the third; numbering the tiles in one dimension cost the first step 3 % for
// the division.
static dim3 cull_tiles(int nR, int nA)
{
    const unsigned ny = (nA + 7) / 8;
    return dim3((nR + 31) / 32, std::min(ny, 65535u), (ny + 65534) / 65535);
}
__device__ __forceinline__ int2 tile_origin()
{
    return make_int2(blockIdx.x * 32, (blockIdx.z * 65535 + blockIdx.y) * 8);
}

// Step 0: every point; a thread each, 32 x 8 points a block.
template <bool SLOW>
__global__ void __launch_bounds__(256) cull_fix_first_kernel(FixArgs a)
{
    chain_begin();
    if (*a.stop) return;  // uniform
    const int2 t = tile_origin();
    const int j = t.x + (threadIdx.x & 31), i = t.y + (threadIdx.x >> 5);
    bool cull = false, ok = false;
    int p = 0;
    if (i < a.nA && j < a.nR) {
        p = i * a.nR + j;
        const float oR = a.offR[p], oA = a.offA[p];
        ok = valid_pt(oR, oA);
        cull = fix_decide<true, SLOW>(a, i, j, oR, oA);
        a.c[p] = cull;
    }
    warp_append(cull && ok, p, a.flipped, a.nFlipped);
}

template <bool SLOW>
__device__ __forceinline__ void fix_decide_list(const FixArgs& a, int step, int tid, int nt)
{
    const unsigned n = __ldcg(a.nList + step);
    const int* list = a.list[step & 1];
    for (unsigned t0 = tid & ~31; t0 < n; t0 += nt) {
        const unsigned t = t0 + (tid & 31);
        bool flip = false;
        int v = 0;
        if (t < n) {
            const int p = __ldcg(list + t);
            const float oR = a.offR[p], oA = a.offA[p];
            flip = fix_decide<false, SLOW>(a, p / a.nR, p % a.nR, oR, oA) != (__ldcg(a.c + p) != 0);
            v = valid_pt(oR, oA) ? p : ~p;
        }
        warp_append(flip, v, a.flipped, a.nFlipped + step);
    }
}

// Applies a step's flips to C (step 0 wrote its own) and lists the points to
// decide next: the later points (raster order) whose box holds a flipped valid
// point, each once per step.  One warp per flipped point.
__device__ __forceinline__ void fix_apply_list(const FixArgs& a, int step, int warp, int nw)
{
    const int lane = threadIdx.x & 31;
    const unsigned nf = __ldcg(a.nFlipped + step);
    const int stamp = a.pass * (kFixSteps + 2) + step + 1;
    for (unsigned k = warp; k < nf; k += nw) {
        int q = __ldcg(a.flipped + k);
        const bool ok = q >= 0;
        q = ok ? q : ~q;
        if (step > 0 && lane == 0) a.c[q] = !__ldcg(a.c + q);
        if (!ok) continue;
        const int i = q / a.nR, j = q % a.nR;
        const int i2 = min(i + a.hA, a.nA - 1);
        const int j1 = max(j - a.hR, 0), j2 = min(j + a.hR, a.nR - 1);
        const int cols = j2 - j1 + 1;
        const int sameRow = j2 - j;                 // (i, j+1 .. j2)
        const int total = sameRow + (i2 - i) * cols;  // then rows i+1 .. i2, columns j1 .. j2
        for (int b = 0; b < total; b += 32) {
            const int e = b + lane;
            int pp = -1;
            if (e < total) {
                const int y = e < sameRow ? i : i + 1 + (e - sameRow) / cols;
                const int x = e < sameRow ? j + 1 + e : j1 + (e - sameRow) % cols;
                pp = y * a.nR + x;
                if (atomicExch(a.mark + pp, stamp) == stamp) pp = -1;  // listed already in this step
            }
            warp_append(pp >= 0, pp, a.list[(step + 1) & 1], a.nList + step + 1);
        }
    }
}

template <bool SLOW>
__global__ void __launch_bounds__(256) cull_fix_list_kernel(FixArgs a, int step)
{
    chain_begin();
    if (*a.stop) return;
    fix_decide_list<SLOW>(a, step, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

__global__ void __launch_bounds__(256) cull_fix_apply_kernel(FixArgs a, int step)
{
    chain_begin();
    if (*a.stop) return;
    fix_apply_list(a, step, (blockIdx.x * blockDim.x + threadIdx.x) >> 5, (gridDim.x * blockDim.x) >> 5);
}

// Steps from `step` on until a list is empty or long or the steps run out, in
// one cluster.  C, the lists and the counters are read past L1 (other CTAs of
// the cluster write them); the cluster barriers order the two halves of a step.
template <bool SLOW>
__global__ void __cluster_dims__(kFixCluster, 1, 1) __launch_bounds__(1024) cull_fix_tail_kernel(FixArgs a, int step)
{
    chain_begin();
    if (*a.stop) return;
    auto sync = [] {
        __threadfence();
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    };
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
    unsigned sum = 0;
    for (;; ++step) {
        const unsigned n = __ldcg(a.nList + step);  // the same value in every thread
        if (n == 0) return;
        sum += n;
        if ((n > kFixLong && sum > kFixSum) || step >= kFixSteps) break;
        fix_decide_list<SLOW>(a, step, tid, nt);
        sync();
        fix_apply_list(a, step, tid >> 5, nt >> 5);
        sync();
    }
    if (tid == 0) {
        *a.resume = step;
        *a.stop = a.pass + 1;
    }
}

// Writes the culls of the converged pass; counts them.
__global__ void cull_apply_kernel(float* offR, float* offA, const uint8_t* c, long long n,
                                  unsigned long long* nCulled, const int* stop)
{
    chain_begin();
    if (*stop) return;
    unsigned long long k = 0;
    for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < n;
         p += (long long)gridDim.x * blockDim.x) {
        if (c[p]) {
            offR[p] = kCulled;
            offA[p] = kCulled;
            k++;
        }
    }
    k = __reduce_add_sync(0xffffffffu, (unsigned)k);
    if ((threadIdx.x & 31) == 0 && k) atomicAdd(nCulled, k);
}

// ---------------------------------------------------------------- stats

// Jacobi eigen-decomposition of a symmetric 3x3 matrix.  A rotation is left
// out where A_PQ^2 <= 1e-34 A_PP A_QQ: its angle, at most 1e-17 sqrt(A_QQ /
// A_PP), changes neither eigenvalues nor vectors in double.  (Rotating until
// the off-diagonals are exactly zero runs into the 60-sweep bound: from about
// 1e-160 on, theta^2 overflows and the rotation does nothing.)
__device__ void jacobi3(double A[3][3], double e[3], double V[3][3])
{
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) V[i][j] = (i == j);
#pragma unroll 1
    for (int sweep = 0; sweep < 60; sweep++) {
        bool any = false;
#pragma unroll
        for (int pq = 0; pq < 3; pq++) {
            const int P = pq == 2 ? 1 : 0, Q = pq == 0 ? 1 : 2;
            if (A[P][Q] * A[P][Q] <= 1e-34 * fabs(A[P][P] * A[Q][Q])) continue;
            any = true;
            const double theta = (A[Q][Q] - A[P][P]) / (2.0 * A[P][Q]);
            const double t = (theta >= 0 ? 1.0 : -1.0) / (fabs(theta) + sqrt(theta * theta + 1.0));
            const double cs = 1.0 / sqrt(t * t + 1.0), sn = t * cs;
#pragma unroll
            for (int k = 0; k < 3; k++) {
                const double akp = A[k][P], akq = A[k][Q];
                A[k][P] = cs * akp - sn * akq;
                A[k][Q] = sn * akp + cs * akq;
            }
#pragma unroll
            for (int k = 0; k < 3; k++) {
                const double apk = A[P][k], aqk = A[Q][k];
                A[P][k] = cs * apk - sn * aqk;
                A[Q][k] = sn * apk + cs * aqk;
            }
#pragma unroll
            for (int k = 0; k < 3; k++) {
                const double vkp = V[k][P], vkq = V[k][Q];
                V[k][P] = cs * vkp - sn * vkq;
                V[k][Q] = sn * vkp + cs * vkq;
            }
        }
        if (!any) break;
    }
#pragma unroll
    for (int i = 0; i < 3; i++) e[i] = A[i][i];
}

// svdfit's solution from the normal equations of the basis (x0, ii, jj):
// sums m = n, ii, jj, ii^2, ii jj, jj^2 (exact) and b = offset, offset ii,
// offset jj over the valid points of a box.
__device__ void plane_solve(double x0, const double (&m)[6], const double (&b)[3], double coef[3])
{
    const double c01 = x0 * m[1], c02 = x0 * m[2];
    double AtA[3][3] = {{x0 * x0 * m[0], c01, c02}, {c01, m[3], m[4]}, {c02, m[4], m[5]}};
    const double Atb[3] = {x0 * b[0], b[1], b[2]};
    double e[3], V[3][3];
    jacobi3(AtA, e, V);
    double s[3], smax = 0;
#pragma unroll
    for (int u = 0; u < 3; u++) {
        s[u] = e[u] > 0 ? sqrt(e[u]) : 0.0;
        smax = s[u] > smax ? s[u] : smax;
    }
    const double thresh = 1.0e-5 * smax;
    coef[0] = coef[1] = coef[2] = 0.0;
#pragma unroll
    for (int u = 0; u < 3; u++) {
        if (s[u] < thresh || s[u] == 0.0) continue;
        const double proj = V[0][u] * Atb[0] + V[1][u] * Atb[1] + V[2][u] * Atb[2];
        const double w = proj / (s[u] * s[u]);
#pragma unroll
        for (int v = 0; v < 3; v++) coef[v] += V[v][u] * w;
    }
}

struct StatsArgs {
    const float* offR;
    const float* offA;
    float* sigmaR;
    float* sigmaA;
    int nR, nA;
    double qvar;  // cullls: quantisation variance (1/NOVER)^2/12 added before the root; 0 for cullst
};

// A thread per point, 32 x 8 points a block, the 40 x 16 offsets they read in
// shared memory (points without a value as kCulled).  Both offsets' fits share
// the position sums, which are integers; one pass over the box gathers what
// means and fits need, a second takes the residuals.  Bound by the double
// divisions and roots of the two eigen-decompositions.
constexpr int ST_BOX = 4;  // 9 x 9, cullStats.c:38-39
__global__ void __launch_bounds__(256) cull_stats_kernel(StatsArgs a)
{
    chain_begin();
    constexpr int TX = 32, TY = 8, SX = TX + 2 * ST_BOX, SY = TY + 2 * ST_BOX;
    __shared__ float2 tile[SY][SX];
    const int2 org = tile_origin();
    const int x0 = org.x, y0 = org.y;
    for (int e = threadIdx.x; e < SX * SY; e += 256) {
        const int x = x0 - ST_BOX + e % SX, y = y0 - ST_BOX + e / SX;
        float2 v = make_float2(kCulled, kCulled);
        if (x >= 0 && x < a.nR && y >= 0 && y < a.nA) {
            v = make_float2(a.offR[(size_t)y * a.nR + x], a.offA[(size_t)y * a.nR + x]);
            if (!valid_pt(v.x, v.y)) v = make_float2(kCulled, kCulled);
        }
        tile[e / SX][e % SX] = v;
    }
    __syncthreads();
    const int tx = threadIdx.x % TX, ty = threadIdx.x / TX;
    const int i = y0 + ty, j = x0 + tx;
    if (i >= a.nA || j >= a.nR) return;
    const size_t k = (size_t)i * a.nR + j;
    unsigned ngood = 0;
    double meanA = 0.0, meanR = 0.0;
    int si = 0, sj = 0, sii = 0, sij = 0, sjj = 0;  // positions from (i, j)
    double bR[2] = {0, 0}, bA[2] = {0, 0};          // offset times position from (i, j)
    for (int y = -ST_BOX; y <= ST_BOX; y++)
#pragma unroll
        for (int x = -ST_BOX; x <= ST_BOX; x++) {
            const float2 v = tile[ty + ST_BOX + y][tx + ST_BOX + x];
            if (v.x > kValidLim) {
                const double r = v.x, z = v.y;
                ngood++;
                meanR += r;
                meanA += z;
                si += y;
                sj += x;
                sii += y * y;
                sij += x * y;
                sjj += x * x;
                bR[0] += r * y;
                bR[1] += r * x;
                bA[0] += z * y;
                bA[1] += z * x;
            }
        }
    const double sumR = meanR, sumA = meanA;
    meanA /= (double)ngood;
    meanR /= (double)ngood;
    double aR[4] = {0, 0, 0, 0}, aA[4] = {0, 0, 0, 0};
    if (ngood > 8) {
        const double n = ngood, di = i, dj = j;
        // sums about the origin from the sums about (i, j); the position sums are exact
        const double m[6] = {n, n * di + si, n * dj + sj, n * di * di + 2.0 * di * si + sii,
                             n * di * dj + di * sj + dj * si + sij, n * dj * dj + 2.0 * dj * sj + sjj};
        const double tR[3] = {sumR, sumR * di + bR[0], sumR * dj + bR[1]};
        const double tA[3] = {sumA, sumA * di + bA[0], sumA * dj + bA[1]};
        double c[3];
        plane_solve((double)(float)meanR, m, tR, c);
        aR[1] = c[0] * meanR;
        aR[2] = c[1];
        aR[3] = c[2];
        plane_solve((double)(float)meanA, m, tA, c);
        aA[1] = c[0] * meanA;
        aA[2] = c[1];
        aA[3] = c[2];
    }
    meanA = meanR = 0.0;
    double varR = 0.0, varA = 0.0;
    for (int y = -ST_BOX; y <= ST_BOX; y++) {
        const double fi = (double)(float)(i + y);
#pragma unroll
        for (int x = -ST_BOX; x <= ST_BOX; x++) {
            const float2 v = tile[ty + ST_BOX + y][tx + ST_BOX + x];
            if (v.x > kValidLim) {
                const double fj = (double)(float)(j + x);
                const float oR = (float)((double)v.x - (aR[1] + aR[2] * fi + aR[3] * fj));
                const float oA = (float)((double)v.y - (aA[1] + aA[2] * fi + aA[3] * fj));
                meanA += oA;
                meanR += oR;
                varA += (double)(oA * oA);
                varR += (double)(oR * oR);
            }
        }
    }
    if (ngood > 8 && a.offR[k] > kValidLim) {
        float sA = (float)(varA / (float)(ngood - 3));
        float sR = (float)(varR / (float)(ngood - 3));
        sA = (float)((double)sA - meanA * meanA / (float)((ngood - 3) * ngood));
        sR = (float)((double)sR - meanR * meanR / (float)((ngood - 3) * ngood));
        sA = (float)(0.00001 > (double)sA ? 0.00001 : (double)sA);
        sR = (float)(0.00001 > (double)sR ? 0.00001 : (double)sR);
        if (a.qvar != 0.0) {  // cullLSStats.c:147-148
            sR = (float)((double)sR + a.qvar);
            sA = (float)((double)sA + a.qvar);
        }
        a.sigmaA[k] = (float)sqrt((double)sA);
        a.sigmaR[k] = (float)sqrt((double)sR);
    } else {
        a.sigmaA[k] = kCulled;
        a.sigmaR[k] = kCulled;
    }
}

// ---------------------------------------------------------------- smooth

struct SmoothArgs {
    const float* offR;
    const float* offA;
    const uint8_t* type;
    float* sigmaR;
    float* sigmaA;
    float* offRS;
    float* offAS;
    int nR, nA, sR, sA;
};

__device__ __forceinline__ float sweight(int m, int s)
{
    const float w2 = (float)((float)s / 2.0 - 0.01);  // cullSmooth.c:10-27
    return (m < -w2 || m > w2) ? 0.5f : 1.0f;
}

__global__ void cull_smooth_kernel(SmoothArgs a)
{
    chain_begin();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= a.nR * a.nA) return;
    const int i = k / a.nR, j = k % a.nR;
    const float nlooks[4] = {0.0f, 1.0f, 0.25f, 0.015f};
    const int i1 = i - a.sA / 2 > 0 ? i - a.sA / 2 : 0, i2 = i + a.sA / 2 < a.nA - 1 ? i + a.sA / 2 : a.nA - 1;
    const int j1 = j - a.sR / 2 > 0 ? j - a.sR / 2 : 0, j2 = j + a.sR / 2 < a.nR - 1 ? j + a.sR / 2 : a.nR - 1;
    double ngood = 0, meanA = 0.0, meanR = 0.0;
    float nLooksEff = 0.0f;
    for (int ii = i1; ii <= i2; ii++) {
        const float wa = sweight(ii - i, a.sA);
        for (int jj = j1; jj <= j2; jj++) {
            const size_t q = (size_t)ii * a.nR + jj;
            if (valid_pt(a.offR[q], a.offA[q])) {
                const double w = (double)(wa * sweight(jj - j, a.sR));
                ngood = __dadd_rn(ngood, w);
                nLooksEff = (float)__dadd_rn((double)nLooksEff, __dmul_rn(w, (double)nlooks[(int)(signed char)a.type[q] & 3]));
                meanA = __dadd_rn(meanA, __dmul_rn(w, (double)a.offA[q]));
                meanR = __dadd_rn(meanR, __dmul_rn(w, (double)a.offR[q]));
            }
        }
    }
    if (((ngood > 1) || (a.sA == 1) || (a.sR == 1)) && a.offR[k] > kValidLim && a.sigmaA[k] > kValidLim) {
        nLooksEff = (float)((double)nLooksEff > 1. ? (double)nLooksEff : 1.);
        a.sigmaA[k] = (float)((double)a.sigmaA[k] / sqrt((double)nLooksEff));
        a.sigmaR[k] = (float)((double)a.sigmaR[k] / sqrt((double)nLooksEff));
        a.offRS[k] = (float)(meanR / (float)ngood);
        a.offAS[k] = (float)(meanA / (float)ngood);
    } else {
        a.offRS[k] = kCulled;
        a.offAS[k] = kCulled;
    }
}

// cullLSSmooth.c:29-70: the unweighted mean over the sA x sR box, one look
// per valid point.
__global__ void cullls_smooth_kernel(SmoothArgs a)
{
    chain_begin();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= a.nR * a.nA) return;
    const int i = k / a.nR, j = k % a.nR;
    const int i1 = i - a.sA / 2 > 0 ? i - a.sA / 2 : 0, i2 = i + a.sA / 2 < a.nA - 1 ? i + a.sA / 2 : a.nA - 1;
    const int j1 = j - a.sR / 2 > 0 ? j - a.sR / 2 : 0, j2 = j + a.sR / 2 < a.nR - 1 ? j + a.sR / 2 : a.nR - 1;
    unsigned ngood = 0;
    float nLooksEff = 0.0f;
    double meanA = 0.0, meanR = 0.0;
    for (int ii = i1; ii <= i2; ii++)
        for (int jj = j1; jj <= j2; jj++) {
            const size_t q = (size_t)ii * a.nR + jj;
            if (valid_pt(a.offR[q], a.offA[q])) {
                ngood++;
                nLooksEff += 1.0f;
                meanA += (double)a.offA[q];
                meanR += (double)a.offR[q];
            }
        }
    if (((ngood > 1) || (a.sA == 1) || (a.sR == 1)) && a.offR[k] > kValidLim && a.sigmaA[k] > kValidLim) {
        nLooksEff = (float)((double)nLooksEff > 1. ? (double)nLooksEff : 1.);
        a.sigmaA[k] = (float)((double)a.sigmaA[k] / sqrt((double)nLooksEff));
        a.sigmaR[k] = (float)((double)a.sigmaR[k] / sqrt((double)nLooksEff));
        a.offRS[k] = (float)(meanR / (float)ngood);
        a.offAS[k] = (float)(meanA / (float)ngood);
    } else {
        a.offRS[k] = kCulled;
        a.offAS[k] = kCulled;
    }
}

// cullLSData.c:36-57 (first pass): valid points and points with data.
__global__ void cullls_count_kernel(const float* offR, const float* offA, const uint8_t* type, unsigned noDataMask,
                                    long long n, unsigned long long* cnt)
{
    chain_begin();
    unsigned long long nv = 0, nd = 0;
    for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < n;
         p += (long long)gridDim.x * blockDim.x) {
        nv += valid_pt(offR[p], offA[p]);
        nd += (type[p] & noDataMask) == 0;
    }
    nv = __reduce_add_sync(0xffffffffu, (unsigned)nv);
    nd = __reduce_add_sync(0xffffffffu, (unsigned)nd);
    if ((threadIdx.x & 31) == 0) {
        if (nv) atomicAdd(&cnt[0], nv);
        if (nd) atomicAdd(&cnt[1], nd);
    }
}

// ---------------------------------------------------------------- sim offsets

__global__ void cull_sim_kernel(float* offR, float* offA, const float* simR, const float* simA, int n, float sign)
{
    chain_begin();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    // cullst.c:109-121 with its local LARGEINT = -2e9: offA < 2e9 + 1
    if ((double)offA[k] < (2e9 + 1) && (double)simA[k] < (2e9 + 1)) {
        offA[k] = offA[k] + sign * simA[k];
        offR[k] = offR[k] + sign * simR[k];
    }
}

// ---------------------------------------------------------------- islands

__device__ __forceinline__ int uf_find(int* par, int x)
{
    int p = par[x];
    while (p != x) {
        const int g = par[p];
        if (g < p) par[x] = g;  // path halving (only towards smaller indices)
        x = p;
        p = par[x];
    }
    return x;
}

__device__ void uf_union(int* par, int a, int b)
{
    bool done = false;
    while (!done) {
        a = uf_find(par, a);
        b = uf_find(par, b);
        if (a == b) return;
        if (a < b) {
            const int t = a;
            a = b;
            b = t;
        }
        // link the larger root a under the smaller root b
        const int old = atomicMin(&par[a], b);
        done = (old == a);
        a = old;
    }
}

struct IslandArgs {
    float* offRS;
    float* offAS;
    int* par;
    int* minX;
    int* maxX;
    int* minY;
    int* maxY;
    int* lastRoot;
    unsigned long long* counts;  // [0] islands culled, [1] points culled
    int nR, nA, conn8, thresh;
};

__global__ void isl_init_kernel(IslandArgs a)
{
    chain_begin();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= a.nR * a.nA) return;
    const float minRegion = (float)(-2000000000 + 1000);  // cullIslands.c:62
    a.par[k] = a.offRS[k] >= minRegion ? k : -1;
    a.minX[k] = a.minY[k] = 0x7fffffff;
    a.maxX[k] = a.maxY[k] = -0x7fffffff;
}

__global__ void isl_union_kernel(IslandArgs a)
{
    chain_begin();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= a.nR * a.nA || a.par[k] < 0) return;
    const int i = k / a.nR, j = k % a.nR;
    if (j > 0 && a.par[k - 1] >= 0) uf_union(a.par, k, k - 1);
    if (i > 0 && a.par[k - a.nR] >= 0) uf_union(a.par, k, k - a.nR);
    if (a.conn8 && i > 0) {
        if (j > 0 && a.par[k - a.nR - 1] >= 0) uf_union(a.par, k, k - a.nR - 1);
        if (j < a.nR - 1 && a.par[k - a.nR + 1] >= 0) uf_union(a.par, k, k - a.nR + 1);
    }
}

__global__ void isl_flatten_kernel(IslandArgs a)
{
    chain_begin();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= a.nR * a.nA || a.par[k] < 0) return;
    int r = k;
    while (a.par[r] != r) r = a.par[r];
    a.par[k] = r;
    const int i = k / a.nR, j = k % a.nR;
    // the bounds only move outwards, so a stale read costs at most an atomic
    // too many: one per new extreme instead of four per pixel of a component
    if (j < a.minX[r]) atomicMin(&a.minX[r], j);
    if (j > a.maxX[r]) atomicMax(&a.maxX[r], j);
    if (i < a.minY[r]) atomicMin(&a.minY[r], i);
    if (i > a.maxY[r]) atomicMax(&a.maxY[r], i);
    if (r == k) atomicMax(a.lastRoot, k);  // the component labelled last
}

__global__ void isl_cull_kernel(IslandArgs a)
{
    chain_begin();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= a.nR * a.nA || a.par[k] < 0) return;
    const int r = a.par[k];
    if (r == *a.lastRoot) return;
    if ((a.maxX[r] - a.minX[r]) > a.thresh || (a.maxY[r] - a.minY[r]) > a.thresh) return;
    a.offRS[k] = kCulled;
    if (a.offAS) a.offAS[k] = kCulled;
    atomicAdd(&a.counts[1], 1ull);
    if (r == k) atomicAdd(&a.counts[0], 1ull);
}

}  // namespace sbk

// ======================================================================= C ABI

using namespace sbk;

namespace {

struct CullDev {
    float *offR, *offA, *corr, *simR, *simA, *offRS, *offAS, *sigmaR, *sigmaA;
    uint8_t *type, *mask;
};

// What the passes read, from either entry point (cullst or cullls).
struct CullJob {
    int nR, nA, bR, bA, sR, sA, islandThresh, connectivity;
    StRule rule;          // rule.slowType is set to the device type grid (cullls)
    bool prepass;         // cullst: corr threshold and mask tests before the median pass
    float corrThresh;
    int singleMT;
    double qvar;          // cullls stats: quantisation variance
    bool lsSmooth;        // cullls smoothing
};

CullJob job_of(const sb_cull_params* p)
{
    CullJob j;
    j.nR = p->nR; j.nA = p->nA; j.bR = p->bR; j.bA = p->bA; j.sR = p->sR; j.sA = p->sA;
    j.islandThresh = p->islandThresh; j.connectivity = p->connectivity;
    j.rule.nGood = p->nGood;
    j.rule.maxR = p->maxR; j.rule.maxA = p->maxA;
    j.rule.slowMaxR = p->maxR; j.rule.slowMaxA = p->maxA;
    j.rule.slowType = nullptr;
    j.rule.slowMask = 0;
    j.rule.selfTest = false;
    j.rule.selfLim = 0.0;
    j.prepass = true;
    j.corrThresh = p->corrThresh;
    j.singleMT = p->singleMT;
    j.qvar = 0.0;
    j.lsSmooth = false;
    return j;
}

// cullLSData.c:99-117: limits where every valid neighbour is slow-moving,
// 40 m/yr over deltaT in pixels, at least 0.2; cullLSStats.c:147-148.
CullJob job_of(const sb_cullls_params* p)
{
    CullJob j;
    j.nR = p->nx; j.nA = p->ny; j.bR = p->boxSize; j.bA = p->boxSize; j.sR = p->sX; j.sA = p->sY;
    j.islandThresh = p->islandThresh; j.connectivity = p->connectivity;
    j.rule.nGood = p->nGood;
    j.rule.maxR = p->maxX; j.rule.maxA = p->maxY;
    double mx = 40.0 / 365. * p->deltaT, my = mx;
    mx /= p->dx;
    my /= p->dy;
    j.rule.slowMaxR = mx > 0.2 ? mx : 0.2;
    j.rule.slowMaxA = my > 0.2 ? my : 0.2;
    j.rule.slowType = nullptr;
    j.rule.slowMask = p->slowVelMask;
    j.rule.selfTest = true;
    j.rule.selfLim = p->noDataLimit;
    j.prepass = false;
    j.corrThresh = 0.0f;
    j.singleMT = 0;
    j.qvar = ((1.0 / p->nOver) * (1.0 / p->nOver)) / 12.;
    j.lsSmooth = true;
    return j;
}

int cull_check(sb_context* c, const sb_cull_params* p, const sb_cull_data* d)
{
    if (!c) return SB_ERR_ARG;
    if (!p || !d) return sb_ctx_fail(c, SB_ERR_ARG, "null params or data");
    if (p->nR <= 0 || p->nA <= 0) return sb_ctx_fail(c, SB_ERR_ARG, "empty grid");
    if ((long long)p->nR * p->nA > (1LL << 30)) return sb_ctx_fail(c, SB_ERR_ARG, "grid too large");
    if (!d->offR || !d->offA || !d->corr || !d->type) return sb_ctx_fail(c, SB_ERR_ARG, "null input grid");
    if (p->bR < 0 || p->bA < 0 || (p->bR / 2 * 2 + 1) * (p->bA / 2 * 2 + 1) > 32 * 32)
        return sb_ctx_fail(c, SB_ERR_UNSUPPORTED, "cull box larger than 32 x 32");
    if (p->useSim && (!d->simR || !d->simA)) return sb_ctx_fail(c, SB_ERR_ARG, "useSim needs simR/simA");
    return SB_OK;
}

#define CKC(call, what)                                              \
    do {                                                             \
        cudaError_t _e = (call);                                     \
        if (_e != cudaSuccess) return sb_ctx_cuda(c, _e, what);      \
    } while (0)

// The grids of a host job that are (also) outputs, in one buffer.
char* grid_block(sb_context* c, size_t n, CullDev* v, cudaError_t* e)
{
    Packed pk;
    size_t at[6];
    for (size_t& a : at) a = pk.add(n * sizeof(float));
    const size_t atT = pk.add(n);
    char* g = (char*)sb_ctx_buf(c, "c_grids", pk.bytes(), e);
    if (!g) return nullptr;
    v->offR = (float*)(g + at[0]);
    v->offA = (float*)(g + at[1]);
    v->offRS = (float*)(g + at[2]);
    v->offAS = (float*)(g + at[3]);
    v->sigmaR = (float*)(g + at[4]);
    v->sigmaA = (float*)(g + at[5]);
    v->type = (uint8_t*)(g + atT);
    return g;
}

// Device views of the job's grids (copies host inputs in).  whole: every pass
// runs, so the outputs are written before anything reads them.
int cull_stage_in(sb_context* c, const sb_cull_params* p, sb_cull_data* d, CullDev* v, bool whole)
{
    const size_t n = (size_t)p->nR * p->nA, fb = n * sizeof(float);
    cudaError_t e;
    if (d->onDevice) {
        v->offR = d->offR; v->offA = d->offA; v->corr = (float*)d->corr; v->type = d->type;
        v->mask = (uint8_t*)d->mask; v->simR = (float*)d->simR; v->simA = (float*)d->simA;
        v->offRS = d->offRS; v->offAS = d->offAS; v->sigmaR = d->sigmaR; v->sigmaA = d->sigmaA;
        if (!v->offRS) v->offRS = (float*)sb_ctx_buf(c, "c_offRS", fb, &e);
        if (!v->offAS) v->offAS = (float*)sb_ctx_buf(c, "c_offAS", fb, &e);
        if (!v->sigmaR) v->sigmaR = (float*)sb_ctx_buf(c, "c_sigmaR", fb, &e);
        if (!v->sigmaA) v->sigmaA = (float*)sb_ctx_buf(c, "c_sigmaA", fb, &e);
        return SB_OK;
    }
    char* grids = grid_block(c, n, v, &e);
    v->corr = (float*)sb_ctx_buf(c, "c_corr", fb, &e);
    v->mask = d->mask ? (uint8_t*)sb_ctx_buf(c, "c_mask", n, &e) : nullptr;
    v->simR = p->useSim ? (float*)sb_ctx_buf(c, "c_simR", fb, &e) : nullptr;
    v->simA = p->useSim ? (float*)sb_ctx_buf(c, "c_simA", fb, &e) : nullptr;
    if (!grids || !v->corr || (d->mask && !v->mask) || (p->useSim && (!v->simR || !v->simA)))
        return sb_ctx_fail(c, SB_ERR_NOMEM, "device allocation failed");
    cudaStream_t s = c->stream;
    CKC(cudaMemcpyAsync(v->offR, d->offR, fb, cudaMemcpyHostToDevice, s), "h2d");
    CKC(cudaMemcpyAsync(v->offA, d->offA, fb, cudaMemcpyHostToDevice, s), "h2d");
    CKC(cudaMemcpyAsync(v->corr, d->corr, fb, cudaMemcpyHostToDevice, s), "h2d");
    CKC(cudaMemcpyAsync(v->type, d->type, n, cudaMemcpyHostToDevice, s), "h2d");
    if (d->mask) CKC(cudaMemcpyAsync(v->mask, d->mask, n, cudaMemcpyHostToDevice, s), "h2d");
    if (p->useSim) {
        CKC(cudaMemcpyAsync(v->simR, d->simR, fb, cudaMemcpyHostToDevice, s), "h2d");
        CKC(cudaMemcpyAsync(v->simA, d->simA, fb, cudaMemcpyHostToDevice, s), "h2d");
    }
    if (whole) return SB_OK;
    // outputs that a single pass reads (stats -> smooth -> islands)
    if (d->sigmaR) CKC(cudaMemcpyAsync(v->sigmaR, d->sigmaR, fb, cudaMemcpyHostToDevice, s), "h2d");
    if (d->sigmaA) CKC(cudaMemcpyAsync(v->sigmaA, d->sigmaA, fb, cudaMemcpyHostToDevice, s), "h2d");
    if (d->offRS) CKC(cudaMemcpyAsync(v->offRS, d->offRS, fb, cudaMemcpyHostToDevice, s), "h2d");
    if (d->offAS) CKC(cudaMemcpyAsync(v->offAS, d->offAS, fb, cudaMemcpyHostToDevice, s), "h2d");
    return SB_OK;
}

int cull_stage_out(OutCopies* oc, const sb_cull_params* p, sb_cull_data* d, const CullDev* v)
{
    if (d->onDevice) return SB_OK;
    const size_t n = (size_t)p->nR * p->nA, fb = n * sizeof(float);
    int rc;
    if ((rc = oc->add(d->offR, v->offR, fb)) != SB_OK) return rc;
    if ((rc = oc->add(d->offA, v->offA, fb)) != SB_OK) return rc;
    if (d->offRS && (rc = oc->add(d->offRS, v->offRS, fb)) != SB_OK) return rc;
    if (d->offAS && (rc = oc->add(d->offAS, v->offAS, fb)) != SB_OK) return rc;
    if (d->sigmaR && (rc = oc->add(d->sigmaR, v->sigmaR, fb)) != SB_OK) return rc;
    if (d->sigmaA && (rc = oc->add(d->sigmaA, v->sigmaA, fb)) != SB_OK) return rc;
    return oc->add(d->type, v->type, n);
}

// Largest float not above t: d > t for a float d is d > float_down(t).
float float_down(double t)
{
    const float f = (float)t;
    return (double)f > t ? nextafterf(f, -INFINITY) : f;
}

// One wavefront pass (after the pre-pass).
int run_st_wavefront(sb_context* c, const CullArgs& a, int nv, int64_t* nCulledOut)
{
    cudaStream_t s = c->stream;
    CKC(cudaMemsetAsync(a.rowCounter, 0, sizeof(int) * 4 + sizeof(unsigned long long) * 2, s), "memset");
    CKC(cudaMemsetAsync(a.progress, 0, sizeof(int) * (size_t)a.nA, s), "memset");
    // one warp per row in flight; enough warps for the wavefront depth
    int warps = c->numSM * 32;
    if (warps > a.nA) warps = a.nA;
    const int threads = 128, blocks = (warps * 32 + threads - 1) / threads;
    const long long spinLimit = c->waitNaps;  // 64 ns naps per wait (sb_set_wait_limit)
    switch (nv) {
    case 1: cull_median_kernel<1><<<blocks, threads, 0, s>>>(a, spinLimit); break;
    case 2: cull_median_kernel<2><<<blocks, threads, 0, s>>>(a, spinLimit); break;
    case 3: cull_median_kernel<3><<<blocks, threads, 0, s>>>(a, spinLimit); break;
    case 4: cull_median_kernel<4><<<blocks, threads, 0, s>>>(a, spinLimit); break;
    case 5: case 6: case 7: case 8: cull_median_kernel<8><<<blocks, threads, 0, s>>>(a, spinLimit); break;
    case 9: case 10: case 11: case 12: case 13: case 14: case 15: case 16:
        cull_median_kernel<16><<<blocks, threads, 0, s>>>(a, spinLimit); break;
    default: cull_median_kernel<32><<<blocks, threads, 0, s>>>(a, spinLimit); break;
    }
    CKC(cudaGetLastError(), "cull_median");
    c->launches++;
    int hostCtl[2];
    unsigned long long culled = 0;
    CKC(cudaMemcpyAsync(hostCtl, a.rowCounter, sizeof(int) * 2, cudaMemcpyDeviceToHost, s), "d2h");
    CKC(cudaMemcpyAsync(&culled, a.nCulled, sizeof(culled), cudaMemcpyDeviceToHost, s), "d2h");
    CKC(cudaStreamSynchronize(s), "cull_median");
    if (hostCtl[1]) return sb_ctx_fail(c, SB_ERR_TIMEOUT, "cullSTData wavefront wait timed out");
    *nCulledOut = (int64_t)culled;
    return SB_OK;
}

// Steps [step, step + n) of a pass over the whole chip (step 0: every point),
// the tail kernel and, when that converged, the culls, without a host round trip.
template <bool SLOW>
cudaError_t launch_fix_steps(sb_context* c, const FixArgs& f, int step, int n, float* offR, float* offA,
                             unsigned long long* nCulled)
{
    cudaStream_t s = c->stream;
    const int wide = c->numSM * 8, end = step + n;
    for (; step < end; ++step) {
        if (step == 0)
            chain(cull_fix_first_kernel<SLOW>, cull_tiles(f.nR, f.nA), 256, 0, s, f);
        else
            chain(cull_fix_list_kernel<SLOW>, wide, 256, 0, s, f, step);
        chain(cull_fix_apply_kernel, wide, 256, 0, s, f, step);
    }
    chain(cull_fix_tail_kernel<SLOW>, kFixCluster, 1024, 0, s, f, end);
    const long long points = (long long)f.nR * f.nA;
    chain(cull_apply_kernel, (int)std::min<long long>((points + 255) / 256, c->numSM * 16), 256, 0, s, offR, offA, f.c,
          points, nCulled, f.stop);
    c->launches += 2 * n + 2;
    return cudaGetLastError();
}

// nPasses median passes, kFixPasses of them enqueued as fixpoints at a time.  A
// pass that its tail kernel leaves unfinished stops the ones behind it and goes
// on by itself; where its steps run out the wavefront kernel does it.  Then the
// rest follow.
int run_st_data(sb_context* c, const CullJob& p, const CullDev* v, int nPasses, int64_t* nCulledOut)
{
    const long long n = (long long)p.nR * p.nA;
    cudaError_t e;
    int* ctl = (int*)sb_ctx_buf(c, "c_ctl", sizeof(int) * 4 + sizeof(unsigned long long) * 2, &e);
    int* progress = (int*)sb_ctx_buf(c, "c_progress", sizeof(int) * (size_t)p.nA, &e);
    if (!ctl || !progress) return sb_ctx_fail(c, SB_ERR_NOMEM, "device allocation failed");
    CullArgs a;
    a.offR = v->offR; a.offA = v->offA; a.corr = v->corr; a.type = v->type; a.mask = v->mask;
    a.nR = p.nR; a.nA = p.nA; a.bR = p.bR; a.bA = p.bA;
    a.rule = p.rule;
    a.corrThresh = p.corrThresh; a.singleMT = p.singleMT;
    a.rowCounter = ctl;
    a.errFlag = ctl + 1;
    a.nCulled = (unsigned long long*)(ctl + 4);
    a.progress = progress;
    cudaStream_t s = c->stream;
    if (p.prepass) {  // of later passes: nothing left to change
        chain(cull_prepass_kernel, (int)((n + 255) / 256), 256, 0, s, a);
        CKC(cudaGetLastError(), "cull_prepass");
        c->launches++;
    }
    const int box = (p.bR / 2 * 2 + 1) * (p.bA / 2 * 2 + 1);
    const int nv = (box + 31) / 32;
    int done = 0, rc;
    if (nv > 4)
        for (; done < nPasses; ++done)
            if ((rc = run_st_wavefront(c, a, nv, nCulledOut)) != SB_OK) return rc;
    if (done == nPasses) return SB_OK;
    // C (bytes), then int arrays: two revisit lists, the flips, the marks
    uint8_t* C = (uint8_t*)sb_ctx_buf(c, "c_fix", (size_t)n + 16 + (size_t)n * 4 * sizeof(int), &e);
    // stop flag, culled counts, then list and flip counts per pass and step
    const int group = std::min(nPasses, kFixPasses);
    const size_t perPass = 2 * (kFixSteps + 2);
    const size_t cntBytes = 16 + (sizeof(unsigned long long) + sizeof(unsigned) * perPass) * group;
    unsigned* cnt = (unsigned*)sb_ctx_buf(c, "c_fixcnt", cntBytes, &e);
    if (!C || !cnt) return sb_ctx_fail(c, SB_ERR_NOMEM, "device allocation failed");
    unsigned long long* culled = (unsigned long long*)(cnt + 4);
    unsigned* steps = (unsigned*)(culled + group);
    int* ibase = (int*)(((uintptr_t)(C + n) + 15) & ~(uintptr_t)15);
    FixArgs f;
    f.offR = v->offR; f.offA = v->offA;
    f.c = C;
    f.list[0] = ibase;
    f.list[1] = ibase + n;
    f.flipped = ibase + 2 * n;
    f.mark = ibase + 3 * n;
    f.stop = (int*)cnt;
    f.resume = f.stop + 1;
    f.nR = p.nR; f.nA = p.nA; f.hR = p.bR / 2; f.hA = p.bA / 2;
    f.nGood = p.rule.nGood;
    f.maxR = float_down(p.rule.maxR);
    f.maxA = float_down(p.rule.maxA);
    f.slowMaxR = float_down(p.rule.slowMaxR);
    f.slowMaxA = float_down(p.rule.slowMaxA);
    f.slowType = p.rule.slowType;
    f.slowMask = p.rule.slowMask;
    f.selfTest = p.rule.selfTest;
    f.selfLim = p.rule.selfLim;
    auto steps_of = [&](int pass, int step, int count) {
        f.pass = pass;
        f.nList = steps + perPass * pass;
        f.nFlipped = f.nList + kFixSteps + 2;
        return f.slowType ? launch_fix_steps<true>(c, f, step, count, v->offR, v->offA, culled + pass)
                          : launch_fix_steps<false>(c, f, step, count, v->offR, v->offA, culled + pass);
    };
    while (done < nPasses) {
        CKC(cudaMemsetAsync(f.mark, 0, (size_t)n * sizeof(int), s), "memset");
        CKC(cudaMemsetAsync(cnt, 0, cntBytes, s), "memset");
        int pass = std::min(group, nPasses - done) - 1;  // the last of the group
        for (int k = 0; k <= pass; ++k) CKC(steps_of(k, 0, 2), "cull_fix");
        for (;;) {
            struct {
                int stop, resume, unused[2];
                unsigned long long culled[kFixPasses];
            } at;
            CKC(cudaMemcpyAsync(&at, cnt, 16 + sizeof(unsigned long long) * group, cudaMemcpyDeviceToHost, s), "d2h");
            CKC(cudaStreamSynchronize(s), "cull_fix");
            if (at.stop) pass = at.stop - 1;
            *nCulledOut = (int64_t)at.culled[pass];
            if (at.stop == 0) break;
            if (at.resume >= kFixSteps) {
                if ((rc = run_st_wavefront(c, a, nv, nCulledOut)) != SB_OK) return rc;
                break;
            }
            CKC(cudaMemsetAsync(f.stop, 0, sizeof(int), s), "memset");
            CKC(steps_of(pass, at.resume, std::min(kFixBatch, kFixSteps - at.resume)), "cull_fix");
        }
        done += pass + 1;
    }
    return SB_OK;
}

int run_stats(sb_context* c, const CullJob& p, const CullDev* v)
{
    StatsArgs a{v->offR, v->offA, v->sigmaR, v->sigmaA, p.nR, p.nA, p.qvar};
    chain(cull_stats_kernel, cull_tiles(p.nR, p.nA), 256, 0, c->stream, a);
    c->launches++;
    return sb_ctx_cuda(c, cudaGetLastError(), "cull_stats");
}

int run_smooth(sb_context* c, const CullJob& p, const CullDev* v)
{
    const int n = p.nR * p.nA;
    SmoothArgs a{v->offR, v->offA, v->type, v->sigmaR, v->sigmaA, v->offRS, v->offAS, p.nR, p.nA, p.sR, p.sA};
    if (p.lsSmooth)
        chain(cullls_smooth_kernel, (n + 127) / 128, 128, 0, c->stream, a);
    else
        chain(cull_smooth_kernel, (n + 127) / 128, 128, 0, c->stream, a);
    c->launches++;
    return sb_ctx_cuda(c, cudaGetLastError(), "cull_smooth");
}

int run_islands(sb_context* c, const CullJob& p, const CullDev* v, int64_t* nIslands, int64_t* nIslandPoints)
{
    const int n = p.nR * p.nA;
    cudaError_t e;
    int* ws = (int*)sb_ctx_buf(c, "c_isl", sizeof(int) * (size_t)n * 5 + 64, &e);
    unsigned long long* cntd = (unsigned long long*)sb_ctx_buf(c, "c_isl_cnt", 4 * sizeof(unsigned long long), &e);
    if (!ws || !cntd) return sb_ctx_fail(c, SB_ERR_NOMEM, "device allocation failed");
    IslandArgs a;
    a.offRS = v->offRS;
    a.offAS = v->offAS;
    a.par = ws;
    a.minX = ws + (size_t)n;
    a.maxX = ws + 2 * (size_t)n;
    a.minY = ws + 3 * (size_t)n;
    a.maxY = ws + 4 * (size_t)n;
    a.lastRoot = ws + 5 * (size_t)n;
    a.counts = cntd;
    a.nR = p.nR;
    a.nA = p.nA;
    a.conn8 = p.connectivity != 4;
    a.thresh = p.islandThresh;
    cudaStream_t s = c->stream;
    CKC(cudaMemsetAsync(a.lastRoot, 0xff, sizeof(int), s), "memset");
    CKC(cudaMemsetAsync(a.counts, 0, 2 * sizeof(unsigned long long), s), "memset");
    const int g = (n + 255) / 256;
    chain(isl_init_kernel, g, 256, 0, s, a);
    chain(isl_union_kernel, g, 256, 0, s, a);
    chain(isl_flatten_kernel, g, 256, 0, s, a);
    chain(isl_cull_kernel, g, 256, 0, s, a);
    c->launches += 4;
    CKC(cudaGetLastError(), "cull_islands");
    unsigned long long cnt[2];
    CKC(cudaMemcpyAsync(cnt, a.counts, sizeof(cnt), cudaMemcpyDeviceToHost, s), "d2h");
    CKC(cudaStreamSynchronize(s), "cull_islands");
    *nIslands = (int64_t)cnt[0];
    *nIslandPoints = (int64_t)cnt[1];
    return SB_OK;
}

int run_sim(sb_context* c, const CullJob& p, const CullDev* v, float sign)
{
    const int n = p.nR * p.nA;
    chain(cull_sim_kernel, (n + 255) / 256, 256, 0, c->stream, v->offR, v->offA, v->simR, v->simA, n, sign);
    c->launches++;
    return sb_ctx_cuda(c, cudaGetLastError(), "cull_sim");
}

// Stage in, run the passes, stage out, with the context's four timing events.
template <typename In, typename F, typename Out>
int cull_run(sb_context* c, In stageIn, F body, Out stageOut)
{
    int rc;
    c->err.clear();
    c->launches = 0;
    CKC(cudaSetDevice(c->device), "cudaSetDevice");
    cudaEventRecord(c->ev[0], c->stream);
    CullDev v;
    if ((rc = stageIn(&v)) != SB_OK) return rc;
    cudaEventRecord(c->ev[1], c->stream);
    if ((rc = body(v)) != SB_OK) return rc;
    cudaEventRecord(c->ev[2], c->stream);
    OutCopies oc(c);
    if ((rc = stageOut(&oc, &v)) != SB_OK) return rc;
    if ((rc = oc.finish("cull")) != SB_OK) return rc;
    cudaEventElapsedTime(&c->timing[0], c->ev[0], c->ev[3]);
    cudaEventElapsedTime(&c->timing[1], c->ev[0], c->ev[1]);
    cudaEventElapsedTime(&c->timing[2], c->ev[1], c->ev[2]);
    cudaEventElapsedTime(&c->timing[3], c->ev[2], c->ev[3]);
    return SB_OK;
}

template <typename F>
int cull_entry(sb_context* c, const sb_cull_params* p, sb_cull_data* d, F body, bool whole = false)
{
    int rc = cull_check(c, p, d);
    if (rc != SB_OK) return rc;
    return cull_run(
        c, [&](CullDev* v) { return cull_stage_in(c, p, d, v, whole); }, body,
        [&](OutCopies* oc, const CullDev* v) { return cull_stage_out(oc, p, d, v); });
}

int cullls_check(sb_context* c, const sb_cullls_params* p, const sb_cullls_data* d)
{
    if (!c) return SB_ERR_ARG;
    if (!p || !d) return sb_ctx_fail(c, SB_ERR_ARG, "null params or data");
    if (p->nx <= 0 || p->ny <= 0) return sb_ctx_fail(c, SB_ERR_ARG, "empty grid");
    if ((long long)p->nx * p->ny > (1LL << 30)) return sb_ctx_fail(c, SB_ERR_ARG, "grid too large");
    if (!d->X || !d->Y || !d->type) return sb_ctx_fail(c, SB_ERR_ARG, "null input grid");
    if (p->boxSize < 0 || (p->boxSize / 2 * 2 + 1) * (p->boxSize / 2 * 2 + 1) > 32 * 32)
        return sb_ctx_fail(c, SB_ERR_UNSUPPORTED, "cull box larger than 32 x 32");
    if (!(p->nOver > 0.0)) return sb_ctx_fail(c, SB_ERR_ARG, "nOver (lstrack's NOVER) must be positive");
    if (!(p->dx > 0.0) || !(p->dy > 0.0)) return sb_ctx_fail(c, SB_ERR_ARG, "pixel sizes dx, dy must be positive");
    return SB_OK;
}

int cullls_stage_in(sb_context* c, const sb_cullls_params* p, sb_cullls_data* d, CullDev* v)
{
    const size_t n = (size_t)p->nx * p->ny, fb = n * sizeof(float);
    cudaError_t e;
    *v = CullDev{};
    if (d->onDevice) {
        v->offR = d->X; v->offA = d->Y; v->type = (uint8_t*)d->type;
        v->offRS = d->XS; v->offAS = d->YS; v->sigmaR = d->sigmaX; v->sigmaA = d->sigmaY;
    } else {
        if (!grid_block(c, n, v, &e)) return sb_ctx_fail(c, SB_ERR_NOMEM, "device allocation failed");
        CKC(cudaMemcpyAsync(v->offR, d->X, fb, cudaMemcpyHostToDevice, c->stream), "h2d");
        CKC(cudaMemcpyAsync(v->offA, d->Y, fb, cudaMemcpyHostToDevice, c->stream), "h2d");
        CKC(cudaMemcpyAsync(v->type, d->type, n, cudaMemcpyHostToDevice, c->stream), "h2d");
    }
    if (!v->offRS) v->offRS = (float*)sb_ctx_buf(c, "c_offRS", fb, &e);
    if (!v->offAS) v->offAS = (float*)sb_ctx_buf(c, "c_offAS", fb, &e);
    if (!v->sigmaR) v->sigmaR = (float*)sb_ctx_buf(c, "c_sigmaR", fb, &e);
    if (!v->sigmaA) v->sigmaA = (float*)sb_ctx_buf(c, "c_sigmaA", fb, &e);
    if (!v->offRS || !v->offAS || !v->sigmaR || !v->sigmaA)
        return sb_ctx_fail(c, SB_ERR_NOMEM, "device allocation failed");
    return SB_OK;
}

int cullls_stage_out(OutCopies* oc, const sb_cullls_params* p, sb_cullls_data* d, const CullDev* v)
{
    if (d->onDevice) return SB_OK;
    const size_t fb = (size_t)p->nx * p->ny * sizeof(float);
    int rc;
    if ((rc = oc->add(d->X, v->offR, fb)) != SB_OK) return rc;
    if ((rc = oc->add(d->Y, v->offA, fb)) != SB_OK) return rc;
    if (d->XS && (rc = oc->add(d->XS, v->offRS, fb)) != SB_OK) return rc;
    if (d->YS && (rc = oc->add(d->YS, v->offAS, fb)) != SB_OK) return rc;
    if (d->sigmaX && (rc = oc->add(d->sigmaX, v->sigmaR, fb)) != SB_OK) return rc;
    if (d->sigmaY && (rc = oc->add(d->sigmaY, v->sigmaA, fb)) != SB_OK) return rc;
    return SB_OK;
}

// nAttempt / nMatch of the first cullLSData pass (cullLSData.c:36-57).
int run_ls_counts(sb_context* c, const sb_cullls_params* p, const CullDev* v, sb_cullls_data* d)
{
    const long long n = (long long)p->nx * p->ny;
    cudaError_t e;
    unsigned long long* cnt = (unsigned long long*)sb_ctx_buf(c, "c_lscnt", 2 * sizeof(unsigned long long), &e);
    if (!cnt) return sb_ctx_fail(c, SB_ERR_NOMEM, "device allocation failed");
    cudaStream_t s = c->stream;
    CKC(cudaMemsetAsync(cnt, 0, 2 * sizeof(unsigned long long), s), "memset");
    long long blocks = (n + 255) / 256;
    if (blocks > (long long)c->numSM * 16) blocks = (long long)c->numSM * 16;
    chain(cullls_count_kernel, (int)blocks, 256, 0, s, v->offR, v->offA, v->type, p->noDataMask, n, cnt);
    CKC(cudaGetLastError(), "cullls_count");
    c->launches++;
    unsigned long long h[2];
    CKC(cudaMemcpyAsync(h, cnt, sizeof(h), cudaMemcpyDeviceToHost, s), "d2h");
    CKC(cudaStreamSynchronize(s), "cullls_count");
    d->nMatch = (int64_t)h[0];
    d->nAttempt = (int64_t)h[1];
    return SB_OK;
}

}  // namespace

extern "C" int sb_cull(sb_context* c, const sb_cull_params* p, sb_cull_data* d)
{
    return cull_entry(c, p, d, [&](const CullDev& v) {
        int rc;
        const CullJob j = job_of(p);
        if (p->useSim && (rc = run_sim(c, j, &v, -1.0f)) != SB_OK) return rc;
        const int passes = p->nCullPasses > 0 ? p->nCullPasses : 3;
        if ((rc = run_st_data(c, j, &v, passes, &d->nCulled)) != SB_OK) return rc;
        if ((rc = run_stats(c, j, &v)) != SB_OK) return rc;
        if (p->useSim && (rc = run_sim(c, j, &v, 1.0f)) != SB_OK) return rc;
        if ((rc = run_smooth(c, j, &v)) != SB_OK) return rc;
        if (p->islandThresh > 0 && (rc = run_islands(c, j, &v, &d->nIslands, &d->nIslandPoints)) != SB_OK)
            return rc;
        return SB_OK;
    }, true);
}

extern "C" int sb_cull_st_data(sb_context* c, const sb_cull_params* p, sb_cull_data* d)
{
    return cull_entry(c, p, d, [&](const CullDev& v) { return run_st_data(c, job_of(p), &v, 1, &d->nCulled); });
}

extern "C" int sb_cull_stats(sb_context* c, const sb_cull_params* p, sb_cull_data* d)
{
    return cull_entry(c, p, d, [&](const CullDev& v) { return run_stats(c, job_of(p), &v); });
}

extern "C" int sb_cull_smooth(sb_context* c, const sb_cull_params* p, sb_cull_data* d)
{
    return cull_entry(c, p, d, [&](const CullDev& v) { return run_smooth(c, job_of(p), &v); });
}

extern "C" int sb_cull_islands(sb_context* c, const sb_cull_params* p, sb_cull_data* d)
{
    return cull_entry(
        c, p, d, [&](const CullDev& v) { return run_islands(c, job_of(p), &v, &d->nIslands, &d->nIslandPoints); });
}

extern "C" int sb_cullls(sb_context* c, const sb_cullls_params* p, sb_cullls_data* d)
{
    int rc = cullls_check(c, p, d);
    if (rc != SB_OK) return rc;
    return cull_run(
        c, [&](CullDev* v) { return cullls_stage_in(c, p, d, v); },
        [&](const CullDev& v) {
            int r;
            CullJob j = job_of(p);
            j.rule.slowType = v.type;
            if ((r = run_ls_counts(c, p, &v, d)) != SB_OK) return r;
            const int passes = p->nCullPasses > 0 ? p->nCullPasses : 3;
            if ((r = run_st_data(c, j, &v, passes, &d->nCulled)) != SB_OK) return r;
            if ((r = run_stats(c, j, &v)) != SB_OK) return r;
            if ((r = run_smooth(c, j, &v)) != SB_OK) return r;
            d->nIslands = d->nIslandPoints = 0;
            if (p->islandThresh > 0 && (r = run_islands(c, j, &v, &d->nIslands, &d->nIslandPoints)) != SB_OK)
                return r;
            return SB_OK;
        },
        [&](OutCopies* oc, const CullDev* v) { return cullls_stage_out(oc, p, d, v); });
}
