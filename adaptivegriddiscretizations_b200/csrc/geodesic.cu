// Geodesic backtracking on B200: the distance-to-seed map used by the stopping
// criteria, and the midpoint ODE on the upwind flow, one warp per tip (and
// seven that help it load).
//
// The reference runs its GeodesicODE kernel in chunks of `typical_len` steps
// and restarts each unfinished geodesic from its last point on the host
// (agd/Eikonal/HFM_CUDA/_GetGeodesics.py:111-134).  Here a warp runs all of
// its chunks in one launch; a chunk boundary resets the same state the
// reference's restart resets (stopping-criteria history, cell cache), so the
// paths are the reference's.  The stepping follows
// cuda/Kernel_GeodesicODE.h:164-412 with the precomputed flow of
// GeodesicODE_Opt.h:236-245, in float.
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "agd_common.cuh"
#include "agd_internal.h"

namespace agd {

// ------------------------------------------------------ distance to seeds ---
struct EGeo {
    int nd, shape[3];
    long long n;  // points of one instance
    int nb;       // instances, one after the other
};

// One min-plus pass: out(x) = min over the 3^d neighbours y of min(255, in(y) + k(y - x)),
// k = round(5 |y - x|) (inf_convolution with distance_kernel(1, ndim, uint8, mult=5)),
// or with l1, k = |y - x|_1 (distance_kernel(1, ndim, uint8, ord=1)).
// FROM_MASK: `in` is the mask, read as 0 at its points and 255 elsewhere (the
// first pass); CUT: values above `cut` become 255 (the last pass).
// Threads run along the last axis, blocks stride over the rows of the others.
template <int D, bool FROM_MASK, bool CUT>
__global__ void __launch_bounds__(256) infconv_kernel(EGeo g, const uint8_t *__restrict__ in, int l1, int cut,
                                                      uint8_t *__restrict__ out) {
    constexpr int NK = D == 2 ? 9 : 27;
    const int nlast = g.shape[D - 1];
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= nlast) return;
    const long long nrows = g.n / nlast;
    long long stride[D];
    stride[D - 1] = 1;
    for (int k = D - 2; k >= 0; --k) stride[k] = stride[k + 1] * g.shape[k + 1];
    // rows of all the instances; a neighbour is one of the same instance
    for (long long r = blockIdx.y * (long long)blockDim.y + threadIdx.y; r < nrows * g.nb;
         r += (long long)gridDim.y * blockDim.y) {
        const long long rr = r % nrows;  // row within the instance
        int x[D];
        x[D - 1] = c;
        if (D == 3) {
            x[0] = (int)(rr / g.shape[1]);
            x[1] = (int)(rr - (long long)x[0] * g.shape[1]);
        } else {
            x[0] = (int)rr;
        }
        const long long p = r * nlast + c;
        int best = 255;
#pragma unroll
        for (int ic = 0; ic < NK; ++ic) {
            int n2 = 0;
            bool ok = true;
            long long m = p;
#pragma unroll
            for (int k = 0, q = ic; k < D; ++k, q /= 3) {
                const int o = q % 3 - 1;
                n2 += o * o;
                const int y = x[k] + o;
                ok = ok && y >= 0 && y < g.shape[k];
                m += o * stride[k];
            }
            if (!ok) continue;
            // offsets in {-1, 0, 1}^d: |o|_1 = |o|^2; round(5 |o|) = 0, 5, 7, 9
            const int kv = l1 ? n2 : (n2 == 0 ? 0 : (n2 == 1 ? 5 : (n2 == 2 ? 7 : 9)));
            const int a = FROM_MASK ? (in[m] ? 0 : 255) : in[m];
            best = min(best, (a >= 255 - kv) ? 255 : a + kv);
        }
        if (CUT && best > cut) best = 255;
        out[p] = (uint8_t)best;
    }
}

template <int D>
static void infconv_pass(const EGeo &g, const uint8_t *in, bool from_mask, bool cut_it, int l1, int cut,
                         uint8_t *out, cudaStream_t st) {
    const dim3 block(32, 8);
    const long long nrows = g.n / g.shape[D - 1] * g.nb;
    const dim3 grid((unsigned)((g.shape[D - 1] + 31) / 32), (unsigned)std::min<long long>((nrows + 7) / 8, 16384));
    if (from_mask && cut_it) infconv_kernel<D, true, true><<<grid, block, 0, st>>>(g, in, l1, cut, out);
    else if (from_mask) infconv_kernel<D, true, false><<<grid, block, 0, st>>>(g, in, l1, cut, out);
    else if (cut_it) infconv_kernel<D, false, true><<<grid, block, 0, st>>>(g, in, l1, cut, out);
    else infconv_kernel<D, false, false><<<grid, block, 0, st>>>(g, in, l1, cut, out);
}

// Distance map of a few seeds given by their indices, in one block: `out` is 255
// everywhere, and the box of npasses points around a seed (clipped to the grid)
// gets the least cost of a path of unit, face- and space-diagonal steps (5, 7, 9):
// for sorted offsets a >= b >= c that is c space diagonals, b - c face diagonals
// and a - b unit steps (a diagonal never costs more than the steps it
// replaces), a steps in all.  The min-plus passes give the same values (they
// stop after npasses steps; a box of the grid holds such a path), at a pass over
// the grid each: 57 us for 1024^2 and 6 passes.
template <int D>
__global__ void __launch_bounds__(512) eucl_seeds_kernel(EGeo g, const int *__restrict__ seeds, int nseeds, int npasses, int cut,
                                                         uint8_t *out) {
    const int side = 2 * npasses + 1, box = D == 2 ? side * side : side * side * side;
    for (int s = 0; s < nseeds; ++s) {
        for (int i = threadIdx.x; i < box; i += blockDim.x) {
            int o[3] = {0, 0, 0}, r = i;
            bool in = true;
            long long p = 0;
#pragma unroll
            for (int k = D - 1; k >= 0; --k) {
                o[k] = r % side - npasses;
                r /= side;
            }
#pragma unroll
            for (int k = 0; k < D; ++k) {
                const int x = __ldg(seeds + s * D + k), y = x + o[k];
                in = in && x >= 0 && x < g.shape[k] && y >= 0 && y < g.shape[k];
                p = p * g.shape[k] + y;
            }
            if (!in) continue;
            int a = abs(o[0]), b = abs(o[1]), c = abs(o[2]);
            int hi = max(a, max(b, c)), lo = min(a, min(b, c)), mid = a + b + c - hi - lo;
            const int v = 9 * lo + 7 * (mid - lo) + 5 * (hi - mid);
            if (v > cut || v >= 255) continue;
            if (v < out[p]) out[p] = (uint8_t)v;
        }
        __syncthreads();
    }
}

__global__ void eucl_init_kernel(EGeo g, const uint8_t *mask, uint8_t *out) {
    const long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (p < g.n * g.nb) out[p] = mask[p] ? 0 : 255;
}

__global__ void eucl_cut_kernel(EGeo g, const uint8_t *in, int cut, uint8_t *out) {
    const long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (p < g.n * g.nb) out[p] = in[p] > cut ? 255 : in[p];
}

// ------------------------------------------------------------ geodesics ---
enum { kContinue = 0, kAtSeed, kInWall, kStationnary, kPastSeed, kVanishingFlow };

struct GeoArgs {
    int nd;
    int shape[3], shape_i[3], shape_o[3];
    int size_i;
    long long size_tot;
    const float *u, *fvec, *fwsum;
    const uint8_t *eucl;
    const float *tips;
    int ntips;
    float step, causality;
    int typical_len, max_chunks, eucl_delay, nymin_delay, pastseed_delay;
    float *paths;
    int cap;
    int *lengths;
    int8_t *stops;
};

constexpr int kMaxHist = 256;  // bound on 1 + max(eucl_delay, nymin_delay)

// The point data around the current cell, in shared memory, one per block: the
// values, flow weight sums, flow planes and distance-to-seed bytes of a W^D
// box of grid points, with the stopping criteria's history.  The first warp of a
// block traces one geodesic; the block's eight warps fill the box together
// (asynchronous 4-byte copies for the floats, batched loads for the bytes), the
// others waiting at a barrier between fills.  All lanes of the first warp step
// the same ODE on the same data, so that the control flow stays warp-uniform and
// the steps read shared memory instead of waiting on global loads.  The box is
// refilled, centred on the current cell, when a cell leaves it: after at least
// W/2 - 1 points of travel.
// What bounds it: the steps' serial chain, so nothing else is left on it.  Two
// flow evaluations a step: the cell tested on the exact differences x - cell;
// corners beyond the causality threshold zeroed once per cell; the norm and its
// reciprocal from one approximate reciprocal square root; the history read before
// the evaluation that it is compared with, its two entries that the PastSeed
// test reads kept in registers.  64 tips on Riemann2 1024^2, 1200 steps: 447 us,
// against 647 us with the integer cell, the comparisons per corner, two
// shared-memory round trips a step and fills by one warp.
constexpr int kGeoWarps = 8;
template <int D>
struct GeoWindow {
    static constexpr int W = D == 2 ? 32 : 12;
    static constexpr int WT = D == 2 ? W * W : W * W * W;
    static constexpr int NJ = (WT + 32 * kGeoWarps - 1) / (32 * kGeoWarps);  // points per thread
    // per point: value (+inf outside the grid), flow (0 outside), weight sum and the
    // causality test's margin causality / weight sum
    float u[WT], wsum[WT], margin[WT], flow[D][WT];
    uint8_t eucl[WT];
    int org[D], next[D];  // next: the origin of the box to fill
    int done;             // the geodesic has ended
    int tq[D][W], tr[D][W];  // per axis: tile and in-tile coordinate of org + t, tq -1 outside the grid
    long long nymin_p[kMaxHist];
};

__device__ __forceinline__ void cp_async4(void *smem, const void *gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// Fills the box at S.next (all threads of the block; barriers on both sides).
template <int D>
__device__ __forceinline__ void fill_box(const GeoArgs &A, GeoWindow<D> &S) {
    using Win = GeoWindow<D>;
    constexpr int W = Win::W;
    const int tid = threadIdx.x;
    if (tid < W) {
#pragma unroll
        for (int k = 0; k < D; ++k) {
            const int y = S.next[k] + tid;
            const bool in = y >= 0 && y < A.shape[k];
            S.tq[k][tid] = in ? y / A.shape_i[k] : -1;
            S.tr[k][tid] = in ? y % A.shape_i[k] : 0;
        }
    }
    if (tid < D) S.org[tid] = S.next[tid];
    __syncthreads();
    int e[Win::NJ];
    float ws[Win::NJ];
#pragma unroll
    for (int j = 0; j < Win::NJ; ++j) {
        e[j] = 255;
        ws[j] = 0.f;
        const int p = j * 32 * kGeoWarps + tid;
        if (p >= Win::WT) continue;
        int t[D], r = p;
#pragma unroll
        for (int k = D - 1; k >= 0; --k) { t[k] = r % W; r /= W; }
        bool in = true;
        long long n_o = 0, g = 0;
        int n_i = 0;
#pragma unroll
        for (int k = 0; k < D; ++k) {
            const int q = S.tq[k][t[k]];
            in = in && q >= 0;
            n_o = n_o * A.shape_o[k] + q;
            n_i = n_i * A.shape_i[k] + S.tr[k][t[k]];
            g = g * A.shape[k] + (S.org[k] + t[k]);
        }
        if (!in) {
            S.u[p] = finf();
#pragma unroll
            for (int k = 0; k < D; ++k) S.flow[k][p] = 0.f;
            continue;
        }
        const long long n = n_o * A.size_i + n_i;
        cp_async4(&S.u[p], A.u + n);
#pragma unroll
        for (int k = 0; k < D; ++k) cp_async4(&S.flow[k][p], A.fvec + k * A.size_tot + n);
        e[j] = __ldg(A.eucl + g);
        ws[j] = __ldg(A.fwsum + n);
    }
#pragma unroll
    for (int j = 0; j < Win::NJ; ++j) {
        const int p = j * 32 * kGeoWarps + tid;
        if (p >= Win::WT) continue;
        S.eucl[p] = (uint8_t)e[j];
        S.wsum[p] = ws[j];
        S.margin[p] = A.causality / ws[j];
    }
    cp_async_wait_all();
    __syncthreads();
}

// sqrt(x) and its reciprocal, each correctly rounded (the values of sqrtf and of
// __frcp_rn of that), by one Newton step from the hardware's approximate
// reciprocal square root and two more for the reciprocal (Markstein's
// fused-multiply-add iterations).  Over every float of two binades, at five
// scales, they differ from sqrtf / __frcp_rn nowhere, but for the reciprocal of
// an all-ones mantissa: for that one, and arguments outside [2^-96, 2^96] (and
// NaN), the result is false and the library functions are to be taken.  Shorter
// on the chain of a geodesic's step than the two calls one after the other.
__device__ __forceinline__ bool inverse_sqrt(float x, float &inv) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    float s = x * r;
    s = fmaf(fmaf(-s, s, x), 0.5f * r, s);
    r = fmaf(fmaf(-s, r, 1.f), r, r);
    inv = fmaf(fmaf(-s, r, 1.f), r, r);
    return x >= 0x1p-96f && x <= 0x1p96f && (__float_as_uint(s) & 0x7fffffu) != 0x7fffffu;
}

template <int D>
struct Walker {
    using Win = GeoWindow<D>;
    static constexpr int NC = 1 << D;
    static constexpr int W = Win::W;
    const GeoArgs &A;
    Win &S;
    float xf[D];      // the current cell (floor of the position)
    int org[D];       // origin of the box
    long long nymin;  // grid index of the retained corner (the reference keeps its
                      // bilevel index: the same point, so the same equality tests)
    int eucl_min;     // distance-to-seed byte at that corner
    float flow_c[NC][D];  // the corners' flow, 0 at those beyond the causality threshold

    __device__ __forceinline__ Walker(const GeoArgs &a, Win &s) : A(a), S(s) {
#pragma unroll
        for (int k = 0; k < D; ++k) org[k] = kIntMax / 2;  // an empty box: the first cell fills it
        reset();
    }
    __device__ __forceinline__ void reset() {
#pragma unroll
        for (int k = 0; k < D; ++k) xf[k] = __int_as_float(0x7fffffff);  // NaN: differs from every cell
        nymin = -1;
        eucl_min = 255;
    }
    // A new cell (xf already set): its corners' data, and the corner and threshold
    // of the causality test (Kernel_GeodesicODE.h:164-260).
    __device__ __forceinline__ int enter(const float *wts) {
        int xq[D], li = 0;
        bool covered = true;
#pragma unroll
        for (int k = 0; k < D; ++k) {
            xq[k] = (int)xf[k];
            covered = covered && xq[k] >= org[k] && xq[k] < org[k] + (W - 1);
        }
        if (!covered) {  // refill the box around the cell: the whole block
            __syncwarp();
#pragma unroll
            for (int k = 0; k < D; ++k) {
                org[k] = xq[k] - (W / 2 - 1);
                if (threadIdx.x == 0) S.next[k] = org[k];
            }
            __syncthreads();
            fill_box<D>(A, S);
        }
#pragma unroll
        for (int k = 0; k < D; ++k) li = li * W + (xq[k] - org[k]);
        float dist[NC], mg[NC];
#pragma unroll
        for (int i = 0; i < NC; ++i) {
            const int c = li + corner(i);
            dist[i] = S.u[c];
            mg[i] = S.margin[c];
#pragma unroll
            for (int k = 0; k < D; ++k) flow_c[i][k] = S.flow[k][c];
        }
        float dmin = finf(), m = 0.f;
        int imin = 0;
        const float wthr = 0.5f / NC;
#pragma unroll
        for (int i = 0; i < NC; ++i) {
            const bool less = !(wts[i] < wthr) && dist[i] < dmin;
            imin = less ? i : imin;
            dmin = less ? dist[i] : dmin;
            m = less ? mg[i] : m;
        }
        if (dmin == finf()) return kInWall;
        long long n = 0;
        int lmin = li;
#pragma unroll
        for (int k = 0; k < D; ++k) {
            n = n * A.shape[k] + (xq[k] + ((imin >> k) & 1));
            lmin += ((imin >> k) & 1) * stride(k);
        }
        nymin = n;
        eucl_min = S.eucl[lmin];
        if (S.wsum[lmin] == 0.f) return kAtSeed;
        const float thr = dmin + m;
#pragma unroll
        for (int i = 0; i < NC; ++i)
            if (dist[i] >= thr)
#pragma unroll
                for (int k = 0; k < D; ++k) flow_c[i][k] = 0.f;
        return kContinue;
    }
    // Offsets in the box: of a step along axis k, and of corner i of a cell.
    __device__ __forceinline__ static constexpr int stride(int k) { return k == D - 1 ? 1 : (k == D - 2 ? W : W * W); }
    __device__ __forceinline__ static constexpr int corner(int i) {
        int c = 0;
        for (int k = 0; k < D; ++k) c += ((i >> k) & 1) * stride(k);
        return c;
    }
    // Kernel_GeodesicODE.h:164-260 (NormalizedFlow).  ok: flow is normalised; else
    // normalise() has to finish it (n2: its squared norm).
    __device__ __forceinline__ int normalized_flow(const float *x, float *flow, float &n2, bool &ok) {
        // Still in the cell xf: 0 <= x - xf < 1, where the difference is exact.
        float dx[D], wts[NC];
        bool inside = true;
#pragma unroll
        for (int k = 0; k < D; ++k) {
            dx[k] = x[k] - xf[k];
            inside = inside && dx[k] >= 0.f && dx[k] < 1.f;
        }
        if (!inside) {
#pragma unroll
            for (int k = 0; k < D; ++k) {
                xf[k] = floorf(x[k]);
                dx[k] = x[k] - xf[k];
            }
            weights(dx, wts);
            const int stop = enter(wts);
            if (stop != kContinue) return stop;
        }
        weights(dx, wts);
#pragma unroll
        for (int k = 0; k < D; ++k) flow[k] = 0.f;
#pragma unroll
        for (int i = 0; i < NC; ++i)
#pragma unroll
            for (int k = 0; k < D; ++k) flow[k] += wts[i] * flow_c[i][k];
        n2 = 0.f;
#pragma unroll
        for (int k = 0; k < D; ++k) n2 += flow[k] * flow[k];
        // The correctly rounded float reciprocal: the reference divides in
        // double and rounds to float, which gives the same value (a double
        // quotient has more than 2 x 24 + 2 bits, so the second rounding is
        // innocuous).
        float l;
        ok = inverse_sqrt(n2, l);
        if (!ok) l = 1.f;
#pragma unroll
        for (int k = 0; k < D; ++k) flow[k] *= l;
        return kContinue;
    }
    __device__ __forceinline__ static bool normalise(float *flow, float n2) {
        const float nrm = sqrtf(n2);
        if (!(nrm > 0.f)) return false;
        const float l = __frcp_rn(nrm);
#pragma unroll
        for (int k = 0; k < D; ++k) flow[k] *= l;
        return true;
    }
    __device__ __forceinline__ static void weights(const float *dx, float *wts) {
#pragma unroll
        for (int i = 0; i < NC; ++i) {
            float w = 1.f;
#pragma unroll
            for (int k = 0; k < D; ++k) w *= ((i >> k) & 1) ? dx[k] : 1.f - dx[k];
            wts[i] = w;
        }
    }
};

// One block per tip: the first warp walks, the others help it fill its box.
template <int D>
__global__ void __launch_bounds__(32 * kGeoWarps) geodesic_kernel(const __grid_constant__ GeoArgs A) {
    __shared__ GeoWindow<D> S;
    const int tip = blockIdx.x;
    const int lane = threadIdx.x;
    if (tip >= A.ntips) return;
    if (threadIdx.x == 0) S.done = 0;
    __syncthreads();
    if (threadIdx.x >= 32) {
        while (true) {
            __syncthreads();  // a box is wanted, or the walk has ended
            if (S.done) return;
            fill_box<D>(A, S);
        }
    }
    float *out = A.paths + (long long)tip * A.cap * D;
    float x[D];
#pragma unroll
    for (int k = 0; k < D; ++k) x[k] = A.tips[tip * D + k];
    if (lane == 0)
        for (int k = 0; k < D; ++k) out[k] = x[k];
    int pos = 1, stop = kContinue;
    const int hlen = 1 + max(A.eucl_delay, A.nymin_delay);
    const float half = 0.5f * A.step;
    Walker<D> Wk(A, S);
    for (int chunk = 0; chunk < A.max_chunks; ++chunk) {
        // a chunk starts afresh from the last point, as the reference's restart does
        for (int l = lane; l < hlen; l += 32) S.nymin_p[l] = -1;
        int eucl0 = 255, eucl1 = 255;  // the entries 0 and 1 of the distance history
        __syncwarp();
        Wk.reset();
        // the PastSeed test waits pastseed_delay steps in the first chunk only
        // (_GetGeodesics.py:107-109,133)
        const int ps_delay = chunk == 0 ? A.pastseed_delay : 0;
        int l = 1 % hlen;  // len % hlen
        int len;
        for (len = 1; len < A.typical_len; ++len) {
            float xm[D], flow[D];
            // The history's entry nymin_delay steps back (the current step's own
            // with no delay), read ahead of the evaluation: it is older.
            int ln = l - A.nymin_delay, le = l - A.eucl_delay;
            if (ln < 0) ln += hlen;
            if (le < 0) le += hlen;
            const long long before = S.nymin_p[ln];
            float n2;
            bool ok;
            stop = Wk.normalized_flow(x, flow, n2, ok);
            if (stop != kContinue) break;
            __syncwarp();  // every lane has read the entry that this one may replace
            S.nymin_p[l] = Wk.nymin;  // (the lanes hold the same values)
            eucl0 = l == 0 ? Wk.eucl_min : eucl0;
            eucl1 = l == 1 ? Wk.eucl_min : eucl1;
            const bool still = Wk.nymin == before || ln == l;
            // The reference's subscript is a boolean expression (cuda/Kernel_GeodesicODE.h:331).
            const int cmp = (le != 0) && (len >= ps_delay);
            const bool past = Wk.eucl_min > (cmp ? eucl1 : eucl0);
            if (!ok || still || past) {
                if (!ok && !Wk.normalise(flow, n2)) stop = kVanishingFlow;
                else if (still) stop = kStationnary;
                else if (past) stop = kPastSeed;
                if (stop != kContinue) break;
            }
#pragma unroll
            for (int k = 0; k < D; ++k) xm[k] = half * flow[k] + x[k];
            stop = Wk.normalized_flow(xm, flow, n2, ok);
            if (stop != kContinue) break;
            if (!ok && !Wk.normalise(flow, n2)) {
                stop = kVanishingFlow;
                break;
            }
#pragma unroll
            for (int k = 0; k < D; ++k) x[k] = A.step * flow[k] + x[k];
            if (pos < A.cap) {
                if (lane < D) {
                    float v = x[0];
#pragma unroll
                    for (int k = 1; k < D; ++k) v = lane == k ? x[k] : v;
                    out[pos * D + lane] = v;
                }
                ++pos;
            }
            l = l + 1 == hlen ? 0 : l + 1;
        }
        if (stop != kContinue) break;
        __syncwarp();  // the history is reset only once every lane has read it
    }
    if (lane == 0) {
        A.lengths[tip] = pos;
        A.stops[tip] = (int8_t)stop;
        S.done = 1;
    }
    __syncthreads();  // ends the helpers
}

static inline unsigned nblocks(long long n, int bs) { return (unsigned)((n + bs - 1) / bs); }

// Min-plus distance map in grid layout: 0 at the mask points, 255 elsewhere,
// then `npasses` passes of infconv_kernel and values above `cut` set to 255.
// The first pass reads the mask and the last one applies the cut; the passes
// alternate between `out` and `tmp` so that the last one writes `out`.
// nb instances one after the other, each its own map.  tmp: scratch of nb
// prod(shape) bytes.
int distance_map(int ndim, const int *shape, const uint8_t *mask, int npasses, int cut, bool l1, uint8_t *out,
                 uint8_t *tmp, cudaStream_t st, int nb) {
    if ((ndim != 2 && ndim != 3) || !shape || !mask || !out || !tmp || npasses < 0 || nb < 1)
        return set_error(AGD_STATUS_INVALID, "distance map: bad arguments");
    EGeo g;
    g.nd = ndim;
    g.nb = nb;
    g.n = 1;
    for (int k = 0; k < 3; ++k) g.shape[k] = 1;
    for (int k = 0; k < ndim; ++k) {
        if (shape[k] <= 0) return set_error(AGD_STATUS_INVALID, "distance map: bad shape");
        g.shape[k] = shape[k];
        g.n *= shape[k];
    }
    const int bs = 256;
    if (npasses == 0) {
        eucl_init_kernel<<<nblocks(g.n * nb, bs), bs, 0, st>>>(g, mask, tmp);
        eucl_cut_kernel<<<nblocks(g.n * nb, bs), bs, 0, st>>>(g, tmp, cut, out);
    } else {
        const uint8_t *src = mask;
        for (int it = 0; it < npasses; ++it) {
            uint8_t *dst = ((npasses - 1 - it) % 2 == 0) ? out : tmp;
            if (ndim == 2) infconv_pass<2>(g, src, it == 0, it == npasses - 1, l1 ? 1 : 0, cut, dst, st);
            else infconv_pass<3>(g, src, it == 0, it == npasses - 1, l1 ? 1 : 0, cut, dst, st);
            src = dst;
        }
    }
    const cudaError_t err = cudaGetLastError();
    return err == cudaSuccess ? AGD_STATUS_OK : set_cuda_error("distance map", err);
}

}  // namespace agd

using namespace agd;

extern "C" {

int agd_eucl_map(int ndim, const int *shape, const uint8_t *seed_mask, int npasses, int cut, uint8_t *eucl,
                 uint8_t *tmp, agd_stream_t stream) {
    clear_error();
    return distance_map(ndim, shape, seed_mask, npasses, cut, false, eucl, tmp, (cudaStream_t)stream);
}

int agd_eucl_map_seeds(int ndim, const int *shape, const int32_t *seed_index, int nseeds, int npasses, int cut,
                       uint8_t *eucl, agd_stream_t stream) {
    clear_error();
    if ((ndim != 2 && ndim != 3) || !shape || !eucl || nseeds < 0 || (nseeds > 0 && !seed_index) || npasses < 0 ||
        npasses > 255)
        return set_error(AGD_STATUS_INVALID, "agd_eucl_map_seeds: bad arguments (npasses in [0, 255])");
    EGeo g;
    g.nd = ndim;
    g.nb = 1;
    g.n = 1;
    for (int k = 0; k < 3; ++k) g.shape[k] = 1;
    for (int k = 0; k < ndim; ++k) {
        if (shape[k] <= 0) return set_error(AGD_STATUS_INVALID, "agd_eucl_map_seeds: bad shape");
        g.shape[k] = shape[k];
        g.n *= shape[k];
    }
    cudaStream_t st = (cudaStream_t)stream;
    cudaError_t err = cudaMemsetAsync(eucl, 255, (size_t)g.n, st);
    if (err != cudaSuccess) return set_cuda_error("distance map clear", err);
    if (nseeds > 0) {
        if (ndim == 2) eucl_seeds_kernel<2><<<1, 512, 0, st>>>(g, seed_index, nseeds, npasses, cut, eucl);
        else eucl_seeds_kernel<3><<<1, 512, 0, st>>>(g, seed_index, nseeds, npasses, cut, eucl);
    }
    err = cudaGetLastError();
    return err == cudaSuccess ? AGD_STATUS_OK : set_cuda_error("eucl_seeds", err);
}

int agd_geodesics(const agd_instance *inst, const float *flow_vector, const float *flow_weightsum, const uint8_t *eucl,
                  const float *tips, int ntips, float step, float causality, int typical_len, int max_chunks,
                  int eucl_delay, int nymin_delay, int pastseed_delay, float *paths, int cap, int32_t *lengths,
                  int8_t *stops, agd_stream_t stream) {
    clear_error();
    if (!inst || (inst->ndim != 2 && inst->ndim != 3) || ntips < 0 || !flow_vector || !flow_weightsum || !eucl ||
        !inst->values || typical_len < 2 || max_chunks < 1 || eucl_delay < 0 || nymin_delay < 0 || pastseed_delay < 0 ||
        1 + (eucl_delay > nymin_delay ? eucl_delay : nymin_delay) > kMaxHist || cap < 1 ||
        (ntips > 0 && (!tips || !paths || !lengths || !stops)))
        return set_error(AGD_STATUS_INVALID, "agd_geodesics: bad arguments");
    if (ntips == 0) return AGD_STATUS_OK;
    GeoArgs A;
    A.nd = inst->ndim;
    A.size_i = 1;
    long long so = 1;
    for (int k = 0; k < 3; ++k) { A.shape[k] = A.shape_i[k] = A.shape_o[k] = 1; }
    for (int k = 0; k < A.nd; ++k) {
        if (inst->shape[k] <= 0 || inst->shape_i[k] <= 0) return set_error(AGD_STATUS_INVALID, "bad shape");
        A.shape[k] = inst->shape[k];
        A.shape_i[k] = inst->shape_i[k];
        A.shape_o[k] = (inst->shape[k] + inst->shape_i[k] - 1) / inst->shape_i[k];
        A.size_i *= inst->shape_i[k];
        so *= A.shape_o[k];
    }
    A.size_tot = so * A.size_i;
    A.u = inst->values;
    A.fvec = flow_vector;
    A.fwsum = flow_weightsum;
    A.eucl = eucl;
    A.tips = tips;
    A.ntips = ntips;
    A.step = step;
    A.causality = causality;
    A.typical_len = typical_len;
    A.max_chunks = max_chunks;
    A.eucl_delay = eucl_delay;
    A.nymin_delay = nymin_delay;
    A.pastseed_delay = pastseed_delay;
    A.paths = paths;
    A.cap = cap;
    A.lengths = lengths;
    A.stops = stops;
    // one geodesic per block: the tips spread over the SMs
    if (A.nd == 2) geodesic_kernel<2><<<(unsigned)ntips, 32 * kGeoWarps, 0, (cudaStream_t)stream>>>(A);
    else geodesic_kernel<3><<<(unsigned)ntips, 32 * kGeoWarps, 0, (cudaStream_t)stream>>>(A);
    const cudaError_t err = cudaGetLastError();
    return err == cudaSuccess ? AGD_STATUS_OK : set_cuda_error("geodesics", err);
}

}  // extern "C"
