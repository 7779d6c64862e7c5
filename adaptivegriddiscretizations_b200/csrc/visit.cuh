// The tile visit of the eikonal solver (Isotropic, Diagonal, Riemann, Rander; 2D
// and 3D) and the visitor that the schedulers of sched.cuh run.
//
#pragma once
#include <cuda_runtime.h>

#include <algorithm>

#include "families.cuh"

namespace agd {

// ------------------------------------------------------- stencil cache ---
// Offsets of the Selling stencil packed in one 32-bit word: two 15-bit signed
// fields in 2D, three 10-bit signed fields in 3D; bits 30 and 31 flag the
// neighbours x - e and x + e hidden by a wall (kHideShift).
constexpr int kHideShift = 30;
template <int D>
__device__ __forceinline__ bool pack_offset(const int *e, int &word) {
    if constexpr (D == 2) {
        if (e[0] < -16384 || e[0] > 16383 || e[1] < -16384 || e[1] > 16383) return false;
        word = (e[0] & 0x7fff) | ((e[1] & 0x7fff) << 15);
        return true;
    } else {
        for (int c = 0; c < 3; ++c)
            if (e[c] < -512 || e[c] > 511) return false;
        word = (e[0] & 0x3ff) | ((e[1] & 0x3ff) << 10) | ((e[2] & 0x3ff) << 20);
        return true;
    }
}
template <int D>
__device__ __forceinline__ void unpack_offset(int word, int *e) {
    if (D == 2) {
        e[0] = (word << 17) >> 17;
        e[1] = (word << 2) >> 17;
    } else {
        e[0] = (word << 22) >> 22;
        e[1] = (word << 12) >> 22;
        e[2] = (word << 2) >> 22;
    }
}

// Bilevel index of grid point y of instance I (tile shape at run time).
__device__ __forceinline__ long long bilevel_index_rt(const Inst &I, int D, const int *y) {
    long long n_o = 0, n_i = 0;
    for (int k = 0; k < D; ++k) {
        const int s = I.a.shape_i[k], yo = y[k] / s;
        n_o = n_o * I.shape_o[k] + yo;
        n_i = n_i * s + (y[k] - yo * s);
    }
    return n_o * I.size_i + n_i;
}

// Wall distance at grid point y (255 outside the grid, as at padding).
template <int D, class Index>
__device__ __forceinline__ int wall_dist_at(const agd_instance &A, const int *y, Index &&index) {
    bool in = true;
#pragma unroll
    for (int c = 0; c < D; ++c) in = in && y[c] >= 0 && y[c] < A.shape[c];
    return in ? (int)__ldg(A.wall_dist + index(y)) : 255;
}

// Hidden-neighbour bits (bit s: the neighbour x + (2s - 1) e) of offset e at
// grid point xt, wd0 the wall distance there (cuda/Walls.h:18-50 for both signs).
template <int D, class Index>
__device__ __forceinline__ unsigned hidden_bits(const agd_instance &A, int wd0, const int *xt, const int *e,
                                                Index &&index) {
    if (wd0 == 255) return 0u;
    unsigned h = 0;
#pragma unroll
    for (int s = 0; s < 2; ++s) {
        int v[3] = {0, 0, 0};
#pragma unroll
        for (int c = 0; c < D; ++c) v[c] = (2 * s - 1) * e[c];
        if (!visible<D>(wd0, xt, v, [&](const int *y) { return wall_dist_at<D>(A, y, index); })) h |= 1u << s;
    }
    return h;
}

// Instance of global tile t (binary search over the tile bases).
__device__ __forceinline__ const Inst &inst_of_tile(const Inst *insts, int ninst, int t) {
    int lo = 0, hi = ninst - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (insts[mid].tile_base <= t) lo = mid; else hi = mid - 1;
    }
    return insts[lo];
}

// Selling stencil of every point of the Riemann instances of a launch, once per
// solve (the reference recomputes it at each visit, cuda/Riemann_.h:23-29).
// One warp per tile.
template <int D>
__global__ void stencil_kernel(const Inst *insts, int ninst, int total_tiles, Ctrl *ctrl) {
    constexpr int SD = D * (D + 1) / 2;
    const int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (t >= total_tiles) return;
    int lo = 0, hi = ninst - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (insts[mid].tile_base <= t) lo = mid; else hi = mid - 1;
    }
    const Inst &I = insts[lo];
    if (!I.stencil) return;
    const long long base = (long long)(t - I.tile_base) * I.size_i;
    const float *__restrict__ geom = I.a.geom;
    float *__restrict__ out = I.stencil + 2 * SD * base;  // the tile's planes, one after the other
    // two points of the lane per step, their loads issued together
    for (int n0 = lane; n0 < I.size_i; n0 += 64) {
        float m[2][SD];
#pragma unroll
        for (int q = 0; q < 2; ++q)
#pragma unroll
            for (int c = 0; c < SD; ++c)
                m[q][c] = n0 + 32 * q < I.size_i ? __ldg(geom + (size_t)c * I.size_tot + base + n0 + 32 * q) : 1.f;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            if (n0 + 32 * q >= I.size_i) break;
            float w[SD];
            int e[SD][3];
            if (D == 2) selling2_fast(m[q], w, e);
            else selling3_fast(m[q], w, e);
#pragma unroll
            for (int r = 0; r < SD; ++r) {
                int word = 0;
                if (!pack_offset<D>(e[r], word)) atomicOr(&ctrl->err, (unsigned)AGD_STATUS_UNSUPPORTED);
                __stcs(out + r * I.size_i + n0 + 32 * q, w[r]);
                __stcs(out + (SD + r) * I.size_i + n0 + 32 * q, __int_as_float(word));
            }
        }
    }
}

// Wall visibility of the cached stencils (cuda/FiniteDifferences.h:51-59): for
// the Riemann instances with walls, the hidden-neighbour bits of every offset,
// set in its packed word.  Only points within the wall distance bound walk
// their offsets (Walls.h:18-50).  One warp per tile, after stencil_kernel.
template <int D>
__global__ void stencil_walls_kernel(const Inst *insts, int ninst, int total_tiles) {
    constexpr int SD = D * (D + 1) / 2;
    const int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (t >= total_tiles) return;
    const Inst &I = inst_of_tile(insts, ninst, t);
    if (!I.stencil || !I.a.wall_dist) return;
    const int n_o = t - I.tile_base;
    const long long base = (long long)n_o * I.size_i;
    for (int n_i = lane; n_i < I.size_i; n_i += 32) {
        const long long n_t = base + n_i;
        const int wd0 = __ldg(I.a.wall_dist + n_t);  // 255 far from the walls and at padding
        if (wd0 == 255) continue;
        int xt[3] = {0, 0, 0}, ro = n_o, ri = n_i;
        for (int k = D - 1; k >= 0; --k) {
            xt[k] = (ro % I.shape_o[k]) * I.a.shape_i[k] + ri % I.a.shape_i[k];
            ro /= I.shape_o[k];
            ri /= I.a.shape_i[k];
        }
        for (int r = 0; r < SD; ++r) {
            float *slot = I.stencil + 2 * SD * base + (SD + r) * I.size_i + n_i;
            const int word = __float_as_int(*slot);
            int e[3] = {0, 0, 0};
            unpack_offset<D>(word, e);
            const unsigned h = hidden_bits<D>(I.a, wd0, xt, e, [&](const int *y) { return bilevel_index_rt(I, D, y); });
            if (h) *slot = __int_as_float(word | (int)(h << kHideShift));
        }
    }
}

// Multiprecision buffers, one warp per tile.  dir 0: first -> second buffers
// (before the solve); dir 1: second -> first buffers for the instances whose
// last epoch was odd (after the solve).
static __global__ void mp_copy_kernel(Sched S, int dir) {
    const int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (t >= 0 && S.ninst > 0) {
        int lo = 0, hi = S.ninst - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (S.inst[mid].tile_base <= t) lo = mid; else hi = mid - 1;
        }
        const Inst &I = S.inst[lo];
        if (t >= I.tile_base + I.size_o || I.a.multip_step == 0.f) return;
        if (dir == 1 && (S.stats[lo].niter_o & 1) == 0) return;
        const long long base = (long long)(t - I.tile_base) * I.size_i;
        float *uf = dir == 0 ? I.a.values : I.a.values_next, *ut = dir == 0 ? I.a.values_next : I.a.values;
        int *qf = dir == 0 ? I.a.valuesq : I.a.valuesq_next, *qt = dir == 0 ? I.a.valuesq_next : I.a.valuesq;
        for (int n_i = lane; n_i < I.size_i; n_i += 32) {
            ut[base + n_i] = uf[base + n_i];
            qt[base + n_i] = qf[base + n_i];
        }
    }
}

// ------------------------------------------------------------- tile visit ---
// MP: multiprecision, u + uq * multip_step with uq an int32 (cuda/HFM.h:12-25):
// Jacobi sweeps inside the tile and double-buffered epochs, as the reference
// forces strict_iter_i and strict_iter_o with it (_Kernel.py:39-45).
// FACT: source factorisation (shifted neighbour values near the seed).
// MODEL Rander: the Riemann stencil of the first symdim geometry planes, and
// the neighbour values at x -/+ e shifted by +/-<w, e> for the drift w of the
// next ndim planes (FiniteDifferences.h:41-45).
// ORD2: second order scheme (neighbours two steps away, cuda/HFM.h:91-138).
// WALLS: neighbours hidden by a wall read +inf (bits of the stencil cache).
// G: warps of the group that visits a tile together (1 for the queue's workers).
template <class TL, int MODEL, bool MP = false, bool FACT = false, bool ORD2 = false, bool WALLS = false, int G = 1>
struct Visit {
    static constexpr int D = TL::D;
    static constexpr int NT = 32 * G;          // threads of the group
    static constexpr int P = TL::SIZE / NT;    // points per thread
    static_assert(TL::SIZE % NT == 0, "a group has at most one thread per point");
    // Phases of a local sweep: the points of a phase are updated from the same
    // state, the phases in turn.  With several points per thread a phase is one
    // point of every thread; with one, the first half of the threads is the
    // first phase.  At second order, whose results depend on the update order, a
    // phase is always 32 points, one warp's.
    static constexpr int NPH = ORD2 ? P * G : (P > 1 ? P : (G > 1 ? 2 : 1));
    static constexpr bool kSelling = MODEL == AGD_MODEL_RIEMANN || MODEL == AGD_MODEL_RANDER;
    static constexpr bool kDrift = MODEL == AGD_MODEL_RANDER;
    static constexpr bool SHIFT = FACT || kDrift;  // neighbour values shifted (fsh)
    static constexpr int NACT = kSelling ? D * (D + 1) / 2 : D;
    static constexpr int NTOT = 2 * NACT;
    static constexpr int SD = D * (D + 1) / 2;

    static constexpr int kBoxed = (int)0xffc00000;  // negative quiet NaN: an in-tile index follows
    // Multiprecision comparison and normalisation (cuda/HFM.h:12-25).
    __device__ __forceinline__ static bool greater(float u, int uq, float v, int vq, float step) {
        return u - v > (float)(vq - uq) * step;
    }
    // inv: 1 / step where that is exact (step a power of two, as _SetGeometry.py:52-56
    // chooses it), so that the quotient is a product; else 0.
    __device__ __forceinline__ static float exact_inverse(float step) {
        return (__float_as_uint(step) & 0x7fffffu) == 0u && step >= 0x1p-100f && step <= 0x1p100f ? 1.f / step : 0.f;
    }
    __device__ __forceinline__ static void normalize(float &u, int &uq, float umax, float step, float inv) {
        if (u < umax) {
            const int n = (int)(inv != 0.f ? u * inv : u / step);
            u -= (float)n * step;
            uq += n;
        }
    }
    __device__ __forceinline__ static void neighbour_mp(float x, int xq, const float *us, const int *uqs, float &v,
                                                        int &vq) {
        const int b = __float_as_int(x);
        const bool in = (b >> 22) == -1;
        const int li = b & (TL::SIZE - 1);
        v = in ? us[li] : x;
        vq = in ? uqs[li] : xq;
    }
    // Shared memory of a warp: the tile's values, then (64-point tiles without
    // multiprecision) one slot per lane and stencil neighbour for the values
    // read from outside the tile, so that every neighbour of a sweep is one
    // shared load; otherwise (kSlots false) the integer parts with multiprecision.
    static constexpr bool kSlots = !MP && (TL::SIZE <= 64 || G >= 4);
    // Point p of a lane: the 8x8 tiles in two checkerboard colours (p = 0 the
    // points with x0 + x1 even), so that a local sweep updates one colour from
    // the other's values of the same sweep and information crosses the tile in
    // fewer sweeps (batch 128 of Riemann2 512^2: +1.7 %, one instance: +5 %,
    // against rows 0-3 then rows 4-7); the 16x16 tiles in bands of four rows
    // (p >> 1), each in the two colours (p & 1), except at second order
    // (Isotropic2 256^2: 3.68 -> 2.97 ms per solve, 38 -> 30 epochs, against
    // bands of two rows); other tiles lane + 32 p.
    // Groups of several warps: the same colours, in 8x8 tiles a warp each, in
    // 16x16 tiles over bands of 4 G rows (the whole tile from 4 warps on).
    __device__ __forceinline__ static int point_of(int tid, int p) {
        if constexpr (D == 2 && TL::SIZE == 64 && TL::S1 == 8) {
            const int c = G == 1 ? p : tid >> 5, r = (tid & 31) >> 2;
            return r * 8 + (((tid & 3) << 1) | ((r ^ c) & 1));
        } else if constexpr (D == 2 && TL::SIZE == 256 && TL::S1 == 16 && !ORD2) {
            const int c = G < 8 ? p : tid >> 7;
            const int r = G < 8 ? 4 * G * (p >> 1) + (tid >> 3) : (tid & 127) >> 3;
            return r * 16 + (((tid & 7) << 1) | ((r ^ c) & 1));
        } else {
            return tid + NT * p;
        }
    }
    __device__ __forceinline__ static void gsync(int group) { group_sync<G>(group); }
    __device__ __forceinline__ static bool gany(int group, bool x) { return group_any<G>(group, x); }
    static constexpr int kSmemFloats = kSlots ? TL::SIZE * (1 + (ORD2 ? 2 : 1) * NTOT) : 2 * TL::SIZE;
    __device__ __forceinline__ static float neighbour(float x, const float *us) {
        const int b = __float_as_int(x);
        const float inside = us[b & (TL::SIZE - 1)];  // index masked into this warp's tile
        return (b >> 22) == -1 ? inside : x;
    }
    // Second order corrections (cuda/HFM.h:91-138): with u0 the point's value and
    // v[k] the smaller neighbour along e_k (on side[k]), where
    // |u0 - 2 v + v2| < thr * max_k (u0 - v_k) and u0 > v, v2 the next neighbour
    // on that side, v becomes v + (v - v2) / 3 and its weight 9/4 of itself.
    // Returns the mask of the corrected neighbours.
    template <class Far>
    __device__ __forceinline__ static unsigned order2(float u0, float *v, float *w, const int *side, Far &&far,
                                                      float thr) {
        float bound = 0.f;
#pragma unroll
        for (int k = 0; k < NACT; ++k) bound = fmaxf(bound, u0 - v[k]);
        unsigned mask = 0;
#pragma unroll
        for (int k = 0; k < NACT; ++k) {
            const float v2 = far(k, side[k]);
            const float d2 = fabsf(u0 - 2.f * v[k] + v2);
            if (d2 < thr * bound && u0 > v[k]) {
                v[k] = (float)((double)v[k] + (double)(v[k] - v2) / 3.0);
                w[k] *= 2.25f;
                mask |= 1u << k;
            }
        }
        return mask;
    }
    __device__ __forceinline__ static float lds(unsigned addr) {
        float v;
        asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
        return v;
    }

    __device__ __forceinline__ static void sts(unsigned addr, float v) {
        asm volatile("st.shared.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
    }
    // Grid point yt seen from point xt of a tile: inside the tile (li: its index
    // there), inside the grid (n_t: its bilevel index; any value otherwise).
    // The tile sides are equal powers of two, so one mask tests all the axes.
    __device__ __forceinline__ static void locate(const int *shape, const int *shape_o, const int *xt, const int *yt,
                                                  bool &intile, bool &indom, int &li, unsigned &n_t) {
        constexpr unsigned SM = TL::S0 - 1;
        static_assert(TL::S0 == TL::S1 && (D == 2 || TL::S0 == TL::S2) && (TL::S0 & SM) == 0, "cubic tiles");
        unsigned diff = 0u, n_o = 0u, n_i = 0u;
        indom = true;
#pragma unroll
        for (int c = 0; c < D; ++c) {
            const unsigned y = (unsigned)yt[c];
            diff |= y ^ (unsigned)xt[c];
            indom = indom && y < (unsigned)shape[c];
            n_o = n_o * (unsigned)shape_o[c] + y / TL::S0;
            n_i = n_i * TL::S0 + (y & SM);
        }
        intile = (diff & ~SM) == 0u;
        li = (int)n_i;
        n_t = n_o * TL::SIZE + n_i;
    }

    // Stencil of the point with bilevel index n_t, in two steps so that the
    // loads of all the points of a lane are in flight together: the raw words
    // (cached weights and packed offsets, or the dual metric; Diagonal: the
    // weights), then the weights and offsets (unpacked, or by Selling's
    // decomposition; unit offsets for Isotropic and Diagonal).
    static constexpr int kRaw = MODEL == AGD_MODEL_ISOTROPIC ? 1 : (MODEL == AGD_MODEL_DIAGONAL ? D : 2 * SD + (kDrift ? D : 0));
    __device__ __forceinline__ static void stencil_load(const Inst &I, size_t base, int n_i, float *raw) {
        const size_t n_t = base + n_i;
        if constexpr (MODEL == AGD_MODEL_ISOTROPIC) return;
        if constexpr (MODEL == AGD_MODEL_DIAGONAL) {
#pragma unroll
            for (int k = 0; k < D; ++k) raw[k] = __ldg(I.a.geom + (size_t)k * I.size_tot + n_t);
            return;
        }
        if (I.stencil) {
#pragma unroll
            for (int r = 0; r < 2 * SD; ++r) raw[r] = __ldg(I.stencil + 2 * SD * base + n_i + r * TL::SIZE);
        } else {
#pragma unroll
            for (int c = 0; c < SD; ++c) raw[c] = __ldg(I.a.geom + (size_t)c * I.size_tot + n_t);
        }
        if constexpr (kDrift) {  // the drift, after the stencil words
#pragma unroll
            for (int c = 0; c < D; ++c) raw[2 * SD + c] = __ldg(I.a.geom + (size_t)(SD + c) * I.size_tot + n_t);
        }
    }
    // Drift shifts <w, e_k> of the offsets (scal_vv order), w = raw[2 SD ..].
    __device__ __forceinline__ static void drift_shifts(const float *raw, const int (*e)[3], float *f) {
#pragma unroll
        for (int k = 0; k < NACT; ++k) {
            float s = 0.f;
#pragma unroll
            for (int c = 0; c < D; ++c) s += raw[2 * SD + c] * float(e[k][c]);
            f[2 * k] += s;
            f[2 * k + 1] -= s;
        }
    }
    // hide[k]: the hidden-neighbour bits of offset k (WALLS: from the cache; else 0).
    // Isotropic offsets are unit vectors, hidden exactly when the neighbour is a
    // wall point, whose value is +inf already: no bits are needed.
    __device__ __forceinline__ static void stencil_decode(const Inst &I, const float *raw, float *w, int (*e)[3],
                                                          unsigned *hide) {
#pragma unroll
        for (int k = 0; k < NACT; ++k) hide[k] = 0u;
        if constexpr (!kSelling) {
#pragma unroll
            for (int k = 0; k < D; ++k) {
                w[k] = MODEL == AGD_MODEL_ISOTROPIC ? I.a.iso_weights[k] : raw[k];
#pragma unroll
                for (int c = 0; c < 3; ++c) e[k][c] = (c == k);
            }
        } else if (I.stencil) {
#pragma unroll
            for (int r = 0; r < SD; ++r) {
                w[r] = raw[r];
                unpack_offset<D>(__float_as_int(raw[SD + r]), e[r]);
                if constexpr (WALLS) hide[r] = (unsigned)__float_as_int(raw[SD + r]) >> kHideShift;
            }
        } else {
            float m[SD];
#pragma unroll
            for (int c = 0; c < SD; ++c) m[c] = raw[c];
            if (D == 2) selling2(m, w, e);
            else selling3(m, w, e);
        }
    }

    __device__ __forceinline__ static void stencil(const Inst &I, size_t n_t, float *w, int (*e)[3]) {
        float raw[kRaw];
        unsigned hide[NACT];
        stencil_load(I, n_t, 0, raw);  // (no cache: planes over the whole grid)
        stencil_decode(I, raw, w, e, hide);
    }

    // Visits tile n_o of instance I (the ii-th) at epoch e; tid: thread of the
    // group, us: the group's shared memory.  Returns whether this thread pushed a tile.
    __device__ static bool run(const Sched &S, const Inst &I, int ii, int n_o, int e, int tid, int group, float *us) {
        const agd_instance &A = I.a;
        const int lane = tid & 31;
        const bool lead = G == 1 || tid < 32;  // the first warp does the tile's bookkeeping
        // (in registers: after a volatile access the compiler would read the descriptor again)
        int shape[D], shape_o[D];
#pragma unroll
        for (int k = 0; k < D; ++k) {
            shape[k] = A.shape[k];
            shape_o[k] = I.shape_o[k];
        }
        const int niter_i = A.niter_i;
        int xo[3] = {0, 0, 0};
        {
            int r = n_o;
#pragma unroll
            for (int k = D - 1; k > 0; --k) {
                const int q = r / shape_o[k];
                xo[k] = r - q * shape_o[k];
                r = q;
            }
            xo[0] = r;
        }
        // Scores of this tile and of its neighbours at epoch e-1 (complete): loaded
        // now, so that their latency overlaps the visit (cuda/Propagation.h:103-167).
        const int t = I.tile_base + n_o;
        int nb = -1;  // neighbour tile handled by this lane (lanes 0..2D-1)
        if (lead && lane < 2 * D) {
            int y[3] = {xo[0], xo[1], xo[2]};
            y[lane >> 1] += 2 * (lane & 1) - 1;
            bool ok = true;
#pragma unroll
            for (int k = 0; k < D; ++k) ok = ok && y[k] >= 0 && y[k] < shape_o[k];
            if (ok) {
                int m = 0;
#pragma unroll
                for (int k = 0; k < D; ++k) m = m * shape_o[k] + y[k];
                nb = I.tile_base + m;
            }
        }
        const int sp_self = lead ? (int)score_at(S, t, e - 1) : 0;
        const int sp_nb = nb >= 0 ? (int)score_at(S, nb, e - 1) : 0;

        const size_t base = (size_t)n_o * TL::SIZE;
        // Epoch e reads buffer (e-1)&1 and writes buffer e&1 with multiprecision.
        const float *u_in = A.values;
        float *u_out = A.values;
        const int *q_in = nullptr;
        int *q_out = nullptr;
        const float step = A.multip_step, umax = A.multip_max, inv = MP ? exact_inverse(step) : 0.f;
        if constexpr (MP) {
            const bool odd = (e & 1) != 0;
            u_in = odd ? A.values : A.values_next;
            u_out = odd ? A.values_next : A.values;
            q_in = odd ? A.valuesq : A.valuesq_next;
            q_out = odd ? A.valuesq_next : A.valuesq;
        }
        int *uqs = reinterpret_cast<int *>(us + TL::SIZE);  // integer parts, after the float parts
        float uold[P], rhs[P];
        // A thread's own values stay in registers where there is one of them.
        constexpr bool kOwn = P == 1;
        float own = 0.f;
        int ownq = 0;
        int qold[P];
        float wts[P][NACT];
        // Neighbour of each stencil offset.  With kSlots: the shared-memory address
        // of its value (the tile slot, or this lane's slot holding the value read
        // from outside).  Otherwise: its value when outside the tile (read once
        // per visit), or its in-tile index boxed as a negative-NaN payload (no
        // solution value is a NaN), so one register holds either.
        float nbv[kSlots ? 1 : P][kSlots ? 1 : NTOT];
        int nbq[MP ? P : 1][MP ? NTOT : 1];
        unsigned nba[kSlots ? P : 1][kSlots ? NTOT : 1];
        float fsh[SHIFT ? P : 1][SHIFT ? NTOT : 1];  // factorisation and drift shifts of the neighbour values
        // second order with factorisation: the shifts of the neighbours two steps away
        float fsh2[FACT && ORD2 ? P : 1][FACT && ORD2 ? NTOT : 1];
        int nbq2[MP && ORD2 ? P : 1][MP && ORD2 ? NTOT : 1];  // their integer parts (multiprecision)
        // second order: the neighbours two steps away, as nba / nbv
        unsigned nba2[ORD2 && kSlots ? P : 1][ORD2 && kSlots ? NTOT : 1];
        float nbv2[ORD2 && !kSlots ? P : 1][ORD2 && !kSlots ? NTOT : 1];
        const unsigned us_addr = (unsigned)__cvta_generic_to_shared(us);
        bool seed[P];
        float raw[P][kRaw];
        // every load of the prologue that does not depend on another one is issued first
#pragma unroll
        for (int p = 0; p < P; ++p) {
            const size_t n_t = base + point_of(tid, p);
            uold[p] = __ldcg(u_in + n_t);
            seed[p] = (__ldg(A.seedbits + (n_t >> 3)) >> (n_t & 7)) & 1;
            rhs[p] = __ldg(A.rhs + n_t);
            if constexpr (MP) qold[p] = __ldcg(q_in + n_t);
            stencil_load(I, base, point_of(tid, p), raw[p]);
        }
#pragma unroll
        for (int p = 0; p < P; ++p) {
            const int n_i = point_of(tid, p);
            int xi[3] = {0, 0, 0}, xt[3] = {0, 0, 0};
            TL::pos(n_i, xi);
#pragma unroll
            for (int k = 0; k < D; ++k) xt[k] = xo[k] * TL::extent(k) + xi[k];
            if constexpr (MP) {
                float u0 = uold[p];
                int q0 = qold[p];
                if (seed[p]) {
                    u0 = rhs[p];
                    q0 = 0;
                    normalize(u0, q0, umax, step, inv);
                }
                us[n_i] = u0;
                uqs[n_i] = q0;
                own = u0;
                ownq = q0;
            } else {
                own = seed[p] ? rhs[p] : uold[p];
                us[n_i] = own;
            }
            int ev[NACT][3];
            unsigned hide[NACT];
            if (seed[p]) continue;  // seeds (and padding) keep their value: no stencil needed
            stencil_decode(I, raw[p], wts[p], ev, hide);
            if constexpr (SHIFT) {
                if constexpr (FACT) {
                    if constexpr (ORD2) factor_shifts<D, NACT, !kSelling>(A, xt, ev, fsh[p], fsh2[p]);
                    else factor_shifts<D, NACT, !kSelling>(A, xt, ev, fsh[p]);
                } else {
#pragma unroll
                    for (int k = 0; k < NTOT; ++k) fsh[p][k] = 0.f;
                }
                if constexpr (kDrift) drift_shifts(raw[p], ev, fsh[p]);
            }
            // Addresses first, then every load of the point, then the stores: a load
            // followed by its own store would make the neighbours' L2 round trips
            // serial.  (The loads of a lane's two points together: the registers
            // spill, batch 128 of Riemann2 512^2 15.2 -> 15.9 ms.)
            float out[kSlots ? NTOT : 1], out2[kSlots && ORD2 ? NTOT : 1];
#pragma unroll
            for (int k = 0; k < NACT; ++k) {
#pragma unroll
                for (int s = 0; s < 2; ++s) {
                    const int q = 2 * k + s;
                    // a neighbour hidden by a wall reads +inf, and so does the one after it
                    // (cuda/FiniteDifferences.h:53-59)
                    const bool hidden = WALLS && ((hide[k] >> s) & 1u);
#pragma unroll
                    for (int far = 0; far < (ORD2 ? 2 : 1); ++far) {  // x + eps e_k, then x + 2 eps e_k
                        int yt[3] = {0, 0, 0}, li;
                        unsigned n_t;
                        bool intile, indom;
#pragma unroll
                        for (int c = 0; c < D; ++c) yt[c] = s ? xt[c] + (far + 1) * ev[k][c] : xt[c] - (far + 1) * ev[k][c];
                        locate(shape, shape_o, xt, yt, intile, indom, li, n_t);
                        if constexpr (kSlots) {
                            const bool in = intile && !hidden;
                            float v = finf();
                            if (!intile && indom && !hidden) v = __ldcg(u_in + n_t);
                            const int slot = in ? li : TL::SIZE + far * P * NTOT * NT + (p * NTOT + q) * NT + tid;
                            if (far == 0) {
                                nba[p][q] = us_addr + 4u * (unsigned)slot;
                                out[q] = v;
                            } else if constexpr (ORD2) {
                                nba2[p][q] = us_addr + 4u * (unsigned)slot;
                                out2[q] = v;
                            }
                        } else {
                            float v = finf();
                            int vq = 0;
                            if (!intile && indom && !hidden) {
                                v = __ldcg(u_in + n_t);
                                if constexpr (MP) vq = __ldcg(q_in + n_t);
                            }
                            if constexpr (FACT && ORD2) {  // outside the tile: value + shift
                                if (far == 1) v += fsh2[p][q];
                            }
                            if (intile && !hidden) v = __int_as_float(kBoxed | li);
                            if (far == 0) {
                                nbv[p][q] = v;
                                if constexpr (MP) nbq[p][q] = vq;
                            } else if constexpr (ORD2) {
                                nbv2[p][q] = v;
                                if constexpr (MP) nbq2[p][q] = vq;
                            }
                        }
                    }
                }
            }
            if constexpr (kSlots) {
#pragma unroll
                for (int q = 0; q < NTOT; ++q) {
                    if (nba[p][q] >= us_addr + 4u * TL::SIZE) sts(nba[p][q], out[q]);
                    if constexpr (ORD2)
                        if (nba2[p][q] >= us_addr + 4u * TL::SIZE) sts(nba2[p][q], out2[q]);
                }
            }
        }
        gsync(group);
        for (int it = 0; it < niter_i; ++it) {
            bool moved = false;
            if constexpr (MP) {
                // strict sweeps: every point from the state at the start of the sweep
                float cand[P];
                int candq[P];
#pragma unroll
                for (int p = 0; p < P; ++p) {
                    cand[p] = finf();
                    candq[p] = 0;
                    if (seed[p]) continue;
                    float v[NACT], w[NACT];
                    int vq[NACT];
                    int side[ORD2 ? NACT : 1];
#pragma unroll
                    for (int k = 0; k < NACT; ++k) {
                        float a, b;
                        int aq, bq;
                        neighbour_mp(nbv[p][2 * k], nbq[p][2 * k], us, uqs, a, aq);
                        neighbour_mp(nbv[p][2 * k + 1], nbq[p][2 * k + 1], us, uqs, b, bq);
                        if constexpr (SHIFT) {  // the float part carries the shift (HFM.h:46-53)
                            a += fsh[p][2 * k];
                            b += fsh[p][2 * k + 1];
                        }
                        const bool take_b = greater(a, aq, b, bq, step);  // HFM.h:52-57
                        v[k] = take_b ? b : a;
                        vq[k] = take_b ? bq : aq;
                        w[k] = wts[p][k];
                        if constexpr (ORD2) side[k] = take_b;
                    }
                    int vqmin = kIntMax;  // HFM.h:79-87
#pragma unroll
                    for (int k = 0; k < NACT; ++k)
                        if (v[k] < finf()) vqmin = min(vqmin, vq[k]);
#pragma unroll
                    for (int k = 0; k < NACT; ++k) v[k] += (float)(vq[k] - vqmin) * step;
                    if constexpr (ORD2) {
                        // second order with multiprecision (HFM.h:89-135): the point's value and
                        // the farther neighbours' relative to the integer part vqmin; a farther
                        // neighbour inside the tile takes its factorisation shift after that,
                        // one outside carries it in its float part already
                        const int n_i = point_of(tid, p);
                        if (vqmin != kIntMax) {
                            const float u0 = (kOwn ? own : us[n_i]) + (float)((kOwn ? ownq : uqs[n_i]) - vqmin) * step;
                            order2(u0, v, w, side, [&](int k, int sd) {
                                const float x = nbv2[p][2 * k + sd];
                                const int b = __float_as_int(x);
                                if ((b >> 22) == -1) {
                                    const int li = b & (TL::SIZE - 1);
                                    float r = us[li] + (float)(uqs[li] - vqmin) * step;
                                    if constexpr (FACT) r += fsh2[p][2 * k + sd];
                                    return r;
                                }
                                return x + (float)(nbq2[p][2 * k + sd] - vqmin) * step;
                            }, A.order2_threshold);
                        }
                    }
                    float c = hfm_update<NACT>(rhs[p], v, w);
                    int cq = vqmin;
                    if (c == finf()) cq = 0;
                    else normalize(c, cq, umax, step, inv);
                    cand[p] = c;
                    candq[p] = cq;
                }
                gsync(group);
#pragma unroll
                for (int p = 0; p < P; ++p) {
                    const int n_i = point_of(tid, p);
                    if (!seed[p] && greater(kOwn ? own : us[n_i], kOwn ? ownq : uqs[n_i], cand[p], candq[p], step)) {
                        us[n_i] = own = cand[p];
                        uqs[n_i] = ownq = candq[p];
                        moved = true;
                    }
                }
            } else {
#pragma unroll
                for (int ph = 0; ph < NPH; ++ph) {
                    const int p = ORD2 ? ph / G : (P > 1 ? ph : 0);
                    const bool mine = !seed[p] && (ORD2   ? (tid >> 5) == ph % G
                                                   : P > 1 || NPH == 1 ? true
                                                                       : tid / (NT / 2) == ph);
                    const int n_i = point_of(tid, p);
                    float cand = finf();
                    if (mine) {
                        float v[NACT], w[NACT];
                        int side[ORD2 ? NACT : 1];
#pragma unroll
                        for (int k = 0; k < NACT; ++k) {
                            float a, b;
                            if constexpr (kSlots) {
                                a = lds(nba[p][2 * k]);
                                b = lds(nba[p][2 * k + 1]);
                            } else {
                                a = neighbour(nbv[p][2 * k], us);
                                b = neighbour(nbv[p][2 * k + 1], us);
                            }
                            if constexpr (SHIFT) {
                                a += fsh[p][2 * k];
                                b += fsh[p][2 * k + 1];
                            }
                            if constexpr (ORD2) v[k] = a > b ? b : a;
                            else v[k] = fminf(a, b);  // (no value is a NaN; one instruction)
                            w[k] = wts[p][k];
                            if constexpr (ORD2) side[k] = a > b;
                        }
                        if constexpr (ORD2) order2(kOwn ? own : us[n_i], v, w, side, [&](int k, int sd) {
                            // (with factorisation, the shift of x +/- 2 e_k; outside the tile
                            // without slots nbv2 carries it already)
                            if constexpr (kSlots) {
                                float r = lds(nba2[p][2 * k + sd]);
                                if constexpr (FACT) r += fsh2[p][2 * k + sd];
                                return r;
                            } else {
                                const float x = nbv2[p][2 * k + sd];
                                if ((__float_as_int(x) >> 22) != -1) return x;
                                float r = us[__float_as_int(x) & (TL::SIZE - 1)];
                                if constexpr (FACT) r += fsh2[p][2 * k + sd];
                                return r;
                            }
                        }, A.order2_threshold);
                        cand = hfm_update<NACT>(rhs[p], v, w);
                    }
                    // Within a warp the points of a phase read one state.  Between the warps of
                    // a group they may read each other's new values (neighbours of one
                    // colour, Riemann offsets): either is a value of this sweep.
                    __syncwarp();
                    if (mine && (kOwn ? own : us[n_i]) > cand) {
                        us[n_i] = own = cand;
                        moved = true;
                    }
                    if (ph + 1 < NPH) gsync(group);
                }
            }
            if (!gany(group, moved)) break;
        }
        bool notconv = false;
#pragma unroll
        for (int p = 0; p < P; ++p) {
            const int n_i = point_of(tid, p);
            const float u = kOwn ? own : us[n_i];
            __stcg(u_out + base + n_i, u);
            float diff, uabs;
            if constexpr (MP) {
                const int q = kOwn ? ownq : uqs[n_i];
                __stcg(q_out + base + n_i, q);
                diff = fabsf(uold[p] - u + (float)(qold[p] - q) * step);  // Update.h:212-216
                uabs = fabsf(u + (float)q * step);
            } else {
                diff = fabsf(uold[p] - u);
                uabs = fabsf(u);
            }
            const float tol = A.atol + A.rtol * uabs;
            if (!(isnan(diff) || diff <= tol)) notconv = true;
        }
        const bool changed = gany(group, notconv);
        if (!lead) return false;

        // Adaptive Gauss-Seidel iteration: a changed tile is visited again with
        // its neighbours (cuda/Propagation.h:151-154, Neighbor() including the
        // tile itself); global iteration: every tile at every epoch until an
        // epoch changes nothing (_solvers.py:77-92, stop test in close_epoch).
        if (A.flags & (AGD_FLAG_SOLVER_AGSI | AGD_FLAG_SOLVER_GLOBAL)) {
            bool pushed;
            if (A.flags & AGD_FLAG_SOLVER_GLOBAL) {
                if (changed && lane == 0) atomicMax(&S.ist[ii].changed, e);
                if (lane == 2 * D) push_tile(S, I, ii, t, e);
                pushed = lane == 2 * D;
            } else {
                const int target = !changed ? -1 : lane == 2 * D ? t : nb;
                if (target >= 0) push_tile(S, I, ii, target, e);
                pushed = target >= 0;
            }
            return pushed;
        }
        // Fast iterative method (cuda/Propagation.h:103-167).
        const int front = A.fim_front_width;
        int sn;
        bool prop;
        if (!changed) {
            const int sp = sp_self;
            if (sp == 0 || sp == front) { sn = 0; prop = false; }
            else { sn = front; prop = true; }
        } else {
            sn = 1;
            if (front > 2) {
                const int sq = nb >= 0 ? sp_nb - 1 : -1;
                int mx = sq;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(kFull, mx, o));
                sn = max(sn, mx);
            }
            prop = sn > 1;
        }
        if (lane == 0) {
            unsigned *arr = (e & 1) ? S.score1 : S.score0;
            __stcg(arr + t, ((unsigned)e << 8) | (unsigned)sn);
        }
        // The pushes of the tile itself (lane 2D, when changed) and of its
        // neighbours (lanes 0..2D-1) go out together.
        const int target = lane == 2 * D ? (changed ? t : -1) : (prop ? nb : -1);
        if (target >= 0) push_tile(S, I, ii, target, e);
        return target >= 0;
    }
};

// variant, tile (D, S0, S1, S2), model, multiprecision, factorisation, second order, walls
#define AGD_VARIANTS(X) \
    X(V_ISO2_8, 2, 8, 8, 1, AGD_MODEL_ISOTROPIC, false, false, false, false) \
    X(V_ISO2_16, 2, 16, 16, 1, AGD_MODEL_ISOTROPIC, false, false, false, false) \
    X(V_RIEM2_8, 2, 8, 8, 1, AGD_MODEL_RIEMANN, false, false, false, false) \
    X(V_ISO3_4, 3, 4, 4, 4, AGD_MODEL_ISOTROPIC, false, false, false, false) \
    X(V_RIEM3_4, 3, 4, 4, 4, AGD_MODEL_RIEMANN, false, false, false, false) \
    X(V_RIEM2_16, 2, 16, 16, 1, AGD_MODEL_RIEMANN, false, false, false, false) \
    X(V_ISO2_8_MP, 2, 8, 8, 1, AGD_MODEL_ISOTROPIC, true, false, false, false) \
    X(V_ISO2_16_MP, 2, 16, 16, 1, AGD_MODEL_ISOTROPIC, true, false, false, false) \
    X(V_RIEM2_8_MP, 2, 8, 8, 1, AGD_MODEL_RIEMANN, true, false, false, true) \
    X(V_ISO3_4_MP, 3, 4, 4, 4, AGD_MODEL_ISOTROPIC, true, false, false, false) \
    X(V_RIEM3_4_MP, 3, 4, 4, 4, AGD_MODEL_RIEMANN, true, false, false, true) \
    X(V_ISO2_8_F, 2, 8, 8, 1, AGD_MODEL_ISOTROPIC, false, true, false, false) \
    X(V_ISO2_16_FMP, 2, 16, 16, 1, AGD_MODEL_ISOTROPIC, true, true, false, false) \
    X(V_RIEM2_8_FMP, 2, 8, 8, 1, AGD_MODEL_RIEMANN, true, true, false, true) \
    X(V_ISO3_4_FMP, 3, 4, 4, 4, AGD_MODEL_ISOTROPIC, true, true, false, false) \
    X(V_RIEM3_4_FMP, 3, 4, 4, 4, AGD_MODEL_RIEMANN, true, true, false, true) \
    X(V_ISO2_16_O2F, 2, 16, 16, 1, AGD_MODEL_ISOTROPIC, false, true, true, false) \
    X(V_RIEM2_8_O2F, 2, 8, 8, 1, AGD_MODEL_RIEMANN, false, true, true, true) \
    X(V_ISO3_4_O2F, 3, 4, 4, 4, AGD_MODEL_ISOTROPIC, false, true, true, false) \
    X(V_RIEM3_4_O2F, 3, 4, 4, 4, AGD_MODEL_RIEMANN, false, true, true, true) \
    X(V_ISO2_16_O2MP, 2, 16, 16, 1, AGD_MODEL_ISOTROPIC, true, false, true, false) \
    X(V_RIEM2_8_O2MP, 2, 8, 8, 1, AGD_MODEL_RIEMANN, true, false, true, true) \
    X(V_ISO3_4_O2MP, 3, 4, 4, 4, AGD_MODEL_ISOTROPIC, true, false, true, false) \
    X(V_RIEM3_4_O2MP, 3, 4, 4, 4, AGD_MODEL_RIEMANN, true, false, true, true) \
    X(V_ISO2_16_O2FMP, 2, 16, 16, 1, AGD_MODEL_ISOTROPIC, true, true, true, false) \
    X(V_RIEM2_8_O2FMP, 2, 8, 8, 1, AGD_MODEL_RIEMANN, true, true, true, true) \
    X(V_ISO3_4_O2FMP, 3, 4, 4, 4, AGD_MODEL_ISOTROPIC, true, true, true, false) \
    X(V_RIEM3_4_O2FMP, 3, 4, 4, 4, AGD_MODEL_RIEMANN, true, true, true, true) \
    X(V_ISO2_16_F, 2, 16, 16, 1, AGD_MODEL_ISOTROPIC, false, true, false, false) \
    X(V_RIEM2_8_F, 2, 8, 8, 1, AGD_MODEL_RIEMANN, false, true, false, true) \
    X(V_ISO3_4_F, 3, 4, 4, 4, AGD_MODEL_ISOTROPIC, false, true, false, false) \
    X(V_RIEM3_4_F, 3, 4, 4, 4, AGD_MODEL_RIEMANN, false, true, false, true) \
    X(V_ISO2_8_O2, 2, 8, 8, 1, AGD_MODEL_ISOTROPIC, false, false, true, false) \
    X(V_ISO2_16_O2, 2, 16, 16, 1, AGD_MODEL_ISOTROPIC, false, false, true, false) \
    X(V_RIEM2_8_O2, 2, 8, 8, 1, AGD_MODEL_RIEMANN, false, false, true, true) \
    X(V_ISO3_4_O2, 3, 4, 4, 4, AGD_MODEL_ISOTROPIC, false, false, true, false) \
    X(V_RIEM3_4_O2, 3, 4, 4, 4, AGD_MODEL_RIEMANN, false, false, true, true) \
    X(V_RIEM2_8_W, 2, 8, 8, 1, AGD_MODEL_RIEMANN, false, false, false, true) \
    X(V_RIEM2_16_W, 2, 16, 16, 1, AGD_MODEL_RIEMANN, false, false, false, true) \
    X(V_RIEM3_4_W, 3, 4, 4, 4, AGD_MODEL_RIEMANN, false, false, false, true) \
    X(V_DIAG2_8, 2, 8, 8, 1, AGD_MODEL_DIAGONAL, false, false, false, false) \
    X(V_DIAG2_16, 2, 16, 16, 1, AGD_MODEL_DIAGONAL, false, false, false, false) \
    X(V_DIAG3_4, 3, 4, 4, 4, AGD_MODEL_DIAGONAL, false, false, false, false) \
    X(V_DIAG2_8_MP, 2, 8, 8, 1, AGD_MODEL_DIAGONAL, true, false, false, false) \
    X(V_DIAG2_16_MP, 2, 16, 16, 1, AGD_MODEL_DIAGONAL, true, false, false, false) \
    X(V_DIAG3_4_MP, 3, 4, 4, 4, AGD_MODEL_DIAGONAL, true, false, false, false) \
    X(V_DIAG2_8_F, 2, 8, 8, 1, AGD_MODEL_DIAGONAL, false, true, false, false) \
    X(V_DIAG2_16_F, 2, 16, 16, 1, AGD_MODEL_DIAGONAL, false, true, false, false) \
    X(V_DIAG3_4_F, 3, 4, 4, 4, AGD_MODEL_DIAGONAL, false, true, false, false) \
    X(V_DIAG2_8_O2, 2, 8, 8, 1, AGD_MODEL_DIAGONAL, false, false, true, false) \
    X(V_DIAG2_16_O2, 2, 16, 16, 1, AGD_MODEL_DIAGONAL, false, false, true, false) \
    X(V_DIAG3_4_O2, 3, 4, 4, 4, AGD_MODEL_DIAGONAL, false, false, true, false) \
    X(V_RAND2_8, 2, 8, 8, 1, AGD_MODEL_RANDER, false, false, false, false) \
    X(V_RAND3_4, 3, 4, 4, 4, AGD_MODEL_RANDER, false, false, false, false) \
    X(V_RAND2_8_W, 2, 8, 8, 1, AGD_MODEL_RANDER, false, false, false, true) \
    X(V_RAND3_4_W, 3, 4, 4, 4, AGD_MODEL_RANDER, false, false, false, true) \
    X(V_RAND2_8_MP, 2, 8, 8, 1, AGD_MODEL_RANDER, true, false, false, true) \
    X(V_RAND3_4_MP, 3, 4, 4, 4, AGD_MODEL_RANDER, true, false, false, true) \
    X(V_RAND2_8_F, 2, 8, 8, 1, AGD_MODEL_RANDER, false, true, false, true) \
    X(V_RAND3_4_F, 3, 4, 4, 4, AGD_MODEL_RANDER, false, true, false, true) \
    X(V_RAND2_8_O2, 2, 8, 8, 1, AGD_MODEL_RANDER, false, false, true, true) \
    X(V_RAND3_4_O2, 3, 4, 4, 4, AGD_MODEL_RANDER, false, false, true, true)

template <unsigned long long VMASK, int G>
__device__ __forceinline__ bool dispatch(const Sched &S, int t, int ii, int e, int tid, int group, float *us) {
    const Inst &I = S.inst[ii];
    const int n_o = t - I.tile_base;
    if constexpr ((VMASK & (VMASK - 1)) == 0) {  // one variant: no switch
#define AGD_CASE(V, D, A, B, C, M, MP, F, O2, W) \
    if constexpr (VMASK == (1ull << V)) return Visit<Tile<D, A, B, C>, M, MP, F, O2, W, G>::run(S, I, ii, n_o, e, tid, group, us);
        AGD_VARIANTS(AGD_CASE)
#undef AGD_CASE
    }
    switch (I.variant) {
#define AGD_CASE(V, D, A, B, C, M, MP, F, O2, W)                                                          \
    case V:                                                                                               \
        if constexpr ((VMASK >> V) & 1)                                                                   \
            return Visit<Tile<D, A, B, C>, M, MP, F, O2, W, G>::run(S, I, ii, n_o, e, tid, group, us);    \
        break;
        AGD_VARIANTS(AGD_CASE)
#undef AGD_CASE
        default:
            break;
    }
    return false;
}

// Shared floats per group of G warps for the variants of VMASK.
template <unsigned long long VMASK, int G>
constexpr int smem_floats() {
    int m = 0;
#define AGD_CASE(V, D, A, B, C, M, MP, F, O2, W) \
    if constexpr ((VMASK >> V) & 1) m = std::max(m, Visit<Tile<D, A, B, C>, M, MP, F, O2, W, G>::kSmemFloats);
    AGD_VARIANTS(AGD_CASE)
#undef AGD_CASE
    return m;
}

template <unsigned long long VMASK>
struct EikonalVisitor {
    static constexpr unsigned long long kTiles16 =
        (1ull << V_RIEM2_16) | (1ull << V_ISO2_16) | (1ull << V_ISO2_16_MP) | (1ull << V_ISO2_16_F) |
        (1ull << V_ISO2_16_FMP) | (1ull << V_ISO2_16_O2F) | (1ull << V_ISO2_16_O2MP) | (1ull << V_ISO2_16_O2FMP) |
        (1ull << V_ISO2_16_O2) | (1ull << V_RIEM2_16_W) | (1ull << V_DIAG2_16) | (1ull << V_DIAG2_16_MP) |
        (1ull << V_DIAG2_16_F) | (1ull << V_DIAG2_16_O2);
    static constexpr unsigned long long kSelling3 =
        (1ull << V_RIEM3_4) | (1ull << V_RIEM3_4_MP) | (1ull << V_RIEM3_4_F) | (1ull << V_RIEM3_4_O2) |
        (1ull << V_RIEM3_4_W) | (1ull << V_RAND3_4) | (1ull << V_RAND3_4_W) | (1ull << V_RAND3_4_MP) |
        (1ull << V_RAND3_4_F) | (1ull << V_RAND3_4_O2) | (1ull << V_RIEM3_4_FMP) | (1ull << V_RIEM3_4_O2F) |
        (1ull << V_RIEM3_4_O2MP) | (1ull << V_RIEM3_4_O2FMP);
    // Resident 4-warp CTAs per SM of the queue's workers that the register
    // budget must allow: 256-point tiles keep 8 points per lane in registers,
    // Riemann3 twelve neighbours per point, multiprecision an integer part
    // beside every value.  Riemann2 8x8: 7 CTAs at up to 72 registers (batch 128
    // of 512^2: 15.2 ms against 15.4 at 8 CTAs and 64 registers).
    static constexpr int kMinCtas = (VMASK & kTiles16)                                            ? 4
                                    : (VMASK & kSelling3)                                         ? 5
                                    : (VMASK & (kMpVariants | kFactorVariants | kOrder2Variants)) ? 7
                                    : (VMASK & (1ull << V_RIEM2_8))                               ? 7
                                                                                                  : 9;
    struct Args {};
    struct Smem {
        float u[smem_floats<VMASK, 1>()];  // values, then out-of-tile neighbours or integer parts
    };
    __device__ __forceinline__ static void visit(const Sched &S, const Args &, int t, int ii, int e, int lane, Smem &sm) {
        dispatch<VMASK, 1>(S, t, ii, e, lane, 0, sm.u);
    }
    // Rounds: groups of kRoundG warps per tile.
    static constexpr bool kQueueless = false;
    static constexpr bool kAll16 = (VMASK & ~kTiles16) == 0;
    // Isotropic and Diagonal 64-point tiles: a warp (Isotropic3 201^3: 4.1 ms against
    // 5.3 with two: a visit has little to compute, and half of a group idles in
    // each phase); Riemann: two, whose points' neighbours fit the registers then
    // (Riemann3 200^3: 9.4 ms against 10.2; Riemann2 512^2 1.39 against 1.59 ms);
    // 16x16 tiles alone in a kernel: eight, a point a thread.
    static constexpr unsigned long long kUnit64 =
        (1ull << V_ISO2_8) | (1ull << V_ISO3_4) | (1ull << V_DIAG2_8) | (1ull << V_DIAG3_4);
    static constexpr int kRoundG = kAll16 ? ((VMASK & kOrder2Variants) ? 1 : 8) : (VMASK & ~kUnit64) ? 2 : 1;
    // A CTA of 16x16 tiles has the whole SM, 4 groups of 8 warps: with two CTAs of
    // two groups, an epoch of few tiles more often gives one of them three
    // (Isotropic2 1203x1501 float64: 4.7 ms, 4.1 with one).
    static constexpr int kRoundWarps = kAll16 ? 32 : 16;
    static constexpr int kRoundCtas = kAll16 ? 1 : 2;
    struct RoundSmem {
        float u[smem_floats<VMASK, kRoundG>()];
    };
    static constexpr bool kOrdered = false;
    __device__ __forceinline__ static bool visit_round(const Sched &S, const Args &, int t, int ii, int e, int tid,
                                                       int group, RoundSmem &sm) {
        return dispatch<VMASK, kRoundG>(S, t, ii, e, tid, group, sm.u);
    }
    // Before the workers: the second buffers of multiprecision instances start
    // as copies of the first (_SetArgs.py:171-177), and the Selling stencils of
    // the Riemann instances are computed.
    static cudaError_t prepare(const Sched &S, const WsLayout &L, cudaStream_t st) {
        constexpr unsigned long long kRiemann = (1ull << V_RIEM2_8) | (1ull << V_RIEM3_4) | (1ull << V_RIEM2_16) |
                                      (1ull << V_RIEM2_8_MP) | (1ull << V_RIEM3_4_MP) | (1ull << V_RIEM2_8_F) |
                                      (1ull << V_RIEM3_4_F) | (1ull << V_RIEM2_8_O2) | (1ull << V_RIEM3_4_O2) |
                                      (1ull << V_RIEM2_8_FMP) | (1ull << V_RIEM3_4_FMP) | kWallVariants |
                                      kRanderVariants | (1ull << V_RIEM2_8_O2F) | (1ull << V_RIEM3_4_O2F) |
                                      (1ull << V_RIEM2_8_O2MP) | (1ull << V_RIEM3_4_O2MP) |
                                      (1ull << V_RIEM2_8_O2FMP) | (1ull << V_RIEM3_4_O2FMP);
        if (VMASK & kMpVariants) mp_copy_kernel<<<(L.total_tiles + 7) / 8, 256, 0, st>>>(S, 0);
        if (!(VMASK & kRiemann) || L.stencil == L.total) return cudaGetLastError();
        // variants that read the hidden-neighbour bits: the walls pass follows
        constexpr unsigned long long kWallCapable = kWallVariants | (1ull << V_RIEM2_8_MP) | (1ull << V_RIEM3_4_MP) |
                                          (1ull << V_RIEM2_8_F) | (1ull << V_RIEM3_4_F) | (1ull << V_RIEM2_8_O2) |
                                          (1ull << V_RIEM3_4_O2) | (1ull << V_RIEM2_8_FMP) | (1ull << V_RIEM3_4_FMP) |
                                          (1ull << V_RIEM2_8_O2F) | (1ull << V_RIEM3_4_O2F) | (1ull << V_RIEM2_8_O2MP) |
                                          (1ull << V_RIEM3_4_O2MP) | (1ull << V_RIEM2_8_O2FMP) | (1ull << V_RIEM3_4_O2FMP) |
                                          (kRanderVariants & ~((1ull << V_RAND2_8) | (1ull << V_RAND3_4)));
        const unsigned grid = (L.total_tiles + 7) / 8;
        if (VMASK & kSelling3) {
            stencil_kernel<3><<<grid, 256, 0, st>>>(S.inst, S.ninst, L.total_tiles, S.ctrl);
            if (VMASK & kWallCapable) stencil_walls_kernel<3><<<grid, 256, 0, st>>>(S.inst, S.ninst, L.total_tiles);
        } else {
            stencil_kernel<2><<<grid, 256, 0, st>>>(S.inst, S.ninst, L.total_tiles, S.ctrl);
            if (VMASK & kWallCapable) stencil_walls_kernel<2><<<grid, 256, 0, st>>>(S.inst, S.ninst, L.total_tiles);
        }
        return cudaGetLastError();
    }
    // After the workers: an instance that ran an odd number of epochs has its
    // result in the second buffers (the reference swaps its argument names).
    static cudaError_t finalize(const Sched &S, const WsLayout &L, cudaStream_t st) {
        if (VMASK & kMpVariants) mp_copy_kernel<<<(L.total_tiles + 7) / 8, 256, 0, st>>>(S, 1);
        return cudaGetLastError();
    }
};

}  // namespace agd
