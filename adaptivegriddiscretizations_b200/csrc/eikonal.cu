// Persistent, device-scheduled block-iterative eikonal solver for B200
// (Isotropic2/3, Riemann2/3), plus the flow pass and the layout kernels.
//
// Scheduling.  The reference iterates on the host: every outer iteration it
// compacts the flags of the tiles to update (cp.flatnonzero), tests for
// termination (np.any, a device->host sync) and launches `Update` on the
// active tiles (agd/Eikonal/HFM_CUDA/_solvers.py:94-120).  Here one launch runs
// all outer iterations ("epochs") of all the instances of a plan, with the
// reference's epoch semantics (the fast-iterative-method scores of
// cuda/Propagation.h:103-167 are epoch-stamped, per instance).  sched.cuh has
// two schedulers:
//   many instances (kPairInstances or more, or release epochs): resident worker
//   warps and one global queue of (tile, epoch) entries, no barrier; the warp
//   that finishes the last tile of an instance's epoch publishes its next one,
//   so instances never wait for one another (sched_worker);
//   fewer: rounds, with every tile owned by one CTA and a barrier of the CTAs
//   between epochs (rounds_worker).
//
// Tile visit (visit.cuh).  A warp, or in rounds a group of warps, per tile, tile
// values in shared memory, niter_i local sweeps in phases, and an
// early exit when a full sweep changes nothing (the state is then a fixed point
// of the visit, so the result equals that of the remaining sweeps).  Values of
// neighbours outside the tile are read once per visit through L2 (ld.cg), as
// other SMs update them concurrently.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <vector>

#include "visit.cuh"

struct agd_plan {
    std::vector<agd::Inst> insts;
    agd::WsLayout L;
    unsigned long long vmask;
    int ndim;
};

namespace agd {

// Checks the instances of one launch; returns the mask of tile-visit variants.
// stencil_cache: whether the launch computes the Riemann stencil cache.
static int validate(const agd_instance *host, const Inst *insts, int n, bool stencil_cache, unsigned long long *vmask) {
    *vmask = 0;
    for (int i = 0; i < n; ++i) {
        const agd_instance &a = host[i];
        const char *bad = nullptr;
        int code = AGD_STATUS_INVALID;
        if (a.ndim != host[0].ndim) bad = "all instances of a plan must share ndim";
        else if (insts[i].variant < 0) { bad = "model/tile shape not built"; code = AGD_STATUS_UNSUPPORTED; }
        else if (a.wall_dist && (a.model == AGD_MODEL_RIEMANN || a.model == AGD_MODEL_RANDER) && !stencil_cache) {
            bad = "walls on a Riemann instance need the stencil cache (agd_eikonal_solve)";
            code = AGD_STATUS_UNSUPPORTED;
        }
        else if (a.multip_step != 0.f && (!a.valuesq || !a.values_next || !a.valuesq_next || !(a.multip_step > 0.f)))
            bad = "multiprecision needs valuesq, values_next, valuesq_next and multip_step > 0";
        else if (!a.values || !a.rhs || !a.seedbits || (a.model != AGD_MODEL_ISOTROPIC && !a.geom)) bad = "missing array";
        else if (reinterpret_cast<uintptr_t>(a.seedbits) % 4 != 0) bad = "seedbits must be 4-byte aligned";
        else if (a.niter_i < 1 || a.fim_front_width < 2 || a.fim_front_width > 255 || a.nitermax_o < 0 ||
                 a.nitermax_o > kMaxEpochs)
            bad = "bad niter_i / fim_front_width / nitermax_o (at most 16000)";
        if (bad) return set_error(code, bad);
        *vmask |= 1ull << insts[i].variant;
    }
    return AGD_STATUS_OK;
}

static int plan_create(const agd_instance *host, int n, agd_plan **out) {
    if (!out) return set_error(AGD_STATUS_INVALID, "null plan pointer");
    *out = nullptr;
    if (n <= 0 || !host) return set_error(AGD_STATUS_INVALID, "no instance");
    agd_plan *P = new agd_plan();
    if (!layout(host, n, P->L, &P->insts)) {
        delete P;
        return set_error(AGD_STATUS_INVALID, "bad instance shape");
    }
    P->ndim = host[0].ndim;
    const int rc = validate(host, P->insts.data(), n, /*stencil_cache=*/true, &P->vmask);
    if (rc != AGD_STATUS_OK) {
        delete P;
        return rc;
    }
    *out = P;
    return AGD_STATUS_OK;
}

// The persistent solve for the variants in vmask, on a workspace laid out by L
// whose descriptors are already uploaded.
static int run_variants(int ndim, unsigned long long vmask, const WsLayout &L, void *ws, int n, agd_stats *stats,
                        const agd_launch *cfg, cudaStream_t st) {
    using namespace fam;
    if (vmask & kRanderVariants) {  // Rander instances run in kernels of their own
        if (vmask & ~kRanderVariants) return set_error(AGD_STATUS_UNSUPPORTED, "Rander instances beside other models in one plan");
        const bool mp = vmask & kMpVariants, f = vmask & kFactorVariants, o2 = vmask & kOrder2Variants;
        if (int(mp) + int(f) + int(o2) > 1)
            return set_error(AGD_STATUS_UNSUPPORTED, "Rander instances of several option families in one plan");
        if (ndim == 2) {
            if (o2) return solve<NO2>(L, ws, n, stats, cfg, st);
            if (f) return solve<NF2>(L, ws, n, stats, cfg, st);
            if (mp) return solve<NMP2>(L, ws, n, stats, cfg, st);
            return solve<N2>(L, ws, n, stats, cfg, st);
        }
        if (o2) return solve<NO3>(L, ws, n, stats, cfg, st);
        if (f) return solve<NF3>(L, ws, n, stats, cfg, st);
        if (mp) return solve<NMP3>(L, ws, n, stats, cfg, st);
        return solve<N3>(L, ws, n, stats, cfg, st);
    }
    if (vmask & kDiagVariants) {  // Diagonal instances run in kernels of their own
        if (vmask & ~kDiagVariants) return set_error(AGD_STATUS_UNSUPPORTED, "Diagonal instances beside other models in one plan");
        const bool mp = vmask & kMpVariants, f = vmask & kFactorVariants, o2 = vmask & kOrder2Variants;
        if (int(mp) + int(f) + int(o2) > 1)
            return set_error(AGD_STATUS_UNSUPPORTED, "Diagonal instances of several option families in one plan");
        if (ndim == 2) {
            if (o2) return solve<DO2>(L, ws, n, stats, cfg, st);
            if (f) return solve<DF2>(L, ws, n, stats, cfg, st);
            if (mp) return solve<DMP2>(L, ws, n, stats, cfg, st);
            return solve<D2>(L, ws, n, stats, cfg, st);
        }
        if (o2) return solve<DO3>(L, ws, n, stats, cfg, st);
        if (f) return solve<DF3>(L, ws, n, stats, cfg, st);
        if (mp) return solve<DMP3>(L, ws, n, stats, cfg, st);
        return solve<D3>(L, ws, n, stats, cfg, st);
    }
    constexpr unsigned long long kO2Combined = kOrder2FactorVariants | kOrder2MpVariants | kOrder2FactorMpVariants;
    if (vmask & kO2Combined) {  // second order with factorisation, multiprecision, or both
        const bool f = vmask & kOrder2FactorVariants, mp = vmask & kOrder2MpVariants,
                   fmp = vmask & kOrder2FactorMpVariants;
        if (int(f) + int(mp) + int(fmp) > 1 || (vmask & ~kO2Combined))
            return set_error(AGD_STATUS_UNSUPPORTED,
                             "second order with factorisation or multiprecision beside other instances in one plan");
        if (ndim == 2) return f ? solve<OF2>(L, ws, n, stats, cfg, st)
                              : mp ? solve<OM2>(L, ws, n, stats, cfg, st)
                                   : solve<OFM2>(L, ws, n, stats, cfg, st);
        return f ? solve<OF3>(L, ws, n, stats, cfg, st)
               : mp ? solve<OM3>(L, ws, n, stats, cfg, st)
                    : solve<OFM3>(L, ws, n, stats, cfg, st);
    }
    if (vmask & kOrder2Variants) {  // second order instances, possibly beside plain ones
        if (vmask & (kMpVariants | kFactorVariants))
            return set_error(AGD_STATUS_UNSUPPORTED, "second order beside multiprecision or factorisation in one plan");
        if (ndim == 2) return solve<O2>(L, ws, n, stats, cfg, st);
        return solve<O3>(L, ws, n, stats, cfg, st);
    }
    if (vmask & kFactorVariants) {  // factored instances, possibly beside plain ones
        if (vmask & kMpVariants)
            return set_error(AGD_STATUS_UNSUPPORTED, "factored instances without and with multiprecision in one plan");
        if (ndim == 2) return solve<F2>(L, ws, n, stats, cfg, st);
        return solve<F3>(L, ws, n, stats, cfg, st);
    }
    if (vmask & kMpVariants) {
        if (ndim == 2) {
            if (vmask == R2MP) return solve<R2MP>(L, ws, n, stats, cfg, st);
            if (vmask == I16MP) return solve<I16MP>(L, ws, n, stats, cfg, st);
            return solve<MP2>(L, ws, n, stats, cfg, st);
        }
        if (vmask == R3MP) return solve<R3MP>(L, ws, n, stats, cfg, st);
        if (vmask == I3MP) return solve<I3MP>(L, ws, n, stats, cfg, st);
        return solve<MP3>(L, ws, n, stats, cfg, st);
    }
    if (ndim == 2) {
        if (vmask == R2) return solve<R2>(L, ws, n, stats, cfg, st);
        if (vmask == R2L) return solve<R2L>(L, ws, n, stats, cfg, st);
        if (vmask == I16) return solve<I16>(L, ws, n, stats, cfg, st);
        if (vmask == I8) return solve<I8>(L, ws, n, stats, cfg, st);
        if (vmask == R2W) return solve<R2W>(L, ws, n, stats, cfg, st);
        return solve<BASE2>(L, ws, n, stats, cfg, st);
    }
    if (vmask == R3) return solve<R3>(L, ws, n, stats, cfg, st);
    if (vmask == I3) return solve<I3>(L, ws, n, stats, cfg, st);
    if (vmask == W3) return solve<W3>(L, ws, n, stats, cfg, st);
    return solve<BASE3>(L, ws, n, stats, cfg, st);
}

static int plan_run(const agd_plan *P, void *ws, size_t ws_bytes, agd_stats *stats, const agd_launch *cfg,
                    cudaStream_t st) {
    if (!P || !ws) return set_error(AGD_STATUS_INVALID, "null plan or workspace");
    const WsLayout &L = P->L;
    if (ws_bytes < L.total) return set_error(AGD_STATUS_WORKSPACE, "workspace too small");
    return run_variants(P->ndim, P->vmask, L, ws, (int)P->insts.size(), stats, cfg, st);
}

// ------------------------------------------------------- fixed scratch ---
// Scratch of agd_eikonal_solve_fixed_scratch: a file-scope device array, so that
// callers which cannot allocate device memory still get a solver.  In host code
// the name g_fixed_scratch is only a host-side stand-in for the symbol; the
// device address is obtained once per device with cudaGetSymbolAddress.
constexpr size_t kFixedScratchBytes = (size_t)AGD_FIXED_SCRATCH_BYTES;
constexpr int kFixedScratchMaxInstances = AGD_FIXED_SCRATCH_MAX_INSTANCES;
static __device__ __align__(256) unsigned char g_fixed_scratch[kFixedScratchBytes];
constexpr int kMaxDevices = 64;
static void *g_fixed_scratch_addr[kMaxDevices];
static std::mutex g_fixed_scratch_lock;
// Host staging of the instance descriptors (about 64 KiB at the maximum count):
// a file-scope array rather than a stack one, since plugin threads may have
// small stacks.  Used under g_fixed_scratch_lock until the upload has read it.
static Inst g_fixed_scratch_insts[kFixedScratchMaxInstances];

static int fixed_scratch_solve(const agd_instance *host, int n, agd_stats *stats, const agd_launch *cfg,
                               cudaStream_t st) {
    if (!host || n <= 0) return set_error(AGD_STATUS_INVALID, "no instance");
    if (n > kFixedScratchMaxInstances)
        return set_error(AGD_STATUS_INVALID, "agd_eikonal_solve_fixed_scratch: more than "
                                             "AGD_FIXED_SCRATCH_MAX_INSTANCES instances");
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess) return set_cuda_error("cudaGetDevice", err);
    if (dev < 0 || dev >= kMaxDevices) return set_error(AGD_STATUS_UNSUPPORTED, "device ordinal too large");
    std::lock_guard<std::mutex> guard(g_fixed_scratch_lock);  // held until the descriptors are staged
    if (!g_fixed_scratch_addr[dev]) {  // first call on this device: resolve the array's device address
        err = cudaGetSymbolAddress(&g_fixed_scratch_addr[dev], g_fixed_scratch);
        if (err != cudaSuccess) {
            g_fixed_scratch_addr[dev] = nullptr;
            return set_cuda_error("cudaGetSymbolAddress(fixed scratch)", err);
        }
    }
    void *scratch = g_fixed_scratch_addr[dev];
    Inst *insts = g_fixed_scratch_insts;
    WsLayout L;
    if (!layout(host, n, L, insts, /*stencil_cache=*/false)) return set_error(AGD_STATUS_INVALID, "bad instance shape");
    unsigned long long vmask = 0;
    const int rc = validate(host, insts, n, /*stencil_cache=*/false, &vmask);
    if (rc != AGD_STATUS_OK) return rc;
    if (L.total > kFixedScratchBytes)
        return set_error(AGD_STATUS_WORKSPACE, "agd_eikonal_solve_fixed_scratch: these instances need more "
                                               "scratch than AGD_FIXED_SCRATCH_BYTES; use agd_eikonal_solve");
    // Pageable host source: the call returns once the descriptors are staged,
    // after which the host array may be reused.
    err = cudaMemcpyAsync(static_cast<char *>(scratch) + L.inst, insts, sizeof(Inst) * n, cudaMemcpyHostToDevice, st);
    if (err != cudaSuccess) return set_cuda_error("descriptor upload", err);
    return run_variants(host[0].ndim, vmask, L, scratch, n, stats, cfg, st);
}

static int plan_upload(const agd_plan *P, void *ws, size_t ws_bytes, cudaStream_t st) {
    if (!P || !ws) return set_error(AGD_STATUS_INVALID, "null plan or workspace");
    if (ws_bytes < P->L.total) return set_error(AGD_STATUS_WORKSPACE, "workspace too small");
    std::vector<Inst> insts(P->insts);
    rebase_stencils(insts.data(), (int)insts.size(), P->L, ws);
    // pageable source: the call returns once the descriptors are staged
    const cudaError_t err = cudaMemcpyAsync(static_cast<char *>(ws) + P->L.inst, insts.data(),
                                            sizeof(Inst) * insts.size(), cudaMemcpyHostToDevice, st);
    return err == cudaSuccess ? AGD_STATUS_OK : set_cuda_error("descriptor upload", err);
}

// ------------------------------------------------------------------ flow ---
// Upwind flow at every point of a solved instance (FLOW_* exports of
// cuda/Update.h:171-209 with one local iteration).  Values are not modified.
template <class TL, int MODEL>
__global__ void flow_kernel(Inst I, float *fvec, float *fwsum, float *fw, int *fidx) {
    using V = Visit<TL, MODEL>;
    constexpr int D = TL::D, P = TL::P, NACT = V::NACT;
    const int lane = threadIdx.x & 31;
    const int n_o = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (n_o >= I.size_o) return;
    const agd_instance &A = I.a;
    int xo[3] = {0, 0, 0};
    {
        int r = n_o;
#pragma unroll
        for (int k = D - 1; k >= 0; --k) { xo[k] = r % I.shape_o[k]; r /= I.shape_o[k]; }
    }
#pragma unroll
    for (int p = 0; p < P; ++p) {
        const int n_i = lane + 32 * p;
        const size_t n_t = (size_t)n_o * TL::SIZE + n_i;
        int xi[3] = {0, 0, 0}, xt[3] = {0, 0, 0};
        TL::pos(n_i, xi);
        bool in = true;
#pragma unroll
        for (int k = 0; k < D; ++k) {
            xt[k] = xo[k] * TL::extent(k) + xi[k];
            in = in && xt[k] < A.shape[k];
        }
        const bool seed = (__ldg(A.seedbits + (n_t >> 3)) >> (n_t & 7)) & 1;
        float w[NACT], fwk[NACT];
        int ev[NACT][3], side[NACT];
        if constexpr (V::kSelling) {
            float m[V::SD];
#pragma unroll
            for (int c = 0; c < V::SD; ++c) m[c] = __ldg(A.geom + (size_t)c * I.size_tot + n_t);
            if (D == 2) selling2_fast(m, w, ev);
            else selling3_fast(m, w, ev);
        } else {
            V::stencil(I, n_t, w, ev);
        }
        unsigned hide[NACT];  // neighbours hidden by a wall (Riemann offsets; see Visit::stencil_decode)
        const int wd0 = (V::kSelling && A.wall_dist && in) ? (int)__ldg(A.wall_dist + n_t) : 255;
#pragma unroll
        for (int k = 0; k < NACT; ++k)
            hide[k] = hidden_bits<D>(A, wd0, xt, ev[k], [&](const int *y) { return bilevel_index<D, TL>(y, I.shape_o); });
        float v[NACT], fsh[2 * NACT], fsh2[2 * NACT];
#pragma unroll
        for (int k = 0; k < 2 * NACT; ++k) fsh2[k] = 0.f;
        if (A.factor_radius2 > 0.f) {
            if (A.order2_threshold > 0.f) factor_shifts<D, NACT, !V::kSelling>(A, xt, ev, fsh, fsh2);
            else factor_shifts<D, NACT, !V::kSelling>(A, xt, ev, fsh);
        } else {
#pragma unroll
            for (int k = 0; k < 2 * NACT; ++k) fsh[k] = 0.f;
        }
        if constexpr (V::kDrift) {
            float raw[V::kRaw];
#pragma unroll
            for (int c = 0; c < D; ++c) raw[2 * V::SD + c] = __ldg(A.geom + (size_t)(V::SD + c) * I.size_tot + n_t);
            V::drift_shifts(raw, ev, fsh);
        }
#pragma unroll
        for (int k = 0; k < NACT; ++k) {
            side[k] = 0;
            fwk[k] = 0.f;
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                int y[3] = {0, 0, 0};
                bool ok = !((hide[k] >> s) & 1u);
#pragma unroll
                for (int c = 0; c < D; ++c) {
                    y[c] = xt[c] + (2 * s - 1) * ev[k][c];
                    ok = ok && y[c] >= 0 && y[c] < A.shape[c];
                }
                const float val = (ok ? __ldg(A.values + bilevel_index<D, TL>(y, I.shape_o)) : finf()) + fsh[2 * k + s];
                if (s == 0) v[k] = val;
                else if (v[k] > val) { v[k] = val; side[k] = 1; }
            }
        }
        if (!seed && in) {
            float vs[NACT], ws[NACT];
#pragma unroll
            for (int k = 0; k < NACT; ++k) { vs[k] = v[k]; ws[k] = w[k]; }
            unsigned o2 = 0;
            if (A.order2_threshold > 0.f) {  // second order: v corrected in place, weights 9/4
                o2 = V::order2(__ldg(A.values + n_t), vs, ws, side, [&](int k, int sd) {
                    int y[3] = {0, 0, 0};
                    bool ok = !((hide[k] >> sd) & 1u);
#pragma unroll
                    for (int c = 0; c < D; ++c) {
                        y[c] = xt[c] + 2 * (2 * sd - 1) * ev[k][c];
                        ok = ok && y[c] >= 0 && y[c] < A.shape[c];
                    }
                    return (ok ? __ldg(A.values + bilevel_index<D, TL>(y, I.shape_o)) : finf()) + fsh2[2 * k + sd];
                }, A.order2_threshold);
#pragma unroll
                for (int k = 0; k < NACT; ++k) v[k] = vs[k];
            }
            const float val = hfm_update<NACT>(__ldg(A.rhs + n_t), vs, ws);
            if (val != finf()) {
#pragma unroll
                for (int k = 0; k < NACT; ++k)
                    fwk[k] = w[k] * fmaxf(0.f, val - v[k]) * (((o2 >> k) & 1) ? 1.5f : 1.f);
            }
        }
        float vec[3] = {0.f, 0.f, 0.f}, sum = 0.f;
#pragma unroll
        for (int k = 0; k < NACT; ++k) {
            sum += fwk[k];
            const int eps = 2 * side[k] - 1;
            int y[3] = {0, 0, 0};
#pragma unroll
            for (int c = 0; c < D; ++c) {
                const int off = eps * ev[k][c];
                vec[c] += fwk[k] * float(off);
                y[c] = xt[c] + off;
            }
            if (fw) fw[(size_t)k * I.size_tot + n_t] = fwk[k];
            if (fidx) fidx[(size_t)k * I.size_tot + n_t] = fwk[k] != 0.f ? bilevel_index<D, TL>(y, I.shape_o) : kIntMax;
        }
        if (fvec)
#pragma unroll
            for (int c = 0; c < D; ++c) fvec[(size_t)c * I.size_tot + n_t] = vec[c];
        if (fwsum) fwsum[n_t] = sum;
    }
}

static int flow_impl(const agd_instance *a, float *fvec, float *fwsum, float *fw, int *fidx, cudaStream_t st) {
    WsLayout L;
    std::vector<Inst> v;
    if (!a || !layout(a, 1, L, &v, /*stencil_cache=*/false)) return set_error(AGD_STATUS_INVALID, "bad instance");
    const Inst &I = v[0];
    const int wpb = 4, grid = (I.size_o + wpb - 1) / wpb;
    switch (base_variant_of(I.a)) {
        case V_ISO2_8: flow_kernel<Tile<2, 8, 8, 1>, AGD_MODEL_ISOTROPIC><<<grid, wpb * 32, 0, st>>>(I, fvec, fwsum, fw, fidx); break;
        case V_ISO2_16: flow_kernel<Tile<2, 16, 16, 1>, AGD_MODEL_ISOTROPIC><<<grid, wpb * 32, 0, st>>>(I, fvec, fwsum, fw, fidx); break;
        case V_RIEM2_8: flow_kernel<Tile<2, 8, 8, 1>, AGD_MODEL_RIEMANN><<<grid, wpb * 32, 0, st>>>(I, fvec, fwsum, fw, fidx); break;
        case V_ISO3_4: flow_kernel<Tile<3, 4, 4, 4>, AGD_MODEL_ISOTROPIC><<<grid, wpb * 32, 0, st>>>(I, fvec, fwsum, fw, fidx); break;
        case V_RIEM3_4: flow_kernel<Tile<3, 4, 4, 4>, AGD_MODEL_RIEMANN><<<grid, wpb * 32, 0, st>>>(I, fvec, fwsum, fw, fidx); break;
        case V_RIEM2_16: flow_kernel<Tile<2, 16, 16, 1>, AGD_MODEL_RIEMANN><<<grid, wpb * 32, 0, st>>>(I, fvec, fwsum, fw, fidx); break;
        case V_DIAG2_8: flow_kernel<Tile<2, 8, 8, 1>, AGD_MODEL_DIAGONAL><<<grid, wpb * 32, 0, st>>>(I, fvec, fwsum, fw, fidx); break;
        case V_DIAG2_16: flow_kernel<Tile<2, 16, 16, 1>, AGD_MODEL_DIAGONAL><<<grid, wpb * 32, 0, st>>>(I, fvec, fwsum, fw, fidx); break;
        case V_DIAG3_4: flow_kernel<Tile<3, 4, 4, 4>, AGD_MODEL_DIAGONAL><<<grid, wpb * 32, 0, st>>>(I, fvec, fwsum, fw, fidx); break;
        case V_RAND2_8: flow_kernel<Tile<2, 8, 8, 1>, AGD_MODEL_RANDER><<<grid, wpb * 32, 0, st>>>(I, fvec, fwsum, fw, fidx); break;
        case V_RAND3_4: flow_kernel<Tile<3, 4, 4, 4>, AGD_MODEL_RANDER><<<grid, wpb * 32, 0, st>>>(I, fvec, fwsum, fw, fidx); break;
        default: return set_error(AGD_STATUS_UNSUPPORTED, "model/tile shape not built");
    }
    const cudaError_t err = cudaGetLastError();
    return err == cudaSuccess ? AGD_STATUS_OK : set_cuda_error("flow_kernel", err);
}

// ---------------------------------------------------------- layout prep ---
struct Geo {
    int nd, shape[3], si[3], so[3], size_i;
    long long size_tot, n;
};
static bool geo_of(int nd, const int *shape, const int *si, Geo &g) {
    if (nd < 1 || nd > 3) return false;
    g.nd = nd;
    g.size_i = 1;
    g.n = 1;
    long long so = 1;
    for (int k = 0; k < 3; ++k) { g.shape[k] = 1; g.si[k] = 1; g.so[k] = 1; }
    for (int k = 0; k < nd; ++k) {
        if (shape[k] <= 0 || si[k] <= 0) return false;
        g.shape[k] = shape[k];
        g.si[k] = si[k];
        g.so[k] = (shape[k] + si[k] - 1) / si[k];
        g.size_i *= si[k];
        so *= g.so[k];
        g.n *= shape[k];
    }
    g.size_tot = so * g.size_i;
    return true;
}

// bilevel index -> grid coordinates (returns false for padding)
__device__ __forceinline__ bool grid_coords(const Geo &g, long long n_t, int *x, long long &flat) {
    long long n_o = n_t / g.size_i;
    int n_i = (int)(n_t - n_o * g.size_i);
    int xo[3], xi[3];
    for (int k = g.nd - 1; k >= 0; --k) {
        xo[k] = (int)(n_o % g.so[k]); n_o /= g.so[k];
        xi[k] = n_i % g.si[k]; n_i /= g.si[k];
    }
    bool in = true;
    flat = 0;
    for (int k = 0; k < g.nd; ++k) {
        x[k] = xo[k] * g.si[k] + xi[k];
        in = in && x[k] < g.shape[k];
        flat = flat * g.shape[k] + x[k];
    }
    return in;
}

// The layout kernels below take four points a thread, neighbours along the last
// axis of a tile, in 32-bit arithmetic with shifts: tile sides that are powers of
// two, the last one at least 4, and fewer than 2^31 points (four_points()).  A
// point a thread with 64-bit divisions, as the kernels beside them for other
// shapes have it, took 107 us for a plane of 201^3 points in either direction,
// 105 us for its seed bits and 169 us for the dual metric of 200^3; four points
// 13 to 29, 10 and 61 us.
struct Geo4 {
    int nd, shape[3], so[3], lsi[3], lsz;
    unsigned size_tot, n;
};
static bool four_points(const Geo &g, Geo4 &q) {
    if (g.size_tot >= (1ll << 31) || g.si[g.nd - 1] % 4) return false;
    q.nd = g.nd;
    q.lsz = 0;
    for (int k = 0; k < 3; ++k) {
        int l = 0;
        while ((1 << l) < g.si[k]) ++l;
        if ((1 << l) != g.si[k]) return false;
        q.shape[k] = g.shape[k];
        q.so[k] = g.so[k];
        q.lsi[k] = l;
        q.lsz += l;
    }
    q.size_tot = (unsigned)g.size_tot;
    q.n = (unsigned)g.n;
    return true;
}

// The points n_t .. n_t + 3 (n_t a multiple of 4): how many of them are in the grid
// (from the first on), and the grid index of the first.
__device__ __forceinline__ int four_coords(const Geo4 &g, unsigned n_t, unsigned &flat) {
    unsigned n_o = n_t >> g.lsz, n_i = n_t & ((1u << g.lsz) - 1u);
    int x[3] = {0, 0, 0};
#pragma unroll
    for (int k = 2; k >= 0; --k) {
        if (k >= g.nd) continue;
        const unsigned q = k == 0 ? 0u : n_o / (unsigned)g.so[k];
        x[k] = (int)(((n_o - q * g.so[k]) << g.lsi[k]) + (n_i & ((1u << g.lsi[k]) - 1u)));
        n_o = q;
        n_i >>= g.lsi[k];
    }
    bool in = true;
    flat = 0;
    int left = 0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        if (k >= g.nd) continue;
        flat = flat * g.shape[k] + x[k];
        left = g.shape[k] - x[k];
        in = in && left > 0;
    }
    return in ? min(left, 4) : 0;
}

// block_expand: grid.y is the plane.  Vector loads where the rows allow them.
__global__ void __launch_bounds__(256) expand4_kernel(Geo4 g, const float *__restrict__ src, int bcast, float pad, int wide,
                                                      float *__restrict__ dst) {
    const unsigned n_t = 4u * (blockIdx.x * blockDim.x + threadIdx.x);
    if (n_t >= g.size_tot) return;
    unsigned flat;
    const int c = four_coords(g, n_t, flat);
    float v[4] = {pad, pad, pad, pad};
    if (bcast) {
        const float b = __ldg(src + blockIdx.y);
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = j < c ? b : pad;
    } else {
        const float *p = src + (size_t)blockIdx.y * g.n + flat;
        if (wide && c == 4) {
            const float4 w = __ldg(reinterpret_cast<const float4 *>(p));
            v[0] = w.x; v[1] = w.y; v[2] = w.z; v[3] = w.w;
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (j < c) v[j] = __ldg(p + j);
        }
    }
    *reinterpret_cast<float4 *>(dst + (size_t)blockIdx.y * g.size_tot + n_t) = make_float4(v[0], v[1], v[2], v[3]);
}

__global__ void __launch_bounds__(256) squeeze4_kernel(Geo4 g, const float *__restrict__ src, int wide, float *__restrict__ dst) {
    const unsigned n_t = 4u * (blockIdx.x * blockDim.x + threadIdx.x);
    if (n_t >= g.size_tot) return;
    unsigned flat;
    const int c = four_coords(g, n_t, flat);
    if (c == 0) return;
    const float4 w = __ldg(reinterpret_cast<const float4 *>(src + (size_t)blockIdx.y * g.size_tot + n_t));
    float *p = dst + (size_t)blockIdx.y * g.n + flat;
    if (wide && c == 4) {
        *reinterpret_cast<float4 *>(p) = w;
    } else {
        const float v[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (j < c) p[j] = v[j];
    }
}

// Seed bits of a grid without seeds: the padding's.
__global__ void __launch_bounds__(256) seedbits4_kernel(Geo4 g, unsigned *__restrict__ bits) {
    const unsigned n_t = 4u * (blockIdx.x * blockDim.x + threadIdx.x);  // (whole warps: size_tot is a multiple of 32)
    unsigned flat, word = 0;
    if (n_t < g.size_tot) word = ((0xfu << four_coords(g, n_t, flat)) & 0xfu) << (n_t & 31u);
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) word |= __shfl_xor_sync(kFull, word, o);
    if (n_t < g.size_tot && (n_t & 31u) == 0u) bits[n_t >> 5] = word;
}

__global__ void block_expand_kernel(Geo g, int nplanes, const float *src, int bcast, float pad, float *dst) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= g.size_tot * nplanes) return;
    const int plane = (int)(i / g.size_tot);
    const long long n_t = i - plane * g.size_tot;
    int x[3];
    long long flat;
    const bool in = grid_coords(g, n_t, x, flat);
    dst[i] = in ? (bcast ? src[plane] : src[plane * g.n + flat]) : pad;
}

__global__ void block_squeeze_kernel(Geo g, int nplanes, const float *src, float *dst) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= g.n * nplanes) return;
    const int plane = (int)(i / g.n);
    long long r = i - plane * g.n;
    int x[3];
    for (int k = g.nd - 1; k >= 0; --k) { x[k] = (int)(r % g.shape[k]); r /= g.shape[k]; }
    long long n_o = 0, n_i = 0;
    for (int k = 0; k < g.nd; ++k) {
        n_o = n_o * g.so[k] + x[k] / g.si[k];
        n_i = n_i * g.si[k] + x[k] % g.si[k];
    }
    dst[i] = src[plane * g.size_tot + n_o * g.size_i + n_i];
}

// Dual metric of M' = diag(h) M diag(h) (Riemann.with_costs, then dual), by the
// adjugate formula, packed [d00, d10, d11(, d20, d21, d22)]; with is_dual, m
// already holds the dual metric and is only rescaled (dualMetric.with_speeds(h)).
__device__ __forceinline__ void geom_at(int nd, const float *m, int is_dual, const float h[3], float *out) {
    if (nd == 2) {
        float a = m[0], b = m[1], c = m[2];
        if (is_dual) {  // entries / (h_i h_j)
            out[0] = a / (h[0] * h[0]); out[1] = b / (h[1] * h[0]); out[2] = c / (h[1] * h[1]);
            return;
        }
        a = a * (h[0] * h[0]); b = b * (h[1] * h[0]); c = c * (h[1] * h[1]);
        const float det = a * c - b * b;
        out[0] = c / det;
        out[1] = -b / det;
        out[2] = a / det;
        return;
    }
    float s[6];
    int k = 0;
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j <= i; ++j, ++k) s[k] = is_dual ? m[k] / (h[i] * h[j]) : m[k] * (h[i] * h[j]);
    if (is_dual) {
        for (int c = 0; c < 6; ++c) out[c] = s[c];
        return;
    }
    // symmetric [[a,b,d],[b,c,e],[d,e,f]] with s = [a, b, c, d, e, f]
    const float a = s[0], b = s[1], c = s[2], d = s[3], e = s[4], f = s[5];
    const float A00 = c * f - e * e, A10 = d * e - b * f, A11 = a * f - d * d;
    const float A20 = b * e - c * d, A21 = b * d - a * e, A22 = a * c - b * b;
    const float det = a * A00 + b * A10 + d * A20;
    out[0] = A00 / det; out[1] = A10 / det; out[2] = A11 / det;
    out[3] = A20 / det; out[4] = A21 / det; out[5] = A22 / det;
}

// Geometry planes in tile layout; +inf at padding points.
__global__ void prep_geom_kernel(Geo g, const float *metric, int bcast, int is_dual, double h0, double h1,
                                 double h2, float *geom) {
    const long long n_t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (n_t >= g.size_tot) return;
    const int sd = g.nd * (g.nd + 1) / 2;
    int x[3];
    long long flat;
    const bool in = grid_coords(g, n_t, x, flat);
    if (!in) {
        for (int c = 0; c < sd; ++c) geom[c * g.size_tot + n_t] = finf();
        return;
    }
    const float h[3] = {(float)h0, (float)h1, (float)h2};
    float out[6];
    geom_at(g.nd, bcast ? metric : metric + flat * sd, is_dual, h, out);
    for (int c = 0; c < sd; ++c) geom[c * g.size_tot + n_t] = out[c];
}

// The solver's arrays of one instance in one launch: values +inf, the right-hand
// side (cost, or 1), the seed bits and the seeds, given by value (bilevel
// indices, in order: a later duplicate wins).
constexpr int kArgSeeds = 32;
struct ArgSeeds {
    int n, at[kArgSeeds];
    float host_value[kArgSeeds];
    const float *value;  // device values, or NULL: host_value
};
__global__ void __launch_bounds__(256) prep_args4_kernel(Geo4 g, const __grid_constant__ ArgSeeds seeds,
                                                         const float *__restrict__ cost, int bcast, int wide,
                                                         float *__restrict__ values, float *__restrict__ rhs,
                                                         unsigned *__restrict__ bits) {
    const unsigned n_t = 4u * (blockIdx.x * blockDim.x + threadIdx.x);
    const bool on = n_t < g.size_tot;
    unsigned word = 0;
    if (on) {
        unsigned flat;
        const int c = four_coords(g, n_t, flat);
        float v[4];
        if (!cost || bcast) {
            const float b = cost ? __ldg(cost) : 1.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = j < c ? b : finf();
        } else if (wide && c == 4) {
            const float4 w = __ldg(reinterpret_cast<const float4 *>(cost + flat));
            v[0] = w.x; v[1] = w.y; v[2] = w.z; v[3] = w.w;
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = j < c ? __ldg(cost + flat + j) : finf();
        }
        unsigned nib = (0xfu << c) & 0xfu;
        for (int s = 0; s < seeds.n; ++s) {
            const unsigned at = (unsigned)seeds.at[s];
            if ((at ^ n_t) & ~3u) continue;
            const float x = seeds.value ? __ldg(seeds.value + s) : seeds.host_value[s];
            nib |= 1u << (at & 3u);
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = (at & 3u) == j ? x : v[j];
        }
        *reinterpret_cast<float4 *>(rhs + n_t) = make_float4(v[0], v[1], v[2], v[3]);
        if (values) *reinterpret_cast<float4 *>(values + n_t) = make_float4(finf(), finf(), finf(), finf());
        word = nib << (n_t & 31u);
    }
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) word |= __shfl_xor_sync(kFull, word, o);
    if (on && (n_t & 31u) == 0u) bits[n_t >> 5] = word;
}

// Sum (double) and number of the values that are not NaN, added to out.
__global__ void __launch_bounds__(256) nan_sum_kernel(const float *__restrict__ x, long long n, double *out) {
    double s = 0.0, c = 0.0;
    for (long long i = blockIdx.x * 256ll + threadIdx.x; i < n; i += gridDim.x * 256ll) {
        const float v = __ldg(x + i);
        if (v == v) {
            s += v;
            c += 1.0;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        s += __shfl_xor_sync(kFull, s, o);
        c += __shfl_xor_sync(kFull, c, o);
    }
    __shared__ double part[2][8];
    if ((threadIdx.x & 31) == 0) {
        part[0][threadIdx.x >> 5] = s;
        part[1][threadIdx.x >> 5] = c;
    }
    __syncthreads();
    if (threadIdx.x < 2) {
        double t = 0.0;
        for (int k = 0; k < 8; ++k) t += part[threadIdx.x][k];
        atomicAdd(out + threadIdx.x, t);
    }
}

template <int D>
__global__ void __launch_bounds__(256) prep_geom4_kernel(Geo4 g, const float *__restrict__ metric, int bcast, int is_dual,
                                                         float h0, float h1, float h2, int wide, float *__restrict__ geom) {
    constexpr int SD = D * (D + 1) / 2;
    const unsigned n_t = 4u * (blockIdx.x * blockDim.x + threadIdx.x);
    if (n_t >= g.size_tot) return;
    unsigned flat;
    const int c = four_coords(g, n_t, flat);
    const float h[3] = {h0, h1, h2};
    float m[4 * SD], out[SD][4];
    if (bcast) {
#pragma unroll
        for (int i = 0; i < 4 * SD; ++i) m[i] = __ldg(metric + i % SD);
    } else if (wide && c == 4) {  // the four points' metrics are 4 SD consecutive floats
#pragma unroll
        for (int i = 0; i < SD; ++i) {
            const float4 w = __ldg(reinterpret_cast<const float4 *>(metric + (size_t)flat * SD) + i);
            m[4 * i] = w.x; m[4 * i + 1] = w.y; m[4 * i + 2] = w.z; m[4 * i + 3] = w.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < 4 * SD; ++i) m[i] = i < c * SD ? __ldg(metric + (size_t)flat * SD + i) : 1.f;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        float o[6];
        geom_at(D, m + j * SD, is_dual, h, o);
#pragma unroll
        for (int k = 0; k < SD; ++k) out[k][j] = j < c ? o[k] : finf();
    }
#pragma unroll
    for (int k = 0; k < SD; ++k)
        *reinterpret_cast<float4 *>(geom + (size_t)k * g.size_tot + n_t) = make_float4(out[k][0], out[k][1], out[k][2], out[k][3]);
}

// Diagonal model: the squared dual costs 1/(c_k h_k)^2 of metric.with_costs(h)
// (or (d_k / h_k)^2 of dualMetric.with_speeds(h)) per axis, in float as the
// reference forms them (_SetGeometry.py:134-135), +inf at padding.
__device__ __forceinline__ void diag_at(int nd, const float *c, int is_dual, const float h[3], float *out) {
    for (int k = 0; k < nd; ++k) {
        const float v = is_dual ? c[k] * (1.f / h[k]) : 1.f / (c[k] * h[k]);
        out[k] = v * v;
    }
}

__global__ void prep_diag_kernel(Geo g, const float *costs, int bcast, int is_dual, double h0, double h1, double h2,
                                 float *geom) {
    const long long n_t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (n_t >= g.size_tot) return;
    int x[3];
    long long flat;
    const bool in = grid_coords(g, n_t, x, flat);
    const float h[3] = {(float)h0, (float)h1, (float)h2};
    float out[3];
    if (in) diag_at(g.nd, bcast ? costs : costs + flat * g.nd, is_dual, h, out);
    for (int k = 0; k < g.nd; ++k) geom[k * g.size_tot + n_t] = in ? out[k] : finf();
}

// Inverse of a packed symmetric matrix [a00, a10, a11(, a20, a21, a22)] by the
// adjugate formula.
__device__ __forceinline__ void sym_inverse(int nd, const float *s, float *out) {
    if (nd == 2) {
        const float det = s[0] * s[2] - s[1] * s[1];
        out[0] = s[2] / det;
        out[1] = -s[1] / det;
        out[2] = s[0] / det;
        return;
    }
    const float a = s[0], b = s[1], c = s[2], d = s[3], e = s[4], f = s[5];
    const float A00 = c * f - e * e, A10 = d * e - b * f, A11 = a * f - d * d;
    const float A20 = b * e - c * d, A21 = b * d - a * e, A22 = a * c - b * b;
    const float det = a * A00 + b * A10 + d * A20;
    out[0] = A00 / det; out[1] = A10 / det; out[2] = A11 / det;
    out[3] = A20 / det; out[4] = A21 / det; out[5] = A22 / det;
}

// Rander model: (inverse of m * outer(h, h), w * h) per point, +inf at padding
// (Metrics/rander.py:61-68).  With is_dual the input (m_d, w_d) is the dual
// metric: scaled by with_speeds(h), then turned into the metric by
// rander.py:35-39, m = (1 + <w_d, s w_d>) s, w = -s w_d with s = (m_d - w_d w_d^T)^-1,
// so that the inverse of m is (m_d - w_d w_d^T) / (1 + <w_d, s w_d>).
// out: the sd planes of the inverse metric, then the nd of the drift.
__device__ __forceinline__ void rander_at(int nd, const float *src, int is_dual, const float hh[3], float *out) {
    const int sd = nd * (nd + 1) / 2;
    float hs[3];  // the grid scales (metric), or their inverses (with_speeds of a dual metric)
    for (int k = 0; k < nd; ++k) hs[k] = is_dual ? 1.f / hh[k] : hh[k];
    float m[6], w[3], mi[6];
    int q = 0;
    for (int i = 0; i < nd; ++i)
        for (int j = 0; j <= i; ++j, ++q) m[q] = src[q] * (hs[i] * hs[j]);  // m * outer(h, h)
    for (int k = 0; k < nd; ++k) w[k] = src[sd + k] * hs[k];
    if (!is_dual) {
        sym_inverse(nd, m, mi);
    } else {
        float t[6], s_[6], om[3] = {0.f, 0.f, 0.f};
        q = 0;
        for (int i = 0; i < nd; ++i)
            for (int j = 0; j <= i; ++j, ++q) t[q] = m[q] - w[i] * w[j];
        sym_inverse(nd, t, s_);
        for (int i = 0; i < nd; ++i)
            for (int j = 0; j < nd; ++j) om[i] += s_[i >= j ? i * (i + 1) / 2 + j : j * (j + 1) / 2 + i] * w[j];
        float wo = 0.f;
        for (int i = 0; i < nd; ++i) wo += w[i] * om[i];
        for (int c = 0; c < sd; ++c) mi[c] = t[c] / (1.f + wo);
        for (int k = 0; k < nd; ++k) w[k] = -om[k];
    }
    for (int c = 0; c < sd; ++c) out[c] = mi[c];
    for (int k = 0; k < nd; ++k) out[sd + k] = w[k];
}

__global__ void prep_rander_kernel(Geo g, const float *metric, int bcast, int is_dual, double h0, double h1,
                                   double h2, float *geom) {
    const long long n_t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (n_t >= g.size_tot) return;
    const int nd = g.nd, sd = nd * (nd + 1) / 2;
    int x[3];
    long long flat;
    const bool in = grid_coords(g, n_t, x, flat);
    const float hh[3] = {(float)h0, (float)h1, (float)h2};
    float out[9];
    if (in) rander_at(nd, bcast ? metric : metric + flat * (sd + nd), is_dual, hh, out);
    for (int c = 0; c < sd + nd; ++c) geom[c * g.size_tot + n_t] = in ? out[c] : finf();
}

// Seed bits: one 32-bit word (32 points) per thread, padding bits set.
__global__ void seedbits_init_kernel(Geo g, unsigned *bits) {
    const long long wi = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (wi * 32 >= g.size_tot) return;
    unsigned word = 0;
    for (int b = 0; b < 32; ++b) {
        int x[3];
        long long flat;
        if (!grid_coords(g, wi * 32 + b, x, flat)) word |= 1u << b;
    }
    bits[wi] = word;
}

// Seeds in order (a later duplicate overrides an earlier one, as numpy assignment does).
// walls (grid layout, or NULL): a seed on a wall keeps the wall's +inf right-hand
// side, since the reference writes the walls after the seeds.
__device__ void place_seeds(const Geo &g, const int *idx, const float *vals, int n, float *rhs, unsigned *bits,
                            unsigned char *trigger, int *bad, const uint8_t *walls = nullptr) {
    for (int s = 0; s < n; ++s) {
        long long n_o = 0, n_i = 0, flat = 0;
        bool ok = true;
        for (int k = 0; k < g.nd; ++k) {
            const int xk = idx[s * g.nd + k];
            ok = ok && xk >= 0 && xk < g.shape[k];
            n_o = n_o * g.so[k] + (ok ? xk / g.si[k] : 0);
            n_i = n_i * g.si[k] + (ok ? xk % g.si[k] : 0);
            flat = flat * g.shape[k] + (ok ? xk : 0);
        }
        if (!ok) {
            if (bad) *bad = 1;
            continue;
        }
        const long long n_t = n_o * g.size_i + n_i;
        if (rhs && !(walls && walls[flat])) rhs[n_t] = vals ? vals[s] : 0.f;
        if (bits) bits[n_t >> 5] |= 1u << (n_t & 31);
        if (trigger) trigger[n_o] = 1;
    }
}

__global__ void seeds_kernel(Geo g, const int *idx, const float *vals, int n, float *rhs, unsigned *bits,
                             unsigned char *trigger, int *bad) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    place_seeds(g, idx, vals, n, rhs, bits, trigger, bad);
}

struct BatchPrep {
    Geo g;
    int si_log2[3];  // log2 of the tile sides, or -1 (all) if one is not a power of two
    int n, model, is_dual, nseeds;
    int nmet, ngeom;  // metric floats per point, geometry planes
    float h[3];
    const float *metric, *cost, *seed_values;
    const int *seed_index;
    float *geom, *rhs, *values;
    unsigned *bits;
    int *bad;
    const uint8_t *walls;
    long long walls_stride;  // 0: one mask for every instance
    uint8_t *trigger;
    long long size_o;  // tiles of an instance
};

// Bilevel index -> grid coordinates for instances of fewer than 2^31 points,
// in 32-bit arithmetic, the in-tile part by shifts when the tile sides are
// powers of two (si_log2 >= 0).  Returns false for padding.
__device__ __forceinline__ bool grid_coords32(const Geo &g, const int *si_log2, int n_t, int &flat) {
    int n_o, n_i, xo[3], xi[3];
    if (si_log2[0] >= 0) {
        const int lsz = si_log2[0] + si_log2[1] + si_log2[2];
        n_o = n_t >> lsz;
        n_i = n_t & ((1 << lsz) - 1);
        for (int k = g.nd - 1; k >= 0; --k) {
            xi[k] = n_i & ((1 << si_log2[k]) - 1);
            n_i >>= si_log2[k];
        }
    } else {
        n_o = n_t / g.size_i;
        n_i = n_t - n_o * g.size_i;
        for (int k = g.nd - 1; k >= 0; --k) {
            xi[k] = n_i % g.si[k];
            n_i /= g.si[k];
        }
    }
    for (int k = g.nd - 1; k >= 0; --k) {
        const int q = n_o / g.so[k];
        xo[k] = n_o - q * g.so[k];
        n_o = q;
    }
    bool in = true;
    flat = 0;
    for (int k = 0; k < g.nd; ++k) {
        const int x = xo[k] * g.si[k] + xi[k];
        in = in && x < g.shape[k];
        flat = flat * g.shape[k] + x;
    }
    return in;
}

// Grid rows of blocks: blockIdx.y is the instance, the blocks of a row stride
// over its points (warps stay 32-aligned because size_tot is a multiple of 32,
// so each warp's ballot is one bit word).
__global__ void prep_batch_kernel(BatchPrep A) {
    const int inst = blockIdx.y;
    const int size_tot = (int)A.g.size_tot;
    for (int n_t = blockIdx.x * blockDim.x + threadIdx.x; n_t < size_tot; n_t += gridDim.x * blockDim.x) {
        const long long i = (long long)inst * size_tot + n_t;
        int flat;
        const bool in = grid_coords32(A.g, A.si_log2, n_t, flat);
        const bool wall = in && A.walls && A.walls[inst * A.walls_stride + flat];
        A.values[i] = finf();
        A.rhs[i] = in && !wall ? (A.cost ? A.cost[inst * A.g.n + flat] : 1.f) : finf();
        if (A.ngeom) {
            float out[9];
            if (in) {
                const float *m = A.metric + (inst * A.g.n + flat) * A.nmet;
                if (A.model == AGD_MODEL_RIEMANN) geom_at(A.g.nd, m, A.is_dual, A.h, out);
                else if (A.model == AGD_MODEL_DIAGONAL) diag_at(A.g.nd, m, A.is_dual, A.h, out);
                else rander_at(A.g.nd, m, A.is_dual, A.h, out);
            }
            float *geo = A.geom + (long long)inst * A.ngeom * A.g.size_tot + n_t;
            for (int c = 0; c < A.ngeom; ++c) geo[c * A.g.size_tot] = in ? out[c] : finf();
        }
        if (A.trigger && n_t % A.g.size_i == 0) A.trigger[inst * A.size_o + n_t / A.g.size_i] = 0;
        const unsigned pad = __ballot_sync(0xffffffffu, !in || wall);
        if ((threadIdx.x & 31) == 0) A.bits[i >> 5] = pad;
    }
}

__global__ void seeds_batch_kernel(BatchPrep A) {
    const int inst = blockIdx.x * blockDim.x + threadIdx.x;
    if (inst >= A.n) return;
    place_seeds(A.g, A.seed_index + (long long)inst * A.nseeds * A.g.nd,
                A.seed_values ? A.seed_values + (long long)inst * A.nseeds : nullptr, A.nseeds,
                A.rhs + inst * A.g.size_tot, A.bits + inst * (A.g.size_tot / 32),
                A.trigger ? A.trigger + inst * A.size_o : nullptr, A.bad,
                A.walls ? A.walls + inst * A.walls_stride : nullptr);
}

// Wall distances in tile layout (255 at padding); with rhs / bits, the wall
// points become seeds of value +inf (_SetArgs.py:124-126).  One thread per
// point; whole warps leave together (size_tot is a multiple of 32), and the
// wall bits of a warp are one seed-bit word, which only that warp writes.
__global__ void walls_kernel(Geo g, const uint8_t *walls, const uint8_t *dist, uint8_t *wall_dist, float *rhs,
                             unsigned *bits) {
    const long long n_t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (n_t >= g.size_tot) return;
    int x[3];
    long long flat;
    const bool in = grid_coords(g, n_t, x, flat);
    const bool wall = in && walls[flat] != 0;
    wall_dist[n_t] = in ? dist[flat] : (uint8_t)255;
    if (wall && rhs) rhs[n_t] = finf();
    const unsigned word = __ballot_sync(kFull, wall);
    if (bits && word && (threadIdx.x & 31) == 0) bits[n_t >> 5] |= word;
}

// Wall distances of nb instances, grid layout (dist) -> tile layout (255 at padding).
__global__ void wall_dist_batch_kernel(Geo g, int nb, const uint8_t *dist, uint8_t *wall_dist) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= g.size_tot * nb) return;
    const long long inst = i / g.size_tot, n_t = i - inst * g.size_tot;
    int x[3];
    long long flat;
    const bool in = grid_coords(g, n_t, x, flat);
    wall_dist[i] = in ? dist[inst * g.n + flat] : (uint8_t)255;
}

// Selling's decomposition of n packed symmetric matrices in the planar layouts
// of the reference's VoronoiDecomposition kernel (Kernel_VoronoiDecomposition.h:45-69):
// m[c * n + p] (lower triangle, row major; FULL: the whole matrices, m[(i D + j)
// n + p], of which the lower triangle is read), weights[r * n + p],
// offsets[(i * SD + r) * n + p] for coordinate i of offset r.  Dimension 1: the
// weight is the matrix, the offset 1.  One thread per matrix, grid stride.
template <int D, class OffT, bool FULL>
__global__ void voronoi_kernel(const float *__restrict__ m, long long n, float *__restrict__ w,
                               OffT *__restrict__ e) {
    constexpr int SD = D * (D + 1) / 2;
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x) {
        float mm[SD], ww[SD];
        int ee[SD][3];
        int c = 0;
#pragma unroll
        for (int i = 0; i < D; ++i)
#pragma unroll
            for (int j = 0; j <= i; ++j, ++c) mm[c] = __ldg(m + (FULL ? i * D + j : c) * n + p);
        if constexpr (D == 1) {
            ww[0] = mm[0];
            ee[0][0] = 1;
        } else if constexpr (D == 2) {
            selling2_fast(mm, ww, ee);
        } else {
            selling3_fast(mm, ww, ee);
        }
#pragma unroll
        for (int r = 0; r < SD; ++r) {
            __stcs(w + r * n + p, ww[r]);
#pragma unroll
            for (int i = 0; i < D; ++i) __stcs(e + (i * SD + r) * n + p, (OffT)ee[r][i]);
        }
    }
}

template <int D, bool FULL>
static void launch_voronoi(const float *m, long long n, float *w, void *e, int offset_bytes, cudaStream_t st) {
    const unsigned blocks = (unsigned)std::min<long long>((n + 127) / 128, 148LL * 64);
    switch (offset_bytes) {
        case 1: voronoi_kernel<D, signed char, FULL><<<blocks, 128, 0, st>>>(m, n, w, static_cast<signed char *>(e)); break;
        case 2: voronoi_kernel<D, short, FULL><<<blocks, 128, 0, st>>>(m, n, w, static_cast<short *>(e)); break;
        case 4: voronoi_kernel<D, int, FULL><<<blocks, 128, 0, st>>>(m, n, w, static_cast<int *>(e)); break;
        default: voronoi_kernel<D, long long, FULL><<<blocks, 128, 0, st>>>(m, n, w, static_cast<long long *>(e)); break;
    }
}

static int voronoi(int ndim, const float *m, long long n, float *weights, void *offsets, int offset_bytes, bool full,
                   cudaStream_t st) {
    if (ndim < 1 || ndim > 3 || n < 0 || (n > 0 && (!m || !weights || !offsets)) ||
        (offset_bytes != 1 && offset_bytes != 2 && offset_bytes != 4 && offset_bytes != 8))
        return set_error(AGD_STATUS_INVALID, "agd_voronoi_decomposition: bad arguments (ndim 1 to 3, "
                                             "offset_bytes 1, 2, 4 or 8)");
    if (n == 0) return AGD_STATUS_OK;
    if (ndim == 1) launch_voronoi<1, false>(m, n, weights, offsets, offset_bytes, st);
    else if (ndim == 2 && full) launch_voronoi<2, true>(m, n, weights, offsets, offset_bytes, st);
    else if (ndim == 2) launch_voronoi<2, false>(m, n, weights, offsets, offset_bytes, st);
    else if (full) launch_voronoi<3, true>(m, n, weights, offsets, offset_bytes, st);
    else launch_voronoi<3, false>(m, n, weights, offsets, offset_bytes, st);
    const cudaError_t err = cudaGetLastError();
    return err == cudaSuccess ? AGD_STATUS_OK : set_cuda_error("voronoi_decomposition", err);
}

__global__ void selling_kernel(int nd, const float *m, int n, float *w, int *e) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    float ww[6];
    int ee[6][3];
    if (nd == 2) {
        float mm[3] = {m[3 * p], m[3 * p + 1], m[3 * p + 2]};
        selling2(mm, ww, ee);
        for (int r = 0; r < 3; ++r) { w[3 * p + r] = ww[r]; e[(3 * p + r) * 2] = ee[r][0]; e[(3 * p + r) * 2 + 1] = ee[r][1]; }
    } else {
        float mm[6];
        for (int c = 0; c < 6; ++c) mm[c] = m[6 * p + c];
        selling3(mm, ww, ee);
        for (int r = 0; r < 6; ++r) { w[6 * p + r] = ww[r]; for (int c = 0; c < 3; ++c) e[(6 * p + r) * 3 + c] = ee[r][c]; }
    }
}

static inline unsigned blocks_for(long long n, int bs) { return (unsigned)((n + bs - 1) / bs); }
static bool on16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace agd

using namespace agd;

extern "C" {

int agd_plan_create(const agd_instance *inst, int n, agd_plan **plan) {
    clear_error();
    return plan_create(inst, n, plan);
}

void agd_plan_destroy(agd_plan *plan) { delete plan; }

size_t agd_plan_workspace_bytes(const agd_plan *plan) { return plan ? plan->L.total : 0; }

int agd_plan_upload(const agd_plan *plan, void *workspace, size_t workspace_bytes, agd_stream_t stream) {
    clear_error();
    return plan_upload(plan, workspace, workspace_bytes, (cudaStream_t)stream);
}

int agd_plan_run(const agd_plan *plan, void *workspace, size_t workspace_bytes, agd_stats *stats,
                 const agd_launch *launch, agd_stream_t stream) {
    clear_error();
    return plan_run(plan, workspace, workspace_bytes, stats, launch, (cudaStream_t)stream);
}

size_t agd_eikonal_workspace_bytes(const agd_instance *inst, int n) {
    WsLayout L;
    if (!inst || n <= 0 || !layout(inst, n, L, static_cast<Inst *>(nullptr))) return 0;
    return L.total;
}

int agd_eikonal_solve(const agd_instance *inst, int n, void *workspace, size_t workspace_bytes, agd_stats *stats,
                      const agd_launch *launch, agd_stream_t stream) {
    clear_error();
    agd_plan *P = nullptr;
    int rc = plan_create(inst, n, &P);
    if (rc != AGD_STATUS_OK) return rc;
    rc = plan_upload(P, workspace, workspace_bytes, (cudaStream_t)stream);
    if (rc == AGD_STATUS_OK) rc = plan_run(P, workspace, workspace_bytes, stats, launch, (cudaStream_t)stream);
    delete P;
    return rc;
}

int agd_eikonal_solve_fixed_scratch(const agd_instance *inst, int n, agd_stats *stats, const agd_launch *launch,
                                    agd_stream_t stream) {
    clear_error();
    return fixed_scratch_solve(inst, n, stats, launch, (cudaStream_t)stream);
}

int agd_flow(const agd_instance *inst, float *flow_vector, float *flow_weightsum, float *flow_weights,
             int32_t *flow_indices, agd_stream_t stream) {
    clear_error();
    return flow_impl(inst, flow_vector, flow_weightsum, flow_weights, flow_indices, (cudaStream_t)stream);
}

int agd_prep_geom(int ndim, const int *shape, const int *shape_i, const float *metric, int broadcast, int is_dual,
                  const double *grid_scales, float *geom, agd_stream_t stream) {
    clear_error();
    Geo g;
    if (ndim < 2 || !geo_of(ndim, shape, shape_i, g) || !metric || !geom || !grid_scales)
        return set_error(AGD_STATUS_INVALID, "agd_prep_geom: bad arguments");
    Geo4 q;
    if (four_points(g, q) && on16(geom)) {
        const int wide = g.shape[ndim - 1] % 4 == 0 && on16(metric);
        const float h0 = (float)grid_scales[0], h1 = (float)grid_scales[1], h2 = ndim == 3 ? (float)grid_scales[2] : 1.f;
        const unsigned nb = blocks_for(g.size_tot / 4, 256);
        if (ndim == 2) prep_geom4_kernel<2><<<nb, 256, 0, (cudaStream_t)stream>>>(q, metric, broadcast, is_dual, h0, h1, h2, wide, geom);
        else prep_geom4_kernel<3><<<nb, 256, 0, (cudaStream_t)stream>>>(q, metric, broadcast, is_dual, h0, h1, h2, wide, geom);
        const cudaError_t err = cudaGetLastError();
        return err == cudaSuccess ? AGD_STATUS_OK : set_cuda_error("prep_geom", err);
    }
    prep_geom_kernel<<<blocks_for(g.size_tot, 256), 256, 0, (cudaStream_t)stream>>>(
        g, metric, broadcast, is_dual, grid_scales[0], grid_scales[1], ndim == 3 ? grid_scales[2] : 1.0, geom);
    const cudaError_t err = cudaGetLastError();
    return err == cudaSuccess ? AGD_STATUS_OK : set_cuda_error("prep_geom", err);
}

int agd_prep_geom_diagonal(int ndim, const int *shape, const int *shape_i, const float *costs, int broadcast,
                           int is_dual, const double *grid_scales, float *geom, agd_stream_t stream) {
    clear_error();
    Geo g;
    if (ndim < 1 || !geo_of(ndim, shape, shape_i, g) || !costs || !geom || !grid_scales)
        return set_error(AGD_STATUS_INVALID, "agd_prep_geom_diagonal: bad arguments");
    prep_diag_kernel<<<blocks_for(g.size_tot, 256), 256, 0, (cudaStream_t)stream>>>(
        g, costs, broadcast, is_dual, grid_scales[0], ndim > 1 ? grid_scales[1] : 1.0, ndim > 2 ? grid_scales[2] : 1.0,
        geom);
    const cudaError_t err = cudaGetLastError();
    return err == cudaSuccess ? AGD_STATUS_OK : set_cuda_error("prep_geom_diagonal", err);
}

int agd_prep_geom_rander(int ndim, const int *shape, const int *shape_i, const float *metric, int broadcast,
                         int is_dual, const double *grid_scales, float *geom, agd_stream_t stream) {
    clear_error();
    Geo g;
    if ((ndim != 2 && ndim != 3) || !geo_of(ndim, shape, shape_i, g) || !metric || !geom || !grid_scales)
        return set_error(AGD_STATUS_INVALID, "agd_prep_geom_rander: bad arguments");
    prep_rander_kernel<<<blocks_for(g.size_tot, 256), 256, 0, (cudaStream_t)stream>>>(
        g, metric, broadcast, is_dual, grid_scales[0], grid_scales[1], ndim == 3 ? grid_scales[2] : 1.0, geom);
    const cudaError_t err = cudaGetLastError();
    return err == cudaSuccess ? AGD_STATUS_OK : set_cuda_error("prep_geom_rander", err);
}

int agd_block_expand(int ndim, const int *shape, const int *shape_i, int nplanes, const float *src, int src_broadcast,
                     float pad, float *dst, agd_stream_t stream) {
    clear_error();
    Geo g;
    if (!geo_of(ndim, shape, shape_i, g) || nplanes < 1 || !src || !dst)
        return set_error(AGD_STATUS_INVALID, "agd_block_expand: bad arguments");
    Geo4 q;
    if (four_points(g, q) && on16(dst) && nplanes <= 65535) {
        const int wide = g.shape[ndim - 1] % 4 == 0 && on16(src);
        expand4_kernel<<<dim3(blocks_for(g.size_tot / 4, 256), nplanes), 256, 0, (cudaStream_t)stream>>>(q, src, src_broadcast, pad,
                                                                                                        wide, dst);
    } else {
        block_expand_kernel<<<blocks_for(g.size_tot * nplanes, 256), 256, 0, (cudaStream_t)stream>>>(
            g, nplanes, src, src_broadcast, pad, dst);
    }
    const cudaError_t err = cudaGetLastError();
    return err == cudaSuccess ? AGD_STATUS_OK : set_cuda_error("block_expand", err);
}

int agd_block_squeeze(int ndim, const int *shape, const int *shape_i, int nplanes, const float *src, float *dst,
                      agd_stream_t stream) {
    clear_error();
    Geo g;
    if (!geo_of(ndim, shape, shape_i, g) || nplanes < 1 || !src || !dst)
        return set_error(AGD_STATUS_INVALID, "agd_block_squeeze: bad arguments");
    Geo4 q;
    if (four_points(g, q) && on16(src) && nplanes <= 65535) {
        const int wide = g.shape[ndim - 1] % 4 == 0 && on16(dst);
        squeeze4_kernel<<<dim3(blocks_for(g.size_tot / 4, 256), nplanes), 256, 0, (cudaStream_t)stream>>>(q, src, wide, dst);
    } else {
        block_squeeze_kernel<<<blocks_for(g.n * nplanes, 256), 256, 0, (cudaStream_t)stream>>>(g, nplanes, src, dst);
    }
    const cudaError_t err = cudaGetLastError();
    return err == cudaSuccess ? AGD_STATUS_OK : set_cuda_error("block_squeeze", err);
}

int agd_prep_seeds(int ndim, const int *shape, const int *shape_i, const int32_t *seed_index, const float *seed_values,
                   int n, float *rhs, uint8_t *seedbits, uint8_t *trigger, agd_stream_t stream) {
    clear_error();
    Geo g;
    if (!geo_of(ndim, shape, shape_i, g) || n < 0 || (n > 0 && !seed_index) || (g.size_tot % 32) != 0)
        return set_error(AGD_STATUS_INVALID, "agd_prep_seeds: bad arguments");
    cudaStream_t st = (cudaStream_t)stream;
    Geo4 q;
    if (seedbits && four_points(g, q))
        seedbits4_kernel<<<blocks_for(g.size_tot / 4, 256), 256, 0, st>>>(q, reinterpret_cast<unsigned *>(seedbits));
    else if (seedbits)
        seedbits_init_kernel<<<blocks_for(g.size_tot / 32, 256), 256, 0, st>>>(g, reinterpret_cast<unsigned *>(seedbits));
    if (trigger) cudaMemsetAsync(trigger, 0, (size_t)(g.size_tot / g.size_i), st);
    if (n > 0) {
        seeds_kernel<<<1, 32, 0, st>>>(g, seed_index, seed_values, n, rhs, reinterpret_cast<unsigned *>(seedbits),
                                       trigger, nullptr);
    }
    const cudaError_t err = cudaGetLastError();
    return err == cudaSuccess ? AGD_STATUS_OK : set_cuda_error("prep_seeds", err);
}

int agd_prep_args(int ndim, const int *shape, const int *shape_i, const float *cost, int cost_broadcast,
                  const int32_t *seed_index, const float *seed_host_values, const float *seed_values, int nseeds,
                  float *values, float *rhs, uint8_t *seedbits, agd_stream_t stream) {
    clear_error();
    Geo g;
    Geo4 q;
    if ((ndim != 2 && ndim != 3) || !shape || !shape_i || !geo_of(ndim, shape, shape_i, g) || (g.size_tot % 32) != 0 ||
        nseeds < 0 || (nseeds > 0 && (!seed_index || (!seed_values && !seed_host_values))) || !rhs || !seedbits)
        return set_error(AGD_STATUS_INVALID, "agd_prep_args: bad arguments");
    if (nseeds > kArgSeeds || !four_points(g, q) || !on16(rhs) || (values && !on16(values)))
        return set_error(AGD_STATUS_UNSUPPORTED, "agd_prep_args: more than 32 seeds, or not a built tile shape");
    ArgSeeds a;
    a.n = nseeds;
    a.value = seed_values;
    for (int s = 0; s < nseeds; ++s) {
        int n_o = 0, n_i = 0;
        for (int k = 0; k < ndim; ++k) {
            const int x = seed_index[s * ndim + k];
            if (x < 0 || x >= shape[k]) return set_error(AGD_STATUS_INVALID, "agd_prep_args: seed outside the grid");
            n_o = n_o * g.so[k] + x / g.si[k];
            n_i = n_i * g.si[k] + x % g.si[k];
        }
        a.at[s] = n_o * g.size_i + n_i;
        a.host_value[s] = seed_host_values ? seed_host_values[s] : 0.f;
    }
    const int wide = g.shape[ndim - 1] % 4 == 0 && on16(cost);
    prep_args4_kernel<<<blocks_for(g.size_tot / 4, 256), 256, 0, (cudaStream_t)stream>>>(
        q, a, cost, cost_broadcast, wide, values, rhs, reinterpret_cast<unsigned *>(seedbits));
    const cudaError_t err = cudaGetLastError();
    return err == cudaSuccess ? AGD_STATUS_OK : set_cuda_error("prep_args", err);
}

int agd_nan_sum(const float *x, long long n, double *out, agd_stream_t stream) {
    clear_error();
    if (!x || !out || n < 0) return set_error(AGD_STATUS_INVALID, "agd_nan_sum: bad arguments");
    cudaStream_t st = (cudaStream_t)stream;
    cudaError_t err = cudaMemsetAsync(out, 0, 2 * sizeof(double), st);
    if (err != cudaSuccess) return set_cuda_error("nan_sum", err);
    if (n > 0) nan_sum_kernel<<<(unsigned)std::min<long long>((n + 2047) / 2048, 148 * 4), 256, 0, st>>>(x, n, out);
    err = cudaGetLastError();
    return err == cudaSuccess ? AGD_STATUS_OK : set_cuda_error("nan_sum", err);
}

int agd_prep_batch(const agd_batch_prep *p, agd_stream_t stream) {
    clear_error();
    Geo g;
    if (!p || (p->ndim != 2 && p->ndim != 3) || !geo_of(p->ndim, p->shape, p->shape_i, g) || p->n < 1 ||
        (g.size_tot % 32) != 0 || p->nseeds < 0 || (p->nseeds > 0 && !p->seed_index) || !p->rhs ||
        !p->values || !p->seedbits)
        return set_error(AGD_STATUS_INVALID, "agd_prep_batch: bad arguments");
    const int sd = p->ndim * (p->ndim + 1) / 2;
    int nmet = 0;
    switch (p->model) {
        case AGD_MODEL_ISOTROPIC: nmet = 0; break;
        case AGD_MODEL_RIEMANN: nmet = sd; break;
        case AGD_MODEL_DIAGONAL: nmet = p->ndim; break;
        case AGD_MODEL_RANDER: nmet = sd + p->ndim; break;
        default: return set_error(AGD_STATUS_INVALID, "agd_prep_batch: unknown model");
    }
    if (nmet && (!p->metric || !p->geom))
        return set_error(AGD_STATUS_INVALID,
                         "agd_prep_batch: Riemann, Diagonal and Rander instances need metric and geom");
    BatchPrep A;
    A.g = g;
    A.n = p->n;
    A.model = p->model;
    A.nmet = nmet;
    A.ngeom = nmet;  // the geometry planes of these models are as many as the metric's floats
    A.is_dual = p->is_dual;
    A.walls = p->walls;
    A.walls_stride = p->walls_shared ? 0 : g.n;
    A.trigger = p->trigger;
    A.size_o = g.size_tot / g.size_i;
    A.nseeds = p->nseeds;
    for (int k = 0; k < 3; ++k) A.h[k] = k < p->ndim ? (float)p->grid_scales[k] : 1.f;
    A.metric = p->metric;
    A.cost = p->cost;
    A.seed_values = p->seed_values;
    A.seed_index = p->seed_index;
    A.geom = p->geom;
    A.rhs = p->rhs;
    A.values = p->values;
    A.bits = reinterpret_cast<unsigned *>(p->seedbits);
    A.bad = p->bad_seed;
    if (g.size_tot >= (1ll << 31) || p->n > 65535)
        return set_error(AGD_STATUS_INVALID, "agd_prep_batch: at most 65535 instances of fewer than 2^31 points");
    bool pow2 = true;
    for (int k = 0; k < 3; ++k) {
        int l = 0;
        while ((1 << l) < g.si[k]) ++l;
        A.si_log2[k] = l;
        pow2 = pow2 && (1 << l) == g.si[k];
    }
    if (!pow2) A.si_log2[0] = A.si_log2[1] = A.si_log2[2] = -1;
    cudaStream_t st = (cudaStream_t)stream;
    // about 16 resident 256-thread blocks per SM over all the instances
    const long long per_inst = std::max<long long>(1, 148LL * 16 / p->n);
    const dim3 grid((unsigned)std::min<long long>((g.size_tot + 255) / 256, per_inst), (unsigned)p->n);
    prep_batch_kernel<<<grid, 256, 0, st>>>(A);
    if (p->nseeds > 0) seeds_batch_kernel<<<blocks_for(p->n, 128), 128, 0, st>>>(A);
    const cudaError_t err = cudaGetLastError();
    return err == cudaSuccess ? AGD_STATUS_OK : set_cuda_error("prep_batch", err);
}

int agd_prep_walls(int ndim, const int *shape, const int *shape_i, const uint8_t *walls, int bound, uint8_t *wall_dist,
                   uint8_t *tmp, float *rhs, uint8_t *seedbits, agd_stream_t stream) {
    clear_error();
    Geo g;
    if ((ndim != 2 && ndim != 3) || !shape || !shape_i || !geo_of(ndim, shape, shape_i, g) || (g.size_tot % 32) != 0 ||
        !walls || !wall_dist || !tmp || bound < 0 || bound > 254)
        return set_error(AGD_STATUS_INVALID, "agd_prep_walls: bad arguments (bound in [0, 254])");
    cudaStream_t st = (cudaStream_t)stream;
    // _SetGeometry.py:271-277: 0 at walls, `bound` passes of the L1 kernel, cut beyond `bound`
    const int rc = distance_map(ndim, shape, walls, bound, bound, true, tmp, tmp + g.n, st);
    if (rc != AGD_STATUS_OK) return rc;
    walls_kernel<<<(unsigned)((g.size_tot + 255) / 256), 256, 0, st>>>(g, walls, tmp, wall_dist, rhs,
                                                                       reinterpret_cast<unsigned *>(seedbits));
    const cudaError_t err = cudaGetLastError();
    return err == cudaSuccess ? AGD_STATUS_OK : set_cuda_error("prep_walls", err);
}

int agd_prep_walls_batch(int ndim, const int *shape, const int *shape_i, int n, const uint8_t *walls, int bound,
                         uint8_t *wall_dist, uint8_t *tmp, agd_stream_t stream) {
    clear_error();
    Geo g;
    if ((ndim != 2 && ndim != 3) || !shape || !shape_i || !geo_of(ndim, shape, shape_i, g) || n < 1 || !walls ||
        !wall_dist || !tmp || bound < 0 || bound > 254)
        return set_error(AGD_STATUS_INVALID, "agd_prep_walls_batch: bad arguments (bound in [0, 254])");
    cudaStream_t st = (cudaStream_t)stream;
    const long long np = g.n * n;  // grid points of all the instances
    const int rc = distance_map(ndim, shape, walls, bound, bound, true, tmp, tmp + np, st, n);
    if (rc != AGD_STATUS_OK) return rc;
    wall_dist_batch_kernel<<<blocks_for(g.size_tot * n, 256), 256, 0, st>>>(g, n, tmp, wall_dist);
    const cudaError_t err = cudaGetLastError();
    return err == cudaSuccess ? AGD_STATUS_OK : set_cuda_error("prep_walls_batch", err);
}

int agd_voronoi_decomposition(int ndim, const float *m, long long n, float *weights, void *offsets, int offset_bytes,
                              agd_stream_t stream) {
    clear_error();
    return voronoi(ndim, m, n, weights, offsets, offset_bytes, false, (cudaStream_t)stream);
}

int agd_voronoi_matrices(int ndim, const float *m, long long n, float *weights, void *offsets, int offset_bytes,
                         agd_stream_t stream) {
    clear_error();
    return voronoi(ndim, m, n, weights, offsets, offset_bytes, true, (cudaStream_t)stream);
}

int agd_selling(int ndim, const float *m, int n, float *weights, int32_t *offsets, agd_stream_t stream) {
    clear_error();
    if ((ndim != 2 && ndim != 3) || n < 0 || (n > 0 && (!m || !weights || !offsets)))
        return set_error(AGD_STATUS_INVALID, "agd_selling: bad arguments");
    if (n == 0) return AGD_STATUS_OK;
    selling_kernel<<<blocks_for(n, 128), 128, 0, (cudaStream_t)stream>>>(ndim, m, n, weights, offsets);
    const cudaError_t err = cudaGetLastError();
    return err == cudaSuccess ? AGD_STATUS_OK : set_cuda_error("selling", err);
}

}  // extern "C"
