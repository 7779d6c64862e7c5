// Forward and reverse-mode differentiation of the eikonal solution on B200.
//
// Linearising sum_k w_k (u - v_k)_+^2 = c^2 at the solution gives, at every
// non-seed point x, diag(x) du(x) - sum_k fw_k(x) du(y_k(x)) = r(x), where
// fw_k are the upwind flow weights, y_k(x) the upwind neighbours and diag the
// weight sum (1 at seeds and outside the domain).  The forward mode solves it
// for r = c dc (dc a variation of the cost; r is the seed value's variation at
// a seed); the reverse mode solves the transposed system
// diag(x) lam(x) - sum_{z: y_k(z) = x} fw_k(z) lam(z) = s(x)
// (agd/Eikonal/HFM_CUDA/_PostProcess.py:155-219).
//
// The reference transposes the graph with an iterative claim loop relaunched
// from the host (graph_reverse.py:10-77, cuda/GraphReverse.h:35-82) and solves
// with the block Gauss-Seidel kernel of cuda/Kernel_LinearUpdate.h under the
// adaptive Gauss-Seidel tile schedule.  Here the tiles run in the rounds of
// sched.cuh, every tile at the first epoch.
//   Reverse: a point whose lam changed adds the change to its upwind neighbours'
//   sums, along the forward planes (no transpose is formed), tile after tile from
//   the tiles where s is not zero, those of late arrival times first
//   (ReverseVisitor).
//   Forward: a counting-sort CSR transpose (rows sorted), then Jacobi sweeps in
//   the tiles until nothing moves; a point whose value moved activates exactly
//   the tiles of the points it is an upwind neighbour of (LinearVisitor).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>

#include "sched.cuh"

namespace agd {

// ------------------------------------------------------------ transpose ---
struct RevGeom {
    long long size_tot;
    int nact;
};

__global__ void rev_count_kernel(RevGeom g, const float *fw, const int *fidx, int *count) {
    const long long n = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (n >= g.size_tot) return;
    for (int k = 0; k < g.nact; ++k) {
        const float w = fw[k * g.size_tot + n];
        const int y = fidx[k * g.size_tot + n];
        if (w != 0.f && y >= 0 && y < g.size_tot) atomicAdd(count + y, 1);
    }
}

__global__ void rev_fill_kernel(RevGeom g, const float *fw, const int *fidx, const int *rowptr, int *cursor, int *src,
                                float *wt) {
    const long long n = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (n >= g.size_tot) return;
    for (int k = 0; k < g.nact; ++k) {
        const float w = fw[k * g.size_tot + n];
        const int y = fidx[k * g.size_tot + n];
        if (w != 0.f && y >= 0 && y < g.size_tot) {
            const int pos = rowptr[y] + atomicAdd(cursor + y, 1);
            src[pos] = (int)n;
            wt[pos] = w;
        }
    }
}

// Rows in increasing source order: the fill order depends on the schedule.
// A row of up to kSortRegs entries is sorted in registers (an insertion
// network with fixed indices, strict comparisons as below); longer rows in
// place in global memory.
constexpr int kSortRegs = 12;
__global__ void rev_sort_kernel(RevGeom g, const int *rowptr, int *src, float *wt) {
    const long long y = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (y >= g.size_tot) return;
    const int a = rowptr[y], b = rowptr[y + 1];
    const int len = b - a;
    if (len <= 1) return;
    if (len <= kSortRegs) {
        int sr[kSortRegs];
        float wr[kSortRegs];
#pragma unroll
        for (int i = 0; i < kSortRegs; ++i)
            if (i < len) {
                sr[i] = src[a + i];
                wr[i] = wt[a + i];
            }
#pragma unroll
        for (int i = 1; i < kSortRegs; ++i) {
#pragma unroll
            for (int j = i; j > 0; --j) {
                if (i < len && sr[j - 1] > sr[j]) {
                    const int ts = sr[j - 1];
                    sr[j - 1] = sr[j];
                    sr[j] = ts;
                    const float tw = wr[j - 1];
                    wr[j - 1] = wr[j];
                    wr[j] = tw;
                }
            }
        }
#pragma unroll
        for (int i = 0; i < kSortRegs; ++i)
            if (i < len) {
                src[a + i] = sr[i];
                wt[a + i] = wr[i];
            }
        return;
    }
    for (int i = a + 1; i < b; ++i) {
        const int s = src[i];
        const float w = wt[i];
        int j = i - 1;
        while (j >= a && src[j] > s) {
            src[j + 1] = src[j];
            wt[j + 1] = wt[j];
            --j;
        }
        src[j + 1] = s;
        wt[j + 1] = w;
    }
}

// Exclusive scan of n ints in three passes (blocks of 1024, block totals, offsets).
__device__ __forceinline__ int warp_incl_scan(int v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(kFull, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

__device__ int block_excl_scan(int v, int *tot) {
    __shared__ int ws[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int inc = warp_incl_scan(v, lane);
    if (lane == 31) ws[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        const int nw = blockDim.x >> 5;
        int x = lane < nw ? ws[lane] : 0;
        x = warp_incl_scan(x, lane);
        if (lane < nw) ws[lane] = x;
    }
    __syncthreads();
    const int off = warp > 0 ? ws[warp - 1] : 0;
    if (tot) *tot = ws[(blockDim.x >> 5) - 1];
    __syncthreads();
    return off + inc - v;
}

__global__ void scan_blocks_kernel(const int *in, int *out, long long n, int *block_tot) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const int v = i < n ? in[i] : 0;
    int tot;
    const int ex = block_excl_scan(v, &tot);
    if (i < n) out[i] = ex;
    if (threadIdx.x == 0) block_tot[blockIdx.x] = tot;
}

__global__ void scan_totals_kernel(int *block_tot, int nb, int *grand) {
    __shared__ int carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int base = 0; base < nb; base += blockDim.x) {
        const int i = base + threadIdx.x;
        const int v = i < nb ? block_tot[i] : 0;
        int tot;
        const int ex = block_excl_scan(v, &tot);
        if (i < nb) block_tot[i] = ex + carry;
        __syncthreads();
        if (threadIdx.x == 0) carry += tot;
        __syncthreads();
    }
    if (threadIdx.x == 0) *grand = carry;
}

__global__ void scan_add_kernel(int *out, long long n, const int *block_off) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i < n) out[i] += block_off[blockIdx.x];
}

// ----------------------------------------------------------- linear visit ---
struct LinArgs {
    const int *rowptr, *src;
    const float *wt;
    const float *wsum, *sens;
    float *lam;
    const float *fw;
    const int *fidx;
    int nact;
    float atol, rtol;
};

// Forward mode: rows from the forward flow planes (fw, fidx), activation through
// the transpose (rowptr, src).
template <int SIZE>
struct LinearVisitor {
    static constexpr int P = SIZE / 32;
    static constexpr int kMaxSweeps = 4 * SIZE;  // in-tile chains are shorter than the tile
    using Args = LinArgs;
    // In-tile entries of each point's row, kept for the sweeps: weight and
    // in-tile index of up to K of them, in row order (a row with more goes on
    // reading the rest from global memory).  Without this cache every sweep
    // re-read the rows through L2: 4.3 us a sweep, 70 % of a visit at 200^3.
    static constexpr int K = SIZE == 256 ? 4 : 8;
    static constexpr int kRowUnroll = K < 6 ? K : 6;  // row entries unrolled in the init (nact <= 6)
    struct Smem {
        float l[SIZE];
        float cw[K][SIZE];
        unsigned char cz[K][SIZE];
    };
    static cudaError_t prepare(const Sched &, const WsLayout &, cudaStream_t) { return cudaSuccess; }
    static cudaError_t finalize(const Sched &, const WsLayout &, cudaStream_t) { return cudaSuccess; }
    // A linear solve is one instance and runs in rounds, a warp per tile.
    static constexpr bool kQueueless = true;
    static constexpr int kMinCtas = 1, kRoundG = 1, kRoundWarps = SIZE == 256 ? 8 : 16, kRoundCtas = 2;
    using RoundSmem = Smem;

    static constexpr bool kOrdered = false;
    __device__ static bool visit_round(const Sched &S, const Args &A, int t, int ii, int e, int lane, int, Smem &sm) {
        const Inst &I = S.inst[ii];
        const int n_o = t - I.tile_base;
        const long long base = (long long)n_o * SIZE;
        float old[P], diag[P], acc[P];
        int r0[P], r1[P];
        unsigned cnt = 0, ovf = 0;  // per point p: cached entries (4 bits at 4p), more than K (bit p)
#pragma unroll
        for (int p = 0; p < P; ++p) {
            const int n_i = lane + 32 * p;
            const long long n_t = base + n_i;
            old[p] = __ldcg(A.lam + n_t);
            sm.l[n_i] = old[p];
            const float d = __ldg(A.wsum + n_t);
            diag[p] = d == 0.f ? 1.f : d;
            float a = __ldg(A.sens + n_t);
            r0[p] = __ldg(A.rowptr + n_t);
            r1[p] = __ldg(A.rowptr + n_t + 1);
            int c = 0;
            // Out-of-tile entries are summed once per visit, in row order; the
            // in-tile ones are cached.  The first kRowUnroll entries of a row are
            // unrolled so that their loads are issued together: a row walked
            // one entry at a time costs two dependent L2 round trips per entry.
#pragma unroll
            for (int k = 0; k < kRowUnroll; ++k) {  // upwind neighbours: nact <= kRowUnroll
                if (k >= A.nact) continue;
                const float w = __ldg(A.fw + k * I.size_tot + n_t);
                const int y = __ldg(A.fidx + k * I.size_tot + n_t);
                if (w == 0.f || y < 0 || (long long)y >= I.size_tot) continue;
                if ((long long)y / SIZE != n_o) {
                    a += w * __ldcg(A.lam + y);
                } else {  // c <= k < K
                    sm.cw[c][n_i] = w;
                    sm.cz[c][n_i] = (unsigned char)(y - (int)base);
                    ++c;
                }
            }
            for (int k = kRowUnroll; k < A.nact; ++k) {  // more neighbours than the unrolled part
                const float w = __ldg(A.fw + k * I.size_tot + n_t);
                const int y = __ldg(A.fidx + k * I.size_tot + n_t);
                if (w == 0.f || y < 0 || (long long)y >= I.size_tot) continue;
                if ((long long)y / SIZE != n_o) {
                    a += w * __ldcg(A.lam + y);
                } else if (c < K) {
                    sm.cw[c][n_i] = w;
                    sm.cz[c][n_i] = (unsigned char)(y - (int)base);
                    ++c;
                } else {
                    ovf |= 1u << p;
                }
            }
            cnt |= (unsigned)c << (4 * p);
            acc[p] = a;
        }
        __syncwarp();
        bool settled = false;
        for (int it = 0; it < kMaxSweeps; ++it) {
            bool moved = false;
#pragma unroll
            for (int p = 0; p < P; ++p) {
                const int n_i = lane + 32 * p;
                float v = acc[p];
                // the in-tile entries in row order: the cached ones, then the rest
                const int c = (int)((cnt >> (4 * p)) & 15u);
#pragma unroll
                for (int k = 0; k < K; ++k)
                    if (k < c) v += sm.cw[k][n_i] * sm.l[sm.cz[k][n_i]];
                if (ovf & (1u << p)) {
                    int seen = 0;
                    const long long n_t = base + n_i;
                    for (int k = 0; k < A.nact; ++k) {
                        const float w = __ldg(A.fw + k * I.size_tot + n_t);
                        const int y = __ldg(A.fidx + k * I.size_tot + n_t);
                        if (w != 0.f && y >= 0 && (long long)y / SIZE == n_o && seen++ >= K)
                            v += w * sm.l[y - (int)base];
                    }
                }
                v = v / diag[p];
                __syncwarp();
                if (v != sm.l[n_i]) {
                    sm.l[n_i] = v;
                    moved = true;
                }
                __syncwarp();
            }
            if (!__any_sync(kFull, moved)) {
                settled = true;
                break;
            }
        }
        bool pushed = false;
#pragma unroll
        for (int p = 0; p < P; ++p) {
            const int n_i = lane + 32 * p;
            const long long n_t = base + n_i;
            const float v = sm.l[n_i];
            __stcg(A.lam + n_t, v);
            const bool changed = fabsf(v - old[p]) > A.atol + A.rtol * fabsf(v);
            if (!changed) continue;
            for (int j = r0[p]; j < r1[p]; ++j) {  // the points that depend on this one
                const int ty = __ldg(A.src + j) / SIZE;
                if (ty == n_o) continue;
                push_round(S, I.tile_base + ty, e);
                pushed = true;
            }
        }
        __syncwarp();
        if (!settled && lane == 0) {
            push_round(S, t, e);
            pushed = true;
        }
        return pushed;
    }
};

// ---------------------------------------------------------- reverse visit ---
struct RevArgs {
    float *acc;        // the right-hand side plus the contributions received
    float *lam;        // acc / diag as of the tile's last visit: what has been passed on
    const float *wsum;
    const float *fw;
    const int *fidx;
    const uint16_t *bin;  // per tile: the first epoch at which it is visited
    float atol, rtol;
};

// Reverse mode, diag lam - W^T lam = s: every point keeps the sum of its
// right-hand side and of the contributions fw_k lam it has received, and what
// it has passed on.  A visit passes the changes of its tile's points on inside
// the tile, in shared memory, until nothing changes, then once to the upwind
// neighbours outside (adds to their sums).  It pushes the tiles of those where
// the change exceeds atol + rtol |lam|, the reference's tolerance; smaller
// changes are added all the same, and rev_finish_kernel forms lam from the sums.
// Contributions go from late to early arrival times, so a tile waits for the
// epoch of its smallest value (due): most of what reaches it has then come.
// What bounds it: the epochs' latency (one dependent load of the sums and the
// planes, the in-tile passes, the adds), and for dense right-hand sides the
// planes' bytes, read once a visit.  Riemann3 200^3, 128 receivers: 5.1 ms (9.9
// without the order), against 14.9 ms as Jacobi sweeps of every tile over a sorted
// transpose, plus 1.0 ms for the transpose.  (Finishing each point once, when
// all the points that depend on it are done, took 861 epochs and 23.8 ms: the
// longest chains cross tiles hundreds of times with contributions far below
// the tolerance.)
template <int SIZE, int NACT>
struct ReverseVisitor {
    using Args = RevArgs;
    static constexpr bool kQueueless = true, kOrdered = true;
    static constexpr int kRoundG = SIZE == 256 ? 4 : 2, kRoundWarps = 16, kRoundCtas = 2;
    static constexpr int NT = 32 * kRoundG, P = SIZE / NT;
    static constexpr int kMaxSweeps = 4 * SIZE;
    struct RoundSmem {
        float acc[SIZE];  // contributions from inside the tile
    };
    static cudaError_t prepare(const Sched &, const WsLayout &, cudaStream_t) { return cudaSuccess; }
    static cudaError_t finalize(const Sched &, const WsLayout &, cudaStream_t) { return cudaSuccess; }
    __device__ __forceinline__ static bool due(const Args &A, int t, int e) { return (int)__ldg(A.bin + t) <= e; }

    __device__ static bool visit_round(const Sched &S, const Args &A, int t, int ii, int e, int tid, int group,
                                       RoundSmem &sm) {
        const Inst &I = S.inst[ii];
        const int n_o = t - I.tile_base;
        const long long base = (long long)n_o * SIZE;
        float acc[P], diag[P], lam[P], lam0[P], w[P][NACT];
        int y[P][NACT];
#pragma unroll
        for (int p = 0; p < P; ++p) {
            const long long n = base + tid + NT * p;
            sm.acc[tid + NT * p] = 0.f;
            acc[p] = __ldcg(A.acc + n);
            lam[p] = lam0[p] = __ldcg(A.lam + n);
            const float d = __ldg(A.wsum + n);
            diag[p] = d == 0.f ? 1.f : d;
#pragma unroll
            for (int k = 0; k < NACT; ++k) {
                w[p][k] = __ldg(A.fw + k * I.size_tot + n);
                y[p][k] = __ldg(A.fidx + k * I.size_tot + n);
            }
        }
#pragma unroll
        for (int p = 0; p < P; ++p)
#pragma unroll
            for (int k = 0; k < NACT; ++k) {
                if (y[p][k] < 0 || (long long)y[p][k] >= I.size_tot) w[p][k] = 0.f;
            }
        group_sync<kRoundG>(group);
        bool settled = false;
        for (int it = 0; it < kMaxSweeps && !settled; ++it) {
            bool moved = false;
#pragma unroll
            for (int p = 0; p < P; ++p) {
                const float v = (acc[p] + sm.acc[tid + NT * p]) / diag[p];
                if (v == lam[p]) continue;
                const float dl = v - lam[p];
                lam[p] = v;
                moved = true;
#pragma unroll
                for (int k = 0; k < NACT; ++k) {
                    const int li = y[p][k] - (int)base;
                    if (w[p][k] != 0.f && li >= 0 && li < SIZE) atomicAdd(&sm.acc[li], w[p][k] * dl);
                }
            }
            settled = !group_any<kRoundG>(group, moved);
        }
        bool pushed = false;
#pragma unroll
        for (int p = 0; p < P; ++p) {
            const int li0 = tid + NT * p;
            const float dl = lam[p] - lam0[p];
            if (sm.acc[li0] != 0.f) atomicAdd(A.acc + base + li0, sm.acc[li0]);
            if (lam[p] == lam0[p]) continue;
            __stcg(A.lam + base + li0, lam[p]);
            const bool far = fabsf(dl) > A.atol + A.rtol * fabsf(lam[p]);
#pragma unroll
            for (int k = 0; k < NACT; ++k) {
                const int li = y[p][k] - (int)base;
                if (w[p][k] == 0.f || (li >= 0 && li < SIZE)) continue;
                atomicAdd(A.acc + y[p][k], w[p][k] * dl);
                if (far) {
                    push_round(S, I.tile_base + y[p][k] / SIZE, e);
                    pushed = true;
                }
            }
        }
        if (!settled && tid == 0) {
            push_round(S, t, e);
            pushed = true;
        }
        group_sync<kRoundG>(group);  // (a later visit reuses sm)
        return pushed;
    }
};

// A float's bits as an unsigned in the same order.
__device__ __forceinline__ unsigned ordered_bits(float x) {
    const unsigned b = __float_as_uint(x);
    return b & 0x80000000u ? ~b : b | 0x80000000u;
}
__device__ __forceinline__ float from_ordered(unsigned b) {
    return __uint_as_float(b & 0x80000000u ? b & 0x7fffffffu : ~b);
}

// Range of the finite values: range[0] the largest (ordered bits), range[1] the
// complement of the smallest; both 0 before.
__global__ void rev_range_kernel(long long n, const float *__restrict__ u, unsigned *range) {
    unsigned hi = 0u, lo = 0u;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float x = __ldg(u + i);
        if (!(fabsf(x) < finf())) continue;
        hi = max(hi, ordered_bits(x));
        lo = max(lo, ~ordered_bits(x));
    }
    hi = __reduce_max_sync(kFull, hi);
    lo = __reduce_max_sync(kFull, lo);
    if ((threadIdx.x & 31) == 0) {
        atomicMax(range, hi);
        atomicMax(range + 1, lo);
    }
}

// The solve's start, a warp per tile: the sums, what has been passed on (nothing),
// the tiles to visit (s not zero somewhere), and their epochs: 1 to nbins, from
// the latest to the earliest arrival time of a tile's first point.
__global__ void rev_start_kernel(int ntiles, int size_i, int nbins, const float *__restrict__ u, const unsigned *range,
                                 const float *__restrict__ sens, float *__restrict__ acc, float *__restrict__ lam,
                                 uint16_t *__restrict__ bin, uint8_t *__restrict__ trigger) {
    const int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (t >= ntiles) return;
    bool any = false;
    unsigned lo = 0u;
    for (int i = lane; i < size_i; i += 32) {
        const long long n = (long long)t * size_i + i;
        const float s = __ldg(sens + n);
        acc[n] = s;
        lam[n] = 0.f;
        any = any || s != 0.f;
        if (u) {
            const float x = __ldg(u + n);
            if (fabsf(x) < finf()) lo = max(lo, ~ordered_bits(x));
        }
    }
    any = __any_sync(kFull, any);
    lo = __reduce_max_sync(kFull, lo);
    if (lane == 0) {
        int b = 1;
        if (u && lo) {
            const float hi = from_ordered(range[0]), min = from_ordered(~range[1]), x = from_ordered(~lo);
            if (hi > min) b = 1 + (int)((hi - x) / (hi - min) * (float)(nbins - 1));
        }
        bin[t] = (uint16_t)b;
        trigger[t] = any;
    }
}

// lam of every point from its sum, changes below the tolerance included.
__global__ void rev_finish_kernel(long long n, const float *__restrict__ acc, const float *__restrict__ wsum,
                                  float *__restrict__ lam) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float d = __ldg(wsum + i);
    lam[i] = acc[i] / (d == 0.f ? 1.f : d);
}

static inline unsigned nb(long long n, int bs) { return (unsigned)((n + bs - 1) / bs); }

struct RevLayout {
    WsLayout L;
    size_t rowptr, cursor, src, wt, btot, grand, total;
    long long size_tot;
    int nact, size_i;
};

static bool rev_layout(const agd_instance *a, RevLayout &R, std::vector<Inst> *insts) {
    agd_instance b = *a;
    b.flags = (b.flags | AGD_FLAG_ACTIVATE_ALL) & ~(AGD_FLAG_SOLVER_AGSI | AGD_FLAG_SOLVER_GLOBAL);
    b.trigger = nullptr;
    b.release = nullptr;  // the linear solves keep the two-list schedule
    if (!layout(&b, 1, R.L, insts, /*stencil_cache=*/false)) return false;
    const Inst &I = (*insts)[0];
    R.size_tot = I.size_tot;
    R.size_i = I.size_i;
    R.nact = (a->model == AGD_MODEL_RIEMANN || a->model == AGD_MODEL_RANDER) ? a->ndim * (a->ndim + 1) / 2 : a->ndim;
    size_t off = R.L.total;
    const long long nblk = (R.size_tot + 1 + 1023) / 1024;
    R.rowptr = off; off = align256(off + sizeof(int) * (R.size_tot + 1));
    R.cursor = off; off = align256(off + sizeof(int) * R.size_tot);
    R.src = off; off = align256(off + sizeof(int) * R.nact * R.size_tot);
    R.wt = off; off = align256(off + sizeof(float) * R.nact * R.size_tot);
    R.btot = off; off = align256(off + sizeof(int) * nblk);
    R.grand = off; off = align256(off + 2 * sizeof(int));
    R.total = off;
    return true;
}

}  // namespace agd

using namespace agd;

extern "C" {

size_t agd_reverse_workspace_bytes(const agd_instance *inst) {
    if (!inst) return 0;
    RevLayout R;
    std::vector<Inst> v;
    if (!rev_layout(inst, R, &v)) return 0;
    return R.total;
}

}  // extern "C"

namespace agd {

// Checks of a linear solve; lays out its workspace.
static int linear_check(const char *who, const agd_instance *inst, const float *flow_weights,
                        const int32_t *flow_indices, const float *flow_weightsum, const float *rhs, const float *sol,
                        const void *workspace, size_t workspace_bytes, RevLayout &R, std::vector<Inst> &insts) {
    char msg[128];
    if (!inst || !flow_weights || !flow_indices || !flow_weightsum || !rhs || !sol || !workspace) {
        snprintf(msg, sizeof(msg), "%s: missing array", who);
        return set_error(AGD_STATUS_INVALID, msg);
    }
    if (!rev_layout(inst, R, &insts)) {
        snprintf(msg, sizeof(msg), "%s: bad instance", who);
        return set_error(AGD_STATUS_INVALID, msg);
    }
    if (insts[0].variant < 0) {
        snprintf(msg, sizeof(msg), "%s: tile shape not built", who);
        return set_error(AGD_STATUS_UNSUPPORTED, msg);
    }
    if (workspace_bytes < R.total) {
        snprintf(msg, sizeof(msg), "%s: workspace too small", who);
        return set_error(AGD_STATUS_WORKSPACE, msg);
    }
    if (R.size_i != 64 && R.size_i != 256) {
        snprintf(msg, sizeof(msg), "%s: tile size not built", who);
        return set_error(AGD_STATUS_UNSUPPORTED, msg);
    }
    return AGD_STATUS_OK;
}

static int reverse_solve(const agd_instance *inst, const float *flow_weights, const int32_t *flow_indices,
                         const float *flow_weightsum, const float *sens, float *lam, float atol, float rtol,
                         void *workspace, size_t workspace_bytes, agd_stats *stats, const agd_launch *launch,
                         cudaStream_t st) {
    RevLayout R;
    std::vector<Inst> insts;
    const int rc = linear_check("agd_reverse", inst, flow_weights, flow_indices, flow_weightsum, sens, lam, workspace,
                                workspace_bytes, R, insts);
    if (rc != AGD_STATUS_OK) return rc;
    char *w = static_cast<char *>(workspace);
    unsigned *range = reinterpret_cast<unsigned *>(w + R.grand);
    uint16_t *bin = reinterpret_cast<uint16_t *>(w + R.cursor);
    uint8_t *trigger = reinterpret_cast<uint8_t *>(w + R.rowptr);
    RevArgs A{reinterpret_cast<float *>(w + R.wt), lam, flow_weightsum, flow_weights, flow_indices, bin, atol, rtol};
    Inst &I = insts[0];
    I.a.flags &= ~AGD_FLAG_ACTIVATE_ALL;
    I.a.trigger = trigger;
    // Epochs of the sweep from late to early tiles: up to 3 per tile of the
    // longest side, in proportion to the tiles of a layer.  Waiting saves
    // visits and costs epochs, which pays where an epoch's tiles fill the GPU:
    // Riemann3 200^3 (2500 tiles a layer) 9.9 ms without order, 8.2 / 5.8 / 5.1 /
    // 5.3 ms with 1 / 2 / 3 / 4 epochs per tile of the side; Riemann3 100 x 90 x 110
    // (600) 2.2 and 2.0 / 1.7 / 1.6 / 1.7; Riemann2 1000 x 800 (100) 1.7 and 1.6 / 2.7 /
    // 3.8; Riemann2 301 x 413 (38) 0.99 and 1.3 / 1.6 / 1.8 ms.
    int side = 1;
    for (int k = 0; k < I.a.ndim; ++k) side = std::max(side, I.shape_o[k]);
    const float per_side = std::min(3.f, (float)I.size_o / (float)side / 200.f);
    const int nbins = std::max(1, std::min((int)(per_side * side), I.a.nitermax_o / 4));
    const float *u = inst->values;
    cudaError_t err = cudaMemsetAsync(range, 0, 2 * sizeof(unsigned), st);
    if (err != cudaSuccess) return set_cuda_error("reverse clear", err);
    if (u) rev_range_kernel<<<std::min(nb(R.size_tot, 1024), 148u * 8u), 256, 0, st>>>(R.size_tot, u, range);
    rev_start_kernel<<<nb(I.size_o, 8), 256, 0, st>>>(I.size_o, R.size_i, nbins, u, range, sens, A.acc, lam, bin, trigger);
    if ((err = cudaGetLastError()) != cudaSuccess) return set_cuda_error("reverse start", err);
    err = cudaMemcpyAsync(w + R.L.inst, insts.data(), sizeof(Inst), cudaMemcpyHostToDevice, st);
    if (err != cudaSuccess) return set_cuda_error("reverse descriptor upload", err);
    int rs;
    if (R.size_i == 256)
        rs = R.nact == 2 ? run_sched<ReverseVisitor<256, 2>>(R.L, workspace, 1, A, stats, launch, st)
                         : run_sched<ReverseVisitor<256, 3>>(R.L, workspace, 1, A, stats, launch, st);
    else
        rs = R.nact == 2   ? run_sched<ReverseVisitor<64, 2>>(R.L, workspace, 1, A, stats, launch, st)
             : R.nact == 3 ? run_sched<ReverseVisitor<64, 3>>(R.L, workspace, 1, A, stats, launch, st)
                           : run_sched<ReverseVisitor<64, 6>>(R.L, workspace, 1, A, stats, launch, st);
    if (rs != AGD_STATUS_OK) return rs;
    rev_finish_kernel<<<nb(R.size_tot, 256), 256, 0, st>>>(R.size_tot, A.acc, flow_weightsum, lam);
    err = cudaGetLastError();
    return err == cudaSuccess ? AGD_STATUS_OK : set_cuda_error("reverse finish", err);
}

// The transpose of the flow graph, then the linear solve on the tiles.
static int forward_solve(const agd_instance *inst, const float *flow_weights, const int32_t *flow_indices,
                         const float *flow_weightsum, const float *rhs, float *sol, float atol, float rtol,
                         void *workspace, size_t workspace_bytes, agd_stats *stats, const agd_launch *launch,
                         cudaStream_t st) {
    RevLayout R;
    std::vector<Inst> insts;
    const int rc = linear_check("agd_forward", inst, flow_weights, flow_indices, flow_weightsum, rhs, sol, workspace,
                                workspace_bytes, R, insts);
    if (rc != AGD_STATUS_OK) return rc;
    char *w = static_cast<char *>(workspace);
    int *rowptr = reinterpret_cast<int *>(w + R.rowptr);
    int *cursor = reinterpret_cast<int *>(w + R.cursor);
    int *src = reinterpret_cast<int *>(w + R.src);
    float *wt = reinterpret_cast<float *>(w + R.wt);
    int *btot = reinterpret_cast<int *>(w + R.btot);
    int *grand = reinterpret_cast<int *>(w + R.grand);
    RevGeom g{R.size_tot, R.nact};
    cudaError_t err = cudaMemsetAsync(cursor, 0, sizeof(int) * R.size_tot, st);
    if (err == cudaSuccess) err = cudaMemsetAsync(sol, 0, sizeof(float) * R.size_tot, st);
    if (err != cudaSuccess) return set_cuda_error("linear solve clear", err);
    // counts (into cursor), exclusive scan into rowptr, then fill
    rev_count_kernel<<<nb(R.size_tot, 256), 256, 0, st>>>(g, flow_weights, flow_indices, cursor);
    const long long n1 = R.size_tot + 1;
    cudaMemsetAsync(rowptr + R.size_tot, 0, sizeof(int), st);
    scan_blocks_kernel<<<nb(n1, 1024), 1024, 0, st>>>(cursor, rowptr, R.size_tot, btot);
    scan_totals_kernel<<<1, 1024, 0, st>>>(btot, (int)nb(n1, 1024), grand);
    scan_add_kernel<<<nb(n1, 1024), 1024, 0, st>>>(rowptr, R.size_tot, btot);
    cudaMemcpyAsync(rowptr + R.size_tot, grand, sizeof(int), cudaMemcpyDeviceToDevice, st);
    cudaMemsetAsync(cursor, 0, sizeof(int) * R.size_tot, st);
    rev_fill_kernel<<<nb(R.size_tot, 256), 256, 0, st>>>(g, flow_weights, flow_indices, rowptr, cursor, src, wt);
    rev_sort_kernel<<<nb(R.size_tot, 256), 256, 0, st>>>(g, rowptr, src, wt);
    if ((err = cudaGetLastError()) != cudaSuccess) return set_cuda_error("linear solve transpose", err);
    // solve on the tiles
    err = cudaMemcpyAsync(w + R.L.inst, insts.data(), sizeof(Inst), cudaMemcpyHostToDevice, st);
    if (err != cudaSuccess) return set_cuda_error("linear solve descriptor upload", err);
    LinArgs A{rowptr, src, wt, flow_weightsum, rhs, sol, flow_weights, flow_indices, R.nact, atol, rtol};
    if (R.size_i == 256) return run_sched<LinearVisitor<256>>(R.L, workspace, 1, A, stats, launch, st);
    return run_sched<LinearVisitor<64>>(R.L, workspace, 1, A, stats, launch, st);
}

}  // namespace agd

extern "C" {

int agd_reverse(const agd_instance *inst, const float *flow_weights, const int32_t *flow_indices,
                const float *flow_weightsum, const float *sens, float *lam, float atol, float rtol, void *workspace,
                size_t workspace_bytes, agd_stats *stats, const agd_launch *launch, agd_stream_t stream) {
    clear_error();
    return reverse_solve(inst, flow_weights, flow_indices, flow_weightsum, sens, lam, atol, rtol, workspace,
                         workspace_bytes, stats, launch, (cudaStream_t)stream);
}

int agd_forward(const agd_instance *inst, const float *flow_weights, const int32_t *flow_indices,
                const float *flow_weightsum, const float *rhs, float *du, float atol, float rtol, void *workspace,
                size_t workspace_bytes, agd_stats *stats, const agd_launch *launch, agd_stream_t stream) {
    clear_error();
    return forward_solve(inst, flow_weights, flow_indices, flow_weightsum, rhs, du, atol, rtol, workspace,
                         workspace_bytes, stats, launch, (cudaStream_t)stream);
}

}  // extern "C"
