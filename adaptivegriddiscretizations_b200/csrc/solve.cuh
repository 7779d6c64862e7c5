// The solve over one set of tile-visit variants, for the solve_*.cu, which
// instantiate it (everything else calls it through its declaration in
// families.cuh).
#pragma once
#include "visit.cuh"

namespace agd {

template <unsigned long long VMASK>
int solve(const WsLayout &L, void *ws, int n, agd_stats *stats, const agd_launch *cfg, cudaStream_t st) {
    return run_sched<EikonalVisitor<VMASK>>(L, ws, n, {}, stats, cfg, st);
}

}  // namespace agd
