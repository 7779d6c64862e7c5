// Eikonal solve kernels: source factorisation (see families.cuh).
#include "solve.cuh"

namespace agd {
template int solve<fam::F2>(const WsLayout &, void *, int, agd_stats *, const agd_launch *, cudaStream_t);
template int solve<fam::F3>(const WsLayout &, void *, int, agd_stats *, const agd_launch *, cudaStream_t);
}  // namespace agd
