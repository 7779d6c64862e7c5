// Eikonal solve kernels: Riemann3, plain and with walls (see families.cuh).
#include "solve.cuh"

namespace agd {
template int solve<fam::R3>(const WsLayout &, void *, int, agd_stats *, const agd_launch *, cudaStream_t);
template int solve<fam::W3>(const WsLayout &, void *, int, agd_stats *, const agd_launch *, cudaStream_t);
}  // namespace agd
