// Eikonal solve kernels: multiprecision, one variant (see families.cuh).
#include "solve.cuh"

namespace agd {
template int solve<fam::R2MP>(const WsLayout &, void *, int, agd_stats *, const agd_launch *, cudaStream_t);
template int solve<fam::I16MP>(const WsLayout &, void *, int, agd_stats *, const agd_launch *, cudaStream_t);
template int solve<fam::R3MP>(const WsLayout &, void *, int, agd_stats *, const agd_launch *, cudaStream_t);
template int solve<fam::I3MP>(const WsLayout &, void *, int, agd_stats *, const agd_launch *, cudaStream_t);
}  // namespace agd
