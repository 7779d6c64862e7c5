// The kernels of the eikonal solve: which tile-visit variants are compiled
// together (a plan runs the smallest set that holds its instances' variants),
// and the solve over them, instantiated in the solve_*.cu.
#pragma once
#include "sched.cuh"

namespace agd {
namespace fam {
using Mask = unsigned long long;
constexpr Mask V(int variant) { return 1ull << variant; }
constexpr Mask R2 = V(V_RIEM2_8), I16 = V(V_ISO2_16), I8 = V(V_ISO2_8), R2L = V(V_RIEM2_16);
constexpr Mask R3 = V(V_RIEM3_4), I3 = V(V_ISO3_4);
// Riemann with walls, beside plain instances of every family
constexpr Mask W2 = V(V_RIEM2_8_W) | V(V_RIEM2_16_W), W3 = V(V_RIEM3_4_W), R2W = V(V_RIEM2_8_W);
constexpr Mask BASE2 = R2 | I16 | I8 | R2L | W2, BASE3 = R3 | I3 | W3;
constexpr Mask R2MP = V(V_RIEM2_8_MP), I16MP = V(V_ISO2_16_MP), R3MP = V(V_RIEM3_4_MP), I3MP = V(V_ISO3_4_MP);
constexpr Mask MP2 = V(V_ISO2_8_MP) | I16MP | R2MP | V(V_ISO2_16_FMP) | V(V_RIEM2_8_FMP) | BASE2;
constexpr Mask MP3 = I3MP | R3MP | V(V_ISO3_4_FMP) | V(V_RIEM3_4_FMP) | BASE3;
constexpr Mask F2 = V(V_ISO2_8_F) | V(V_ISO2_16_F) | V(V_RIEM2_8_F) | BASE2;
constexpr Mask F3 = V(V_ISO3_4_F) | V(V_RIEM3_4_F) | BASE3;
constexpr Mask O2 = V(V_ISO2_8_O2) | V(V_ISO2_16_O2) | V(V_RIEM2_8_O2) | BASE2;
constexpr Mask O3 = V(V_ISO3_4_O2) | V(V_RIEM3_4_O2) | BASE3;
// second order with factorisation, with multiprecision, with both
constexpr Mask OF2 = V(V_ISO2_16_O2F) | V(V_RIEM2_8_O2F), OF3 = V(V_ISO3_4_O2F) | V(V_RIEM3_4_O2F);
constexpr Mask OM2 = V(V_ISO2_16_O2MP) | V(V_RIEM2_8_O2MP), OM3 = V(V_ISO3_4_O2MP) | V(V_RIEM3_4_O2MP);
constexpr Mask OFM2 = V(V_ISO2_16_O2FMP) | V(V_RIEM2_8_O2FMP), OFM3 = V(V_ISO3_4_O2FMP) | V(V_RIEM3_4_O2FMP);
constexpr Mask D2 = V(V_DIAG2_8) | V(V_DIAG2_16), D3 = V(V_DIAG3_4);
constexpr Mask DMP2 = V(V_DIAG2_8_MP) | V(V_DIAG2_16_MP) | D2, DMP3 = V(V_DIAG3_4_MP) | D3;
constexpr Mask DF2 = V(V_DIAG2_8_F) | V(V_DIAG2_16_F) | D2, DF3 = V(V_DIAG3_4_F) | D3;
constexpr Mask DO2 = V(V_DIAG2_8_O2) | V(V_DIAG2_16_O2) | D2, DO3 = V(V_DIAG3_4_O2) | D3;
constexpr Mask N2 = V(V_RAND2_8) | V(V_RAND2_8_W), N3 = V(V_RAND3_4) | V(V_RAND3_4_W);
constexpr Mask NMP2 = V(V_RAND2_8_MP) | N2, NMP3 = V(V_RAND3_4_MP) | N3;
constexpr Mask NF2 = V(V_RAND2_8_F) | N2, NF3 = V(V_RAND3_4_F) | N3;
constexpr Mask NO2 = V(V_RAND2_8_O2) | N2, NO3 = V(V_RAND3_4_O2) | N3;
}  // namespace fam

template <unsigned long long VMASK>
int solve(const WsLayout &L, void *ws, int n, agd_stats *stats, const agd_launch *cfg, cudaStream_t st);

}  // namespace agd
