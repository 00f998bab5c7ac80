// elem_volume.h -- the reference volume of a hexahedron, for the host's set-up
// and the device's (Real: double there, an operator-by-operator rounded double
// here, so that both give the same bits).
#pragma once

#ifdef __CUDACC__
#define LULESH_HD __host__ __device__
#else
#define LULESH_HD
#endif

namespace lulesh {

// CalcElemVolume (LULESH-OMP.cc:1706-1790), same association as the reference.
template <class Real>
LULESH_HD inline Real elem_volume(const Real x[8], const Real y[8], const Real z[8])
{
    const Real dx61 = x[6] - x[1], dy61 = y[6] - y[1], dz61 = z[6] - z[1];
    const Real dx70 = x[7] - x[0], dy70 = y[7] - y[0], dz70 = z[7] - z[0];
    const Real dx63 = x[6] - x[3], dy63 = y[6] - y[3], dz63 = z[6] - z[3];
    const Real dx20 = x[2] - x[0], dy20 = y[2] - y[0], dz20 = z[2] - z[0];
    const Real dx50 = x[5] - x[0], dy50 = y[5] - y[0], dz50 = z[5] - z[0];
    const Real dx64 = x[6] - x[4], dy64 = y[6] - y[4], dz64 = z[6] - z[4];
    const Real dx31 = x[3] - x[1], dy31 = y[3] - y[1], dz31 = z[3] - z[1];
    const Real dx72 = x[7] - x[2], dy72 = y[7] - y[2], dz72 = z[7] - z[2];
    const Real dx43 = x[4] - x[3], dy43 = y[4] - y[3], dz43 = z[4] - z[3];
    const Real dx57 = x[5] - x[7], dy57 = y[5] - y[7], dz57 = z[5] - z[7];
    const Real dx14 = x[1] - x[4], dy14 = y[1] - y[4], dz14 = z[1] - z[4];
    const Real dx25 = x[2] - x[5], dy25 = y[2] - y[5], dz25 = z[2] - z[5];
    auto triple = [](Real x1, Real y1, Real z1, Real x2, Real y2, Real z2, Real x3, Real y3, Real z3) {
        return x1 * (y2 * z3 - z2 * y3) + x2 * (z1 * y3 - y1 * z3) + x3 * (y1 * z2 - z1 * y2);
    };
    const Real vol = triple(dx31 + dx72, dx63, dx20, dy31 + dy72, dy63, dy20, dz31 + dz72, dz63, dz20) +
                     triple(dx43 + dx57, dx64, dx70, dy43 + dy57, dy64, dy70, dz43 + dz57, dz64, dz70) +
                     triple(dx14 + dx25, dx61, dx50, dy14 + dy25, dy61, dy50, dz14 + dz25, dz61, dz50);
    return vol * Real(1.0 / 12.0);
}

}  // namespace lulesh
