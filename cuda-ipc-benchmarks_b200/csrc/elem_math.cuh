// elem_math.cuh -- the element volume in the reference's written form (same
// operands, same association), for the mixed-precision kinematics: fewer FP64
// operations than the modal form where only the volume is wanted in FP64.
#pragma once

namespace lulesh {

// TRIPLE_PRODUCT of lulesh.cu:287-288, with its argument binding
template <typename T>
__device__ __forceinline__ T triple_product(T x1, T y1, T z1, T x2, T y2, T z2,
                                            T x3, T y3, T z3)
{
    return ((x1) * ((y2) * (z3) - (z2) * (y3)) + (x2) * ((z1) * (y3) - (y1) * (z3)) +
            (x3) * ((y1) * (z2) - (z1) * (y2)));
}

// CalcElemVolume, lulesh.cu:221-307
template <typename T>
__device__ __forceinline__ T elem_volume(const T x[8], const T y[8], const T z[8])
{
    const T twelveth = T(1.0) / T(12.0);
    T dx61 = x[6] - x[1], dy61 = y[6] - y[1], dz61 = z[6] - z[1];
    T dx70 = x[7] - x[0], dy70 = y[7] - y[0], dz70 = z[7] - z[0];
    T dx63 = x[6] - x[3], dy63 = y[6] - y[3], dz63 = z[6] - z[3];
    T dx20 = x[2] - x[0], dy20 = y[2] - y[0], dz20 = z[2] - z[0];
    T dx50 = x[5] - x[0], dy50 = y[5] - y[0], dz50 = z[5] - z[0];
    T dx64 = x[6] - x[4], dy64 = y[6] - y[4], dz64 = z[6] - z[4];
    T dx31 = x[3] - x[1], dy31 = y[3] - y[1], dz31 = z[3] - z[1];
    T dx72 = x[7] - x[2], dy72 = y[7] - y[2], dz72 = z[7] - z[2];
    T dx43 = x[4] - x[3], dy43 = y[4] - y[3], dz43 = z[4] - z[3];
    T dx57 = x[5] - x[7], dy57 = y[5] - y[7], dz57 = z[5] - z[7];
    T dx14 = x[1] - x[4], dy14 = y[1] - y[4], dz14 = z[1] - z[4];
    T dx25 = x[2] - x[5], dy25 = y[2] - y[5], dz25 = z[2] - z[5];
    T volume = triple_product(dx31 + dx72, dx63, dx20, dy31 + dy72, dy63, dy20,
                              dz31 + dz72, dz63, dz20) +
               triple_product(dx43 + dx57, dx64, dx70, dy43 + dy57, dy64, dy70,
                              dz43 + dz57, dz64, dz70) +
               triple_product(dx14 + dx25, dx61, dx50, dy14 + dy25, dy61, dy50,
                              dz14 + dz25, dz61, dz50);
    volume *= twelveth;
    return volume;
}

}  // namespace lulesh
