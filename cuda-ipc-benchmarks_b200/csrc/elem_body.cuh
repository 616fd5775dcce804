// elem_body.cuh -- per-element bodies of the FP64 force and kinematics
// kernels.  Each body receives the element's eight gathered node values and
// does the rest: element loads, arithmetic, stores.  The launch that
// gathers (kernels.cu) issues all 48 node loads before any arithmetic.
#pragma once

#include <climits>

#include "elem_math.cuh"
#include "elem_modal.cuh"
#include "kernels.cuh"

namespace lulesh {

// Corner forces are written once and read once: with LULESH_CORNER_STREAM
// (the default) they use evict-first stores and loads, leaving L2 to the
// node and element arrays (nodal 67.6 -> 61.3 us at -s 100 on B200).
#ifndef LULESH_CORNER_STREAM
#define LULESH_CORNER_STREAM 1
#endif

__device__ __forceinline__ void st_corner(double *p, double v)
{
#if LULESH_CORNER_STREAM
    __stcs(p, v);
#else
    *p = v;
#endif
}

__device__ __forceinline__ double ld_corner(const double *p)
{
#if LULESH_CORNER_STREAM
    return __ldcs(p);
#else
    return *p;
#endif
}

// Velocities gathered into registers at kernel start, handed to the body
// where its arithmetic first needs them.
struct VelRegs {
    const double (&xd)[8];
    const double (&yd)[8];
    const double (&zd)[8];
    __device__ __forceinline__ void fetch(double (&x)[8], double (&y)[8], double (&z)[8]) const
    {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            x[i] = xd[i];
            y[i] = yd[i];
            z[i] = zd[i];
        }
    }
};

// The eight node indices of element el on the structured mesh, in the
// nodelist order of BuildMesh (lulesh.cu:730-737): corner j sits at lattice
// offset (x: bits 0x66, y: 0xCC, z: 0xF0 of j) from corner 0.
template <bool U = false>
__device__ __forceinline__ void elem_nodes(const DomDev &D, int el, int n[8])
{
    if (U) {  // an unstructured mesh's own nodelist (stride padded_numElem)
#pragma unroll
        for (int k = 0; k < 8; ++k) n[k] = D.nodelist[(size_t)k * D.Ep + el];
        return;
    }
    const int nx = D.nx, en = D.en;
    const int ix = el % nx;
    const int t = el / nx;
    const int iy = t % nx;
    const int iz = t / nx;
    const int n0 = (iz * en + iy) * en + ix;
    n[0] = n0;
    n[1] = n0 + 1;
    n[2] = n0 + en + 1;
    n[3] = n0 + en;
    n[4] = n0 + en * en;
    n[5] = n0 + en * en + 1;
    n[6] = n0 + en * en + en + 1;
    n[7] = n0 + en * en + en;
}

// CalcVolumeForceForElems_kernel (lulesh.cu:2080-2259) after the coordinate
// gathers, in the element's modes (elem_modal.cuh): stress + FB hourglass
// corner forces, one component at a time, handed to store(component, f[8]).
// vel(component, v[8]) gives the corner velocities, asked for only when HG
// (hourglass coefficient > 0); elem_error() is called when the volume or the
// centre Jacobian is negative.
//
// A component needs the geometry (78 registers of it) and its own eight
// velocities, nothing of the other components, so the three run one after the
// other in few registers.
template <bool HG, class Vel, class Store, class Error>
__device__ __forceinline__ void force_modal(const double (&xn)[8], const double (&yn)[8],
                                            const double (&zn)[8], double volo, double v, double p,
                                            double q, double ss, double mass, double hourg,
                                            const Vel &vel, const Store &store,
                                            const Error &elem_error)
{
    ElemModes<double> m;
    elem_modes(xn, yn, zn, m);
    ForceGeometry<double> g;
    force_geometry<double, HG>(m, g);
    const double det = volo * v;
    if (v < 0. || g.det < 0.) elem_error();
    const double press = (p + q) * (1.0 / 64.0);
    const double vol64 = (1.0 / 64.0) / det;
    const double coef = HG ? -hourg * 0.01 * ss * mass * rcbrt(det) : 0.0;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        double vc[8], f[8];
        if (HG) vel(c, vc);
        force_component<double, HG>(m, g, c, vc, press, vol64, coef, f);
        store(c, f);
    }
}

// the corner arrays at elem + Ep * corner
struct CornerStore {
    double *fx, *fy, *fz;
    int elem, Ep;
    __device__ __forceinline__ void operator()(int c, const double (&f)[8]) const
    {
        double *p = (c == 0 ? fx : c == 1 ? fy : fz) + elem;
#pragma unroll
        for (int k = 0; k < 8; ++k) st_corner(p + Ep * k, f[k]);
    }
};

// CalcKinematicsAndMonotonicQGradient_kernel (lulesh.cu:3343-3507) after
// the node gathers, for element k.
template <class Vel>
__device__ __forceinline__ void kin_elem(const DomDev &D, TimeCtl &T, int k, double (&x_local)[8],
                                         double (&y_local)[8], double (&z_local)[8],
                                         const Vel &vel)
{
    double B[3][8];
    double Dv[3];
    const double volume = elem_volume(x_local, y_local, z_local);
    const double relativeVolume = volume / D.volo[k];
    D.vnew[k] = relativeVolume;
    D.delv[k] = relativeVolume - D.v[k];
    D.arealg[k] = elem_characteristic_length(x_local, y_local, z_local, volume);

    double xd_local[8], yd_local[8], zd_local[8];
    vel.fetch(xd_local, yd_local, zd_local);
    const double dt2 = 0.5 * T.deltatime;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        x_local[j] -= dt2 * xd_local[j];
        y_local[j] -= dt2 * yd_local[j];
        z_local[j] -= dt2 * zd_local[j];
    }
    double detJ;
    shape_function_derivatives(x_local, y_local, z_local, B, &detJ);
    elem_velocity_divergence(xd_local, yd_local, zd_local, B, detJ, Dv);
    const double vdovNew = Dv[0] + Dv[1] + Dv[2];
    D.vdov[k] = vdovNew;

    const double vol = D.volo[k] * relativeVolume;
    // undo the half-step shift exactly as the reference does (the restored
    // coordinates can differ from the originals in the last bit)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        x_local[j] += dt2 * xd_local[j];
        y_local[j] += dt2 * yd_local[j];
        z_local[j] += dt2 * zd_local[j];
    }
    double dxz, dvz, dxx, dvx, dxe, dve;
    mono_gradient(x_local, y_local, z_local, xd_local, yd_local, zd_local, vol, &dxz, &dvz,
                  &dxx, &dvx, &dxe, &dve);
    D.delx_zeta[k] = dxz;
    D.delv_zeta[k] = dvz;
    D.delx_xi[k] = dxx;
    D.delv_xi[k] = dvx;
    D.delx_eta[k] = dxe;
    D.delv_eta[k] = dve;
    if (relativeVolume < 0) atomicMin(&T.bad_vol, k);
}

}  // namespace lulesh
