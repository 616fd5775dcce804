// elem_body.cuh -- per-element bodies of the FP64 force and kinematics
// kernels, in the modes of elem_modal.cuh.  Each body receives the element's
// eight gathered node values and does the rest: element loads, arithmetic,
// stores.
#pragma once

#include <climits>

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
    const int en = D.en;
    int ix, iy, iz;
    lattice(D.by_nx, el, ix, iy, iz);
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
    const double coef = HG ? over_cbrt(-hourg * 0.01 * ss * mass, det) : 0.0;
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
// the coordinate gathers, for element k, in the element's modes.  The
// velocities enter through their A, B, C modes only; vel(component, v[8])
// gives the corner values.  The monotonic-Q gradients are those of the
// coordinates themselves (the reference shifts them by half a step and back).
template <class Vel>
__device__ __forceinline__ void kin_modal(const DomDev &D, TimeCtl &T, double dt, int k,
                                          const double (&xn)[8], const double (&yn)[8],
                                          const double (&zn)[8], const Vel &vel)
{
    ElemModes<double> m;
    elem_modes(xn, yn, zn, m);
    FaceCrosses<double> c;
    face_crosses(m, c);
    const double volume = modal_volume(m, c);
    const double relativeVolume = volume / D.volo[k];
    D.vnew[k] = relativeVolume;
    D.delv[k] = relativeVolume - D.v[k];
    if (relativeVolume < 0) atomicMin(&T.bad_vol, k);
    D.arealg[k] = modal_length(m, c, volume);

    double va[3], vb[3], vc[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        double v[8], vg;
        vel(i, v);
        odd_modes(v, va[i], vb[i], vc[i], vg);
    }
    D.vdov[k] = modal_divergence(m, va, vb, vc, 0.5 * dt);

    const double norm = 1.0 / (volume + 1.e-36);
    double delx, delv;
    modal_mono(c.ab, vc, volume, norm, &delx, &delv);
    D.delx_zeta[k] = delx;
    D.delv_zeta[k] = delv;
    modal_mono(c.bc, va, volume, norm, &delx, &delv);
    D.delx_xi[k] = delx;
    D.delv_xi[k] = delv;
    modal_mono(c.ca, vb, volume, norm, &delx, &delv);
    D.delx_eta[k] = delx;
    D.delv_eta[k] = delv;
}

}  // namespace lulesh
