// mixed.cu -- mixed-precision variants of the force, nodal and kinematics
// kernels (LULESH_FLAG_MIXED).
//
// FP32: the element-local stress / FB-hourglass arithmetic of
//   CalcVolumeForceForElems_kernel (lulesh.cu:2080-2259) and the
//   characteristic length, velocity divergence and monotonic-Q gradients of
//   CalcKinematicsAndMonotonicQGradient_kernel (lulesh.cu:3343-3507), in the
//   element's modes (elem_modal.cuh).  Every one of these is a function of
//   coordinate and velocity DIFFERENCES, so the kernels form x[k] - x[0] and
//   xd[k] - xd[0] in FP64 and hand FP32 only those: a velocity gradient then
//   keeps FP32's digits where the flow is fast and its differences small.
// FP32 storage, compensated sum: corner forces are stored as FP32 and each
//   node adds its eight corners with Neumaier's compensated summation, then
//   converts (sum + compensation) to FP64.
// FP64 (unchanged): element volume, relative volume and delv (delv is a
//   difference of two numbers near 1, which FP32 would leave with 3-5
//   digits), the node update, the EOS, and the dt reduction.
#include <climits>

#include <type_traits>

#include "elem_math.cuh"
#include "elem_modal.cuh"
#include "kernels.cuh"

namespace lulesh {

// Resident blocks per SM asked of the compiler for the mixed kernels, measured
// on B200 at -s 120 (1.7e6 elements), identical results: force 5 (96
// registers) 87 us, 94 at 3 and 4; kinematics 5 (94 registers) 78 us, the
// same at 4 and 6.  The corner-by-corner forms took 131 us and 113 us at 128
// registers.  What is left in both is the 48 gathers and their conversions to
// FP32, and in the kinematics the FP64 volume.
#ifndef LULESH_MIXED_FORCE_MINB
#define LULESH_MIXED_FORCE_MINB 5
#endif
#ifndef LULESH_MIXED_KIN_MINB
#define LULESH_MIXED_KIN_MINB 5
#endif

__device__ __forceinline__ void elem_nodes_m(const DomDev &D, int el, int n[8])
{
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

// The FP32 corner arrays of a domain: by value with the domain's record, from
// the device table otherwise.
template <class W>
__device__ __forceinline__ CornerF32 corner_arrays(const W &, const CornerF32 *table,
                                                   const CornerF32 &one, int d)
{
    return W::kTable ? table[d] : one;
}

template <bool HG, class W>
__global__ void __launch_bounds__(kElemBlock, LULESH_MIXED_FORCE_MINB)
    k_force_mixed(const __grid_constant__ W w, Params P, const CornerF32 *cfs, CornerF32 cf1)
{
    pdl_enter();
    const int2 blk = w.template block<kElemBlock, false>();
    const DomDev &D = w.domain(blk.x);
    TimeCtl &T = w.time(D);
    if (W::kTable && !T.active) return;
    const int elem = blk.y + threadIdx.x;
    if (elem >= D.numElem) return;
    const CornerF32 cf = corner_arrays(w, cfs, cf1, blk.x);

    int n[8];
    elem_nodes_m(D, elem, n);
#pragma unroll
    for (int i = 0; i < 8; ++i) n[i] = chk_index(n[i], D.numNode, &T, kChkNode);
    // all node gathers first: the velocities arrive while the coordinate
    // arithmetic runs
    float v[3][8];
    if (HG) {
        const double u0 = D.xd[n[0]], v0 = D.yd[n[0]], w0 = D.zd[n[0]];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            v[0][i] = (float)(D.xd[n[i]] - u0);
            v[1][i] = (float)(D.yd[n[i]] - v0);
            v[2][i] = (float)(D.zd[n[i]] - w0);
        }
    }
    const double x0 = D.x[n[0]], y0 = D.y[n[0]], z0 = D.z[n[0]];
    float xn[8], yn[8], zn[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        xn[i] = (float)(D.x[n[i]] - x0);
        yn[i] = (float)(D.y[n[i]] - y0);
        zn[i] = (float)(D.z[n[i]] - z0);
    }
    const double volume = D.v[elem];
    const float det = (float)(D.volo[elem] * volume);
    const float coef =
        over_cbrt((float)(-P.hgcoef * 0.01 * D.ss[elem] * D.elemMass[elem]), det);
    const float press = (float)(D.p[elem] + D.q[elem]) * (1.0f / 64.0f);
    const float vol64 = (1.0f / 64.0f) / det;
    if (!W::kTable && !T.active) return;

    ElemModes<float> m;
    elem_modes(xn, yn, zn, m);
    ForceGeometry<float> g;
    force_geometry<float, HG>(m, g);
    if (volume < 0. || g.det < 0.f) atomicMin(&T.bad_vol, elem);
    // written once, read once by the nodal gather: evict-first
    const int Ep = D.Ep;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        float f[8];
        force_component<float, HG>(m, g, c, v[c], press, vol64, coef, f);
        float *to = (c == 0 ? cf.fx : c == 1 ? cf.fy : cf.fz) + elem;
#pragma unroll
        for (int k = 0; k < 8; ++k) __stcs(to + Ep * k, f[k]);
    }
}

// launch(where, the only domain's corner arrays)
template <class Launch>
static void launch_mixed(const SetArgs &a, int nblocks, const Launch &launch)
{
    launch_where<true, false>(a, nblocks, [&](const auto &w) {
        launch(w, a.corner32 ? *a.corner32 : CornerF32{});
    });
}

void launch_force_mixed(const SetArgs &a, int nblocks, Params P, const CornerF32 *cf,
                        cudaStream_t s)
{
    launch_mixed(a, nblocks, [&](const auto &w, const CornerF32 &one) {
        using W = std::decay_t<decltype(w)>;
        if (P.hgcoef > 0.0)
            launch_k(k_force_mixed<true, W>, nblocks, kElemBlock, s, a.pdl != 0, w, P, cf, one);
        else
            launch_k(k_force_mixed<false, W>, nblocks, kElemBlock, s, a.pdl != 0, w, P, cf, one);
    });
}

// Neumaier's compensated addition: s + c carries the sum of all terms
__device__ __forceinline__ void comp_add(float &s, float &c, float v)
{
    const float t = s + v;
    if (fabsf(s) >= fabsf(v))
        c += (s - t) + v;
    else
        c += (v - t) + s;
    s = t;
}

// Resident blocks per SM for the mixed node update, whose 24 corner loads
// are all issued before the compensated sums: 10 (48 registers) measured
// best on B200 at -s 120 (57.4 us against 57.7 at 8, 59.2 at 12 and 75.5
// at 16; 83.7 us with the loads interleaved with the sums at 16).
#ifndef LULESH_MIXED_NODAL_MINB
#define LULESH_MIXED_NODAL_MINB 10
#endif

template <class W>
__global__ void __launch_bounds__(kNodeBlock, min_blocks(LULESH_MIXED_NODAL_MINB, kNodeBlock))
    k_nodal_mixed(const __grid_constant__ W w, Params P, const CornerF32 *cfs, CornerF32 cf1)
{
    pdl_enter();
    const int2 blk = w.template block<kNodeBlock, LULESH_NODAL_REVERSE && !W::kTable>();
    const DomDev &D = w.domain(blk.x);
    TimeCtl &T = w.time(D);
    if (W::kTable && !T.active) return;
    const int i = blk.y + threadIdx.x;
    if (i >= D.numNode) return;
    const CornerF32 cf = corner_arrays(w, cfs, cf1, blk.x);
    const int nx = D.nx;
    int px, py, pz;
    lattice(D.by_en, i, px, py, pz);
    float sx = 0.f, sy = 0.f, sz = 0.f, cx = 0.f, cy = 0.f, cz = 0.f;
    const int ox[8] = {0, 1, 1, 0, 0, 1, 1, 0}, oy[8] = {0, 0, 1, 1, 0, 0, 1, 1},
              oz[8] = {0, 0, 0, 0, 1, 1, 1, 1};
    // all 24 corner loads first, then the compensated sums in corner order
    float vx[8], vy[8], vz[8];
    bool in[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int ex = px - ox[j], ey = py - oy[j], ez = pz - oz[j];
        in[j] = (unsigned)ex < (unsigned)nx && (unsigned)ey < (unsigned)nx &&
                (unsigned)ez < (unsigned)nx;
        vx[j] = vy[j] = vz[j] = 0.f;
        if (in[j]) {
            const int idx = chk_index(j * D.Ep + (ez * nx + ey) * nx + ex, 8LL * D.Ep,
                                      &T, kChkCorner);
            vx[j] = __ldcs(cf.fx + idx);
            vy[j] = __ldcs(cf.fy + idx);
            vz[j] = __ldcs(cf.fz + idx);
        }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        if (in[j]) {
            comp_add(sx, cx, vx[j]);
            comp_add(sy, cy, vy[j]);
            comp_add(sz, cz, vz[j]);
        }
    }
    const double fx = (double)sx + (double)cx;
    const double fy = (double)sy + (double)cy;
    const double fz = (double)sz + (double)cz;
    if (!W::kTable && !T.active) return;
    const double one_over_nMass = 1. / D.nodalMass[i];
    double xdd = fx * one_over_nMass, ydd = fy * one_over_nMass, zdd = fz * one_over_nMass;
    if (D.col == 0 && px == 0) xdd = 0.0;
    if (D.row == 0 && py == 0) ydd = 0.0;
    if (D.plane == 0 && pz == 0) zdd = 0.0;
    const double dt = T.deltatime, u_cut = P.u_cut;
    double xdtmp = D.xd[i] + xdd * dt;
    double ydtmp = D.yd[i] + ydd * dt;
    double zdtmp = D.zd[i] + zdd * dt;
    if (fabs(xdtmp) < u_cut) xdtmp = 0.0;
    if (fabs(ydtmp) < u_cut) ydtmp = 0.0;
    if (fabs(zdtmp) < u_cut) zdtmp = 0.0;
    D.x[i] += xdtmp * dt;
    D.y[i] += ydtmp * dt;
    D.z[i] += zdtmp * dt;
    D.xd[i] = xdtmp;
    D.yd[i] = ydtmp;
    D.zd[i] = zdtmp;
    if (w.materialize()) {
        D.fx[i] = fx;
        D.fy[i] = fy;
        D.fz[i] = fz;
        D.xdd[i] = xdd;
        D.ydd[i] = ydd;
        D.zdd[i] = zdd;
    }
}

void launch_nodal_mixed(const SetArgs &a, int nblocks, Params P, const CornerF32 *cf,
                        cudaStream_t s)
{
    launch_mixed(a, nblocks, [&](const auto &w, const CornerF32 &one) {
        launch_k(k_nodal_mixed<std::decay_t<decltype(w)>>, nblocks, kNodeBlock, s, a.pdl != 0, w,
                 P, cf, one);
    });
}

template <class W>
__global__ void __launch_bounds__(kElemBlock, LULESH_MIXED_KIN_MINB)
    k_kinematics_mixed(const __grid_constant__ W w)
{
    pdl_enter();
    const int2 blk = w.template block<kElemBlock, LULESH_KIN_REVERSE>();
    const DomDev &D = w.domain(blk.x);
    TimeCtl &T = w.time(D);
    if (W::kTable && !T.active) return;
    const int k = blk.y + threadIdx.x;
    if (k >= D.numElem) return;
    int n[8];
    elem_nodes_m(D, k, n);
#pragma unroll
    for (int l = 0; l < 8; ++l) n[l] = chk_index(n[l], D.numNode, &T, kChkNode);
    // FP64: volume and relative volume (they feed delv)
    double x64[8], y64[8], z64[8];
#pragma unroll
    for (int l = 0; l < 8; ++l) {
        x64[l] = D.x[n[l]];
        y64[l] = D.y[n[l]];
        z64[l] = D.z[n[l]];
    }
    if (!W::kTable && !T.active) return;
    const double volume = elem_volume(x64, y64, z64);
    const double relativeVolume = volume / D.volo[k];
    D.vnew[k] = relativeVolume;
    D.delv[k] = relativeVolume - D.v[k];
    if (relativeVolume < 0) atomicMin(&T.bad_vol, k);
    // FP32: everything else, on coordinates relative to corner 0
    float xl[8], yl[8], zl[8];
#pragma unroll
    for (int l = 0; l < 8; ++l) {
        xl[l] = (float)(x64[l] - x64[0]);
        yl[l] = (float)(y64[l] - y64[0]);
        zl[l] = (float)(z64[l] - z64[0]);
    }
    const float vol = (float)volume;
    ElemModes<float> m;
    elem_modes(xl, yl, zl, m);
    FaceCrosses<float> c;
    face_crosses(m, c);
    D.arealg[k] = (double)modal_length(m, c, vol);
    // the velocities' A, B, C modes are all the step needs
    float va[3], vb[3], vc[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const double *from = c == 0 ? D.xd : c == 1 ? D.yd : D.zd;
        const double v0 = from[n[0]];
        float v[8], vg;
#pragma unroll
        for (int l = 0; l < 8; ++l) v[l] = (float)(from[n[l]] - v0);
        odd_modes(v, va[c], vb[c], vc[c], vg);
    }
    D.vdov[k] = (double)modal_divergence(m, va, vb, vc, (float)(0.5 * T.deltatime));
    const float norm = 1.0f / (vol + 1.e-36f);
    float delx, delv;
    modal_mono(c.ab, vc, vol, norm, &delx, &delv);
    D.delx_zeta[k] = delx;
    D.delv_zeta[k] = delv;
    modal_mono(c.bc, va, vol, norm, &delx, &delv);
    D.delx_xi[k] = delx;
    D.delv_xi[k] = delv;
    modal_mono(c.ca, vb, vol, norm, &delx, &delv);
    D.delx_eta[k] = delx;
    D.delv_eta[k] = delv;
}

void launch_kinematics_mixed(const SetArgs &a, int nblocks, Params P, cudaStream_t s)
{
    (void)P;
    launch_where<true, false>(a, nblocks, [&](const auto &w) {
        launch_k(k_kinematics_mixed<std::decay_t<decltype(w)>>, nblocks, kElemBlock, s,
                 a.pdl != 0, w);
    });
}

}  // namespace lulesh
