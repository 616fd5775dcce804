// elem_modal.cuh -- the hexahedron arithmetic of the force and kinematics
// kernels in the element's trilinear modes.
//
// A trilinear hexahedron is x(xi,eta,zeta) = sum over its eight modes.  With
// the corner signs (xi,eta,zeta) of the nodelist order, the signed corner sums
//   A, B, C     sum of xi x, eta x, zeta x            (the Jacobian)
//   D, E, F     sum of eta zeta x, xi zeta x, xi eta x (hourglass)
//   G           sum of xi eta zeta x                   (hourglass)
// carry everything the step needs:
//   * the hourglass base vectors of CalcFBHourglassForceForElems
//     (lulesh.cu:2017-2071) ARE the sign patterns of D, E, F, G, so the mode
//     sums hx, hy, hz of CalcHourglassModes are D, E, F, G themselves;
//   * the volume is 1/64 [A.(BxC) + (A.(FxE) + B.(DxF) + C.(ExD)) / 3], the
//     integral of the Jacobian determinant (CalcElemVolume, lulesh.cu:221-307,
//     gives the same number), and VoluDer (lulesh.cu:1756-1784) its gradient:
//     linear in the mode gradients W below;
//   * the face normal sums of CalcElemNodeNormals (lulesh.cu:1657-1711) have
//     components in the modes A, B, C only, BxC + FxE and its rotations.
// The reference evaluates all of these corner by corner: 934 FP64 operations
// per element for the force and 649 for the kinematics, with 32 hourglass
// coefficients and 24 volume derivatives alive at once.  In modes the same
// results take about 600 and 350, and a third of the registers.
//
// Coordinates enter through differences of corners only (diagonals for A, B,
// C, G; edges for D, E, F), so no sum of coordinates near 1 is rounded.
// Every product that feeds a sum is an explicit fma: the bits do not depend
// on the kernel the functions are inlined into.  The modes, the crosses and
// the kinematics' cancelling sums give the same bits with x and y (and xi and
// eta) exchanged, as the problem does: the symmetry check of a run compares
// elements across that diagonal, and its largest relative difference at
// -s 100 after 505 cycles is 5e-14 this way and 8e-12 with dot3 throughout,
// for 0 of 225 us a cycle.
#pragma once

namespace lulesh {

__device__ __forceinline__ double fma_t(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float fma_t(float a, float b, float c) { return fmaf(a, b, c); }
// a sum and a product that no compiler joins into one fma
__device__ __forceinline__ double sum_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float sum_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
// a / sqrt(s) and a / cbrt(s) through the reciprocal roots, a third of the
// operations of a root and a quotient: within 2 ulp in FP64.  Against 80-bit
// arithmetic from -s 5 to -s 45 the lengths and delx are as near either way (rms
// 1.0-1.2 units of 2^-53; 1.2-34 in the corner form) and the corner forces equal;
// roots and quotients take -s 100 from 185 to 192 us per cycle.  The FP32
// reciprocal square root is off by 2 ulp by itself and gets one Newton step
// (but not at 0 and infinity, where the step is not a number): with it the
// mixed kernels' lengths are as near FP64 as with the rounded root and quotient.
__device__ __forceinline__ double over_sqrt(double a, double s) { return a * rsqrt(s); }
__device__ __forceinline__ float over_sqrt(float a, float s)
{
    const float r = rsqrtf(s);
    const float e = fmaf(-s * r, r, 1.0f);
    return a * (e == e ? fmaf(0.5f * r, e, r) : r);
}
__device__ __forceinline__ double over_cbrt(double a, double s) { return a * rcbrt(s); }
__device__ __forceinline__ float over_cbrt(float a, float s) { return a * rcbrtf(s); }
__device__ __forceinline__ double fmax_t(double a, double b) { return fmax(a, b); }
__device__ __forceinline__ float fmax_t(float a, float b) { return fmaxf(a, b); }
__device__ __forceinline__ double abs_t(double a) { return fabs(a); }
__device__ __forceinline__ float abs_t(float a) { return fabsf(a); }

// r = a x b
template <typename T>
__device__ __forceinline__ void cross(const T a[3], const T b[3], T r[3])
{
    r[0] = fma_t(a[1], b[2], -(a[2] * b[1]));
    r[1] = fma_t(a[2], b[0], -(a[0] * b[2]));
    r[2] = fma_t(a[0], b[1], -(a[1] * b[0]));
}

// r = a x b + c x d
template <typename T>
__device__ __forceinline__ void cross2(const T a[3], const T b[3], const T c[3], const T d[3],
                                       T r[3])
{
    T s[3];
    cross(c, d, s);
    r[0] = fma_t(a[1], b[2], fma_t(-a[2], b[1], s[0]));
    r[1] = fma_t(a[2], b[0], fma_t(-a[0], b[2], s[1]));
    r[2] = fma_t(a[0], b[1], fma_t(-a[1], b[0], s[2]));
}

template <typename T>
__device__ __forceinline__ T dot3(const T a[3], const T b[3])
{
    return fma_t(a[0], b[0], fma_t(a[1], b[1], a[2] * b[2]));
}

// a . b, the same bits with x and y exchanged
template <typename T>
__device__ __forceinline__ T dot3_sym(const T a[3], const T b[3])
{
    return fma_t(a[2], b[2], sum_rn(mul_rn(a[0], b[0]), mul_rn(a[1], b[1])));
}

// A, B, C and G of one component from its diagonals (n6-n0, n7-n1, n4-n2,
// n5-n3)
template <typename T>
__device__ __forceinline__ void odd_modes(const T v[8], T &a, T &b, T &c, T &g)
{
    const T u0 = v[6] - v[0], u1 = v[7] - v[1], u2 = v[4] - v[2], u3 = v[5] - v[3];
    const T p = u0 - u2, q = u1 - u3, s = u0 + u2, t = u1 + u3;
    a = p - q;
    b = p + q;
    c = s + t;
    g = s - t;
}

// D, E, F of one component from its edges
template <typename T>
__device__ __forceinline__ void even_modes(const T v[8], T &d, T &e, T &f)
{
    const T q0 = v[3] - v[0], q1 = v[2] - v[1], q2 = v[7] - v[4], q3 = v[6] - v[5];
    const T s = q3 - q0, t = q2 - q1;
    d = s + t;
    f = s - t;
    const T p0 = v[1] - v[0], p1 = v[2] - v[3], p2 = v[5] - v[4], p3 = v[6] - v[7];
    e = (p3 - p0) + (p2 - p1);
}

// Modes of one element's coordinates, [component] each.
template <typename T>
struct ElemModes {
    T A[3], B[3], C[3], D[3], E[3], F[3], G[3];
};

template <typename T>
__device__ __forceinline__ void elem_modes(const T x[8], const T y[8], const T z[8],
                                           ElemModes<T> &m)
{
    odd_modes(x, m.A[0], m.B[0], m.C[0], m.G[0]);
    odd_modes(y, m.A[1], m.B[1], m.C[1], m.G[1]);
    odd_modes(z, m.A[2], m.B[2], m.C[2], m.G[2]);
    even_modes(x, m.D[0], m.E[0], m.F[0]);
    even_modes(y, m.D[1], m.E[1], m.F[1]);
    even_modes(z, m.D[2], m.E[2], m.F[2]);
}

// The face-area crosses of one element, x64: BxC, CxA, AxB and the hourglass
// parts FxE, DxF, ExD that complete them to face normals and volume.
template <typename T>
struct FaceCrosses {
    T bc[3], ca[3], ab[3], fe[3], df[3], ed[3];
};

template <typename T>
__device__ __forceinline__ void face_crosses(const ElemModes<T> &m, FaceCrosses<T> &c)
{
    cross(m.B, m.C, c.bc);
    cross(m.C, m.A, c.ca);
    cross(m.A, m.B, c.ab);
    cross(m.F, m.E, c.fe);
    cross(m.D, m.F, c.df);
    cross(m.E, m.D, c.ed);
}

// What the corner forces of one element need of its geometry: the volume
// gradient by mode W (x64), the face normal sums N in modes A, B, C (x64),
// and A.(BxC), whose sign is the Jacobian determinant's at the centre.
template <typename T>
struct ForceGeometry {
    T WA[3], WB[3], WC[3], WD[3], WE[3], WF[3], NA[3], NB[3], NC[3], det;
};

template <typename T, bool HG>
__device__ __forceinline__ void force_geometry(const ElemModes<T> &m, ForceGeometry<T> &g)
{
    const T third = T(1.0) / T(3.0);
    FaceCrosses<T> x;
    face_crosses(m, x);
    g.det = dot3(m.A, x.bc);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        g.NA[i] = x.bc[i] + x.fe[i];
        g.NB[i] = x.ca[i] + x.df[i];
        g.NC[i] = x.ab[i] + x.ed[i];
    }
    if (HG) {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            g.WA[i] = fma_t(third, x.fe[i], x.bc[i]);
            g.WB[i] = fma_t(third, x.df[i], x.ca[i]);
            g.WC[i] = fma_t(third, x.ed[i], x.ab[i]);
        }
        cross2(m.F, m.B, m.C, m.E, g.WD);
        cross2(m.A, m.F, m.D, m.C, g.WE);
        cross2(m.E, m.A, m.B, m.D, g.WF);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            g.WD[i] *= third;
            g.WE[i] *= third;
            g.WF[i] *= third;
        }
    }
}

// Corner values of one component from its modes: r[k] = sum of the modes
// with corner k's signs.
template <typename T>
__device__ __forceinline__ void corners_from_modes(T a, T b, T c, T d, T e, T f, T g, T r[8])
{
    const T s = d + e, t = d - e;
    const T e0 = s + f, e2 = f - s, e1 = t - f, e3 = -(t + f);  // corners 0/6, 2/4, 1/7, 3/5
    const T ab = a + b, cg = c + g, amb = a - b, cmg = c - g;
    const T o0 = ab + cg, o2 = ab - cg, o1 = amb - cmg, o3 = amb + cmg;
    r[0] = e0 - o0;
    r[6] = e0 + o0;
    r[2] = e2 + o2;
    r[4] = e2 - o2;
    r[1] = e1 + o1;
    r[7] = e1 - o1;
    r[3] = e3 - o3;
    r[5] = e3 + o3;
}

// One component of an element's corner forces: the stress -sigma N of
// SumElemStressesToNodeForces (lulesh.cu:1604-1652) and, with HG, the
// Flanagan-Belytschko hourglass force of CalcElemFBHourglassForce
// (lulesh.cu:1833-2013) for the velocity component v.
//   press   (p + q) / 64          vol64   1 / (64 volume)
//   coef    the hourglass coefficient
template <typename T, bool HG>
__device__ __forceinline__ void force_component(const ElemModes<T> &m, const ForceGeometry<T> &w,
                                                int j, const T v[8], T press, T vol64, T coef,
                                                T f[8])
{
    const T na = press * w.NA[j], nb = press * w.NB[j], nc = press * w.NC[j];
    if (!HG) {
        corners_from_modes(na, nb, nc, T(0), T(0), T(0), T(0), f);
        return;
    }
    T va, vb, vc, vd, ve, vf, vg;
    odd_modes(v, va, vb, vc, vg);
    even_modes(v, vd, ve, vf);
    // M = (1/volume) (volume gradient . velocity): one column of the
    // volume-weighted velocity gradient
    T M[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const T s = fma_t(w.WA[i], va, fma_t(w.WB[i], vb, w.WC[i] * vc));
        const T t = fma_t(w.WD[i], vd, fma_t(w.WE[i], ve, w.WF[i] * vf));
        M[i] = (s + t) * vol64;
    }
    // hourglass-shaped part of the velocity, mode by mode
    const T sd = fma_t(-m.D[0], M[0], fma_t(-m.D[1], M[1], fma_t(-m.D[2], M[2], vd)));
    const T se = fma_t(-m.E[0], M[0], fma_t(-m.E[1], M[1], fma_t(-m.E[2], M[2], ve)));
    const T sf = fma_t(-m.F[0], M[0], fma_t(-m.F[1], M[1], fma_t(-m.F[2], M[2], vf)));
    const T sg = fma_t(-m.G[0], M[0], fma_t(-m.G[1], M[1], fma_t(-m.G[2], M[2], vg)));
    const T cv = -(coef * vol64);
    T Q[3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
        Q[i] = cv * fma_t(m.D[i], sd, fma_t(m.E[i], se, fma_t(m.F[i], sf, m.G[i] * sg)));
    const T fa = fma_t(w.WA[0], Q[0], fma_t(w.WA[1], Q[1], fma_t(w.WA[2], Q[2], na)));
    const T fb = fma_t(w.WB[0], Q[0], fma_t(w.WB[1], Q[1], fma_t(w.WB[2], Q[2], nb)));
    const T fc = fma_t(w.WC[0], Q[0], fma_t(w.WC[1], Q[1], fma_t(w.WC[2], Q[2], nc)));
    const T fd = fma_t(w.WD[0], Q[0], fma_t(w.WD[1], Q[1], fma_t(w.WD[2], Q[2], coef * sd)));
    const T fe = fma_t(w.WE[0], Q[0], fma_t(w.WE[1], Q[1], fma_t(w.WE[2], Q[2], coef * se)));
    const T ff = fma_t(w.WF[0], Q[0], fma_t(w.WF[1], Q[1], fma_t(w.WF[2], Q[2], coef * sf)));
    corners_from_modes(fa, fb, fc, fd, fe, ff, coef * sg, f);
}

// CalcElemVolume (lulesh.cu:221-307)
template <typename T>
__device__ __forceinline__ T modal_volume(const ElemModes<T> &m, const FaceCrosses<T> &c)
{
    const T h = (dot3_sym(m.A, c.fe) + dot3_sym(m.B, c.df)) + dot3_sym(m.C, c.ed);
    return T(1.0 / 64.0) * fma_t(T(1.0) / T(3.0), h, dot3_sym(m.C, c.ab));
}

// The larger |N + M|^2, |N - M|^2 of a pair of opposite faces
template <typename T>
__device__ __forceinline__ T larger_face(const T a[3], const T b[3], const T mm[3])
{
    T n[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) n[i] = a[i] + b[i];
    return fma_t(T(2.0), abs_t(dot3(n, mm)), dot3(n, n) + dot3(mm, mm));
}

// CalcElemCharacteristicLength (lulesh.cu:3126-3166): 4 volume over the
// root of the largest AreaFace (lulesh.cu:3103-3122).  AreaFace is
// (f.f)(g.g) - (f.g)^2 = |f x g|^2 of the face's centre tangents, and f x g
// is (N +- M)/4 with N = BxC + FxE, M = BxE + FxC on the xi faces and their
// rotations on the others (the three M add up to zero).
template <typename T>
__device__ __forceinline__ T modal_length(const ElemModes<T> &m, const FaceCrosses<T> &c, T volume)
{
    T ma[3], mb[3], mc[3];
    cross2(m.B, m.E, m.F, m.C, ma);
    cross2(m.D, m.A, m.C, m.F, mb);
#pragma unroll
    for (int i = 0; i < 3; ++i) mc[i] = -(ma[i] + mb[i]);
    T area = fmax_t(larger_face(c.bc, c.fe, ma), T(0.0));
    area = fmax_t(larger_face(c.ca, c.df, mb), area);
    area = fmax_t(larger_face(c.ab, c.ed, mc), area);
    return over_sqrt(T(16.0) * volume, area);
}

// dxx + dyy + dzz of CalcElemVelocityGradient (lulesh.cu:3171-3248) at the
// half step: (cofactors of J) : (velocity modes) / det J, with
// J = J(x) - dt2 J(v).  The step's strain rates are used nowhere else.
template <typename T>
__device__ __forceinline__ T modal_divergence(const ElemModes<T> &m, const T va[3], const T vb[3],
                                              const T vc[3], T dt2)
{
    T a[3], b[3], c[3], bc[3], ca[3], ab[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        a[i] = fma_t(-dt2, va[i], m.A[i]);
        b[i] = fma_t(-dt2, vb[i], m.B[i]);
        c[i] = fma_t(-dt2, vc[i], m.C[i]);
    }
    cross(b, c, bc);
    cross(c, a, ca);
    cross(a, b, ab);
    return ((dot3_sym(bc, va) + dot3_sym(ca, vb)) + dot3_sym(ab, vc)) / dot3_sym(c, ab);
}

// One direction of CalcMonoGradient (lulesh.cu:3251-3334): n the cross of
// the two other directions' modes, v the direction's velocity modes
template <typename T>
__device__ __forceinline__ void modal_mono(const T n[3], const T v[3], T volume, T norm, T *delx,
                                           T *delv)
{
    const T ptiny = T(1.e-36);
    *delx = over_sqrt(T(16.0) * volume, dot3(n, n) + T(256.0) * ptiny);
    *delv = (T(1.0 / 64.0) * norm) * dot3_sym(n, v);
}

}  // namespace lulesh
