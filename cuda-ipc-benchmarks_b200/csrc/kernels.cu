// kernels.cu -- the per-cycle kernels of the LULESH Lagrange leapfrog step.
//
// One cycle is five launches (captured in CUDA graphs), four in small sets,
// whose kernels make the time increment themselves:
//   time_increment  TimeIncrement on the device (lulesh.cu:1400-1461)
//   force           CalcVolumeForceForElems_kernel (lulesh.cu:2080-2259):
//                   stress + FB hourglass corner forces per element
//   nodal           AddNodeForcesFromElems + CalcAccelerationForNodes +
//                   ApplyAccelerationBoundaryConditionsForNodes +
//                   CalcPositionAndVelocityForNodes (lulesh.cu:1715-1751,
//                   2925-3044) fused: corners summed in corner order with
//                   no atomics, then the node update
//   kinematics      CalcKinematicsAndMonotonicQGradient_kernel
//                   (lulesh.cu:3343-3507)
//   eos             CalcMonotonicQRegionForElems_kernel +
//                   ApplyMaterialPropertiesAndUpdateVolume_kernel +
//                   CalcTimeConstraintsForElems (lulesh.cu:3554-3725,
//                   3988-4097, 4216-4403) fused; the dt minimum is reduced
//                   with warp shuffles and one 64-bit atomicMin per block
// Two halo kernels follow CommSyncPosVel and CommMonoQ: the PosVel sync
// copies a neighbour's max-side node layer, the MonoQ ghost kernel its
// boundary element layer of delv_*.  A subdomain set's fused cycle needs
// neither (every corner of every node is summed in single-domain order, and
// k_eos<..., SUB> reads comm-face neighbours in place), and the parts of a
// multi-GPU problem read their proxies in place after the MONOQ messages.
// Unstructured (lmesh) domains run force and kinematics with Mesh::kLists and
// EOS with U = true, which read nodelist, the face links and elemBC from memory
// instead of computing them from the element index, and k_nodal_u for the nodal
// step; scattered ones Mesh::kPacked, k_begin_packed and k_nodal_packed.
#include <climits>
#include <cstdint>
#include <type_traits>

#include "elem_body.cuh"
#include "kernels.cuh"
#include "lulesh_b200.h"

namespace lulesh {

// ---------------------------------------------------------------------------
// time increment

__device__ __forceinline__ unsigned long long dbits(double v)
{
    return (unsigned long long)__double_as_longlong(v);
}

__device__ __forceinline__ void time_increment(TimeCtl &T, const Params &P)
{
    T.active = 0;
    if (T.done) return;
    // checkErrors (lulesh.cu:2879-2892): a cycle that raised an error ends
    // the job before the next one starts
    if (T.bad_vol != INT_MAX) {
        T.status = -1;
        T.done = 1;
        return;
    }
    if (T.bad_q != INT_MAX) {
        T.status = -2;
        T.done = 1;
        return;
    }
#if LULESH_CHECKED
    if (T.chk != 0) {
        T.status = LULESH_BOUNDS_ERROR;
        T.done = 1;
        return;
    }
#endif
    // while (time < stoptime) ... if (its == num_iters) break (lulesh.cu:4858-4873)
    if (!(T.time < P.stoptime) || (T.its_cap > 0 && T.cycle >= T.its_cap)) {
        T.done = 1;
        return;
    }
    if (T.cycle != 0) {
        // the previous cycle's CalcTimeConstraintsForElems result
        T.dtcourant = __longlong_as_double((long long)T.min_courant);
        T.dthydro = __longlong_as_double((long long)T.min_hydro);
    }
    T.min_courant = dbits(1.0e+20);
    T.min_hydro = dbits(1.0e+20);

    double targetdt = P.stoptime - T.time;
    if ((P.dtfixed <= 0.0) && (T.cycle != 0)) {
        double ratio;
        double gnewdt = 1.0e+20;
        double newdt;
        if (T.dtcourant < gnewdt) gnewdt = T.dtcourant / 2.0;
        if (T.dthydro < gnewdt) gnewdt = T.dthydro * 2.0 / 3.0;
        newdt = gnewdt;
        const double olddt = T.deltatime;
        ratio = newdt / olddt;
        if (ratio >= 1.0) {
            if (ratio < P.deltatimemultlb)
                newdt = olddt;
            else if (ratio > P.deltatimemultub)
                newdt = olddt * P.deltatimemultub;
        }
        if (newdt > P.dtmax) newdt = P.dtmax;
        T.deltatime = newdt;
    }
    // try to prevent very small scaling on the next cycle
    if ((targetdt > T.deltatime) && (targetdt < (4.0 * T.deltatime / 3.0)))
        targetdt = 2.0 * T.deltatime / 3.0;
    if (targetdt < T.deltatime) T.deltatime = targetdt;
    T.time += T.deltatime;
    ++T.cycle;
    T.active = 1;
}

// The time increment inside the cycle's own kernels (SetArgs::next), for sets
// small enough that a launch more is felt.  T, the job's time state, stands
// still while force and nodal run; N is scratch between cycles.
//   force       runs where the increment will find the job due; its errors go
//               to N, so that no block sees another's and stops
//   nodal       one extra warp a block makes the increment from T, for the
//               block's own use; the job's first block leaves it in N
//   kinematics  works from N; the job's first block copies N to T and adds
//               force's errors
//   EOS         as after a k_time_increment launch
// Measured on B200 in graphs of 4 cycles, us per cycle with a launch -> inside:
// -s 10 17.5 -> 16.7, -s 30 20.1 -> 18.6, 2x2x2 of -s 12 23.1 -> 21.6; the sizes
// around the lines up to which it is done: kInlineIncrementNodes, kernels.cuh.
__device__ __forceinline__ bool increment_due(const TimeCtl &T, const Params &P)
{
#if LULESH_CHECKED
    if (T.chk != 0) return false;
#endif
    return !T.done && T.bad_vol == INT_MAX && T.bad_q == INT_MAX && T.time < P.stoptime &&
           !(T.its_cap > 0 && T.cycle >= T.its_cap);
}

// what time_increment sets, from one record to the other
__device__ __forceinline__ void copy_increment(TimeCtl &to, const TimeCtl &from)
{
    to.time = from.time;
    to.deltatime = from.deltatime;
    to.dtcourant = from.dtcourant;
    to.dthydro = from.dthydro;
    to.min_courant = from.min_courant;
    to.min_hydro = from.min_hydro;
    to.cycle = from.cycle;
    to.active = from.active;
    to.done = from.done;
    to.status = from.status;
}

__device__ __forceinline__ void commit_increment(TimeCtl &T, TimeCtl &N)
{
    copy_increment(T, N);
    if (N.bad_vol != INT_MAX) {
        atomicMin(&T.bad_vol, N.bad_vol);
        N.bad_vol = INT_MAX;
    }
    if (N.chk != 0) {
        atomicCAS(&T.chk, 0, N.chk);
        N.chk = 0;
    }
}

// the block that speaks for its job: the first items of its first domain
__device__ __forceinline__ bool first_of_job(const DomDev &D, int first)
{
    return first == 0 && (D.col | D.row | D.plane) == 0;
}

__global__ void k_time_increment(TimeCtl *tcs, int ntc, Params P)
{
    pdl_enter();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < ntc) time_increment(tcs[i], P);
}

void launch_time_increment(TimeCtl *tcs, int ntc, Params P, cudaStream_t s, bool pdl)
{
    const int b = 128;
    launch_k(k_time_increment, (ntc + b - 1) / b, b, s, pdl, tcs, ntc, P);
}

// ---------------------------------------------------------------------------
// structured-mesh indexing helpers

// corner j of an element sits at lattice offset (CX[j], CY[j], CZ[j]) from
// the element's corner 0 (nodelist order of BuildMesh, lulesh.cu:730-737)
__device__ __constant__ int kCX[8] = {0, 1, 1, 0, 0, 1, 1, 0};
__device__ __constant__ int kCY[8] = {0, 0, 1, 1, 0, 0, 1, 1};
__device__ __constant__ int kCZ[8] = {0, 0, 0, 0, 1, 1, 1, 1};

// ---------------------------------------------------------------------------
// scattered meshes

// 32 bytes in one access (32-byte aligned); the volatile form keeps its place
// after griddepcontrol.wait
__device__ __forceinline__ void ld4(const double *p, double &a, double &b, double &c, double &d)
{
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
                 : "=d"(a), "=d"(b), "=d"(c), "=d"(d)
                 : "l"(p));
}

__device__ __forceinline__ void st4(double *p, double a, double b, double c, double d)
{
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(a), "d"(b), "d"(c),
                 "d"(d)
                 : "memory");
}

__device__ __forceinline__ void load_node(const DomDev &D, int n, double &x, double &y, double &z,
                                          double &xd, double &yd, double &zd)
{
    const double *p = D.nodePack + 8 * (size_t)n;
    ld4(p, x, y, z, xd);
    const double2 t = *reinterpret_cast<const double2 *>(p + 4);
    yd = t.x;
    zd = t.y;
}

__device__ __forceinline__ void store_node(const DomDev &D, int n, double x, double y, double z,
                                           double xd, double yd, double zd)
{
    double *p = D.nodePack + 8 * (size_t)n;
    st4(p, x, y, z, xd);
    *reinterpret_cast<double2 *>(p + 4) = make_double2(yd, zd);
}

// Start of a scattered mesh's cycle: the time increment, and every node's six
// values side by side.  The first cycle of a graph: what the caller wrote to the
// node arrays before it counts, and the node update keeps both forms from there.
__global__ void __launch_bounds__(kNodeBlock)
    k_begin_packed(const __grid_constant__ OneDomain w, Params P)
{
    pdl_enter();
    const DomDev &D = w.D[0];
    const int i = blockIdx.x * kNodeBlock + threadIdx.x;
    if (i == 0) time_increment(*w.tc, P);
    if (i < D.numNode) store_node(D, i, D.x[i], D.y[i], D.z[i], D.xd[i], D.yd[i], D.zd[i]);
}

void launch_begin_packed(const SetArgs &a, int nblocks, Params P, cudaStream_t s)
{
    launch_k(k_begin_packed, nblocks, kNodeBlock, s, a.pdl != 0, by_value<1>(a, nblocks), P);
}

// The fourth value of a corner's sector: kNewCorner where fx_elem, fy_elem and
// fz_elem do not have the corner force yet, else 0.
constexpr double kNewCorner = 1.0;

// An element's packed corner forces to the arrays that callers read
__device__ __forceinline__ void show_element(const DomDev &D, int e)
{
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        double *p = D.cornerPack + 4 * (8 * (size_t)e + k);
        double fx, fy, fz, state;
        ld4(p, fx, fy, fz, state);
        if (state != kNewCorner) continue;
        D.fx_elem[e + D.Ep * k] = fx;
        D.fy_elem[e + D.Ep * k] = fy;
        D.fz_elem[e + D.Ep * k] = fz;
        p[3] = 0.0;
    }
}

__global__ void __launch_bounds__(kElemBlock) k_show_corners(const __grid_constant__ OneDomain w)
{
    const int e = blockIdx.x * kElemBlock + threadIdx.x;
    if (e < w.D[0].numElem) show_element(w.D[0], e);
}

void launch_show_corners(const SetArgs &a, int nblocks, cudaStream_t s)
{
    launch_k(k_show_corners, nblocks, kElemBlock, s, /*pdl=*/false, by_value<1>(a, nblocks));
}

// ---------------------------------------------------------------------------
// force: CalcVolumeForceForElems_kernel, lulesh.cu:2080-2259

// One element of the force phase: the node gathers, then force_modal.
//
// Bound by the corner stores (192 B of the 290 B an element moves) and by
// FP64 issue, about evenly: 63 us at -s 100 (1.0e6 elements) on B200, where
// the stores and loads take 44 us at the measured copy rate and the 588
// operations 32 us at the FP64 peak (70 us with the records read from memory).
// The form that evaluated the reference's expressions corner by corner took
// 125 us (934 operations, 254 registers, 8 warps per SM).  All 48 gathers go out
// before any arithmetic: with the velocities gathered component by component,
// where force_modal asks for them, the kernel fits 128 registers (16 warps) but
// took 73 against 70 us, and 312 against 272 us at -s 160.
template <bool HG, Mesh M, bool TABLE, bool SHOW>
__device__ __forceinline__ void force_one(const DomDev &D, bool active, TimeCtl &E, const Params &P,
                                          int elem, int (&n)[8])
{
#pragma unroll
    for (int i = 0; i < 8; ++i) n[i] = chk_index(n[i], D.numNode, &E, kChkNode);
    double vn[3][8], xn[8], yn[8], zn[8];
    if constexpr (M == Mesh::kPacked) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
            load_node(D, n[i], xn[i], yn[i], zn[i], vn[0][i], vn[1][i], vn[2][i]);
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            if (HG) {
                vn[0][i] = D.xd[n[i]];
                vn[1][i] = D.yd[n[i]];
                vn[2][i] = D.zd[n[i]];
            } else {
                vn[0][i] = vn[1][i] = vn[2][i] = 0.0;
            }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) xn[i] = D.x[n[i]];
#pragma unroll
        for (int i = 0; i < 8; ++i) yn[i] = D.y[n[i]];
#pragma unroll
        for (int i = 0; i < 8; ++i) zn[i] = D.z[n[i]];
    }
    if (!TABLE && !active) {
        // the graph's last cycle with work was an earlier one
        if (SHOW) show_element(D, elem);
        return;
    }
    double fx[8], fy[8];  // held for cornerPack, whose corners take all three
    force_modal<HG>(
        xn, yn, zn, D.volo[elem], D.v[elem], D.p[elem], D.q[elem], D.ss[elem], D.elemMass[elem],
        P.hgcoef,
        [&](int c, double (&v)[8]) {
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = vn[c][i];
        },
        [&](int c, const double (&f)[8]) {
            if constexpr (M == Mesh::kPacked) {
                double *p = D.cornerPack + 32 * (size_t)elem;
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    if (c == 0) fx[k] = f[k];
                    if (c == 1) fy[k] = f[k];
                    if (c == 2) st4(p + 4 * k, fx[k], fy[k], f[k], SHOW ? 0.0 : kNewCorner);
                }
            }
            if (M != Mesh::kPacked || SHOW)
                CornerStore{D.fx_elem, D.fy_elem, D.fz_elem, elem, D.Ep}(c, f);
        },
        [&] { atomicMin(&E.bad_vol, elem); });
}

// SHOW (kPacked): the corner forces in both forms
template <bool HG, int BS, Mesh M, class W, bool SHOW = false>
__global__ void __launch_bounds__(BS, min_blocks(kForceMinBlocks, BS))
    k_force(const __grid_constant__ W w, Params P)
{
    // an lmesh cycle begins with another kernel: the node ids may come early
    if (M == Mesh::kBox) pdl_enter();
    const int2 blk = w.template block<BS, LULESH_FORCE_REVERSE>();
    const DomDev &D = w.domain(blk.x);
    const int elem = blk.y + threadIdx.x;
    int n[8];
    if (M != Mesh::kBox) {
        if (elem < D.numElem) elem_nodes<true>(D, elem, n);
        pdl_enter();
    }
    const TimeCtl &T = w.time(D);
    const bool active = w.increments() ? increment_due(T, P) : T.active != 0;
    if (W::kTable && !active) return;
    if (elem >= D.numElem) return;
    if (M == Mesh::kBox) elem_nodes<false>(D, elem, n);
    force_one<HG, M, W::kTable, SHOW>(D, active, w.next(D), P, elem, n);
}

template <int BS, Mesh M, bool SHOW = false, class W>
static void launch_force_w(const W &w, bool pdl, int nblocks, Params P, cudaStream_t s)
{
    if (P.hgcoef > 0.0)
        launch_k(k_force<true, BS, M, W, SHOW>, nblocks, BS, s, pdl, w, P);
    else
        launch_k(k_force<false, BS, M, W, SHOW>, nblocks, BS, s, pdl, w, P);
}

template <int BS>
static void launch_force_bs(const SetArgs &a, int nblocks, Params P, cudaStream_t s)
{
    launch_where<true, BS == kElemBlock>(a, nblocks, [&](const auto &w) {
        launch_force_w<BS, Mesh::kBox>(w, a.pdl != 0, nblocks, P, s);
    });
}

void launch_force(const SetArgs &a, int nblocks, Params P, cudaStream_t s, int bs, bool u)
{
    if (u) {  // an lmesh set is one domain
        const OneDomain w = by_value<1>(a, nblocks);
        if (w.D[0].nodePack && a.show)
            launch_force_w<kElemBlock, Mesh::kPacked, true>(w, a.pdl != 0, nblocks, P, s);
        else if (w.D[0].nodePack)
            launch_force_w<kElemBlock, Mesh::kPacked>(w, a.pdl != 0, nblocks, P, s);
        else
            launch_force_w<kElemBlock, Mesh::kLists>(w, a.pdl != 0, nblocks, P, s);
        return;
    }
    switch (bs) {
        case 64: launch_force_bs<64>(a, nblocks, P, s); break;
        case 256: launch_force_bs<256>(a, nblocks, P, s); break;
        default: launch_force_bs<kElemBlock>(a, nblocks, P, s); break;
    }
}

// ---------------------------------------------------------------------------
// nodal: corner gather (in nodeElemCornerList order) + node update

// Sum the corner forces around node (px,py,pz) of domain D in corner order
// j = 0..7, the order nodeElemCornerList has on a structured mesh
// (lulesh.cu:1082-1091).  A corner whose element lies in a neighbouring
// subdomain is read from that subdomain's corner array: the result equals
// the undecomposed mesh's sum bit for bit.
// NEIGHBOURS false: this domain's own corners only.
template <bool NEIGHBOURS>
__device__ __forceinline__ void gather_corners(const DomDev *doms, const DomDev &D, int px,
                                               int py, int pz, double &fx, double &fy,
                                               double &fz, TimeCtl *T)
{
    const int nx = D.nx;
    fx = fy = fz = 0.0;
    if (NEIGHBOURS && D.tp > 1) {
        // subdomains: the source domain of each corner first (this one or
        // a neighbour), then one load path that the warp shares
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int ex = px - kCX[j], ey = py - kCY[j], ez = pz - kCZ[j];
            const int sx = (ex < 0) ? -1 : (ex >= nx ? 1 : 0);
            const int sy = (ey < 0) ? -1 : (ey >= nx ? 1 : 0);
            const int sz = (ez < 0) ? -1 : (ez >= nx ? 1 : 0);
            const DomDev *S = &D;
            bool use = (sx | sy | sz) == 0;
            if (!use) {
                const int nb = D.nbr[(sx + 1) + 3 * (sy + 1) + 9 * (sz + 1)];
                if (nb >= 0) {
                    S = &doms[nb];
                    use = true;
                }
            }
            if (use) {
                const int lx = ex - sx * nx, ly = ey - sy * nx, lz = ez - sz * nx;
                const int idx = chk_index(j * S->Ep + (lz * nx + ly) * nx + lx, 8LL * S->Ep, T,
                                          kChkCorner);
                fx += ld_corner(S->fx_elem + idx);
                fy += ld_corner(S->fy_elem + idx);
                fz += ld_corner(S->fz_elem + idx);
            }
        }
        return;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int ex = px - kCX[j], ey = py - kCY[j], ez = pz - kCZ[j];
        const bool inside = (unsigned)ex < (unsigned)nx && (unsigned)ey < (unsigned)nx &&
                            (unsigned)ez < (unsigned)nx;
        if (inside) {
            const int idx = chk_index(j * D.Ep + (ez * nx + ey) * nx + ex, 8LL * D.Ep, T,
                                      kChkCorner);
            fx += ld_corner(D.fx_elem + idx);
            fy += ld_corner(D.fy_elem + idx);
            fz += ld_corner(D.fz_elem + idx);
        }
    }
}

// Node i's state where the update reads it
struct NodeNow {
    const DomDev &D;
    int i;
    __device__ __forceinline__ double mass() const { return D.nodalMass[i]; }
    __device__ __forceinline__ double x() const { return D.x[i]; }
    __device__ __forceinline__ double y() const { return D.y[i]; }
    __device__ __forceinline__ double z() const { return D.z[i]; }
    __device__ __forceinline__ double xd() const { return D.xd[i]; }
    __device__ __forceinline__ double yd() const { return D.yd[i]; }
    __device__ __forceinline__ double zd() const { return D.zd[i]; }
};

// or before pdl_enter
struct NodeEarly {
    double vm, vx, vy, vz, vxd, vyd, vzd;
    __device__ __forceinline__ void read(const DomDev &D, int i)
    {
        vm = __ldcg(D.nodalMass + i);
        vxd = __ldcg(D.xd + i), vyd = __ldcg(D.yd + i), vzd = __ldcg(D.zd + i);
        vx = __ldcg(D.x + i), vy = __ldcg(D.y + i), vz = __ldcg(D.z + i);
    }
    __device__ __forceinline__ double mass() const { return vm; }
    __device__ __forceinline__ double x() const { return vx; }
    __device__ __forceinline__ double y() const { return vy; }
    __device__ __forceinline__ double z() const { return vz; }
    __device__ __forceinline__ double xd() const { return vxd; }
    __device__ __forceinline__ double yd() const { return vyd; }
    __device__ __forceinline__ double zd() const { return vzd; }
};

// The same for the 2x2x2 subdomains of a problem: their corner arrays lie at
// equal distances (even_records, set.hpp), so a corner's place follows from its
// position in the whole mesh, without its owner's record.  For sets of one wave,
// where the records are links of the chain: 2x2x2 of -s 12 22.6 -> 20.5 us per
// cycle on B200; past it the gather waits for its sectors either way, and the
// lookups need fewer registers (-s 50 197.9 against 198.9, -s 70 541 against 545).
__device__ __forceinline__ void gather_corners_few(const FewDomains &w, const DomDev &D, int px,
                                                   int py, int pz, double &fx, double &fy,
                                                   double &fz, TimeCtl *T)
{
    const DomDev &D0 = w.D[0];
    const int nx = D0.nx;
    // along each axis: the element before and after the node, its place in its
    // subdomain's row, and that subdomain's part of the distance
    const int at[3] = {D.col * nx + px, D.row * nx + py, D.plane * nx + pz};
    int local[3][2], owner[3][2];
    bool in[3][2];
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const int e = at[a] - c;
            in[a][c] = (unsigned)e < (unsigned)(2 * nx);
            owner[a][c] = e >= nx ? 1 : 0;
            local[a][c] = e - owner[a][c] * nx;
        }
    fx = fy = fz = 0.0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int cx = (j & 1) ^ ((j >> 1) & 1), cy = (j >> 1) & 1, cz = j >> 2;  // kCX, kCY, kCZ
        if (in[0][cx] && in[1][cy] && in[2][cz]) {
            const int d = owner[0][cx] + 2 * owner[1][cy] + 4 * owner[2][cz];
            const int idx = chk_index(j * D0.Ep + (local[2][cz] * nx + local[1][cy]) * nx +
                                          local[0][cx],
                                      8LL * D0.Ep, T, kChkCorner);
            const long long off = d * w.stride + idx;
            fx += ld_corner(D0.fx_elem + off);
            fy += ld_corner(D0.fy_elem + off);
            fz += ld_corner(D0.fz_elem + off);
        }
    }
}

// CalcAccelerationForNodes (lulesh.cu:2926-2939), the symmetry-plane zeroing
// of ApplyAccelerationBoundaryConditionsForNodes (bc bits 0/1/2 zero the
// x/y/z acceleration) and CalcPositionAndVelocityForNodes (lulesh.cu:
// 2999-3028) for node i with the summed force (fx, fy, fz)
template <class Node>
__device__ __forceinline__ void advance_node(const DomDev &D, double dt, const Params &P, int i,
                                             int bc, double fx, double fy, double fz,
                                             int materialize, bool write_f, const Node &n,
                                             bool pack = false)
{
    const double one_over_nMass = 1. / n.mass();
    double xdd = fx * one_over_nMass;
    double ydd = fy * one_over_nMass;
    double zdd = fz * one_over_nMass;
    if (bc & 1) xdd = 0.0;
    if (bc & 2) ydd = 0.0;
    if (bc & 4) zdd = 0.0;

    const double u_cut = P.u_cut;
    double xdtmp = n.xd() + xdd * dt;
    double ydtmp = n.yd() + ydd * dt;
    double zdtmp = n.zd() + zdd * dt;
    if (fabs(xdtmp) < u_cut) xdtmp = 0.0;
    if (fabs(ydtmp) < u_cut) ydtmp = 0.0;
    if (fabs(zdtmp) < u_cut) zdtmp = 0.0;
    const double x = n.x() + xdtmp * dt;
    const double y = n.y() + ydtmp * dt;
    const double z = n.z() + zdtmp * dt;
    D.x[i] = x;
    D.y[i] = y;
    D.z[i] = z;
    D.xd[i] = xdtmp;
    D.yd[i] = ydtmp;
    D.zd[i] = zdtmp;
    if (pack) store_node(D, i, x, y, z, xdtmp, ydtmp, zdtmp);
    if (materialize) {
        if (write_f) {
            D.fx[i] = fx;
            D.fy[i] = fy;
            D.fz[i] = fz;
        }
        D.xdd[i] = xdd;
        D.ydd[i] = ydd;
        D.zdd[i] = zdd;
    }
}

// MODE 0: gather every corner (neighbour subdomains included) and update
//         the node: the fused form of the SBN exchange + node update.
// MODE 1: AddNodeForcesFromElems over this domain's own corners only,
//         writing fx/fy/fz (the partial sums the reference exchanges).
// MODE 2: the node update from fx/fy/fz (after CommSBN added neighbours).
// INCR (MODE 0): a warp more than BS threads makes the time increment while
// the others gather.
template <int MODE, int BS, class W, bool INCR = false>
__global__ void __launch_bounds__(INCR ? BS + 32 : BS,
                                  min_blocks(INCR ? kNodalIncrMinBlocks
                                             : std::is_same_v<W, FewDomains>
                                                 ? kNodalFewMinBlocks
                                                 : kNodalMinBlocks,
                                             BS))
    k_nodal(const __grid_constant__ W w, Params P)
{
    if (!INCR) pdl_enter();
    const int2 blk = w.template block<BS, LULESH_NODAL_REVERSE && !W::kTable>();
    const DomDev &D = w.domain(blk.x);
    TimeCtl &T = w.time(D);
    const int i = blk.y + threadIdx.x;
    if constexpr (INCR) {
        NodeEarly node;
        if (!W::kTable && threadIdx.x < BS && i < D.numNode) node.read(D, i);
        pdl_enter();
        __shared__ double s_dt;
        __shared__ int s_active;
        const bool speaks = first_of_job(D, blk.y);
        if (W::kTable && !speaks && !increment_due(T, P)) return;
        const bool mine = threadIdx.x < BS && i < D.numNode;
        int px, py, pz;
        lattice(D.by_en, i, px, py, pz);
        double fx, fy, fz;
        if (threadIdx.x >= BS) {
            TimeCtl n = T;
            time_increment(n, P);
            if (threadIdx.x == BS) {
                s_dt = n.deltatime;
                s_active = n.active;
                if (speaks) copy_increment(w.next(D), n);
            }
        } else if (mine) {
            if constexpr (std::is_same_v<W, FewDomains>)
                gather_corners_few(w, D, px, py, pz, fx, fy, fz, &w.next(D));
            else
                gather_corners<!std::is_same_v<W, OneDomain>>(w.doms(), D, px, py, pz, fx, fy, fz,
                                                              &w.next(D));
        }
        __syncthreads();
        if (!mine || !s_active) return;
        if (W::kTable) node.read(D, i);
        const int bc = (D.col == 0 && px == 0 ? 1 : 0) | (D.row == 0 && py == 0 ? 2 : 0) |
                       (D.plane == 0 && pz == 0 ? 4 : 0);
        advance_node(D, s_dt, P, i, bc, fx, fy, fz, w.materialize(), true, node);
        return;
    }
    if (W::kTable && !T.active) return;
    if (i >= D.numNode) return;
    int px, py, pz;
    lattice(D.by_en, i, px, py, pz);

    double fx, fy, fz;
    if (MODE == 0) {
        gather_corners<!std::is_same_v<W, OneDomain>>(w.doms(), D, px, py, pz, fx, fy, fz, &T);
    } else if (MODE == 1) {
        gather_corners<false>(w.doms(), D, px, py, pz, fx, fy, fz, &T);  // own corners only
        D.fx[i] = fx;
        D.fy[i] = fy;
        D.fz[i] = fz;
        return;
    } else {
        fx = D.fx[i];
        fy = D.fy[i];
        fz = D.fz[i];
    }

    // ApplyAccelerationBoundaryConditionsForNodes: symmetry planes are the
    // px/py/pz == 0 node sets of the domains at the mesh origin faces
    const int bc = (D.col == 0 && px == 0 ? 1 : 0) | (D.row == 0 && py == 0 ? 2 : 0) |
                   (D.plane == 0 && pz == 0 ? 4 : 0);
    if (!W::kTable && !T.active) return;
    advance_node(D, T.deltatime, P, i, bc, fx, fy, fz, w.materialize(), MODE == 0,
                 NodeNow{D, i});
}

// Scattered meshes: the corner forces of a node, one sector each, summed in
// run order, then the node update.
__global__ void __launch_bounds__(kNodeBlock)
    k_nodal_packed(const __grid_constant__ OneDomain w, Params P)
{
    const DomDev &D = w.D[0];
    TimeCtl &T = *w.tc;
    const int i = blockIdx.x * kNodeBlock + threadIdx.x;
    int k[8], bc = 0;
    NodeEarly node;
    if (i < D.numNode) {
#pragma unroll
        for (int j = 0; j < 8; ++j) k[j] = D.packedCornerEll[(size_t)j * D.numNode + i];
        bc = D.nodeBC[i];
        node.read(D, i);
    }
    pdl_enter();
    if (i >= D.numNode) return;
    double vx[8], vy[8], vz[8], pad;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        vx[j] = vy[j] = vz[j] = 0.0;
        if (k[j] >= 0)
            ld4(D.cornerPack + 4 * (size_t)chk_index(k[j], 8LL * D.Ep, &T, kChkCorner), vx[j],
                vy[j], vz[j], pad);
    }
    if (!T.active) return;
    double fx = 0.0, fy = 0.0, fz = 0.0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        if (k[j] >= 0) {  // a run is a prefix of the slots
            fx += vx[j];
            fy += vy[j];
            fz += vz[j];
        }
    }
    advance_node(D, T.deltatime, P, i, bc, fx, fy, fz, w.mat, true, node, /*pack=*/true);
}

// Unstructured meshes: AddNodeForcesFromElems (lulesh.cu:1715-1751) over
// each node's run of nodeElemCornerList, in list order, then the node
// update.  The runs of a block's consecutive nodes are contiguous in the
// list; when they fit, the block stages them in shared memory with
// coalesced loads (read straight from the list, each thread's run is an
// 8-int stride: one sector per thread per load), and the corner loads go
// out four corners at a time.
template <int BS>
__global__ void __launch_bounds__(BS, min_blocks(kNodalUMinBlocks, BS))
    k_nodal_u(const __grid_constant__ OneDomain w, Params P)
{
    __shared__ int s_list[8 * BS];
    const int2 blk = w.template block<BS, LULESH_NODAL_REVERSE>();
    const DomDev &D = w.D[0];
    const TimeCtl &T = *w.tc;
    const int first = blk.y;
    const int last = min(first + BS, D.numNode) - 1;
    int slot[8];
    if (D.nodeCornerEll && first + (int)threadIdx.x <= last) {
#pragma unroll
        for (int j = 0; j < 8; ++j)
            slot[j] = D.nodeCornerEll[(size_t)j * D.numNode + first + threadIdx.x];
    }
    pdl_enter();
    if (!T.active) return;  // the whole block
    if (D.nodeCornerEll) {
        // the run slot-major (uniform per block: no staging, no barrier):
        // eight coalesced loads, then the corners, summed in run order
        const int i = first + threadIdx.x;
        if (i > last) return;
        const int(&k)[8] = slot;
        double fx = 0.0, fy = 0.0, fz = 0.0;
#pragma unroll
        for (int h = 0; h < 8; h += 4) {
            double vx[4], vy[4], vz[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                vx[q] = vy[q] = vz[q] = 0.0;
                if (k[h + q] >= 0) {
                    const int c = chk_index(k[h + q], 8LL * D.Ep, const_cast<TimeCtl *>(&T),
                                            kChkCorner);
                    vx[q] = ld_corner(D.fx_elem + c);
                    vy[q] = ld_corner(D.fy_elem + c);
                    vz[q] = ld_corner(D.fz_elem + c);
                }
            }
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (k[h + q] >= 0) {  // a run is a prefix of the slots
                    fx += vx[q];
                    fy += vy[q];
                    fz += vz[q];
                }
        }
        advance_node(D, T.deltatime, P, i, D.nodeBC[i], fx, fy, fz, w.mat, true, NodeNow{D, i});
        return;
    }
    const long long list_len = 8LL * D.numElem;  // corner-list entries
    const int lo = chk_index(D.nodeElemStart[first], list_len, const_cast<TimeCtl *>(&T),
                             kChkCornerRun);
    const int len = D.nodeElemStart[last] + D.nodeElemCount[last] - lo;
    const bool staged = len <= 8 * BS && lo + (long long)len <= list_len;
    if (staged)
        for (int k = threadIdx.x; k < len; k += BS) s_list[k] = D.nodeElemCornerList[lo + k];
    __syncthreads();
    const int i = first + threadIdx.x;
    if (i > last) return;
    int start = D.nodeElemStart[i], count = D.nodeElemCount[i];
#if LULESH_CHECKED
    if (start < 0 || count < 0 || start + (long long)count > list_len ||
        (staged && (start < lo || start + count > lo + len))) {
        atomicCAS(&const_cast<TimeCtl &>(T).chk, 0, (int)kChkCornerRun);
        start = lo;
        count = 0;
    }
#endif
    const int *list = staged ? s_list + (start - lo) : D.nodeElemCornerList + start;

    double fx = 0.0, fy = 0.0, fz = 0.0;
    int j = 0;
    for (; j + 4 <= count; j += 4) {
        int k[4];
        double vx[4], vy[4], vz[4];
#pragma unroll
        for (int q = 0; q < 4; ++q)
            k[q] = chk_index(list[j + q], 8LL * D.Ep, const_cast<TimeCtl *>(&T), kChkCorner);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            vx[q] = ld_corner(D.fx_elem + k[q]);
            vy[q] = ld_corner(D.fy_elem + k[q]);
            vz[q] = ld_corner(D.fz_elem + k[q]);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            fx += vx[q];
            fy += vy[q];
            fz += vz[q];
        }
    }
    for (; j < count; ++j) {
        const int k = chk_index(list[j], 8LL * D.Ep, const_cast<TimeCtl *>(&T), kChkCorner);
        fx += ld_corner(D.fx_elem + k);
        fy += ld_corner(D.fy_elem + k);
        fz += ld_corner(D.fz_elem + k);
    }
    // symmetry nodes of the mesh's X/Y/Z sets: nodeBC bits 0/1/2
    advance_node(D, T.deltatime, P, i, D.nodeBC[i], fx, fy, fz, w.mat, true, NodeNow{D, i});
}

template <int BS>
static void launch_nodal_bs(const SetArgs &a, int nblocks, Params P, cudaStream_t s)
{
    launch_where<true, BS == kNodeBlock>(a, nblocks, [&](const auto &w) {
        using W = std::decay_t<decltype(w)>;
        if (a.next)
            launch_k(k_nodal<0, BS, W, true>, nblocks, BS + 32, s, a.pdl != 0, w, P);
        else
            launch_k(k_nodal<0, BS, W>, nblocks, BS, s, a.pdl != 0, w, P);
    });
}

void launch_nodal(const SetArgs &a, int nblocks, Params P, cudaStream_t s, int bs, bool u)
{
    if (u) {
        const OneDomain w = by_value<1>(a, nblocks);
        launch_k(w.D[0].nodePack ? k_nodal_packed : k_nodal_u<kNodeBlock>, nblocks, kNodeBlock, s,
                 a.pdl != 0, w, P);
        return;
    }
    switch (bs) {
        case 256: launch_nodal_bs<256>(a, nblocks, P, s); break;
        case 512: launch_nodal_bs<512>(a, nblocks, P, s); break;
        default: launch_nodal_bs<kNodeBlock>(a, nblocks, P, s); break;
    }
}

void launch_nodal_gather_local(const SetArgs &a, int nblocks, cudaStream_t s)
{
    k_nodal<1, kNodeBlock, ManyDomains><<<nblocks, kNodeBlock, 0, s>>>(ManyDomains{a}, Params{});
}

void launch_nodal_update(const SetArgs &a, int nblocks, Params P, cudaStream_t s)
{
    k_nodal<2, kNodeBlock, ManyDomains><<<nblocks, kNodeBlock, 0, s>>>(ManyDomains{a}, P);
}

// ---------------------------------------------------------------------------
// kinematics: CalcKinematicsAndMonotonicQGradient_kernel, lulesh.cu:3343-3507

// Bound by latency and FP64 issue at 20 warps per SM: 43 us at -s 100
// (1.0e6 elements) on B200, against 22 us for its 144 B per element at the
// measured copy rate and 20 us for its 367 operations (51.6 us with the
// records read from memory); 80 us with the reference's corner-by-corner
// expressions (649 operations, 168 registers).
// The velocities are gathered where kin_modal asks for them, after the volume
// and length stores, at 96 registers (5 blocks); 6 us more at 4 blocks.  Up
// front took 8 us more at 3 blocks, and between the coordinates and the volume
// 2 us more at 4 blocks and 4 at 5 (with spills).
template <int BS, Mesh M, class W>
__global__ void __launch_bounds__(BS, min_blocks(M == Mesh::kPacked ? kKinPackedMinBlocks
                                                                    : kKinMinBlocks, BS))
    k_kinematics(const __grid_constant__ W w)
{
    const int2 blk = w.template block<BS, LULESH_KIN_REVERSE>();
    const DomDev &D = w.domain(blk.x);
    TimeCtl &T = w.time(D), &N = w.next(D);
    int n[8];
    if (M != Mesh::kBox && blk.y + (int)threadIdx.x < D.numElem)
        elem_nodes<true>(D, blk.y + threadIdx.x, n);
    pdl_enter();
    if (w.increments() && threadIdx.x == 0 && first_of_job(D, blk.y)) commit_increment(T, N);
    if (W::kTable && !N.active) return;
    const int k = blk.y + threadIdx.x;
    if (k >= D.numElem) return;

    if (M == Mesh::kBox) elem_nodes<false>(D, k, n);
#pragma unroll
    for (int l = 0; l < 8; ++l) n[l] = chk_index(n[l], D.numNode, &T, kChkNode);
    double xn[8], yn[8], zn[8];
    if constexpr (M == Mesh::kPacked) {
        double vn[3][8];
#pragma unroll
        for (int l = 0; l < 8; ++l)
            load_node(D, n[l], xn[l], yn[l], zn[l], vn[0][l], vn[1][l], vn[2][l]);
        if (!W::kTable && !N.active) return;
        kin_modal(D, T, N.deltatime, k, xn, yn, zn, [&](int c, double (&v)[8]) {
#pragma unroll
            for (int l = 0; l < 8; ++l) v[l] = vn[c][l];
        });
        return;
    } else {
#pragma unroll
        for (int l = 0; l < 8; ++l) xn[l] = D.x[n[l]];
#pragma unroll
        for (int l = 0; l < 8; ++l) yn[l] = D.y[n[l]];
#pragma unroll
        for (int l = 0; l < 8; ++l) zn[l] = D.z[n[l]];
        if (!W::kTable && !N.active) return;
        kin_modal(D, T, N.deltatime, k, xn, yn, zn, [&](int c, double (&v)[8]) {
            const double *a = c == 0 ? D.xd : c == 1 ? D.yd : D.zd;
#pragma unroll
            for (int l = 0; l < 8; ++l) v[l] = a[n[l]];
        });
    }
}

template <int BS>
static void launch_kinematics_bs(const SetArgs &a, int nblocks, cudaStream_t s)
{
    launch_where<true, BS == kElemBlock>(a, nblocks, [&](const auto &w) {
        launch_k(k_kinematics<BS, Mesh::kBox, std::decay_t<decltype(w)>>, nblocks, BS, s, a.pdl != 0,
                 w);
    });
}

void launch_kinematics(const SetArgs &a, int nblocks, Params P, cudaStream_t s, int bs, bool u)
{
    (void)P;
    if (u) {
        const OneDomain w = by_value<1>(a, nblocks);
        launch_k(w.D[0].nodePack ? k_kinematics<kElemBlock, Mesh::kPacked, OneDomain>
                                 : k_kinematics<kElemBlock, Mesh::kLists, OneDomain>,
                 nblocks, kElemBlock, s, a.pdl != 0, w);
        return;
    }
    switch (bs) {
        case 64: launch_kinematics_bs<64>(a, nblocks, s); break;
        case 256: launch_kinematics_bs<256>(a, nblocks, s); break;
        default: launch_kinematics_bs<kElemBlock>(a, nblocks, s); break;
    }
}

// ---------------------------------------------------------------------------
// eos: monotonic Q region + EOS + volume update + dt constraints

// Boundary-condition mask and the six face-neighbour indices of element z,
// computed from its position: the values SetupConnectivityBC stores in
// elemBC and lxim..lzetap (lulesh.cu:537-686).  Interior neighbours are the
// adjacent elements; a face on the mesh boundary is a symmetry plane at the
// minimum and a free surface at the maximum; a face against another
// subdomain is a comm face whose neighbour is a ghost element (ghost face
// offsets in the order planeMin, planeMax, rowMin, rowMax, colMin, colMax).
// Indices the limiter does not read for a given mask are left as is.
__device__ __forceinline__ void elem_face_links(const DomDev &D, int z, int &bc, int &xm,
                                                int &xp, int &em, int &ep, int &zm, int &zp)
{
    const int nx = D.nx, nn = nx * nx;
    int ix, iy, iz;
    lattice(D.by_nx, z, ix, iy, iz);
    bc = 0;
    xm = z - 1;
    xp = z + 1;
    em = z - nx;
    ep = z + nx;
    zm = z - nn;
    zp = z + nn;
    const int last = D.tp - 1;
    if (iz == 0) {
        if (D.plane == 0) bc |= ZETA_M_SYMM;
        else { bc |= ZETA_M_COMM; zm = D.ghost[0] + iy * nx + ix; }
    }
    if (iz == nx - 1) {
        if (D.plane == last) bc |= ZETA_P_FREE;
        else { bc |= ZETA_P_COMM; zp = D.ghost[1] + iy * nx + ix; }
    }
    if (iy == 0) {
        if (D.row == 0) bc |= ETA_M_SYMM;
        else { bc |= ETA_M_COMM; em = D.ghost[2] + iz * nx + ix; }
    }
    if (iy == nx - 1) {
        if (D.row == last) bc |= ETA_P_FREE;
        else { bc |= ETA_P_COMM; ep = D.ghost[3] + iz * nx + ix; }
    }
    if (ix == 0) {
        if (D.col == 0) bc |= XI_M_SYMM;
        else { bc |= XI_M_COMM; xm = D.ghost[4] + iz * nx + iy; }
    }
    if (ix == nx - 1) {
        if (D.col == last) bc |= XI_P_FREE;
        else { bc |= XI_P_COMM; xp = D.ghost[5] + iz * nx + iy; }
    }
}

// One direction of the monotonic limiter, lulesh.cu:3595-3624, from the
// element's gradient d and those of its minus and plus neighbours (the
// element's own at a symmetry plane, 0 at a free surface).
__device__ __forceinline__ double mono_limiter(double d, double delvm, double delvp, double mult,
                                               double maxslope)
{
    const double ptiny = 1.e-36;
    const double norm = 1. / (d + ptiny);
    delvm = delvm * norm;
    delvp = delvp * norm;
    double phi = .5 * (delvm + delvp);
    delvm *= mult;
    delvp *= mult;
    if (delvm < phi) phi = delvm;
    if (delvp < phi) phi = delvp;
    if (phi < 0.) phi = 0.;
    if (phi > maxslope) phi = maxslope;
    return phi;
}

// CalcPressureForElems_device, lulesh.cu:3764-3791
__device__ __forceinline__ void calc_pressure(double &p_new, double &bvc, double &pbvc,
                                              double &e_old, double &compression,
                                              double &vnewc, double pmin, double p_cut,
                                              double eosvmax)
{
    const double c1s = 2.0 / 3.0;
    double p_temp;
    bvc = c1s * (compression + 1.);
    pbvc = c1s;
    p_temp = bvc * e_old;
    if (fabs(p_temp) < p_cut) p_temp = 0.0;
    if (vnewc >= eosvmax) p_temp = 0.0;
    if (p_temp < pmin) p_temp = pmin;
    p_new = p_temp;
}

// x / rho0 (the reference density).  With RHO1 the density is 1.0, and
// x / 1.0 is x exactly in IEEE-754 arithmetic, so the division is left
// out; the results are the same bits either way.
template <bool RHO1>
__device__ __forceinline__ double per_rho0(double x, double rho0)
{
    return RHO1 ? x : x / rho0;
}

// CalcEnergyForElems_device, lulesh.cu:3867-3974
template <bool RHO1>
__device__ __forceinline__ void calc_energy(double &p_new, double &e_new, double &q_new,
                                            double &bvc, double &pbvc, double &p_old,
                                            double &e_old, double &q_old, double &compression,
                                            double &compHalfStep, double &vnewc, double &work,
                                            double &delvc, double pmin, double p_cut,
                                            double e_cut, double q_cut, double emin,
                                            double &qq, double &ql, double &rho0,
                                            double &eosvmax)
{
    const double sixth = 1.0 / 6.0;
    double pHalfStep;
    e_new = e_old - 0.5 * delvc * (p_old + q_old) + 0.5 * work;
    if (e_new < emin) e_new = emin;
    calc_pressure(pHalfStep, bvc, pbvc, e_new, compHalfStep, vnewc, pmin, p_cut, eosvmax);
    const double vhalf = 1. / (1. + compHalfStep);
    if (delvc > 0.) {
        q_new = 0.;
    } else {
        double ssc = per_rho0<RHO1>(pbvc * e_new + vhalf * vhalf * bvc * pHalfStep, rho0);
        if (ssc <= .1111111e-36)
            ssc = .3333333e-18;
        else
            ssc = sqrt(ssc);
        q_new = (ssc * ql + qq);
    }
    e_new = e_new + 0.5 * delvc * (3.0 * (p_old + q_old) - 4.0 * (pHalfStep + q_new));
    e_new += 0.5 * work;
    if (fabs(e_new) < e_cut) e_new = 0.;
    if (e_new < emin) e_new = emin;
    calc_pressure(p_new, bvc, pbvc, e_new, compression, vnewc, pmin, p_cut, eosvmax);
    double q_tilde;
    if (delvc > 0.) {
        q_tilde = 0.;
    } else {
        double ssc = per_rho0<RHO1>(pbvc * e_new + vnewc * vnewc * bvc * p_new, rho0);
        if (ssc <= .1111111e-36)
            ssc = .3333333e-18;
        else
            ssc = sqrt(ssc);
        q_tilde = (ssc * ql + qq);
    }
    e_new = e_new - (7.0 * (p_old + q_old) - 8.0 * (pHalfStep + q_new) + (p_new + q_tilde)) *
                        delvc * sixth;
    if (fabs(e_new) < e_cut) e_new = 0.;
    if (e_new < emin) e_new = emin;
    calc_pressure(p_new, bvc, pbvc, e_new, compression, vnewc, pmin, p_cut, eosvmax);
    if (delvc <= 0.) {
        double ssc = per_rho0<RHO1>(pbvc * e_new + vnewc * vnewc * bvc * p_new, rho0);
        if (ssc <= .1111111e-36)
            ssc = .3333333e-18;
        else
            ssc = sqrt(ssc);
        q_new = (ssc * ql + qq);
        if (fabs(q_new) < q_cut) q_new = 0.;
    }
}

// The rep loop of ApplyMaterialPropertiesAndUpdateVolume_kernel
// (lulesh.cu:4045-4083), the reference's cost model: every rep re-evaluates
// the EOS from the same inputs (the loop is pure).
template <bool RHO1>
__device__ __forceinline__ void eos_reps(int rep, double e_temp, double p_temp, double q_temp,
                                         double qq_temp, double ql_temp, double delvc_temp,
                                         double vnewc, double eosvmin, double eosvmax,
                                         double rho0, const Params &P, double &p_new,
                                         double &e_new, double &q_new, double &bvc,
                                         double &pbvc)
{
    double e_old, delvc, p_old, q_old, compression, compHalfStep, qq_old, ql_old, work;
    for (int r = 0; r < rep; r++) {
        e_old = e_temp;
        p_old = p_temp;
        q_old = q_temp;
        qq_old = qq_temp;
        ql_old = ql_temp;
        delvc = delvc_temp;
        work = 0.;
        double vchalf;
        compression = 1. / vnewc - 1.;
        vchalf = vnewc - delvc * .5;
        compHalfStep = 1. / vchalf - 1.;
        if (eosvmin != 0.) {
            if (vnewc <= eosvmin) compHalfStep = compression;
        }
        if (eosvmax != 0.) {
            if (vnewc >= eosvmax) {
                p_old = 0.;
                compression = 0.;
                compHalfStep = 0.;
            }
        }
        calc_energy<RHO1>(p_new, e_new, q_new, bvc, pbvc, p_old, e_old, q_old, compression,
                          compHalfStep, vnewc, work, delvc, P.pmin, P.p_cut, P.e_cut, P.q_cut,
                          P.emin, qq_old, ql_old, rho0, eosvmax);
    }
}

__device__ __forceinline__ double warp_max(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

__device__ __forceinline__ double warp_min(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Block b's turn among a domain's EOS blocks.  The slots are grouped by rep
// class, the costliest first; walked in that order, the first third of the
// kernel computes and the rest waits for memory.  One block in kEosMix is
// therefore a costly one until those run out (a permutation of the blocks; the
// blocks' own order where the costly class is more than 1/kEosMix of them).
// EOS on B200, us, class order -> 2, 3, 4 of a kind: -s 100 55.9 -> 52.1 (3 and
// 4), -s 133 with 20 regions and cost 4 135.8 -> 127.4 (3), 129.4 (4).
constexpr int kEosMix = 3;
template <int BS>
__device__ __forceinline__ int eos_block(const DomDev &D, int b)
{
    const int heavy = D.eosClassEnd[0] / BS;
    if (heavy * kEosMix > (D.numElem + BS - 1) / BS || b >= heavy * kEosMix) return b;
    return b % kEosMix == 0 ? b / kEosMix : heavy + b - b / kEosMix - 1;
}

// Lanes that share the reps of an element of a domain's costliest class: a
// power of two, at most kRepLanes and the class's reps, while the kernel stays
// one wave of blocks; 1 otherwise.  In one wave the costliest class's reps, 20
// by default, are the kernel's longest chain while lanes stand idle.  Every rep
// is still evaluated: lane k has reps k, k + lanes, ..., and the lane of the
// last one writes.  Cycle on B200, us, 1 -> 4, 8, 16 lanes: -s 10 15.6 -> 14.6,
// 14.6, 14.6; -s 20 16.9 -> 16.0, 16.0, 16.2; -s 30 17.7 -> 16.7, 18.7, 18.7;
// -s 45 26.1 -> 25.3 (all); with cost 3 18.1 -> 15.5, 18.1 -> 15.1, 20.3 ->
// 17.7, 28.3 -> 25.3 (4 lanes).  Past one wave the class's warps run beside the
// others', and its loads would be made by more of them.
#ifndef LULESH_REP_LANES
#define LULESH_REP_LANES 4
#endif
constexpr int kRepLanes = LULESH_REP_LANES;

// blocks of the costliest class with its reps shared, and of the other slots
__host__ __device__ __forceinline__ int shared_blocks(const DomDev &D, int lanes, int bs)
{
    return (int)(((long long)D.eosClassEnd[0] * lanes + bs - 1) / bs);
}
__host__ __device__ __forceinline__ int other_blocks(const DomDev &D, int bs)
{
    return (D.numElem - D.eosClassEnd[0] + bs - 1) / bs;
}

static int rep_lanes(const DomDev &D, int bs)
{
    const int wave = 148 * min_blocks(kEosMinBlocks, bs);
    int lanes = kRepLanes;
    while (lanes > 1 && (lanes > D.eosClassRep[0] ||
                         shared_blocks(D, lanes, bs) + other_blocks(D, bs) > wave))
        lanes /= 2;
    return lanes;
}

// A thread's place in the EOS kernel: its slot, the reps it evaluates, and
// whether it writes the element's results (the thread that has the last rep).
struct EosPlace {
    int slot, rep;
    bool writes;
};

template <int BS, bool SHARE>
__device__ __forceinline__ EosPlace eos_place(const DomDev &D, int b, int lanes)
{
    EosPlace p{eos_block<BS>(D, b) * BS + (int)threadIdx.x, 0, true};
    if (SHARE) {
        const int shared = shared_blocks(D, lanes, BS), costly = D.eosClassEnd[0];
        if (b < shared) {
            const int t = b * BS + threadIdx.x, part = t & (lanes - 1);
            const int rep = D.eosClassRep[0];
            p.slot = t >> (31 - __clz(lanes));
            if (p.slot >= costly) p.slot = D.numElem;  // past the class: none
            p.rep = (rep - part + lanes - 1) >> (31 - __clz(lanes));
            p.writes = part == ((rep - 1) & (lanes - 1));
            return p;
        }
        p.slot = costly + (b - shared) * BS + threadIdx.x;
    }
    int cls = 0;
    while (cls < D.eosNumClass - 1 && p.slot >= D.eosClassEnd[cls]) ++cls;
    p.rep = D.eosClassRep[cls];
    return p;
}

// SUB: a subdomain set's fused cycle, which reads a comm face's neighbour
// element in the neighbouring subdomain (no MonoQ ghost copy)
//
// Bound by the latency of its 22 loads an element and their scattered sectors
// (487 B of L2 traffic for 196 B of data), not by the reps: 52 us at -s 100
// (1.0e6 elements) on B200, against 30 us for the 196 B at the measured copy
// rate; 40 more reps for the costliest class add 8 us.  With each load beside
// its use, between branches, atomics and stores that no load can pass, it took
// 70.5 us at 40 registers and 12 blocks per SM.  All loads first want 64
// registers: 8 blocks 55.9 us, 6 64.4, 7 59.8, 10 59.9 (spills), 12 72.5.
// Elements in natural order instead of class order: 57.8 us at 8 blocks,
// 53.7 at 9, but 150 against 136 us at -s 133 with cost 4, where every warp
// runs its costliest element's reps.
template <int BS, bool U, bool SUB, class W, bool SHARE = false>
__global__ void __launch_bounds__(BS, min_blocks(kEosMinBlocks, BS))
    k_eos(const __grid_constant__ W w, Params P, int lanes)
{
    const int2 blk = w.template block<BS, LULESH_EOS_REVERSE>();
    const DomDev &D = w.domain(blk.x);
    TimeCtl &T = w.time(D);
    const EosPlace place = eos_place<BS, SHARE>(D, blk.y / BS, lanes);
    // before pdl_enter: the element, and where the kernel is one wave what the
    // kinematics kernel does not write
    int zidx = 0;
    double mass_z, volo_z, q_old_z, v_z, e_temp, p_temp;
    if (place.slot < D.numElem) {
        zidx = chk_index(D.eosOrder[place.slot], D.numElem, &T, kChkSlot);
        if (SHARE) {
            mass_z = __ldcg(D.elemMass + zidx), volo_z = __ldcg(D.volo + zidx);
            q_old_z = __ldcg(D.q + zidx), v_z = __ldcg(D.v + zidx);
            e_temp = __ldcg(D.e + zidx), p_temp = __ldcg(D.p + zidx);
        }
    }
    pdl_enter();
    if (!T.active) return;  // uniform per block
    double dtc = 1.0e+20, vmax = 0.0;
    if (place.slot < D.numElem) {
        // The element of this slot and its rep count.  The reference visits
        // regElemlist and finds the rep by region (giveMyRegion,
        // lulesh.cu:3976-3984); here slots are grouped by rep class
        // (HostDomain::eosOrder), which keeps the trip count uniform per warp
        // with denser loads (measured 98 us vs 99 us regElemlist order and
        // 108 us natural order at -s 100).
        const int rep = place.rep;

        // Every array the element needs, before any arithmetic, branch or
        // store.  A face on the mesh boundary reads the element itself: its
        // neighbour's value is then the element's own (symmetry plane) or
        // replaced by 0 (free surface).
        int bcMask, lm[3], lp[3];
        if (U) {  // the mesh's own links and boundary mask
            bcMask = D.elemBC[zidx];
            lm[0] = D.lxim[zidx];
            lp[0] = D.lxip[zidx];
            lm[1] = D.letam[zidx];
            lp[1] = D.letap[zidx];
            lm[2] = D.lzetam[zidx];
            lp[2] = D.lzetap[zidx];
        } else {
            elem_face_links(D, zidx, bcMask, lm[0], lp[0], lm[1], lp[1], lm[2], lp[2]);
        }
        const auto is = [&](int mask, int symm, int free) {
            return (bcMask & mask) == symm || (bcMask & mask) == free;
        };
        if (is(XI_M, XI_M_SYMM, XI_M_FREE)) lm[0] = zidx;
        if (is(XI_P, XI_P_SYMM, XI_P_FREE)) lp[0] = zidx;
        if (is(ETA_M, ETA_M_SYMM, ETA_M_FREE)) lm[1] = zidx;
        if (is(ETA_P, ETA_P_SYMM, ETA_P_FREE)) lp[1] = zidx;
        if (is(ZETA_M, ZETA_M_SYMM, ZETA_M_FREE)) lm[2] = zidx;
        if (is(ZETA_P, ZETA_P_SYMM, ZETA_P_FREE)) lp[2] = zidx;
        const DomDev *sm[3] = {&D, &D, &D}, *sp[3] = {&D, &D, &D};
        if (SUB) {
            // comm faces: the mirrored element of the neighbour's opposite
            // face layer, where k_monoq_ghost would copy it from
            const int nx = D.nx;
            int ix, iy, iz;
            lattice(D.by_nx, zidx, ix, iy, iz);
            if (bcMask & XI_M_COMM) {
                sm[0] = &w.doms()[D.nbr[0 + 3 + 9]];
                lm[0] = (iz * nx + iy) * nx + (nx - 1);
            }
            if (bcMask & XI_P_COMM) {
                sp[0] = &w.doms()[D.nbr[2 + 3 + 9]];
                lp[0] = (iz * nx + iy) * nx;
            }
            if (bcMask & ETA_M_COMM) {
                sm[1] = &w.doms()[D.nbr[1 + 0 + 9]];
                lm[1] = (iz * nx + (nx - 1)) * nx + ix;
            }
            if (bcMask & ETA_P_COMM) {
                sp[1] = &w.doms()[D.nbr[1 + 6 + 9]];
                lp[1] = (iz * nx) * nx + ix;
            }
            if (bcMask & ZETA_M_COMM) {
                sm[2] = &w.doms()[D.nbr[1 + 3 + 0]];
                lm[2] = ((nx - 1) * nx + iy) * nx + ix;
            }
            if (bcMask & ZETA_P_COMM) {
                sp[2] = &w.doms()[D.nbr[1 + 3 + 18]];
                lp[2] = iy * nx + ix;
            }
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            lm[c] = chk_index(lm[c], SUB ? sm[c]->allElem : D.allElem, &T, kChkLink);
            lp[c] = chk_index(lp[c], SUB ? sp[c]->allElem : D.allElem, &T, kChkLink);
        }
        const double dxi = D.delv_xi[zidx], deta = D.delv_eta[zidx], dzeta = D.delv_zeta[zidx];
        double xim = sm[0]->delv_xi[lm[0]], xip = sp[0]->delv_xi[lp[0]];
        double etam = sm[1]->delv_eta[lm[1]], etap = sp[1]->delv_eta[lp[1]];
        double zetam = sm[2]->delv_zeta[lm[2]], zetap = sp[2]->delv_zeta[lp[2]];
        const double vdov_z = D.vdov[zidx];
        const double vnew_z = D.vnew[zidx];
        const double xxi = D.delx_xi[zidx], xeta = D.delx_eta[zidx], xzeta = D.delx_zeta[zidx];
        if (!SHARE) {
            mass_z = D.elemMass[zidx], volo_z = D.volo[zidx];
            q_old_z = D.q[zidx], v_z = D.v[zidx];
            e_temp = D.e[zidx], p_temp = D.p[zidx];
        }
        const double delvc_temp = D.delv[zidx];
        const double area_tmp = D.arealg[zidx];

        // ---- CalcMonotonicQRegionForElems_kernel, lulesh.cu:3586-3724
        if ((bcMask & XI_M) == XI_M_FREE) xim = 0.0;
        if ((bcMask & XI_P) == XI_P_FREE) xip = 0.0;
        if ((bcMask & ETA_M) == ETA_M_FREE) etam = 0.0;
        if ((bcMask & ETA_P) == ETA_P_FREE) etap = 0.0;
        if ((bcMask & ZETA_M) == ZETA_M_FREE) zetam = 0.0;
        if ((bcMask & ZETA_P) == ZETA_P_FREE) zetap = 0.0;
        const double mult = P.monoq_limiter_mult, maxs = P.monoq_max_slope;
        const double phixi = mono_limiter(dxi, xim, xip, mult, maxs);
        const double phieta = mono_limiter(deta, etam, etap, mult, maxs);
        const double phizeta = mono_limiter(dzeta, zetam, zetap, mult, maxs);
        double qlin, qquad;
        if (vdov_z > 0.) {
            qlin = 0.;
            qquad = 0.;
        } else {
            double delvxxi = dxi * xxi;
            double delvxeta = deta * xeta;
            double delvxzeta = dzeta * xzeta;
            if (delvxxi > 0.) delvxxi = 0.;
            if (delvxeta > 0.) delvxeta = 0.;
            if (delvxzeta > 0.) delvxzeta = 0.;
            const double rho = mass_z / (volo_z * vnew_z);
            qlin = -P.qlc_monoq * rho *
                   (delvxxi * (1. - phixi) + delvxeta * (1. - phieta) +
                    delvxzeta * (1. - phizeta));
            qquad = P.qqc_monoq * rho *
                    (delvxxi * delvxxi * (1. - phixi * phixi) +
                     delvxeta * delvxeta * (1. - phieta * phieta) +
                     delvxzeta * delvxzeta * (1. - phizeta * phizeta));
        }
        const bool writes = !SHARE || place.writes;
        if (writes && q_old_z > P.qstop) atomicMin(&T.bad_q, zidx);
        if (writes && w.materialize()) {
            D.qq[zidx] = qquad;
            D.ql[zidx] = qlin;
        }

        // ---- ApplyMaterialPropertiesAndUpdateVolume_kernel, lulesh.cu:4025-4096
        double eosvmin = P.eosvmin, eosvmax = P.eosvmax;
        double vnewc = vnew_z;
        if (eosvmin != 0.) {
            if (vnewc < eosvmin) vnewc = eosvmin;
        }
        if (eosvmax != 0.) {
            if (vnewc > eosvmax) vnewc = eosvmax;
        }
        double vc = v_z;
        if (eosvmin != 0.) {
            if (vc < eosvmin) vc = eosvmin;
        }
        if (eosvmax != 0.) {
            if (vc > eosvmax) vc = eosvmax;
        }
        if (writes && vc <= 0.) atomicMin(&T.bad_vol, zidx);

        double p_new = 0., e_new = 0., q_new = 0., bvc = 0., pbvc = 0.;
        const double rho0 = P.refdens;
        // the reference density is 1.0 in every sedov problem (uniform branch)
        const bool rho1 = rho0 == 1.0;
        if (rho1)
            eos_reps<true>(rep, e_temp, p_temp, q_old_z, qquad, qlin, delvc_temp, vnewc,
                           eosvmin, eosvmax, rho0, P, p_new, e_new, q_new, bvc, pbvc);
        else
            eos_reps<false>(rep, e_temp, p_temp, q_old_z, qquad, qlin, delvc_temp, vnewc,
                            eosvmin, eosvmax, rho0, P, p_new, e_new, q_new, bvc, pbvc);
        if (writes) {
            D.p[zidx] = p_new;
            D.e[zidx] = e_new;
            D.q[zidx] = q_new;
        }

        // CalcSoundSpeedForElems_device, lulesh.cu:3795-3809
        double ssTmp = pbvc * e_new + vnewc * vnewc * bvc * p_new;
        if (!rho1) ssTmp = ssTmp / rho0;
        if (ssTmp <= .1111111e-36)
            ssTmp = .3333333e-18;
        else
            ssTmp = sqrt(ssTmp);
        if (writes) D.ss[zidx] = ssTmp;

        // UpdateVolumesForElems_device, lulesh.cu:3850-3861
        double tmpV = vnew_z;
        if (fabs(tmpV - 1.0) < P.v_cut) tmpV = 1.0;
        if (writes) D.v[zidx] = tmpV;

        // CalcTimeConstraintsForElems_kernel body, lulesh.cu:4246-4279
        const double qqc2 = 64.0 * P.qqc * P.qqc;
        const double vdov_tmp = vdov_z;
        vmax = fabs(vdov_tmp);
        const double ss_tmp = ssTmp;
        double dtf = ss_tmp * ss_tmp;
        dtf += ((vdov_tmp < 0.) ? qqc2 * area_tmp * area_tmp * vdov_tmp * vdov_tmp : 0.);
        dtf = area_tmp * rsqrt(dtf);
        if (writes && vdov_tmp != 0. && dtf < dtc) dtc = dtf;
    }
    // block minimum (exact, order-free), one atomic per block.  The hydro
    // limit dvovmax / (|vdov| + tiny) falls as |vdov| grows, also after
    // rounding, so its minimum is that of the block's largest |vdov|: one
    // division per block.
    __shared__ double s_c[BS / 32], s_v[BS / 32];
    dtc = warp_min(dtc);
    vmax = warp_max(vmax);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) {
        s_c[warp] = dtc;
        s_v[warp] = vmax;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double c = s_c[0], v = s_v[0];
#pragma unroll
        for (int k = 1; k < BS / 32; ++k) {
            c = fmin(c, s_c[k]);
            v = fmax(v, s_v[k]);
        }
        if (c < 1.0e+20) atomicMin(&T.min_courant, dbits(c));
        if (v != 0.) {
            const double h = P.dvovmax / (v + 1.e-20);
            if (h < 1.0e+20) atomicMin(&T.min_hydro, dbits(h));
        }
    }
}

template <int BS, bool U, bool SUB>
static void launch_eos_bs(const SetArgs &a, int nblocks, Params P, cudaStream_t s)
{
    const int lanes = !SUB && a.records && a.ndom == 1 ? rep_lanes(a.records[0], BS) : 1;
    if constexpr (!SUB) {
        if (lanes > 1) {
            const int n = shared_blocks(a.records[0], lanes, BS) + other_blocks(a.records[0], BS);
            launch_k(k_eos<BS, U, false, OneDomain, true>, n, BS, s, a.pdl != 0, by_value<1>(a, n),
                     P, lanes);
            return;
        }
    }
    if constexpr (U)
        launch_k(k_eos<BS, true, false, OneDomain>, nblocks, BS, s, a.pdl != 0,
                 by_value<1>(a, nblocks), P, 1);
    else
        launch_where<!SUB, SUB>(a, nblocks, [&](const auto &w) {
            launch_k(k_eos<BS, false, SUB, std::decay_t<decltype(w)>>, nblocks, BS, s, a.pdl != 0,
                     w, P, 1);
        });
}

void launch_eos(const SetArgs &a, int nblocks, Params P, cudaStream_t s, int bs, bool u,
                bool sub)
{
    if (u) {
        launch_eos_bs<kElemBlock, true, false>(a, nblocks, P, s);
        return;
    }
    if (sub) {  // subdomain sets take 128-element blocks only
        launch_eos_bs<kElemBlock, false, true>(a, nblocks, P, s);
        return;
    }
    switch (bs) {
        case 64: launch_eos_bs<64, false, false>(a, nblocks, P, s); break;
        case 256: launch_eos_bs<256, false, false>(a, nblocks, P, s); break;
        default: launch_eos_bs<kElemBlock, false, false>(a, nblocks, P, s); break;
    }
}

// ---------------------------------------------------------------------------
// fused halo kernels of a subdomain set

// CommSyncPosVel semantics (lulesh-comms-gpu.cu:1231-1661): a node shared by
// several subdomains takes x,y,z,xd,yd,zd from the subdomain that holds it
// on its minimum faces only (the "+side owner"), which never writes it here.
// Blocks cover the max-side faces only (sync blocks, build_tables): block b
// takes face blocks[b].y >> 24 of domain blocks[b].x from item
// (blocks[b].y & 0xffffff) on.  Face 0 holds the nodes with px = nx, face 1
// those with py = nx and px < nx, face 2 those with pz = nx and px, py < nx,
// so every node of a max-side face is visited once; the copy itself is
// decided from the node's position, as for the whole node range.
__global__ void k_posvel_sync(SetArgs a)
{
    pdl_enter();
    const int2 blk = a.blocks[blockIdx.x];
    const DomDev &D = a.doms[blk.x];
    const TimeCtl &T = a.tcs[D.tc];
    if (!T.active) return;
    const int face = blk.y >> 24;
    const int item = (blk.y & 0xffffff) + threadIdx.x;
    const int en = D.en, nx = D.nx, tp = D.tp;
    int px, py, pz;
    if (face == 0) {
        if (item >= en * en) return;
        px = nx, py = item % en, pz = item / en;
    } else if (face == 1) {
        if (item >= nx * en) return;
        px = item % nx, py = nx, pz = item / nx;
    } else {
        if (item >= nx * nx) return;
        px = item % nx, py = item / nx, pz = nx;
    }
    const int i = (pz * en + py) * en + px;
    const int sx = (px == nx && D.col < tp - 1) ? 1 : 0;
    const int sy = (py == nx && D.row < tp - 1) ? 1 : 0;
    const int sz = (pz == nx && D.plane < tp - 1) ? 1 : 0;
    if ((sx | sy | sz) == 0) return;
    const int nb = D.nbr[(sx + 1) + 3 * (sy + 1) + 9 * (sz + 1)];
    if (nb < 0) return;
    const DomDev &O = a.doms[nb];
    const int j = chk_index(((pz - sz * nx) * en + (py - sy * nx)) * en + (px - sx * nx),
                            O.numNode, &a.tcs[D.tc], kChkNode);
    D.x[i] = O.x[j];
    D.y[i] = O.y[j];
    D.z[i] = O.z[j];
    D.xd[i] = O.xd[j];
    D.yd[i] = O.yd[j];
    D.zd[i] = O.zd[j];
}

void launch_posvel_sync(const SetArgs &a, int nblocks, cudaStream_t s)
{
    launch_k(k_posvel_sync, nblocks, kNodeBlock, s, a.pdl != 0, a);
}

// CommMonoQ semantics (lulesh-comms-gpu.cu:1665-1806): the delv_* ghost
// faces (offsets of SetupConnectivityBC, lulesh.cu:581-615) receive the
// neighbour's boundary element layer.  Block b covers face blocks[b].y>>24
// of domain blocks[b].x, items (blocks[b].y & 0xffffff) onward.
__global__ void k_monoq_ghost(SetArgs a)
{
    pdl_enter();
    const int2 blk = a.blocks[blockIdx.x];
    const DomDev &D = a.doms[blk.x];
    const TimeCtl &T = a.tcs[D.tc];
    if (!T.active) return;
    const int f = blk.y >> 24;
    const int item = (blk.y & 0xffffff) + threadIdx.x;
    const int nx = D.nx;
    if (item >= nx * nx || D.ghost[f] < 0) return;
    const int a0 = item / nx, b0 = item % nx;  // (plane|row, row|col) of the face
    int dxn = 0, dyn = 0, dzn = 0, src;
    switch (f) {
        case 0: dzn = -1; src = ((nx - 1) * nx + a0) * nx + b0; break;  // row a0, col b0
        case 1: dzn = 1; src = (0 * nx + a0) * nx + b0; break;
        case 2: dyn = -1; src = (a0 * nx + (nx - 1)) * nx + b0; break;  // plane a0, col b0
        case 3: dyn = 1; src = (a0 * nx + 0) * nx + b0; break;
        case 4: dxn = -1; src = (a0 * nx + b0) * nx + (nx - 1); break;  // plane a0, row b0
        default: dxn = 1; src = (a0 * nx + b0) * nx + 0; break;
    }
    const int nb = D.nbr[(dxn + 1) + 3 * (dyn + 1) + 9 * (dzn + 1)];
    if (nb < 0) return;
    const DomDev &N = a.doms[nb];
    const int g = chk_index(D.ghost[f] + item, D.allElem, &a.tcs[D.tc], kChkLink);
    src = chk_index(src, N.numElem, &a.tcs[D.tc], kChkLink);
    D.delv_xi[g] = N.delv_xi[src];
    D.delv_eta[g] = N.delv_eta[src];
    D.delv_zeta[g] = N.delv_zeta[src];
}

void launch_monoq_ghost(const SetArgs &a, int nblocks, cudaStream_t s)
{
    launch_k(k_monoq_ghost, nblocks, kElemBlock, s, a.pdl != 0, a);
}

}  // namespace lulesh
