// kernels.cuh -- launch interface of the per-cycle kernels.
#pragma once

#include <cuda_runtime.h>

#include "lulesh_dev.h"

// Block order of the kinematics and EOS launches.  Kinematics walks its
// block table last to first: its last outputs are then those of the first
// elements, where each rep class of the EOS walk starts, and they are still
// in L2 (measured on B200 at -s 100: EOS 91 -> 86 us, cycle 329 -> 325 us,
// the same results).  Reversing the EOS walk instead gained nothing.
#ifndef LULESH_KIN_REVERSE
#define LULESH_KIN_REVERSE 1
#endif
#ifndef LULESH_FORCE_REVERSE
#define LULESH_FORCE_REVERSE 0
#endif
#ifndef LULESH_EOS_REVERSE
#define LULESH_EOS_REVERSE 0
#endif

// Node blocks last to first: the nodal kernel follows the force kernel,
// whose last-written corner forces are the ones still in L2 (measured on
// B200 at -s 100: nodal 53.7 -> 48.9 us, the same results).
#ifndef LULESH_NODAL_REVERSE
#define LULESH_NODAL_REVERSE 1
#endif

namespace lulesh {

constexpr int kElemBlock = 128;  // threads per block, element kernels
constexpr int kNodeBlock = 128;  // threads per block, node kernels

// Resident blocks per SM asked of the compiler (the register budget of the
// element kernels), chosen by measurement on B200 at -s 100: force 3 (164
// registers, 69.8 us; 86 us at 4 blocks with spills, 88 at 5), kinematics 5
// (96 registers, 51.6 us; 57.8 at 4, and 2 us more at 6 with spills), EOS 8
// (64 registers, 55.9 us; 59.8 at 7 and at 10, 64.4 at 6, 72.5 at 12).
#ifndef LULESH_FORCE_MINB
#define LULESH_FORCE_MINB 3
#endif
#ifndef LULESH_KIN_MINB
#define LULESH_KIN_MINB 5
#endif
#ifndef LULESH_EOS_MINB
#define LULESH_EOS_MINB 8
#endif
// nodal: 12 blocks (40 registers) for the streaming corner gather, 41.6 us at
// -s 100 and 188 at -s 160; 44.6 and 195 at 16 (32 registers, spills), 41.6 and
// 187 at 10.  The subdomain gather, whose neighbour records add latency, wants
// every warp slot: 54.8 us at 16, 56.6 at 12, 59.3 at 10 (2x2x2 of -s 50).
#ifndef LULESH_NODAL_MINB
#define LULESH_NODAL_MINB 12
#endif
constexpr int kNodalMinBlocks = LULESH_NODAL_MINB;
constexpr int kNodalFewMinBlocks = 16;
// with the time increment's warp (small sets): registers for all
// corner loads of a node at once beside its state (55; 16 B of spills at 8
// blocks, and -s 30 16.6 us per cycle against 16.1, -s 60 42.7 against 41.7)
#ifndef LULESH_NODAL_INCR_MINB
#define LULESH_NODAL_INCR_MINB 7
#endif
constexpr int kNodalIncrMinBlocks = LULESH_NODAL_INCR_MINB;
// unstructured nodal kernel: four corners x 3 components in flight
#ifndef LULESH_NODAL_U_MINB
#define LULESH_NODAL_U_MINB 12
#endif
constexpr int kNodalUMinBlocks = LULESH_NODAL_U_MINB;
constexpr int kForceMinBlocks = LULESH_FORCE_MINB;
constexpr int kKinMinBlocks = LULESH_KIN_MINB;
// packed meshes: 128 registers, 12.6 us at -s 40; 14.8 at 3 and 5 blocks
#ifndef LULESH_KIN_PACKED_MINB
#define LULESH_KIN_PACKED_MINB 4
#endif
constexpr int kKinPackedMinBlocks = LULESH_KIN_PACKED_MINB;
constexpr int kEosMinBlocks = LULESH_EOS_MINB;

// Minimum resident blocks of a kernel launched with BS threads per block
// that keeps the per-SM thread target of `minb` blocks of 128 threads.
constexpr int min_blocks(int minb, int bs)
{
    return (minb * 128 / bs) > 0 ? (minb * 128 / bs) : 1;
}

// Largest set (nodes) whose cycle kernels make the time increment.  Every block
// of the node update then makes it, to save a launch: 1 to 2 us of a cycle while
// the blocks run in one wave, less and less beyond it.  B200, graphs of four
// cycles, us per cycle, launch -> inside:
//   one domain        -s 36 23.1 -> 21.7   50 31.0 -> 28.3   51 32.2 -> 31.6
//                     60 44.8 -> 43.3   66 56.9 -> 56.0   70 66.2 -> 65.6
//                     80 97.1 -> 97.0   90 137.2 -> 137.1   100 183.9 -> 185.0
//   2x2x2 of          -s 18 27.2 -> 25.5   24 36.1 -> 32.7   25 38.0 -> 38.0
//                     26 39.8 -> 40.3   28 46.6 -> 46.0   30 52.5 -> 52.8
//                     32 58.9 -> 62.6
//   3x3x3 of          -s 14 33.8 -> 32.5   18 45.7 -> 50.2   20 61.3 -> 60.4
//   batches of -s 28  2 jobs 26.6 -> 25.5   4 32.8 -> 31.6   6 39.9 -> 41.4
//                     8 47.2 -> 48.6   12 67.8 -> 69.4
// One domain's line is past its gains of more than 1% (-s 66).  Sets of several
// domains read neighbours' or their own records in those blocks as well; theirs
// is where the first wave of that kernel ends, kNodalIncrMinBlocks blocks of 128
// nodes on each of 148 SMs (2x2x2 of -s 24, five jobs of -s 28).
constexpr long long kInlineIncrementNodes = 148 * 16 * 128;
constexpr long long kInlineIncrementNodesMany = 148 * kNodalIncrMinBlocks * 128;

// Block shapes the FP64 element kernels (force, kinematics, EOS) and the
// nodal kernel are compiled for; a set's block tables use one of each.
constexpr bool valid_elem_block(int bs) { return bs == 64 || bs == 128 || bs == 256; }
constexpr bool valid_node_block(int bs) { return bs == 128 || bs == 256 || bs == 512; }

// What the element kernels read the mesh from: the element's position in a
// structured box, an unstructured mesh's lists, or those lists and the packed
// nodes and corners of a scattered mesh.
enum class Mesh { kBox, kLists, kPacked };

// A kernel launch over all domains of a set: block b works on domain
// blocks[b].x starting at item blocks[b].y (element, node or region slot).
struct SetArgs {
    const DomDev *doms;
    TimeCtl *tcs;
    const int2 *blocks;
    int materialize;  // also write the per-cycle transients
    // launch with programmatic stream serialisation (host side only; the
    // kernels launched this way wait for the previous grid first)
    int pdl = 0;
    // host side only: the records of a set of 1 or kFewDomains equal domains,
    // which the kernels then take by value (OneDomain, FewDomains)
    const DomDev *records = nullptr;
    int ndom = 0;
    // one record per job beside tcs: the cycle's kernels make the time
    // increment themselves (inline_increment, set.hpp); null after a
    // k_time_increment launch
    TimeCtl *next = nullptr;
    const CornerF32 *corner32 = nullptr;  // a mixed set's first domain (host side only)
    int show = 0;  // a scattered mesh's corner forces to fx_elem ... too (host side only)
};

// Where a block of a cycle kernel works: its domain's record, the time state
// (time) and the first item.  next is where the cycle's own time state is
// formed when its kernels increment the time themselves, else time again.
//
// ManyDomains reads them from memory: block table -> domain record -> array
// pointers, three dependent loads before the first gather, and the pointers
// again after every store (which the compiler cannot tell from the table).
// A set of one domain, or of the 2x2x2 equal subdomains of a problem, passes
// its records as the kernel's parameter instead: pointers and sizes come from
// the constant bank and the place from the block index.  Measured on B200, us
// per cycle, ManyDomains -> by value: -s 100 225 -> 204 (force 70 -> 64,
// kinematics 50 -> 43, nodal 47 -> 43), -s 160 897 -> 826, -s 30 28.9 -> 25.0,
// 2x2x2 of -s 50 237 -> 218.5.  Batches and servers have up to hundreds of
// uneven domains and keep the tables.  (Copying ManyDomains' record through the
// read-only path made a 24-job batch 2% slower.)
struct ManyDomains {
    SetArgs a;
    template <int BS, bool REVERSE>
    __device__ __forceinline__ int2 block() const
    {
        return a.blocks[REVERSE ? gridDim.x - 1 - blockIdx.x : blockIdx.x];
    }
    __device__ __forceinline__ const DomDev &domain(int d) const { return a.doms[d]; }
    __device__ __forceinline__ TimeCtl &time(const DomDev &D) const { return a.tcs[D.tc]; }
    __device__ __forceinline__ TimeCtl &next(const DomDev &D) const
    {
        return a.next ? a.next[D.tc] : a.tcs[D.tc];
    }
    __device__ __forceinline__ bool increments() const { return a.next != nullptr; }
    __device__ __forceinline__ const DomDev *doms() const { return a.doms; }
    __device__ __forceinline__ int materialize() const { return a.materialize; }
    // The node block table is already laid out last to first.  A job that is
    // done skips its gathers: the time state is read first.
    static constexpr bool kTable = true;
};

// N equal domains of one problem, in block table order (build_tables)
template <int N>
struct ByValue {
    DomDev D[N];
    TimeCtl *tc, *tn;
    int mat;
    int per;  // blocks per domain of this launch
    long long stride;  // doubles from one domain's corner forces to the next's
    template <int BS, bool REVERSE>
    __device__ __forceinline__ int2 block() const
    {
        const int b = REVERSE ? gridDim.x - 1 - blockIdx.x : blockIdx.x;
        const int d = N == 1 ? 0 : b / per;
        return make_int2(d, (b - d * per) * BS);
    }
    __device__ __forceinline__ const DomDev &domain(int d) const { return D[N == 1 ? 0 : d]; }
    __device__ __forceinline__ TimeCtl &time(const DomDev &) const { return *tc; }
    __device__ __forceinline__ TimeCtl &next(const DomDev &) const { return *tn; }
    __device__ __forceinline__ bool increments() const { return tn != tc; }
    __device__ __forceinline__ const DomDev *doms() const { return D; }
    __device__ __forceinline__ int materialize() const { return mat; }
    // the time state is read beside the gathers, and checked before any store
    static constexpr bool kTable = false;
};
using OneDomain = ByValue<1>;
// (3x3x3, 27 records of 21 KB, would fit the 32,764 B a kernel may take; it reads
// the table, not measured the other way)
constexpr int kFewDomains = 8;
using FewDomains = ByValue<kFewDomains>;

template <int N>
inline ByValue<N> by_value(const SetArgs &a, int nblocks)
{
    ByValue<N> w;
    for (int d = 0; d < N; ++d) w.D[d] = a.records[d];
    w.tc = a.tcs;
    w.tn = a.next ? a.next : a.tcs;
    w.mat = a.materialize;
    w.per = nblocks / N;
    w.stride = N > 1 ? a.records[1].fx_elem - a.records[0].fx_elem : 0;
    return w;
}

// launch(where) with the cheapest form the set allows, of those the call can
// be for: ONE a single domain, FEW the 2x2x2 subdomains (128-wide blocks only).
template <bool ONE, bool FEW, class Launch>
inline void launch_where(const SetArgs &a, int nblocks, const Launch &launch)
{
    if constexpr (ONE) {
        if (a.records && a.ndom == 1) return launch(by_value<1>(a, nblocks));
    }
    if constexpr (FEW) {
        if (a.records && a.ndom == kFewDomains) return launch(by_value<kFewDomains>(a, nblocks));
    }
    launch(ManyDomains{a});
}

// ---------------------------------------------------------------------------
// checked builds
//
// With -DLULESH_CHECKED=1 the FP64 cycle kernels range-check every index
// they compute or load before using it: node indices, corner indices,
// corner-list runs, EOS slots and face links.  An index out of range is
// replaced by 0, which every array holds, so no access leaves its array and
// no thread leaves the kernel's control flow.  The first failing check's
// code is kept in TimeCtl::chk, and the next time increment ends the job
// with LULESH_BOUNDS_ERROR.  This build stands in for a memory checker.
#ifndef LULESH_CHECKED
#define LULESH_CHECKED 0
#endif
enum CheckCode { kChkNode = 1, kChkCorner = 2, kChkCornerRun = 3, kChkSlot = 4, kChkLink = 5 };

__device__ __forceinline__ int chk_index(long long i, long long n, TimeCtl *T, int code)
{
#if LULESH_CHECKED
    if (i < 0 || i >= n) {
        atomicCAS(&T->chk, 0, code);
        return 0;
    }
#else
    (void)n;
    (void)T;
    (void)code;
#endif
    return (int)i;
}

// ---------------------------------------------------------------------------
// programmatic dependent launch
//
// The cycle kernels may be launched with programmatic stream serialisation
// (SetArgs::pdl): the next kernel's blocks are then scheduled while this
// one's last wave drains.  Every kernel launched that way calls pdl_enter()
// before it reads what the previous grid may write, or writes anything: it
// waits until that grid has completed and its writes are visible, then lets
// its own dependents be scheduled.  Without the attribute both pass at once.
//
// What the previous kernel cannot write may be read before pdl_enter(), while
// that kernel runs: the mesh's tables (node ids, corner slots, the EOS order)
// in every set, and in small sets, whose kernels are chains of loads, the node
// update's own node and the EOS's element values.  Their last writer is
// several grids back: every kernel waits before it lets its dependents in, so
// all grids but the previous one have ended, and __ldcg takes their values
// from L2.  Only kernels that always follow another kernel of the set do this:
// nothing of the caller's can lie between.  Measured on B200, us per cycle:
// -s 10 15.0 -> 14.1, -s 30 16.6 -> 16.1, -s 45 25.3 -> 24.2, -s 60 42.5 ->
// 41.3, a scattered -s 40 mesh 38.3 -> 37.3, -s 100 182.7 -> 181.4.  The force
// kernel's gathers done the same way (past L1) gained 3% at -s 10 and lost 2%
// at -s 60.

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void pdl_enter()
{
    pdl_wait();
    pdl_trigger();
}

template <typename... KArgs, typename... Args>
inline void launch_k(void (*kernel)(KArgs...), int grid, int block, cudaStream_t s, bool pdl,
                     Args... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = pdl ? attr : nullptr;
    cfg.numAttrs = pdl ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, args...);  // errors: cudaGetLastError
}

// start of a scattered mesh's cycle: time increment and node packing (node blocks)
void launch_begin_packed(const SetArgs &a, int nblocks, Params P, cudaStream_t s);
// a scattered mesh's corner forces to fx_elem, fy_elem, fz_elem (element blocks)
void launch_show_corners(const SetArgs &a, int nblocks, cudaStream_t s);
void launch_time_increment(TimeCtl *tcs, int ntc, Params P, cudaStream_t s, bool pdl = false);
// u: the set's domains are unstructured (lmesh): 128-wide blocks, mesh
// arrays read instead of structured indexing
void launch_force(const SetArgs &a, int nblocks, Params P, cudaStream_t s,
                  int bs = kElemBlock, bool u = false);
void launch_nodal(const SetArgs &a, int nblocks, Params P, cudaStream_t s,
                  int bs = kNodeBlock, bool u = false);
// staged comm path: own-corner partial sums, then the update from fx/fy/fz
void launch_nodal_gather_local(const SetArgs &a, int nblocks, cudaStream_t s);
void launch_nodal_update(const SetArgs &a, int nblocks, Params P, cudaStream_t s);
void launch_kinematics(const SetArgs &a, int nblocks, Params P, cudaStream_t s,
                       int bs = kElemBlock, bool u = false);
// sub: a subdomain set's fused cycle, comm-face neighbours read in the
// neighbouring subdomain (k_monoq_ghost not needed)
void launch_eos(const SetArgs &a, int nblocks, Params P, cudaStream_t s, int bs = kElemBlock,
                bool u = false, bool sub = false);
// fused halo kernels of a subdomain set (direct reads of neighbour memory)
void launch_posvel_sync(const SetArgs &a, int nblocks, cudaStream_t s);
void launch_monoq_ghost(const SetArgs &a, int nblocks, cudaStream_t s);

// mixed precision variants of the element kernels
void launch_force_mixed(const SetArgs &a, int nblocks, Params P, const CornerF32 *cf,
                        cudaStream_t s);
void launch_nodal_mixed(const SetArgs &a, int nblocks, Params P, const CornerF32 *cf,
                        cudaStream_t s);
void launch_kinematics_mixed(const SetArgs &a, int nblocks, Params P, cudaStream_t s);

}  // namespace lulesh
