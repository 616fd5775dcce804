// set.hpp -- host-side state of a lulesh_set (one GPU, one stream).
#pragma once

#include <cuda_runtime.h>

#include <string>
#include <vector>

#include "block_cache.hpp"
#include "host_setup.hpp"
#include "kernels.cuh"
#include "lulesh_b200.h"
#include "lulesh_dev.h"

// The fused subdomain cycle needs no PosVel sync (CommSyncPosVel,
// lulesh-comms.cu:115-168).  The reference syncs because each rank sums a
// shared node's forces as its own partial sum plus the neighbour's, in its
// own order, so the two copies of the node can differ in the last bits.
// Here every subdomain gathers every corner of its nodes, the neighbours'
// included, in the single-domain corner order, and the node masses are the
// single-domain sums: both copies of a shared node take the same operations
// on the same values and stay equal bit for bit (checked against the single
// domain, every field, 2^3, 3^3 and 4^3 subdomains, up to 400 cycles).
// Leaving the copy out takes 2x2x2 of -s 50 from 349.5 to 343.9 us per
// cycle.  1 puts the k_posvel_sync launch back in the fused cycle.  The
// staged Comm* path keeps the reference's exchange; the parts of a
// multi-GPU problem exchange POSVEL only when their driver asks for it.
#ifndef LULESH_FUSED_POSVEL_SYNC
#define LULESH_FUSED_POSVEL_SYNC 0
#endif

// The EOS of a subdomain set's fused cycle, and of a part of a multi-GPU
// problem, reads a comm face's neighbour element in the neighbouring
// subdomain or its proxy (k_eos<..., SUB>): the value k_monoq_ghost would
// copy into this subdomain's ghost face (CommMonoQ semantics,
// lulesh-comms-gpu.cu:1665-1806).  1 copies the ghost faces and reads them.
#ifndef LULESH_FUSED_MONOQ_GHOST
#define LULESH_FUSED_MONOQ_GHOST 0
#endif

// 0 launches every cycle kernel with plain stream order
#ifndef LULESH_PDL
#define LULESH_PDL 1
#endif

struct lulesh_set {
    int device = 0;
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    int flags = 0;
    lulesh::Params P{};
    int tp = 1;  // subdomains per axis of each job (1 for batches)
    // one unstructured domain read from this lmesh file (empty: -s meshes)
    std::string mesh_path;
    bool unstructured = false;
    // FNV-1a of an unstructured mesh's sizes, connectivity and coordinates
    // (identifies the mesh in checkpoints; 0 for -s meshes)
    unsigned long long mesh_hash = 0;
    int ndom = 0, njobs = 0;

    // per-domain metadata kept on the host
    std::vector<lulesh::DomDev> hdoms;
    std::vector<int> dom_rank;         // rank of each domain inside its job
    std::vector<int> dom_job;          // job of each domain
    std::vector<int> job_origin;       // domain holding the job's origin
    std::vector<lulesh_job> jobs;
    std::vector<size_t> corner_list_len;

    // block shapes and block-table order (lulesh_set_tuning): elements per
    // block of the FP64 element kernels, nodes per block of the nodal
    // kernel, 0 = domains in creation order / 1 = largest domain first
    int eb = lulesh::kElemBlock, nb = lulesh::kNodeBlock, order = 0;

    // device tables (elem_blocks is the base of one allocation holding all)
    lulesh::DomDev *ddoms = nullptr;
    lulesh::TimeCtl *dtc = nullptr;   // njobs records, then njobs more (args().next)
    lulesh::TimeCtl *htc_pinned = nullptr;  // pinned mirror for readback
    int2 *elem_blocks = nullptr, *node_blocks = nullptr, *ghost_blocks = nullptr;
    int n_elem_blocks = 0, n_node_blocks = 0, n_ghost_blocks = 0;
    // subdomain sets: blocks over the max-side node faces (PosVel sync)
    int2 *sync_blocks = nullptr;
    int n_sync_blocks = 0;

    // mixed precision corner buffers
    lulesh::CornerF32 *dcorner32 = nullptr;
    std::vector<lulesh::CornerF32> hcorner32;  // host copy

    // L2 access-policy window set on `stream` (single domains)
    bool l2_window = false;
    // launch the cycle kernels with programmatic dependent launch
    bool pdl = LULESH_PDL != 0;

    // the arena; subdomain sets start it with the node region (every
    // domain's x..zd, node_region_bytes), single domains carve in place
    void *arena = nullptr;
    size_t arena_bytes = 0;
    // what the device pointers above and htc_pinned lie in
    lulesh::Block arena_block, tables_block, ctl_block, pinned_block;
    // a caller has had pointers to the arena, or may have kernels of the set in
    // a graph of its own: work on the set's memory may run on streams unknown
    // here
    bool handed_out = false;
    bool graphs_show = false;  // handed_out when the graphs were captured
    void *pack = nullptr;  // nodePack and cornerPack of a scattered mesh
    size_t node_region_bytes = 0;

    // captured cycle, and a graph of graph_cycles consecutive cycles
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    bool graph_ready = false;
    int graph_cycles = 1;
    cudaGraph_t graph_k = nullptr;
    cudaGraphExec_t exec_k = nullptr;
    bool graph_k_ready = false;
    // exec_k for launches with others of the call after them, where that makes a
    // difference (show_corners)
    cudaGraphExec_t exec_quiet_k = nullptr;
    long long cycles_run = 0;  // by one-cycle launches (cycles_per_launch, set.cu)
    // graph_cycles taken at its word, whatever the set has run (lulesh_autotune,
    // whose trials do not count as cycles of the set)
    bool tuning = false;
    // whole-run graph: a WHILE conditional node around a few cycles
    // (rungraph.cu); run_ctl[0] counts its turns, run_ctl[1] is their cap
    cudaGraph_t graph_run = nullptr;
    cudaGraphExec_t exec_run = nullptr;
    unsigned long long *run_ctl = nullptr;

    // one part of a problem split over several GPUs (lulesh_create_part):
    // the local domains hold ranks [first_rank, first_rank + ndom); proxies
    // of the remote neighbours follow them in the device domain table
    // (index ndom + k), with their arrays in proxy_arena
    int nparts = 1, part = 0, first_rank = 0;
    std::vector<lulesh::DomDev> hproxies;
    std::vector<int> proxy_rank;
    void *proxy_arena = nullptr;
    bool mass_pending = false;  // nodal mass waits for the MASS exchange
    // pointer tables of the halo pack (send) and unpack (recv) kernels, per
    // (kind, peer part)
    struct HaloTable {
        double **ptrs = nullptr;
        long long n = 0;
    };
    std::vector<int> peers;
    std::vector<HaloTable> halo_send, halo_recv;  // [kind * peers.size() + peer slot]
    // direct transport: this part's mailbox (every message it receives, at
    // the offsets of mailbox_layout, then one arrival flag per message) and
    // the mailboxes of its peers (mapped through CUDA IPC, or device
    // pointers of parts in the same process)
    void *mailbox = nullptr;
    size_t mailbox_bytes = 0;
    std::vector<void *> peer_mailbox;  // by peer slot
    std::vector<bool> peer_mailbox_ipc;

    // staged comm state: receive-buffer capacity per domain (doubles)
    long com_buf_doubles = 0;
    int max_plane = 0, max_edge = 0;
    int posted_msg = 0, posted_fields = 0, posted_do_recv = 1, posted_plane_only = 0;

    // memory of the set that is no longer used
    void give_back(lulesh::Block *b) const
    {
        if (handed_out)
            lulesh::block_free(b);
        else
            lulesh::block_put(b);
    }

    // The cycle's kernels make the time increment (kernels.cu) in place of a
    // launch of its own.
    bool inline_increment() const
    {
        if (nparts > 1 || unstructured || (flags & (LULESH_FLAG_COMM_STAGED | LULESH_FLAG_MIXED)))
            return false;
        // k_posvel_sync reads the job's time state before kinematics commits it
        if (LULESH_FUSED_POSVEL_SYNC && tp > 1) return false;
        long long nodes = 0;
        for (const lulesh::DomDev &D : hdoms) nodes += D.numNode;
        return nodes <= (ndom == 1 ? lulesh::kInlineIncrementNodes
                                   : lulesh::kInlineIncrementNodesMany);
    }

    // 2x2x2 subdomains in the order of their ranks, their corner forces at
    // equal distances (one arena of equal parts)
    bool even_records() const
    {
        if (ndom != lulesh::kFewDomains || tp != 2) return false;
        const lulesh::DomDev &a = hdoms[0];
        const auto step = hdoms[1].fx_elem - a.fx_elem;
        for (int d = 0; d < ndom; ++d) {
            const lulesh::DomDev &b = hdoms[d];
            if (b.fx_elem != a.fx_elem + d * step || b.fy_elem != a.fy_elem + d * step ||
                b.fz_elem != a.fz_elem + d * step || b.col + 2 * b.row + 4 * b.plane != d)
                return false;
        }
        return true;
    }

    lulesh::SetArgs args(const int2 *blocks) const
    {
        lulesh::SetArgs a;
        a.doms = ddoms;
        a.tcs = dtc;
        a.blocks = blocks;
        a.materialize = (flags & LULESH_FLAG_MATERIALIZE) ? 1 : 0;
        a.pdl = pdl ? 1 : 0;
        // not for parts: their records are followed by proxies
        a.ndom = ndom;
        a.records = nparts == 1 && njobs == 1 && (ndom == 1 || even_records()) ? hdoms.data()
                                                                               : nullptr;
        if (inline_increment()) a.next = dtc + njobs;
        a.corner32 = hcorner32.empty() ? nullptr : hcorner32.data();
        return a;
    }
};

namespace lulesh {
void set_error(const std::string &msg);
int cuda_status(cudaError_t e, const char *what);
// enqueue one cycle (no graph); follows: straight after another one, with
// nothing of the caller's between; last: the caller's may come straight after
int enqueue_cycle(lulesh_set *s, bool follows = false, bool last = true);
// the start of a cycle: the time increment (and a scattered mesh's packing)
void launch_begin(lulesh_set *s, cudaStream_t st, bool follows = false);
// A scattered mesh's newest corner forces lie in cornerPack.  show_corners puts
// them into fx_elem, fy_elem and fz_elem, where callers read them, before the
// library reads these itself; hide_corners: fx_elem ... are the newest, written
// by the library.  Both on the set's stream.  Once a caller may read them without
// the library's doing (handed_out) the last cycle of a graph runs the force kernel
// that writes both forms, but not in launches of longer graphs with others of
// the call after them.  A -s 40 mesh on B200, us per call of 16 cycles: 614, 618
// this way, 624 with both forms in each graph; a launch of show_corners after
// each call adds 25.  refresh_graphs drops the graphs that were captured without.
int show_corners(lulesh_set *s);
int hide_corners(lulesh_set *s);
int refresh_graphs(lulesh_set *s);
// the FP64 force phase of every domain of the set
void launch_force_fp64(lulesh_set *s, cudaStream_t st, bool last = true);
// staged comm path of one cycle (comm.cu)
int enqueue_cycle_staged(lulesh_set *s);
// free the comm message tables of a set (comm.cu)
void comm_release(const lulesh_set *s);
// allocate the staged cycle's message tables ahead of graph capture
int comm_prepare(lulesh_set *s);
// (re)build the block tables from s->eb, s->nb, s->order
int build_tables(lulesh_set *s);
// release the captured cycle graphs (rebuilt at the next step)
void drop_graph(lulesh_set *s);
// read every job's time state back and return the first job's non-OK
// status (LULESH_OK when all are fine); synchronises the stream
int run_status(lulesh_set *s);
// prepare what enqueue_cycle needs before a capture (staged comm tables)
int prepare_capture(lulesh_set *s);
// nodal mass of every subdomain over the whole problem (setup.cu): each node
// adds volume/8 of the elements touching it in ascending global element
// index, reading neighbouring subdomains (or their proxies) through nbr
int nodal_mass_on_device(lulesh_set *s);
// a part of a multi-GPU problem: the proxies and halo tables (part.cu)
int part_build(lulesh_set *s);
void part_release(lulesh_set *s);
}  // namespace lulesh
