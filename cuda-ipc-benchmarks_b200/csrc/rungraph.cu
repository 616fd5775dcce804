// rungraph.cu -- the whole run as one CUDA graph launch.
//
// The reference drives its main loop from the host (lulesh.cu:4858-4873):
// TimeIncrement, LagrangeLeapFrog, and a check of the stop condition every
// cycle.  Here the loop is a WHILE conditional node: its body is a few cycles
// (the same launches lulesh_step captures) followed by k_run_continue,
// which keeps the loop going while any job of the set is not done.  A batch
// of jobs, or a single job, then runs to completion in a single launch with
// no host involvement.  Every turn is counted and the loop stops at a cap, so
// it ends even if a job could never reach its stop condition.
#include "set.hpp"

namespace lulesh {

namespace {

constexpr unsigned long long kDefaultRunCap = 1000000ull;

// Cycles per turn of the loop.  A turn's end (k_run_continue, then the
// conditional node's own decision) costs about as much as two kernels of a
// small mesh; cycles after the last job is done skip their work.  Measured on
// B200, us per cycle, 1 -> 4 per turn: -s 10 23.6 -> 19.0, -s 30 26.8 -> 21.7, a
// batch of 24 jobs 194 -> 185.
constexpr int kCyclesPerTurn = 4;

// ctl[0]: turns so far, ctl[1]: cap
__global__ void k_run_continue(cudaGraphConditionalHandle h, const TimeCtl *tcs, int ntc,
                               unsigned long long *ctl)
{
    __shared__ int any;
    if (threadIdx.x == 0) any = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < ntc; i += blockDim.x)
        if (!tcs[i].done) atomicOr(&any, 1);
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned long long n = ++ctl[0];
        cudaGraphSetConditional(h, (any && n < ctl[1]) ? 1u : 0u);
    }
}

#define RCHECK(call)                                            \
    do {                                                        \
        int _st = cuda_status((call), #call);                   \
        if (_st != LULESH_OK) return _st;                       \
    } while (0)

int ensure_run_graph(lulesh_set *s)
{
    int st = refresh_graphs(s);
    if (st != LULESH_OK || s->exec_run) return st;
    st = prepare_capture(s);
    if (st != LULESH_OK) return st;
    cudaGraph_t g = nullptr;
    RCHECK(cudaGraphCreate(&g, 0));
    cudaGraphConditionalHandle h;
    st = cuda_status(cudaGraphConditionalHandleCreate(&h, g, 1, cudaGraphCondAssignDefault),
                     "conditional handle");
    cudaGraphNodeParams p = {};
    p.type = cudaGraphNodeTypeConditional;
    p.conditional.handle = h;
    p.conditional.type = cudaGraphCondTypeWhile;
    p.conditional.size = 1;
    cudaGraphNode_t node;
    if (st == LULESH_OK)
        st = cuda_status(cudaGraphAddNode(&node, g, nullptr, 0, &p), "while node");
    if (st == LULESH_OK) {
        cudaGraph_t body = p.conditional.phGraph_out[0];
        st = cuda_status(cudaStreamBeginCaptureToGraph(s->stream, body, nullptr, nullptr, 0,
                                                       cudaStreamCaptureModeThreadLocal),
                         "capture loop body");
        if (st == LULESH_OK) {
            int est = LULESH_OK;
            for (int c = 0; c < kCyclesPerTurn && est == LULESH_OK; ++c)
                est = enqueue_cycle(s, c > 0, c + 1 == kCyclesPerTurn);
            k_run_continue<<<1, 128, 0, s->stream>>>(h, s->dtc, s->njobs, s->run_ctl);
            cudaGraph_t captured = nullptr;
            const int cst = cuda_status(cudaStreamEndCapture(s->stream, &captured), "end capture");
            st = (est != LULESH_OK) ? est : cst;
        }
    }
    if (st == LULESH_OK) st = cuda_status(cudaGraphInstantiate(&s->exec_run, g, 0), "instantiate");
    if (st != LULESH_OK) {
        cudaGraphDestroy(g);
        return st;
    }
    s->graph_run = g;
    return LULESH_OK;
}

}  // namespace
}  // namespace lulesh

using namespace lulesh;

extern "C" int lulesh_run_graph(lulesh_set *s, long long max_cycles)
{
    if (!s) return LULESH_INVALID_ARG;
    int st = ensure_run_graph(s);
    if (st != LULESH_OK) return st;
    const unsigned long long cap = max_cycles > 0 ? (unsigned long long)max_cycles : kDefaultRunCap;
    const unsigned long long ctl[2] = {0ull, cap / kCyclesPerTurn};
    if (ctl[1] > 0) {
        RCHECK(cudaMemcpyAsync(s->run_ctl, ctl, sizeof ctl, cudaMemcpyHostToDevice, s->stream));
        RCHECK(cudaGraphLaunch(s->exec_run, s->stream));
    }
    // the cap's last cycles, fewer than a turn (no work where all jobs are done)
    for (unsigned long long c = 0; c < cap % kCyclesPerTurn; ++c)
        if ((st = enqueue_cycle(s)) != LULESH_OK) return st;
    return run_status(s);  // synchronises the stream
}
