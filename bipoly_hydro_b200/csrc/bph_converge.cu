// bph_converge.cu -- the cycle loop of the converged solves on the device.
//
// A converged solve repeats an ADI cycle until the potential stops
// changing: FP64 (bph_solve_converged) copies the slot array, runs nsteps
// ADI steps and measures ||phi - phi_prev|| / ||phi||; the mixed form
// (bph_solve_converged_mixed) runs one FP32 refinement cycle that reports
// ||delta|| / ||phi|| itself.  Instead of a host round trip per cycle, the
// loop is one CUDA graph: a cycle, then a `while` node whose body holds the
// further ones.  After each cycle k_conv_check reduces the per-slot norms,
// applies the stopping rule and sets the node's condition; the host
// reads the cycle count once at the end.  The graph is built by stream
// capture of the same launchers the host loop uses, once per context,
// schedule and kernel choice.
#include <cmath>
#include <vector>

#include "bph_internal.cuh"

namespace bph {
namespace {

constexpr int kCheckThreads = 256;
// The first cycle runs ahead of the while node, which a solve of one cycle then
// does not enter.  Cycles per pass of the node's body where a cycle can be
// skipped: an iteration of the node costs more than the two launches of a
// skipped cycle, and most solves take three or four cycles.  (All four in the
// body: 127 us for the one cycle of a solve that starts converged at
// 66 x 66 x 64, 112 mixed; one ahead: 119, by now 110, and 104.)
constexpr int kBodyCycles = 3;

__global__ void k_conv_init(ConvState *st, double tol, int max_cycles, int mixed, double least) {
    st->tol = tol;
    st->prev = INFINITY;
    st->upd = INFINITY;
    st->max_cycles = max_cycles;
    st->cycles = 0;
    st->mixed = mixed;
    st->least = least;
    st->done = 0;
}

// red[2 i] = sum over slot i of |update|^2, red[2 i + 1] = |phi|^2 (Parseval
// weights included).  Fixed-order reduction (deterministic).
__global__ void __launch_bounds__(kCheckThreads) k_conv_check(const double *__restrict__ red, int N, ConvState *st,
                                                              cudaGraphConditionalHandle cond, bool last) {
    __shared__ double sn[kCheckThreads], sd[kCheckThreads];
    if (st->done) {
        if (last && threadIdx.x == 0) cudaGraphSetConditional(cond, 0u);
        return;
    }
    double num = 0.0, den = 0.0;
    for (int i = threadIdx.x; i < N; i += kCheckThreads) {
        num += red[2 * i];
        den += red[2 * i + 1];
    }
    sn[threadIdx.x] = num;
    sd[threadIdx.x] = den;
    __syncthreads();
    for (int w = kCheckThreads / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) {
            sn[threadIdx.x] += sn[threadIdx.x + w];
            sd[threadIdx.x] += sd[threadIdx.x + w];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        const double upd = sd[0] > 0.0 ? sqrt(sn[0] / sd[0]) : sqrt(sn[0]);
        const int cyc = st->cycles + 1;
        // Stop at the tolerance or the cycle limit; the mixed form also when a
        // cycle no longer halves the update (its FP32 solves are then at
        // their accuracy; FP64 cycles: at the least update) or the update is
        // not finite.
        bool stop = (upd <= st->tol) || (cyc >= st->max_cycles);
        if (st->mixed) stop = stop || !(upd == upd) || (upd > 0.5 * st->prev) || upd <= st->least;
        st->cycles = cyc;
        st->upd = upd;
        st->prev = upd;
        st->done = stop ? 1 : 0;
        if (last) cudaGraphSetConditional(cond, stop ? 0u : 1u);
    }
}

}  // namespace

// Captures reps cycles of a converged form and their checks on cs into graph g;
// past the first, a cycle returns at once when the loop has stopped.
static cudaError_t capture_cycles(bph_ctx *c, Schedule &s, bool mixed, bool modal, int reps, cudaStream_t cs,
                                  cudaGraph_t g, cudaGraphConditionalHandle cond,
                                  std::vector<cudaGraphNode_t> *last_nodes) {
    cudaError_t e = cudaStreamBeginCaptureToGraph(cs, g, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) return e;
    cudaStream_t keep = c->stream;
    const bool keep_pdl = c->pdl;
    c->stream = cs;
    c->pdl = false;  // plain serial edges between the cycles
    cudaError_t ce = cudaSuccess;
    for (int r = 0; r < reps && ce == cudaSuccess; ++r) {
        const int *skip = r > 0 ? &c->d_conv->done : nullptr;
        if (modal) {
            ce = launch_modal_cycle(c, s, c->d_modY, c->d_prev, mixed ? nullptr : c->d_modpre, 1, c->d_modnorm, skip);
        } else if (mixed) {
            ce = launch_adi_defect(c, s, skip);
        } else if (c->adi_seg) {  // the update norms come from the sweep's write-back
            ce = launch_adi(c, s, 0, s.nsteps, false, nullptr, nullptr, 1, nullptr, c->d_red);
        } else {
            ce = cudaMemcpyAsync(c->d_prev, c->d_P, sizeof(double) * (size_t)c->N * c->nplane,
                                 cudaMemcpyDeviceToDevice, cs);
            if (ce == cudaSuccess) ce = launch_adi(c, s, 0, s.nsteps, false);
            if (ce == cudaSuccess) ce = launch_update_norm(c, c->d_red);
        }
        if (ce == cudaSuccess) {
            k_conv_check<<<1, kCheckThreads, 0, cs>>>(modal ? c->d_modnorm : c->d_red,
                                                      modal ? c->N * modal_groups(c) : c->N, c->d_conv, cond,
                                                      r + 1 == reps);
            ce = cudaGetLastError();
        }
        ++c->launches;
    }
    c->stream = keep;
    c->pdl = keep_pdl;
    if (ce == cudaSuccess && last_nodes) {
        cudaStreamCaptureStatus status;
        const cudaGraphNode_t *nodes = nullptr;
        size_t count = 0;
        ce = cudaStreamGetCaptureInfo(cs, &status, nullptr, nullptr, &nodes, &count);
        if (ce == cudaSuccess) last_nodes->assign(nodes, nodes + count);
    }
    cudaGraph_t into = nullptr;
    e = cudaStreamEndCapture(cs, &into);
    return e == cudaSuccess ? ce : e;
}

// Builds the graph of one converged form on the context's current arrays and
// schedule s (the cycles captured from the launchers): a cycle, then a while
// node over further ones.
static int build_conv_graph(bph_ctx *c, Schedule &s, bool mixed, cudaGraphExec_t *out) {
    *out = nullptr;
    const bool modal = modal_converged(c, s, mixed) && (mixed || c->d_modpre);
    cudaGraph_t g = nullptr;
    cudaStream_t cs = nullptr;
    cudaGraphExec_t exec = nullptr;
    cudaError_t e = cudaGraphCreate(&g, 0);
    cudaGraphConditionalHandle cond = 0;
    if (e == cudaSuccess) e = cudaGraphConditionalHandleCreate(&cond, g, 1, cudaGraphCondAssignDefault);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking);
    std::vector<cudaGraphNode_t> after;
    if (e == cudaSuccess) e = capture_cycles(c, s, mixed, modal, 1, cs, g, cond, &after);
    cudaGraphNodeParams p = {};
    cudaGraphNode_t node = nullptr;
    if (e == cudaSuccess) {
        p.type = cudaGraphNodeTypeConditional;
        p.conditional.handle = cond;
        p.conditional.type = cudaGraphCondTypeWhile;
        p.conditional.size = 1;
        e = cudaGraphAddNode(&node, g, after.data(), after.size(), &p);
    }
    const bool skips = modal || (mixed && c->mixed_kind == BPH_MIXED_DIRECT);
    if (e == cudaSuccess)
        e = capture_cycles(c, s, mixed, modal, skips ? kBodyCycles : 1, cs, p.conditional.phGraph_out[0], cond, nullptr);
    if (e == cudaSuccess) e = cudaGraphInstantiate(&exec, g, 0);
    if (cs) cudaStreamDestroy(cs);
    if (g) cudaGraphDestroy(g);
    if (e != cudaSuccess) {
        cudaGetLastError();
        if (exec) cudaGraphExecDestroy(exec);
        return cuda_fail(e, "converged-loop graph");
    }
    *out = exec;
    return BPH_OK;
}

int conv_loop_device(bph_ctx *c, Schedule &s, bool mixed, double tol, int max_cycles) {
    int rc;
    if (!c->d_conv) {
        cudaError_t e = cudaMalloc((void **)&c->d_conv, sizeof(ConvState));
        if (e != cudaSuccess) {
            cudaGetLastError();
            return cuda_fail(e, "cudaMalloc(converged-loop state)");
        }
        c->bytes += sizeof(ConvState);
    }
    ConvGraph &cg = c->conv[mixed ? 1 : 0];
    const bool modal = modal_converged(c, s, mixed) && (mixed || c->d_modpre);
    const int kind = modal ? -2 : mixed ? (c->mixed_kind * 2 + (c->mixed_pf ? 1 : 0)) : 0;
    if (!cg.exec || cg.build_id != s.build_id || cg.kind != kind) {
        if (cg.exec) cudaGraphExecDestroy(cg.exec);
        cg.exec = nullptr;
        if ((rc = build_conv_graph(c, s, mixed, &cg.exec))) return rc;
        cg.build_id = s.build_id;
        cg.kind = kind;
    }
    ++c->launches;
    k_conv_init<<<1, 1, 0, c->stream>>>(c->d_conv, tol, max_cycles, mixed ? 1 : 0, modal ? kLeastUpdate : 0.0);
    BPH_CUDA(cudaGetLastError());
    BPH_CUDA(cudaGraphLaunch(cg.exec, c->stream));
    return BPH_OK;
}

void conv_graph_drop(ConvGraph &cg) {
    if (cg.exec) cudaGraphExecDestroy(cg.exec);
    cg = ConvGraph();
}

void conv_graphs_free(bph_ctx *c) {
    for (ConvGraph &cg : c->conv) conv_graph_drop(cg);
    if (c->d_conv) cudaFree(c->d_conv);
    c->d_conv = nullptr;
}

}  // namespace bph
