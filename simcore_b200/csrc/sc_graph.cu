// sc_step_graph: the reference step loop without host round trips, rebuilds
// decided on the device: captured as one CUDA graph, a WHILE loop of
// Brownian-dynamics steps, or, of small contexts, launched as a chain.
#include "sc_context.h"

#include <optional>

using namespace scapi;

// Contexts whose steps are chained (enqueue_chain) instead of looped in a
// graph.  Per BD step, chain against graph: 2,000 bonds 34.7 us against 40.9
// (FP64) and 24.1 against 30.5 (mixed), 12,000 bonds 38.1 and 39.6, 29.3 and
// 31.8, 16,000 bonds the same; beyond, one cluster's rebuild (125 us at 20,000
// bonds) costs more than the loop's conditional nodes.  The cluster also scans
// one counter per 32 cells; the suspensions of these sizes have up to 11,000.
// A rebuild's candidate pairs cost the cluster about 3 ns each more than the
// rebuild's own kernels, so dense lists take the graph: 12,000 bonds with 8,000
// pairs 28.7 us chained, 31.1 in the graph (mixed), with 34,000 44.1 and 42.8,
// with 160,000 in a buckling network, rebuilt every step, 777 and 334; 2,000
// bonds with 9,300 pairs 44.0 and 48.1, with 23,500 rebuilt every step 293 and
// 259; 300 bonds with 3,600, rebuilt every step, 213 and 202.  64 systems of
// 12,200 bonds and 5,000 pairs, rebuilt every step: 59.9 and 63.5.
static const int kChainBonds = 12288;
static const int kChainGroups = 32768;
static const int kChainPairs = 16384;
static const int kChainPairsPerBond = 6;
// BD steps queued at a time: what a run that stops early still launches for
// nothing (about 2 us a launch), against a synchronisation and an empty queue
// (about 15 us) per 9 ms or more of steps.
static const int kChainPiece = 512;

extern "C" {

// The launches of one BD step after its rebuild decision.
static int bd_step(sc_ctx *c, bool fuse, bool chain) {
  const int interaction = c->desc.interaction_flag ? 1 : 0;
  int n = 0;
  for (int half = 0; half < 2; ++half) {
    const int rb = half == 0 ? c->rbuf : 1 - c->rbuf;
    // A graph body's first kernel follows a conditional rebuild node (or the
    // body's start), not a kernel: it is launched without the programmatic
    // attribute.  A chained step's follows the control kernel, which may write
    // the pair list: the pair kernel then waits first.
    // The second half is the even (full) step: crosslink tethers first.
    if (half == 1 && interaction) n += sc::launch_tether(c->k, c->d, c->st);
    if (interaction && !fuse) {
      std::optional<sc::PdlOff> alone;
      if (half == 0 && !chain) alone.emplace();
      n += sc::launch_pairs(c->k, c->d, rb, c->prec, (int)(c->np + c->np / 8), c->st, c->npx,
                            c->pair_block, half == 0 && chain, chain);
    }
    if (interaction && c->k.thermo) n += sc::launch_thermo(c->k, c->d, c->prec, c->st);
    if (half == 0 && (!interaction || fuse)) {
      sc::PdlOff off;
      n += sc::launch_integrate(c->k, c->d, c->nblocks, c->C, 1, rb, interaction, c->capture, c->prec,
                           c->fast, c->st, fuse);
    } else {
      n += sc::launch_integrate(c->k, c->d, c->nblocks, c->C, half == 0 ? 1 : 0, rb, interaction,
                           c->capture, c->prec, c->fast, c->st, fuse);
    }
  }
  return n;
}

// Steps launched one after another with a control kernel between them, for
// small contexts: no conditional nodes.
static void enqueue_chain(sc_ctx *c, int bd) {
  const bool fuse = fused_pairs(c);
  const int stoch = c->desc.stoch_flag ? 1 : 0;
  c->graph_fused = fuse;
  for (int i = 0; i <= bd; ++i) {
    c->launches += sc::launch_step_control(c->k, c->d, c->rb, c->prec, stoch, i == 0 ? bd : 0,
                                           i > 0, i < bd, host_report(c), c->st);
    if (i < bd) c->launches += bd_step(c, fuse, true);
  }
  c->launches += sc::launch_report(c->d, host_report(c), 1, c->st);
}

// Captures one graph: head (loop condition, first rebuild decision) ->
// WHILE (loop_count > 0) { IF(rebuild) -> midstep -> full step -> tail (next
// rebuild decision) } -> report to the host.  Built for the current geometry-buffer parity; every
// BD step returns the parity to where it started.
static sc_status build_graph(sc_ctx *c) {
  drop_graph(c);
  cudaGraph_t g = nullptr;
  CK(cudaGraphCreate(&g, 0));
  const int interaction = c->desc.interaction_flag ? 1 : 0;
  cudaGraphConditionalHandle h_loop, h_if = 0;
  CK(cudaGraphConditionalHandleCreate(&h_loop, g, 0, 0));
  // The rebuild condition is set by the head and by every tail (the decision
  // for the step after), so it belongs to the outer graph, like the loop's.
  if (interaction) CK(cudaGraphConditionalHandleCreate(&h_if, g, 0, 0));
  // head kernel: sets the loop condition and decides the first rebuild
  CK(cudaStreamBeginCaptureToGraph(c->st, g, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed));
  sc::launch_loop_head(c->d, host_report(c), h_loop, h_if, interaction, c->st);
  cudaStreamCaptureStatus cs;
  const cudaGraphNode_t *deps = nullptr;
  size_t ndeps = 0;
  CK(cudaStreamGetCaptureInfo(c->st, &cs, nullptr, nullptr, &deps, &ndeps));
  std::vector<cudaGraphNode_t> head(deps, deps + ndeps);
  CK(cudaStreamEndCapture(c->st, &g));
  // WHILE node
  cudaGraphNodeParams wp = {};
  wp.type = cudaGraphNodeTypeConditional;
  wp.conditional.handle = h_loop;
  wp.conditional.type = cudaGraphCondTypeWhile;
  wp.conditional.size = 1;
  cudaGraphNode_t wnode;
  CK(cudaGraphAddNode(&wnode, g, head.data(), head.size(), &wp));
  cudaGraph_t body = wp.conditional.phGraph_out[0];
  std::vector<cudaGraphNode_t> tail;
  if (interaction) {
    cudaGraphNodeParams ip = {};
    ip.type = cudaGraphNodeTypeConditional;
    ip.conditional.handle = h_if;
    ip.conditional.type = cudaGraphCondTypeIf;
    ip.conditional.size = 1;
    cudaGraphNode_t inode;
    CK(cudaGraphAddNode(&inode, body, nullptr, 0, &ip));
    cudaGraph_t rb = ip.conditional.phGraph_out[0];
    CK(cudaStreamBeginCaptureToGraph(c->st, rb, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed));
    long long launches = c->launches;
    rebuild_enqueue(c, true);
    c->launches = launches;
    CK(cudaStreamEndCapture(c->st, &rb));
    tail.push_back(inode);
  }
  CK(cudaStreamBeginCaptureToGraph(c->st, body, tail.empty() ? nullptr : tail.data(), nullptr,
                                   tail.size(), cudaStreamCaptureModeRelaxed));
  const bool fuse = fused_pairs(c);
  c->graph_fused = fuse;
  bd_step(c, fuse, false);
  sc::launch_loop_tail(c->d, c->desc.stoch_flag ? 1 : 0, h_loop, h_if, interaction, c->st);
  CK(cudaStreamEndCapture(c->st, &body));
  // What the host reads afterwards.
  CK(cudaStreamBeginCaptureToGraph(c->st, g, &wnode, nullptr, 1, cudaStreamCaptureModeRelaxed));
  sc::launch_report(c->d, host_report(c), 1, c->st);
  CK(cudaStreamEndCapture(c->st, &g));
  CK(cudaGetLastError());
  cudaError_t e = cudaGraphInstantiate(&c->graph_exec, g, 0);
  cudaGraphDestroy(g);
  if (e != cudaSuccess) {
    c->graph_exec = nullptr;
    return fail(c, SC_ERR_CUDA, "graph instantiation failed: %s", cudaGetErrorString(e));
  }
  c->graph_rbuf = c->rbuf;
  return SC_OK;
}

// Whether a captured run, whose pair count is known, is launched as a chain.
static bool chained(const sc_ctx *c) {
  if (!c->desc.interaction_flag || c->run_form == SC_RUN_GRAPH) return false;
  return c->run_form == SC_RUN_CHAIN ||
         (c->nb <= kChainBonds && c->rb.n_groups <= kChainGroups && c->np <= kChainPairs &&
          c->np <= (long long)kChainPairsPerBond * c->nb);
}

sc_status sc_set_run_form(sc_ctx *c, sc_run_form form) {
  if (!c || (form != SC_RUN_AUTO && form != SC_RUN_GRAPH && form != SC_RUN_CHAIN))
    return SC_ERR_INVALID_ARG;
  c->run_form = form;
  return SC_OK;
}

sc_status sc_step_graph(sc_ctx *c, int n) {
  if (!c || !c->loaded || n < 0) return SC_ERR_INVALID_ARG;
  CK(cudaSetDevice(c->desc.device));
  // Align to a midstep with the host-driven loop, then run whole BD steps.
  if (!c->midstep && n > 0) {
    CKS(step_once(c));
    --n;
  }
  int bd = n / 2;
  if (bd > 0) {
    CKS(thermo_reserve(c, 2 * (long long)bd));
    // The list must have room to grow by half before a captured run.
    if (!c->np_known) CKS(sync_pair_count(c));
    if (c->reps.size() == 1 && c->np + c->np / 2 > c->pcap)
      CKS(ensure_pair_capacity(c, c->np + c->np / 2));
    if (!c->gev0) {
      CK(cudaEventCreate(&c->gev0));
      CK(cudaEventCreate(&c->gev1));
    }
    c->graph_ms = 0.0;
    // A rebuild whose list outgrows its segment stops the run at that BD
    // step, with nothing past the rebuild done; the list then grows, the
    // rebuild is redone host-side and the run resumes with that step.
    // (A chain of more than kChainPiece steps is queued in pieces.)
    for (int attempt = 0; bd > 0;) {
      if (attempt == 8) return fail(c, SC_ERR_LIST_OVERFLOW, "pair list kept overflowing inside captured runs");
      const bool chain = chained(c);
      if (!chain && (!c->graph_exec || c->graph_rbuf != c->rbuf)) CKS(build_graph(c));
      // The head reads the step count and the last node writes everything
      // the host looks at, both in pinned memory: no copies, one
      // synchronisation per launch.
      const int queued = chain ? std::min(bd, kChainPiece) : bd;
      *c->h_loop = queued;
      CK(cudaEventRecord(c->gev0, c->st));
      if (chain) {
        enqueue_chain(c, queued);
        CK(cudaGetLastError());
      } else {
        CK(cudaGraphLaunch(c->graph_exec, c->st));
      }
      CK(cudaEventRecord(c->gev1, c->st));
      c->pairs_ready = false;
      CK(cudaStreamSynchronize(c->st));
      take_pair_count(c);
      const unsigned st = c->hb->status;
      const long long nr0 = c->hb->rebuilds[0], nr1 = c->hb->rebuilds[1];
      const bool overflow = (st & sc::ST_LIST_OVERFLOW) != 0u;
      // BD steps completed: all of them, or those before the stopped one.  (A run
      // that an error ends counts as run to its end.)
      const int done = overflow ? queued - *c->h_loop : st ? bd : queued;
      if (c->graph_fused && done > 0) c->slots_stale = true;
      c->i_step += 2 * (long long)done;
      if (c->desc.stoch_flag) c->mcount += done;
      {
        float ms = 0.f;
        CK(cudaEventElapsedTime(&ms, c->gev0, c->gev1));
        c->graph_ms += ms;
      }
      // Kernels the graph ran: loop head and report, per BD step the two tether
      // kernels (mesh lambdas, anchor forces) + 2 steps + tail (the stopped
      // step's too), per rebuild the captured sequence.  A step is its pair
      // kernel (unless fused; near-parallel pairs are evaluated in place),
      // thermo and one or two integrator kernels.
      const int int_l = (c->d.n_tm > 0 ? 1 : 0) + (c->nblocks > 0 ? 1 : 0);
      const long long per_bd =
          c->desc.interaction_flag
              ? 1 + (c->d.nx ? 2 : 0) +
                    2 * ((c->graph_fused ? 0 : 1) + int_l + (c->k.thermo ? 1 : 0))
              : 1 + 2 * int_l;
      if (!chain)
        c->launches += 2 + (long long)(done + (overflow ? 1 : 0)) * per_bd +
                       (nr1 - nr0) * c->rebuild_kernels;
      bd -= done;
      if (!overflow) {
        CKS(check_status(c));  // status and maxima were read with the counters
        continue;
      }
      ++attempt;
      if (st & ~sc::ST_LIST_OVERFLOW) {
        CKS(readback(c));  // reports the other error
        return fail(c, SC_ERR_LIST_OVERFLOW, "pair list overflow inside a captured run");
      }
      if (c->reps.size() != 1)
        return fail(c, SC_ERR_LIST_OVERFLOW, "a system's pair list outgrew its segment inside a captured run");
      const unsigned clear = 0u;
      CK(cudaMemcpyAsync(c->d.status, &clear, sizeof(unsigned), cudaMemcpyHostToDevice, c->st));
      CKS(sync_pair_count(c));
      CKS(grow_after_overflow(c));
      // The stopped step's due flag is still set: redo its rebuild, with
      // headroom for the rest of the run.
      CKS(rebuild(c));
      if (c->np + c->np / 2 > c->pcap) CKS(ensure_pair_capacity(c, c->np + c->np / 2));
    }
    unsigned st = c->hb->status;
    if (st & sc::ST_UNPHYSICAL) return fail(c, SC_ERR_UNPHYSICAL, "Unphysical result");
  }
  if (n % 2) CKS(step_once(c));
  return SC_OK;
}

}  // extern "C"
