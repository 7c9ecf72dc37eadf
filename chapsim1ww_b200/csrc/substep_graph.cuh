// Substep calls (chapsim_rk3_mom_tg / _mom_io / _eng_io) replayed as captured
// graphs.  Host code over the runtime API only; the context is a template
// parameter, so that the rules below are tested without a device.
#pragma once
#include <cuda_runtime_api.h>
#include <stdint.h>

namespace chapsim {

// The captured launches of one kind of substep call.
struct SubGraph {
  cudaGraphExec_t exec = nullptr;
  int64_t kernels = 0;
  int calls = 0, replays = 0;
  bool off = false;  // capturing failed: launched directly
};

// A context's captures by NS and the IO's io_cur, and the calls of a kind that
// are launched directly before it is captured.
struct SubGraphs {
  static constexpr int kWait = 2, kWaitMax = 64, kPaid = 8;
  SubGraph mom[4][2], eng[4][2];
  int wait = kWait;
  // The captures go stale when a launch shape, a table or DT changes.  A
  // capture with its instantiation costs about seven replays' gain (60-70 us
  // against 10 us a call on a 32x24x16 IO section), so where one is dropped
  // before kPaid replays the next waits twice as long: with DT changed every
  // 6 steps that section took 362 us a step when every kind was captured at
  // its third call, against 215 this way.
  void drop() {
    bool paid = false, unpaid = false;
    for (auto *set : {mom, eng})
      for (int ns = 0; ns < 4; ++ns)
        for (int par = 0; par < 2; ++par) {
          SubGraph &g = set[ns][par];
          if (g.exec) {
            (g.replays < kPaid ? unpaid : paid) = true;
            cudaGraphExecDestroy(g.exec);
          }
          g = SubGraph();
        }
    if (unpaid)
      wait = wait < kWaitMax ? 2 * wait : kWaitMax;
    else if (paid)
      wait = kWait;
  }
};

// One substep call.  A host's time loop makes the same calls every step, and
// launching a substep's ten to fifteen kernels one by one costs it 2.5 us
// each (on the smallest grids more than they run), so after the first calls of
// a kind the launches are captured once and replayed as one graph.  Those
// first calls, timed phases, the coupled section (its launches reach into the
// TG context) and a stream that the caller is capturing launch directly, and
// so does a kind whose capture fails (a graph takes device memory that a
// launch does not).
template <typename Ctx, typename F> int run_substep(Ctx *ctx, SubGraph &g, F launch) {
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (g.off || ctx->timing || ctx->xnp || g.calls < ctx->sub.wait ||
      cudaStreamIsCapturing(ctx->stream, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) {
    ++g.calls;
    return launch();
  }
  const int par = ctx->io_cur;
  cudaError_t e = cudaSuccess;
  if (!g.exec) {
    cudaGraph_t graph = nullptr;
    const int64_t before = ctx->launches;
    int rc = 0;
    // The caller's thread, or another one in the global mode, may be capturing
    // a stream of its own, and cudaGraphInstantiate is a call that would end
    // that capture: this one has nothing to do with it.
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    cudaThreadExchangeStreamCaptureMode(&mode);
    e = cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) {
      rc = launch();
      e = cudaStreamEndCapture(ctx->stream, &graph);
    }
    g.kernels = ctx->launches - before;
    ctx->launches = before;
    ctx->io_cur = par;  // captured, not run
    if (e == cudaSuccess) e = rc ? cudaErrorUnknown : cudaGraphInstantiate(&g.exec, graph, 0);
    if (graph) cudaGraphDestroy(graph);
    cudaThreadExchangeStreamCaptureMode(&mode);
    if (e != cudaSuccess) g.exec = nullptr;
  }
  if (g.exec) e = cudaGraphLaunch(g.exec, ctx->stream);
  if (e != cudaSuccess) {
    cudaGetLastError();
    if (g.exec) cudaGraphExecDestroy(g.exec);
    g.exec = nullptr;
    g.off = true;
    return launch();
  }
  ++g.replays;
  ctx->launches += g.kernels;
  return 0;
}

}  // namespace chapsim
