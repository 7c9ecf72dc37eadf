"""When a substep call is captured and when it is launched directly
(csrc/substep_graph.cuh), on the CPU: the header runs against a fake of the
runtime calls that it makes, in a small host program."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

FAKE = r"""
#include <cstdio>
#include <cstdlib>
#include <string>
#include "substep_graph.cuh"

static int begins, captures, graph_launches, fail_begin, fail_inst, fail_launch, user_capture, live, in_capture;
extern "C" {
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *s) {
  *s = user_capture ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
  if (fail_begin) return cudaErrorUnknown;
  ++begins;
  in_capture = 1;
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) {
  in_capture = 0;
  *g = (cudaGraph_t)8;
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t, unsigned long long) {
  if (fail_inst) return cudaErrorMemoryAllocation;
  ++captures;
  ++live;
  *e = (cudaGraphExec_t)16;
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { --live; return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) {
  if (fail_launch) return cudaErrorMemoryAllocation;
  ++graph_launches;
  return cudaSuccess;
}
static cudaStreamCaptureMode thread_mode = cudaStreamCaptureModeGlobal;
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode *m) {
  const cudaStreamCaptureMode was = thread_mode;
  thread_mode = *m;
  *m = was;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "fake"; }
}

struct Ctx {
  cudaStream_t stream = nullptr;
  bool timing = false;
  int xnp = 0, io_cur = 0;
  int64_t launches = 0;
  std::string err;
  chapsim::SubGraphs sub;
  int direct = 0;
  // a momentum call: three kernels, the G buffers change places
  int call(int ns) {
    const int par = io_cur;
    const int rc = chapsim::run_substep(this, sub.mom[ns][par], [&] {
      if (!in_capture) ++direct;
      launches += 3;
      io_cur = 1 - par;
      return 0;
    });
    if (!rc) io_cur = 1 - par;
    return rc;
  }
  int step() { return call(1) | call(2) | call(3); }
};
#define CHECK(x) do { if (!(x)) { printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)

int main(int argc, char **argv) {
  const std::string what = argv[1];
  Ctx c;
  if (what == "steady") {  // six kinds: two direct calls each, then replays
    for (int s = 0; s < 40; ++s) CHECK(c.step() == 0);
    CHECK(captures == 6 && c.direct == 12 && graph_launches == 120 - 12);
    CHECK(c.launches == 3 * 120 && c.io_cur == 0);
    c.sub.drop();
    CHECK(live == 0);
  } else if (what == "dropped") {  // every `period` steps, 100 times
    const int period = atoi(argv[2]), most = atoi(argv[3]);
    for (int s = 0; s < 100 * period; ++s) {
      if (s % period == 0) c.sub.drop();
      CHECK(c.step() == 0);
    }
    printf("%d captures\n", captures);
    CHECK(most < 0 ? captures == 600 : captures <= most);
    CHECK(c.launches == 900 * period);
  } else if (what == "direct") {  // the caller captures, phases are timed, the coupled section
    user_capture = 1;
    for (int s = 0; s < 10; ++s) CHECK(c.step() == 0);
    user_capture = 0;
    c.timing = true;
    for (int s = 0; s < 10; ++s) CHECK(c.step() == 0);
    c.timing = false;
    c.xnp = 1;
    for (int s = 0; s < 10; ++s) CHECK(c.step() == 0);
    CHECK(captures == 0 && c.direct == 90 && c.launches == 270);
  } else if (what == "fails") {  // no memory for a graph: the calls go on, and capture again after a drop
    int &f = argv[2] == std::string("begin") ? fail_begin : argv[2] == std::string("instantiate") ? fail_inst : fail_launch;
    f = 1;
    for (int s = 0; s < 10; ++s) CHECK(c.step() == 0);
    CHECK(c.direct == 30 && c.launches == 90 && c.io_cur == 0 && graph_launches == 0 && live == 0);
    CHECK(begins <= 6);  // one try a kind
    f = 0;
    c.sub.drop();
    for (int s = 0; s < 10; ++s) CHECK(c.step() == 0);
    CHECK(c.direct == 30 + 12 && graph_launches == 30 - 12 && c.launches == 180);
  }
  CHECK(thread_mode == cudaStreamCaptureModeGlobal);
  return 0;
}
"""


@pytest.fixture(scope="module")
def prog(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("substep_graph")
    src = d / "check.cpp"
    src.write_text(FAKE)
    exe = str(d / "check")
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "chapsim1ww_b200", "csrc"), "-I",
                    os.path.join(CUDA, "include"), str(src), "-o", exe], check=True, capture_output=True)
    return exe


def run(prog, *args):
    r = subprocess.run([prog, *map(str, args)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def test_steady_calls_are_captured_once(prog):
    run(prog, "steady")


@pytest.mark.parametrize("period,most", [(3, 0), (5, 6), (6, 6), (10, 18), (24, -1)])
def test_captures_that_do_not_pay_are_given_up(prog, period, most):
    """DT changed every `period` steps: a kind that is called too few times in
    between is captured a bounded number of times, not each time again."""
    run(prog, "dropped", period, most)


def test_calls_that_launch_directly(prog):
    run(prog, "direct")


@pytest.mark.parametrize("call", ["begin", "instantiate", "launch"])
def test_failed_captures_launch_directly(prog, call):
    run(prog, "fails", call)
