"""A capture whose work throws is ended and its graph destroyed: the stream is
not left capturing, so the engine's later calls fail or succeed by themselves.
The capture of csrc/capture.h runs here against a fake runtime."""
import os
import re
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "web-exoplasim_b200", "csrc")

FAKE = r"""
#include "capture.h"
#include <cstdio>
static int begun, ended, destroyed, cleared, graphs[4];
static cudaError_t begin_status, end_status;
cudaError_t cudaStreamBeginCapture(cudaStream_t, enum cudaStreamCaptureMode) {
  if (begin_status == cudaSuccess) ++begun;
  return begin_status;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  *g = end_status == cudaSuccess ? (cudaGraph_t)&graphs[ended] : nullptr;
  ++ended;
  return end_status;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { ++destroyed; return cudaSuccess; }
cudaError_t cudaGetLastError() { ++cleared; return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }

// begun, ended and destroyed after a capture whose work throws or not
static void report(const char* name, cudaError_t at_begin, cudaError_t at_end, bool throws, bool keep) {
  begun = ended = destroyed = 0;
  begin_status = at_begin, end_status = at_end;
  bool caught = false;
  try {
    exogcm::Graph graph;
    exogcm::Capture capture(nullptr);
    if (throws) throw exogcm::Error(-3, "work");
    capture.end(graph);
    if (keep) graph.release();
  } catch (const exogcm::Error&) { caught = true; }
  std::printf("%s %d %d %d %d\n", name, begun, ended, destroyed, (int)caught);
}
int main() {
  report("kept", cudaSuccess, cudaSuccess, false, true);
  report("dropped", cudaSuccess, cudaSuccess, false, false);
  report("work_throws", cudaSuccess, cudaSuccess, true, true);
  report("work_throws_and_end_fails", cudaSuccess, cudaErrorUnknown, true, true);
  report("end_fails", cudaSuccess, cudaErrorUnknown, false, true);
  report("begin_fails", cudaErrorUnknown, cudaSuccess, false, true);
}
"""


def test_a_capture_is_ended_whatever_its_work_does(tmp_path):
    source, program = tmp_path / "fake.cpp", tmp_path / "fake"
    source.write_text(FAKE)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, "-I", "/usr/local/cuda/include", str(source), "-o", str(program)],
                   check=True)
    out = subprocess.run([str(program)], check=True, capture_output=True, text=True).stdout
    got = {line.split()[0]: [int(v) for v in line.split()[1:]] for line in out.splitlines()}
    # captures begun, ended, graphs destroyed, errors raised
    assert got == {"kept": [1, 1, 0, 0], "dropped": [1, 1, 1, 0], "work_throws": [1, 1, 1, 1],
                   "work_throws_and_end_fails": [1, 1, 0, 1], "end_fails": [1, 1, 0, 1], "begin_fails": [0, 0, 0, 1]}


def test_every_capture_is_one_that_ends():
    for name in os.listdir(CSRC):
        if name != "capture.h":
            assert not re.search(r"cudaStream(?:Begin|End)Capture\s*\(", open(os.path.join(CSRC, name)).read()), name
