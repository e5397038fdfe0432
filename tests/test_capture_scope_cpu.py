"""Graph capture in the solvers (csrc/gbfe_capture.h) on pretended streams: an exception on the way ends the capture,
drops the graph and puts the context's flags back; no kernel is launched."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "dft-efe_gb300" / "csrc"
CUDA = Path(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc").resolve().parent.parent / "include"

SOURCE = r"""
#include "gbfe_capture.h"
#include <cstdio>
#include <stdexcept>
using namespace gbfe;
static bool open_capture = false, refuse = false;
static int graphs = 0;
extern "C" cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
  if (refuse) return cudaErrorStreamCaptureUnsupported;
  open_capture = true;
  return cudaSuccess;
}
extern "C" cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) {
  open_capture = false;
  *g = reinterpret_cast<cudaGraph_t>(&graphs);
  ++graphs;
  return cudaSuccess;
}
extern "C" cudaError_t cudaGraphDestroy(cudaGraph_t) { --graphs; return cudaSuccess; }
extern "C" cudaError_t cudaGetLastError() { return cudaSuccess; }
#define CHECK(c) do { if (!(c)) { printf("line %d: %s\n", __LINE__, #c); return 1; } } while (0)
int main() {
  bool capturing = false;
  int profiling = 1;
  bool thrown = false;
  try {
    const Restore<int> off(profiling, 0);
    CaptureScope c(nullptr, capturing);
    CHECK(c.begin() == cudaSuccess && capturing && open_capture && profiling == 0);
    throw std::runtime_error("a launch failed");
  } catch (const std::exception &) {
    thrown = true;
  }
  CHECK(thrown && !capturing && !open_capture && graphs == 0 && profiling == 1);
  cudaGraph_t g = nullptr;
  {
    CaptureScope c(nullptr, capturing);
    CHECK(c.begin() == cudaSuccess);
    CHECK(c.end(&g) == cudaSuccess && g && !capturing);
  }
  CHECK(graphs == 1 && !open_capture);
  refuse = true;
  {
    CaptureScope c(nullptr, capturing);
    CHECK(c.begin() != cudaSuccess && !capturing);
  }
  CHECK(graphs == 1);
  return 0;
}
"""


def test_an_exception_ends_the_capture(tmp_path):
    if not shutil.which("g++") or not (CUDA / "cuda_runtime_api.h").exists():
        pytest.skip("g++ or the CUDA headers are not available")
    (tmp_path / "t.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{CSRC}", f"-I{CUDA}", str(tmp_path / "t.cpp"), "-o",
                    str(tmp_path / "t")], check=True)
    r = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.parametrize("path", sorted(CSRC.glob("*.cu")), ids=lambda p: p.name)
def test_captures_go_through_the_scope(path):
    text = path.read_text()
    assert "cudaStreamBeginCapture" not in text and "capturing = true" not in text
