"""What the launchers keep from one launch to the next, against fakes of the runtime calls that they make (no GPU)."""
import os
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "fluidmoe_b200" / "csrc"
CUDA = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda")) / "include"

pytestmark = pytest.mark.skipif(shutil.which("g++") is None or not (CUDA / "cuda_runtime.h").exists(),
                                reason="needs g++ and the CUDA headers")


def _run(tmp_path, program):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(program)
    subprocess.run(["g++", "-std=c++17", "-Wno-deprecated-declarations", f"-I{CSRC}", f"-I{CUDA}", str(src), "-o", str(exe),
                    "-lpthread"], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert res.returncode == 0, res.stdout + res.stderr


CHECK = """
#include <cstdio>
#include <cstdlib>
#define CHECK(x) do { if (!(x)) { printf("line %d: %s\\n", __LINE__, #x); exit(1); } } while (0)
"""


def test_state_of_a_stream(tmp_path):
    """A state for each device and stream id: not shared by a stream that got a destroyed one's handle, none under
    capture, for a stream without an id or for the 65th stream, and the same one at every later launch."""
    _run(tmp_path, CHECK + """
#include "include/stream_table.h"
static int dev = 0;
static unsigned long long id = 1;
static cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
static cudaError_t capturing = cudaSuccess, ids = cudaSuccess;
extern "C" cudaError_t cudaGetDevice(int* d) { *d = dev; return cudaSuccess; }
extern "C" cudaError_t cudaStreamGetId(cudaStream_t, unsigned long long* i) { *i = id; return ids; }
extern "C" cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* c) { *c = cap; return capturing; }
extern "C" cudaError_t cudaGetLastError() { return cudaSuccess; }
struct State { int n = 0; };
int main() {
  fm::StreamTable<State> t;
  const cudaStream_t handle = (cudaStream_t)0x1234;
  State *a = nullptr, *b = nullptr;
  CHECK(t.find(handle, &a) && a != nullptr);
  a->n = 7;
  CHECK(t.find(handle, &b) && b == a);
  id = 2;                                      // destroyed, and the handle given to another stream
  CHECK(t.find(handle, &b) && b != nullptr && b != a && b->n == 0);
  dev = 1;
  id = 1;
  CHECK(t.find(handle, &b) && b != nullptr && b != a);
  dev = 0;
  cap = cudaStreamCaptureStatusActive;
  CHECK(t.find(handle, &b) && b == nullptr);
  cap = cudaStreamCaptureStatusNone;
  capturing = cudaErrorStreamCaptureImplicit;
  CHECK(!t.find(handle, &b) && b == nullptr);
  capturing = cudaSuccess;
  ids = cudaErrorInvalidResourceHandle;
  CHECK(t.find(handle, &b) && b == nullptr);
  ids = cudaSuccess;
  for (id = 3; id <= 63; ++id) CHECK(t.find(handle, &b) && b != nullptr);
  id = 64;                                     // the 65th
  CHECK(t.find(handle, &b) && b == nullptr);
  id = 1;
  CHECK(t.find(handle, &b) && b == a && a->n == 7);
}
""")


def test_shared_memory_limit_of_every_device(tmp_path):
    """The limit is raised on each device that launches the kernel, once; a refusal is tried again."""
    _run(tmp_path, CHECK + """
#include "include/fm_smem.h"
static int dev = 0, raised = 0;
static cudaError_t answer = cudaSuccess;
extern "C" cudaError_t cudaGetDevice(int* d) { *d = dev; return cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { ++raised; return answer; }
int main() {
  static std::atomic<unsigned long long> done{0}, other[2];
  answer = cudaErrorInvalidValue;
  CHECK(fm::allow_smem(&dev, 1, done) == cudaErrorInvalidValue && raised == 1);
  answer = cudaSuccess;
  for (int i = 0; i < 2; ++i) CHECK(fm::allow_smem(&dev, 1, done) == cudaSuccess && raised == 2);
  dev = 1;
  for (int i = 0; i < 2; ++i) CHECK(fm::allow_smem(&dev, 1, done) == cudaSuccess && raised == 3);
  dev = 63;
  for (int i = 0; i < 2; ++i) CHECK(fm::allow_smem(&dev, 1, done) == cudaSuccess && raised == 4);
  dev = 64;
  for (int i = 0; i < 2; ++i) CHECK(fm::allow_smem(&dev, 1, done) == cudaSuccess && raised == 5 + i);
  dev = 0;
  CHECK(fm::allow_smem(&dev, 1, done) == cudaSuccess && raised == 6);
  CHECK(fm::allow_smem(&dev, 1, other[1]) == cudaSuccess && raised == 7);
}
""")
