"""The context's host side (csrc/ctx.h) on the CPU, against a CUDA runtime of stubs
that record what they are asked and fail where told to."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
GXX = shutil.which("g++")
pytestmark = pytest.mark.skipif(GXX is None, reason="no C++ compiler")

STUBS = r"""
#include <cstdio>
#include <cstdlib>
#include <set>
#include <string>
#include "ctx.h"
static std::set<void *> waited;
static bool pinned_fails = false;
static size_t handles = 0;
extern "C" {
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { waited.insert(s); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = (cudaStream_t)(++handles * 64); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { *e = (cudaEvent_t)(++handles * 64); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaMalloc(void **p, size_t n) { *p = std::malloc(n); return cudaSuccess; }
cudaError_t cudaFree(void *p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMallocHost(void **p, size_t n) {
  if (pinned_fails) return cudaErrorMemoryAllocation;
  *p = std::malloc(n);
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) { std::free(p); return cudaSuccess; }
}
#define CHECK(c) do { if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); return 1; } } while (0)
int main() {
  pt_ctx x;
  x.stream = (cudaStream_t)32;
"""


def run(tmp_path, body):
    from paintop_b200 import build
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc()))), "include")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(STUBS + body + "\n  return 0;\n}\n")
    r = subprocess.run([GXX, "-std=c++17", "-Wall", "-I", os.path.join(ROOT, "paintop_b200", "csrc"), "-I", cuda,
                        str(src), "-o", str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout


def test_waiting_for_a_failed_call_covers_the_side_streams(tmp_path):
    run(tmp_path, """
  CHECK(x.make_sides(3) == cudaSuccess);
  x.wait_all();
  CHECK(waited.count(x.stream) && waited.size() == 4);
  for (int k = 0; k < 3; ++k) CHECK(waited.count(x.side[k]));
  waited.clear();  // the arena is not freed before they are done
  CHECK(x.reserve(100) && x.reserve(100000) && waited.size() == 4);
  x.release();""")


def test_a_failed_solve_waits_for_the_whole_context():
    text = open(os.path.join(ROOT, "paintop_b200", "csrc", "solver_host.cu")).read()
    settle = text[text.index("~Settle() {"):]
    assert "ctx->wait_all();" in settle[:settle.index("}")]


def test_staging_without_page_locked_memory(tmp_path):
    """A call needs the staging; page-locked memory is a matter of speed."""
    run(tmp_path, """
  pinned_fails = true;
  CHECK(x.reserve_pin(1000) && x.pin && x.pin_cap >= 1000);
  static_cast<char *>(x.pin)[999] = 1;
  CHECK(x.reserve_pin(5000) && x.pin_cap >= 5000);
  pinned_fails = false;
  CHECK(x.reserve_pin(50000) && x.pin_cap >= 50000);
  x.release();
  CHECK(!x.pin && !x.pin_cap);""")
