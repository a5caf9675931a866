"""CPU tests of the pools of streams and device blocks (``csrc/pools.cu``) against a fake CUDA runtime.

The file is compiled as plain C++ with fakes of the runtime calls that it makes; a fake can be told
to fail, and counts what is alive.
"""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "gbasis_b200", "csrc")

FAKES = r"""
#include <cstdio>
#include <cstdlib>
#include <map>
#include <vector>
#include "pools.h"
#include "errors.h"
static int fail_event = -1, events = 0, streams = 0;  // fail_event: calls until one fails
static size_t capacity = 0, used = 0;
static std::map<void*, size_t> blocks;
static cudaError_t last = cudaSuccess;
static char next_handle[1 << 16];
static int handles = 0;
extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  ++streams; *s = (cudaStream_t)(next_handle + handles++); return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { --streams; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  if (fail_event == 0) { fail_event = -1; return last = cudaErrorMemoryAllocation; }
  if (fail_event > 0) --fail_event;
  ++events; *e = (cudaEvent_t)(next_handle + handles++); return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t) { --events; return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) {
  if (used + n > capacity) return last = cudaErrorMemoryAllocation;
  used += n; *p = next_handle + handles++; blocks[*p] = n; return cudaSuccess;
}
cudaError_t cudaFree(void* p) { used -= blocks.at(p); blocks.erase(p); return cudaSuccess; }
}
namespace gbx {
int set_error(int code, const char*, ...) { return code; }
int cuda_status(cudaError_t e, const char*) {
  return e == cudaSuccess ? GBX_OK : e == cudaErrorMemoryAllocation ? GBX_ERR_OOM : GBX_ERR_CUDA;
}
}
using namespace gbx;
#define CHECK(c) do { if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); return 1; } } while (0)
"""


def _run(tmp_path, body):
    from gbasis_b200.build import nvcc
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc()))), "include")
    src = tmp_path / "t.cpp"
    src.write_text(FAKES + "int main() {\n" + body + "\n  return 0;\n}\n")
    exe = tmp_path / "t"
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", include, "-I", CSRC, "-I", os.path.join(ROOT, "include"),
                    "-x", "c++", str(src), os.path.join(CSRC, "pools.cu"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout


def test_a_set_stays_usable_after_a_failed_event(tmp_path):
    """Every auxiliary stream has its event, also when an event could not be created once and the
    set is used again, by its owner or through the pool."""
    _run(tmp_path, r"""
  std::unique_ptr<StreamSet> s;
  CHECK(streams_take(0, &s) == GBX_OK);
  for (int n = 0; n < 4; ++n) {
    fail_event = n;  // fails at the (n + 1)-th event of the growth
    CHECK(s->ensure_aux((int)s->aux.size() + 6) != GBX_OK);
    CHECK(s->aux.size() == s->join.size());
    CHECK(s->ensure_aux((int)s->aux.size()) == GBX_OK);
    CHECK(s->aux.size() == s->join.size());
  }
  streams_give(std::move(s), true);
  CHECK(streams_take(0, &s) == GBX_OK);
  CHECK(s->ensure_aux(16) == GBX_OK);
  CHECK(s->aux.size() == 16 && s->join.size() == 16);
  s.reset();
  CHECK(streams == 0 && events == 0);
""")


def test_a_full_device_takes_the_idle_blocks(tmp_path):
    """An allocation that fits without the cache's idle blocks succeeds, leaves no error behind and
    frees them; one that does not fit fails as before, and blocks in use stay."""
    _run(tmp_path, r"""
  capacity = 1000;
  void *a, *b, *c;
  size_t na, nb, nc;
  CHECK(block_alloc(0, &a, 300, &na, "a") == GBX_OK && na == 300);
  CHECK(block_alloc(0, &b, 500, &nb, "b") == GBX_OK);
  block_give(0, b, nb);  // idle: 500 of the 800 in use
  CHECK(block_alloc(0, &c, 600, &nc, "c") == GBX_OK && nc == 600);
  CHECK(cudaGetLastError() == cudaSuccess && used == 900);
  block_give(0, c, nc);
  CHECK(block_alloc(0, &b, 900, &nb, "b") == GBX_ERR_OOM);
  CHECK(used == 300 && blocks.count(a));
  block_give(0, a, na);
  CHECK(block_alloc(0, &b, 200, &nb, "b") == GBX_OK && b == a && nb == 300);  // reused
  block_give(0, b, nb);
  release_pools();
  CHECK(used == 0);
""")
