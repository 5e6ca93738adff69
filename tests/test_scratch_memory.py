"""Device scratch kept between stage calls (geye_gb300/csrc/memory.cu), run on the host against a
device of 100 MB that counts: an allocation that does not fit takes what idle contexts keep, never what
a call has in use; a call that needs less than an earlier one fits where that one would not; everything
is given back; contexts on several threads."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = "/usr/local/cuda/include"

HARNESS = r"""
#include <assert.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <thread>
#include "runtime.h"
using namespace geye;

static std::mutex mu;
static std::map<void *, size_t> live;
static size_t in_use = 0;
static thread_local cudaError_t last = cudaSuccess;
static const size_t MB = 1 << 20, kRoom = 100 * MB;
extern "C" {
cudaError_t cudaMalloc(void **p, size_t n) {
  std::lock_guard<std::mutex> g(mu);
  if (in_use + n > kRoom) return last = cudaErrorMemoryAllocation;
  *p = malloc(n);
  live[*p] = n;
  in_use += n;
  return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
  std::lock_guard<std::mutex> g(mu);
  auto it = live.find(p);
  if (it == live.end()) abort();   // (freed twice)
  in_use -= it->second;
  live.erase(it);
  free(p);
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaGetLastError(void) { const cudaError_t e = last; last = cudaSuccess; return e; }
const char *cudaGetErrorString(cudaError_t) { return "out of memory"; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaFreeHost(void *) { return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
}
namespace geye {
void set_error(const std::string &) {}
bool injected(geye_ctx *, const char *) { return false; }
}
#define CHECK(c) do { if (!(c)) { fprintf(stderr, "line %d: %s\n", __LINE__, #c); exit(1); } } while (0)

int main() {
  {
    geye_ctx a, b;
    DevBuf x(&a.scratch), big;
    CHECK(x.alloc(&a, 60 * MB) == GEYE_OK);
    memset(x.p, 1, 60 * MB);
    CHECK(big.alloc(&b, 80 * MB) == GEYE_ERR_NOMEM);   // a's call has it
    CHECK(in_use == 60 * MB && static_cast<char *>(x.p)[60 * MB - 1] == 1);
    cudaGetLastError();
    a.scratch.reset();
    CHECK(in_use == 60 * MB);                          // kept
    CHECK(big.alloc(&b, 80 * MB) == GEYE_OK);          // taken
    CHECK(last == cudaSuccess && in_use == 80 * MB);
    // a's next call is smaller than the one before: 60 MB do not fit, what it needs does
    DevBuf y(&a.scratch), z(&a.scratch);
    CHECK(y.alloc(&a, 10 * MB) == GEYE_OK && last == cudaSuccess);
    CHECK(z.alloc(&a, 30 * MB) == GEYE_ERR_NOMEM);
    a.scratch.reset();
    big.release();
    DevBuf w(&a.scratch);
    CHECK(w.alloc(&a, 5 * MB) == GEYE_OK);
    a.scratch.reset();
  }
  CHECK(in_use == 0 && live.empty());
  {   // the scratch of a context that another device's call cannot use stays
    geye_ctx a, b;
    a.device = 1;
    DevBuf x(&a.scratch), big;
    CHECK(x.alloc(&a, 60 * MB) == GEYE_OK);
    a.scratch.reset();
    CHECK(big.alloc(&b, 80 * MB) == GEYE_ERR_NOMEM && in_use == 60 * MB);
  }
  CHECK(in_use == 0);
  {   // stage calls of four contexts and plans that come and go
    std::vector<std::thread> threads;
    for (int t = 0; t < 4; t++)
      threads.emplace_back([t] {
        geye_ctx c;
        unsigned s = t + 1;
        auto rnd = [&s](unsigned n) { return (s = s * 1664525u + 1013904223u) >> 8, (s >> 8) % n; };
        for (int k = 0; k < 3000; k++) {
          if (t < 2) {
            char *held[4];
            size_t size[4];
            int n = 0;
            for (int i = 0; i < 4; i++) {
              DevBuf x(&c.scratch);
              const size_t want = 1000 + rnd(10 * MB);
              if (x.alloc(&c, want) != GEYE_OK) break;
              held[n] = x.as<char>();
              size[n++] = want;
              held[i][0] = held[i][want - 1] = (char)(16 * t + i);
            }
            for (int i = 0; i < n; i++) CHECK(held[i][0] == 16 * t + i && held[i][size[i] - 1] == 16 * t + i);
            c.scratch.reset();
          } else {
            DevBuf p;
            if (p.alloc(&c, 1000 + rnd(60 * MB)) == GEYE_OK) p.as<char>()[p.bytes - 1] = 1;
          }
        }
      });
    for (auto &t : threads) t.join();
  }
  CHECK(in_use == 0 && live.empty());
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None or not os.path.isdir(CUDA), reason="no C++ compiler or no CUDA headers")
def test_scratch_is_given_back(tmp_path):
    src = tmp_path / "harness.cpp"
    src.write_text(HARNESS)
    csrc = os.path.join(ROOT, "geye_gb300", "csrc")
    exe = str(tmp_path / "harness")
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-pthread", "-I", csrc, "-I", os.path.join(ROOT, "include"), "-I", CUDA,
                        "-o", exe, "-x", "c++", os.path.join(csrc, "memory.cu"), str(src)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr[-2000:]
