"""The pool of device blocks that a prepare takes over from the last one (DevicePool in
csrc/common.cuh), compiled for the host against a cudaMalloc of 2 MB pages with a fixed capacity."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.path.dirname(os.path.dirname(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"))

PROGRAM = r"""
#include <cstdio>
#include <map>
#include "common.cuh"

static const size_t PAGE = 2 << 20;
static size_t total = 0, used = 0;
static int mallocs = 0;
static std::map<void*, size_t> blocks;
extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) {
  const size_t b = (n + PAGE - 1) / PAGE * PAGE;
  if (used + b > total) return cudaErrorMemoryAllocation;
  used += b;
  mallocs++;
  *p = ::operator new(1);
  blocks[*p] = b;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  used -= blocks.at(p);
  blocks.erase(p);
  ::operator delete(p);
  return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) {
  *f = total - used;
  *t = total;
  return cudaSuccess;
}
}
using namespace msbg;

// first: sizes (bytes) of the last problem's buffers; then the next one's, under a pool.
static bool next_problem(size_t pages, int n1, size_t b1, int n2, size_t b2) {
  total = pages * PAGE;
  std::vector<DeviceBuffer> a(n1), b(n2);
  for (auto& x : a)
    if (x.ensure(b1) != cudaSuccess) return false;
  mallocs = 0;
  PoolScope pool;
  for (auto& x : a) x.release();
  bool ok = true;
  for (auto& x : b) ok = ok && x.ensure(b2) == cudaSuccess && x.bytes == b2;
  std::printf("%d mallocs, %d left\n", mallocs, (int)((total - used) / PAGE));
  return ok;
}
int main() {
  int bad = 0;
  // a card nearly full: 12 x 75 pages fit, and must after 10 x 90 too, which would serve them
  bad |= !next_problem(1000, 10, 90 * PAGE, 12, 75 * PAGE) << 0;
  // the same sizes again, and sizes within a page of them: nothing is allocated
  bad |= !(next_problem(1000, 10, 90 * PAGE, 10, 90 * PAGE) && mallocs == 0) << 1;
  bad |= !(next_problem(1000, 10, 90 * PAGE - 5, 10, 90 * PAGE - 4096) && mallocs == 0) << 2;
  // a card nearly empty: somewhat smaller buffers take the blocks, up to 1/64 of what is free
  bad |= !(next_problem(100000, 10, 90 * PAGE, 10, 80 * PAGE) && mallocs == 0) << 3;
  bad |= !(next_problem(8000, 10, 90 * PAGE, 10, 75 * PAGE) && mallocs == 3) << 4;
  // small buffers on a nearly full card
  bad |= !next_problem(10, 8, PAGE / 2, 8, PAGE / 2 - 9) << 5;
  if (used || !blocks.empty()) bad |= 64;
  return bad;
}
"""


def test_a_pool_refuses_nothing_that_fits_without_it(tmp_path):
    if not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")) or not shutil.which("g++"):
        pytest.skip("no CUDA headers or no g++")
    src, exe = tmp_path / "pool.cpp", tmp_path / "pool"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + os.path.join(CUDA, "include"),
                    "-I" + os.path.join(ROOT, "include"),
                    "-I" + os.path.join(ROOT, "msbg-flip_b200", "csrc"), str(src), "-o", str(exe)],
                   check=True, capture_output=True, text=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, (r.returncode, r.stdout)
