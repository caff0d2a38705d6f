"""The library's device arrays (csrc/common.cuh) on a fake CUDA runtime with a set amount of memory: no
GPU, no libcudart, only the header's own code."""
import os
import shutil
import subprocess

import pytest

from matlab_ufvm_b200 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

RUNTIME = r'''
#include <cstdlib>
#include <map>
std::map<void*, size_t> live;
size_t total = 1 << 20, used = 0, idle = 0;
long mallocs = 0, pooled = 0;
static int give(void** p, size_t n) {
  if (used + idle + n > total) return 2;  // cudaErrorMemoryAllocation
  *p = malloc(1);
  live[*p] = n;
  used += n;
  return 0;
}
static int take(void* p, bool keep) {
  const size_t n = live.at(p);
  live.erase(p);
  free(p);
  used -= n;
  if (keep) idle += n;
  return 0;
}
extern "C" {
int cudaMalloc(void** p, size_t n) { ++mallocs; return give(p, n); }
int cudaFree(void* p) { return take(p, false); }
int cudaMallocAsync(void** p, size_t n, void*) { return give(p, n); }
int cudaMallocFromPoolAsync(void** p, size_t n, void*, void*) {
  ++pooled;
  if (n <= idle) idle -= n;
  return give(p, n);
}
int cudaFreeAsync(void* p, void*) { return take(p, true); }
int cudaDeviceSynchronize() { return 0; }
int cudaGetLastError() { return 0; }
const char* cudaGetErrorString(int) { return "fake"; }
int cudaStreamIsCapturing(void*, int* s) { *s = 0; return 0; }
void** __cudaRegisterFatBinary(void*) { return nullptr; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
char __cudaInitModule(void**) { return 1; }
}
'''

MAIN = r'''
#include <cstdio>
#include "common.cuh"
extern size_t total, used, idle;
extern long mallocs, pooled;
namespace ufvm {
void set_error(const std::string&) {}
const char* get_error() { return ""; }
double host_ms_now() { return 0; }
void trim_scratch_pool() { idle = 0; }
}
using namespace ufvm;
#define REQUIRE(c) if (!(c)) { printf("line %d: %s\n", __LINE__, #c); return 1; }
int main() { BODY return 0; }
'''


def run(body, tmp_path):
    nvcc = build.NVCC if os.path.exists(build.NVCC) else shutil.which("nvcc")
    if nvcc is None:
        pytest.skip("no nvcc")
    (tmp_path / "runtime.cpp").write_text(RUNTIME)
    (tmp_path / "main.cu").write_text(MAIN.replace("BODY", body))
    subprocess.run(["g++", "-std=c++17", "-c", "runtime.cpp", "-o", "runtime.o"], check=True, cwd=tmp_path)
    subprocess.run([nvcc, *build.ARCH, "-std=c++17", "-cudart", "none", "-I", os.path.join(ROOT, "include"), "-I", build.CSRC,
                    "main.cu", "runtime.o", "-o", "t"], check=True, cwd=tmp_path)
    r = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def test_growth_falls_back_to_what_was_asked_for(tmp_path):
    run(r'''
  DArr<char> a, b;
  REQUIRE(dalloc(a, 300000) == UFVM_OK && a.n == 300000)
  REQUIRE(dalloc(a, 400000) == UFVM_OK && a.n == 500000)   // grows by a quarter more
  REQUIRE(dalloc(a, 1000000) == UFVM_OK && a.n == 1000000) // 1,250,000 would not fit
  REQUIRE(t_dev_bytes == 1000000 && used == 1000000)
  REQUIRE(dalloc(b, 100000) == UFVM_E_OOM && b.p == nullptr && b.n == 0)
  dfree(a);
  REQUIRE(t_dev_bytes == 0 && used == 0)
''', tmp_path)


def test_idle_scratch_is_given_back_before_an_allocation_fails(tmp_path):
    run(r'''
  DArr<char> s, a;
  {
    AllocStreamScope scope(nullptr, (cudaMemPool_t)1);
    REQUIRE(dalloc(s, 600000) == UFVM_OK && s.async)
    dfree(s);
  }
  REQUIRE(idle == 600000)
  REQUIRE(dalloc(a, 900000) == UFVM_OK && idle == 0)
  dfree(a);
''', tmp_path)


def test_large_scratch_does_not_come_from_the_pool(tmp_path):
    run(r'''
  DArr<char> s, a;
  total = 1ull << 40;
  AllocStreamScope scope(nullptr, (cudaMemPool_t)1);
  REQUIRE(dalloc(s, kPoolArray - 1) == UFVM_OK && s.async && pooled == 1 && mallocs == 0)
  REQUIRE(dalloc(a, kPoolArray) == UFVM_OK && !a.async && pooled == 1 && mallocs == 1)
  dfree(a);
  REQUIRE(idle == 0)
  dfree(s);
  REQUIRE(idle == kPoolArray - 1 && used == 0)
''', tmp_path)
