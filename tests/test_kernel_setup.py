"""CPU: what is remembered of a kernel, per context (csrc/kernel_setup.cuh), against a runtime made of counters.

The header is compiled for the host with the runtime functions that it calls defined in the test: they count, and keep what has been set
per context as the driver does."""
import shutil
import subprocess
from pathlib import Path

import pytest

from baselinebenchmark_b200 import build

CSRC = Path(__file__).resolve().parent.parent / "baselinebenchmark_b200" / "csrc"
CUDA_INCLUDE = Path("/usr/local/cuda/include")

PROGRAM = r'''
#include "kernel_setup.cuh"
#include <cassert>
#include <cstdio>
#include <cstring>
#include <map>
#include <utility>

static unsigned long long current = 0;                 // number of the current context, 0: none
static std::map<std::pair<unsigned long long, const void*>, size_t> limit;
static std::map<std::pair<unsigned long long, const void*>, int> carveout;
static int sets = 0, gets = 0, fail = 0;

static CUresult get_current(CUcontext* c) { *c = current ? (CUcontext)0x1000 : nullptr; return CUDA_SUCCESS; }   // one address for all
static CUresult get_number(CUcontext, unsigned long long* n) {
  if (current == ~0ull) return CUDA_ERROR_CONTEXT_IS_DESTROYED;
  *n = current;
  return CUDA_SUCCESS;
}
extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) { *v = (int)a; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void* k, cudaFuncAttribute a, int v) {
  ++sets;
  if (fail) return cudaErrorInvalidValue;
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) limit[{current, k}] = (size_t)v; else carveout[{current, k}] = v;
  return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void* k) { ++gets; memset(a, 0, sizeof *a); a->numRegs = 1 + (int)((uintptr_t)k & 127); return cudaSuccess; }
cudaError_t cudaGetDriverEntryPoint(const char* name, void** f, unsigned long long, cudaDriverEntryPointQueryResult* r) {
  *f = strcmp(name, "cuCtxGetId") ? (void*)get_current : (void*)get_number;
  *r = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
}
using moba::KernelSetup;
KernelSetup& KernelSetup::instance() { static KernelSetup s; return s; }
static const void* kernel(int i) { return (const void*)(uintptr_t)(0x400000 + 48 * i); }
// a launch may rely on this much: what the call leaves behind is what the current context has
static void use(int i, size_t smem, bool carve = false) {
  int regs = 0;
  assert(KernelSetup::instance().prepare(kernel(i), smem, carve ? &regs : nullptr, carve) == cudaSuccess);
  const size_t has = limit[{current, kernel(i)}];
  assert(has >= smem);
  if (carve) { const int c = carveout[{current, kernel(i)}]; assert(c == 100); assert(regs == 1 + (int)((uintptr_t)kernel(i) & 127)); }
}
static int sets_of(int i, size_t smem, bool carve = false) { const int was = sets; use(i, smem, carve); return sets - was; }

int main() {
  current = 1;
  assert(sets_of(0, 100) == 1 && sets_of(0, 100) == 0 && sets_of(0, 60) == 0);
  assert(sets_of(0, 200) == 1 && sets_of(0, 150) == 0);              // more than before: set again, and kept
  assert(sets_of(1, 100, true) == 2 && sets_of(1, 100, true) == 0 && gets == 1);
  current = 2;                                                      // another context, at the same address
  assert(sets_of(0, 100) == 1 && sets_of(1, 100, true) == 2 && sets_of(1, 100, true) == 0);
  current = 1;
  assert(sets_of(0, 200) == 0);                                     // both are remembered
  current = 0;                                                      // none: nothing to remember it by
  assert(sets_of(0, 100) == 1 && sets_of(0, 100) == 1);
  current = ~0ull;                                                  // one that is gone
  assert(sets_of(0, 100) == 1 && sets_of(0, 100) == 1);
  current = 3;
  fail = 1;
  assert(KernelSetup::instance().prepare(kernel(0), 100, nullptr, false) == cudaErrorInvalidValue);
  fail = 0;
  assert(sets_of(0, 100) == 1 && sets_of(0, 100) == 0);              // a refused setting is not remembered
  for (int i = 0; i < 400; ++i) use(i, 100 + i);                    // more kernels than places
  for (int i = 0; i < 400; ++i) use(i, 100 + i);
  for (unsigned long long c = 10; c < 60; ++c) { current = c; use(0, 100); use(0, 100); }   // more contexts than tables
  current = 1;
  use(0, 200);
  assert(sets_of(0, 200) == 0);
  assert(KernelSetup::instance().device().sms == (int)cudaDevAttrMultiProcessorCount);
  puts("ok");
}
'''


@pytest.mark.skipif(shutil.which("g++") is None or not (CUDA_INCLUDE / "cuda_runtime.h").exists(),
                    reason="needs g++ and the CUDA headers")
def test_what_is_set_is_set_in_every_context(tmp_path):
    source = tmp_path / "setup.cpp"
    source.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(CSRC), "-I", str(CUDA_INCLUDE), "-x", "c++", str(source), "-o",
                    str(tmp_path / "setup")], check=True)
    assert subprocess.run([str(tmp_path / "setup")], capture_output=True, text=True, check=True).stdout == "ok\n"


@pytest.mark.skipif(shutil.which("nm") is None, reason="needs nm")
def test_the_library_shares_no_object_with_another_build_of_it():
    """A symbol of type u (STB_GNU_UNIQUE) is one object for the whole process, whichever library it is in: two builds of this one that are
    loaded side by side would work on one table."""
    symbols = subprocess.run(["nm", "-D", str(build.build())], capture_output=True, text=True, check=True).stdout
    assert "moba_forward" in symbols
    assert [line for line in symbols.splitlines() if line.split()[-2] == "u"] == []
