"""Kernel attributes are set on every device that launches, and a launch that
the runtime refuses ends the solve with an error.  The failing CUDA calls are
fakes on the host: no kernel runs with anything missing."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "specfem3d_geotech_gb300", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

FAKES = r"""
#include <cassert>
#include <cstdio>
#include <thread>
#include <vector>
#include "sg_kernels.cuh"

static thread_local int device = 0;
static bool refuse = false;
static std::atomic<int> sets{0};
static cudaLaunchConfig_t seen;
static float a0; static int a1; static const void* a2;
extern "C" cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute a, int v) {
  assert(a == cudaFuncAttributeMaxDynamicSharedMemorySize && v == 200000);
  if (refuse) return cudaErrorInvalidValue;
  ++sets;
  return cudaSuccess;
}
extern "C" cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** args) {
  seen = *c;
  a2 = f; a0 = *(float*)args[0]; a1 = *(int*)args[1];
  return cudaSuccess;
}
static void kernel(float, int) {}

int main() {
  std::atomic<unsigned long long> done{};
  const void* k = (const void*)kernel;
  assert(sg::allow_smem(done, k, 200000) && sets == 1);
  assert(sg::allow_smem(done, k, 200000) && sets == 1);      // once per device
  device = 1;
  assert(sg::allow_smem(done, k, 200000) && sets == 2);      // and on the next one again
  device = 2;
  refuse = true;
  assert(!sg::allow_smem(done, k, 200000));
  refuse = false;
  assert(sg::allow_smem(done, k, 200000) && sets == 3);      // a refusal is not remembered
  device = 64;
  assert(sg::allow_smem(done, k, 200000) && sg::allow_smem(done, k, 200000) && sets == 5);
  std::vector<std::thread> ts;
  for (int i = 0; i < 8; ++i)
    ts.emplace_back([&, i] { device = 8 + i; for (int n = 0; n < 1000; ++n) assert(sg::allow_smem(done, k, 200000)); });
  for (auto& t : ts) t.join();
  assert(sets == 13);
  sg::launch_chained(kernel, 5, 96, 7000, nullptr, 3, 4.9);  // arguments convert to the kernel's types
  assert(a2 == k && a0 == 3.f && a1 == 4 && seen.gridDim.x == 5 && seen.blockDim.x == 96);
  assert(seen.dynamicSmemBytes == 7000 && seen.numAttrs == 1);
  std::puts("ok");
}
"""

# a launch that needs more shared memory than the default is refused, as on a
# device where the kernel's limit was not raised
SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <cuda_runtime_api.h>
static __thread cudaError_t pending = cudaSuccess;
static void* real_of(const char* name) { return dlsym(dlopen("libcudart.so.13", RTLD_LAZY), name); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** args) {
  static cudaError_t (*real)(const cudaLaunchConfig_t*, const void*, void**);
  if (c->dynamicSmemBytes > 49152) return pending = cudaErrorInvalidValue;
  if (!real) *(void**)&real = real_of("cudaLaunchKernelExC");
  return real(c, f, args);
}
cudaError_t cudaGetLastError(void) {
  static cudaError_t (*real)(void);
  cudaError_t e = pending;
  pending = cudaSuccess;
  if (e != cudaSuccess) return e;
  if (!real) *(void**)&real = real_of("cudaGetLastError");
  return real();
}
"""


def test_attributes_are_per_device_and_chained_launches_pass_their_arguments(tmp_path):
    src = tmp_path / "fakes.cpp"
    src.write_text(FAKES)
    exe = str(tmp_path / "fakes")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, "-I", CUDA + "/include", str(src), "-o", exe, "-lpthread"],
                   check=True, timeout=300)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=60)
    assert out.stdout.strip() == "ok"


@pytest.mark.gpu
def test_a_refused_launch_ends_the_solve(tmp_path):
    src = tmp_path / "shim.c"
    src.write_text(SHIM)
    shim = str(tmp_path / "shim.so")
    subprocess.run(["gcc", "-shared", "-fPIC", "-I", CUDA + "/include", str(src), "-o", shim, "-ldl"], check=True,
                   timeout=300)
    code = """if 1:
        import sys; sys.path.insert(0, %r)
        import specfem3d_geotech_gb300 as sg
        from specfem3d_geotech_gb300 import meshgen
        model = sg.Model(meshgen.slope3d(9, 4, 5), precision=sg.PREC_MIXED)
        ctl = sg.make_control(nl_maxiter=2, cg_maxiter=300, precision=sg.PREC_MIXED)
        model.ctx.profile(True)
        try:
            model.trials([1.0, 1.1, 1.2, 1.3], ctl)
        except sg.SgError as e:
            assert e.code == sg.SG_ERR_CUDA and "pcg" in str(e), (e.code, str(e))
            assert model.ctx.profile_read()["pcg_iters"] == 0      # before iterations on stale products
        else:
            raise AssertionError("the solve went on")
    """ % ROOT
    subprocess.run([sys.executable, "-c", code], check=True, timeout=300,
                   env=dict(os.environ, LD_PRELOAD=shim, SG_PERSIST="0"))
