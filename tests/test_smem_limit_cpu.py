"""The dynamic shared memory that a kernel is allowed belongs to the kernel, not to a launch: a launch that lowered it would
take it from another host thread between that one's set and launch.  Run without a GPU against a stand-in for the runtime
calls of a launch, which writes down what they are given."""
import os
import subprocess
import sys

import pytest

torch = pytest.importorskip("torch")
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
INCLUDE = "/usr/local/cuda/include"

RUNTIME = r"""
#include <cuda_runtime_api.h>
#include <stdio.h>
#include <string.h>
#undef cudaGetDeviceProperties
extern "C" {
cudaError_t cudaGetDevice(int* dev) { *dev = 0; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
static cudaError_t props(cudaDeviceProp* p) {
  memset(p, 0, sizeof(*p));
  p->multiProcessorCount = 148;
  p->sharedMemPerBlockOptin = 232448;
  return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) { return props(p); }
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp* p, int) { return props(p); }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute, int v) { printf("set %p %d\n", f, v); return cudaSuccess; }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
  printf("launch %p %zu\n", f, c->dynamicSmemBytes);
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void**, size_t smem, cudaStream_t) {
  printf("launch %p %zu\n", f, smem);
  return cudaSuccess;
}
}
"""

CALLS = r"""
import ctypes as C
import sys
sys.path.insert(0, sys.argv[1])
from cherryq_b200 import _cabi
lib = _cabi.lib()
at = C.c_void_p(1 << 20)                     # never read: nothing is launched
for bits, K, N in ((3, 4096, 1024), (4, 1024, 264)):
    L = _cabi.tlayer_init(bits, K, N, 16, 128)
    L.blob = 1 << 20
    for M in (300, 16, 4096, 100, 1, 300):
        assert lib.cq_tlayer_gemm(C.byref(L), at, K, at, N, M, 0, at, at, None) == 0
for K, N, M in ((8192, 8192, 16), (512, 256, 16), (4096, 13824, 16), (1024, 512, 4), (16384, 256, 8)):
    Kc = K - 16
    assert lib.cq_vecquant3matmul_cherryq(at, at, at, at, at, at, M, K, Kc // 8 * 3, N, 16, 128, 0, 0, None) == 0
"""


@pytest.mark.skipif(not os.path.exists(os.path.join(INCLUDE, "cuda_runtime_api.h")), reason="needs the CUDA headers")
def test_the_limit_of_a_kernel_is_never_lowered(tmp_path):
    src, shim = tmp_path / "runtime.cpp", tmp_path / "runtime.so"
    src.write_text(RUNTIME)
    subprocess.run(["g++", "-shared", "-fPIC", f"-I{INCLUDE}", str(src), "-o", str(shim)], check=True)
    res = subprocess.run([sys.executable, "-c", CALLS, ROOT], env=dict(os.environ, LD_PRELOAD=str(shim)), capture_output=True,
                         text=True, timeout=300)
    assert res.returncode == 0, res.stderr[-2000:]
    limit, launches = {}, 0
    for line in res.stdout.splitlines():
        what, fn, size = line.split()
        if what == "set":
            assert int(size) >= limit.get(fn, 0), line
            limit[fn] = int(size)
        else:
            launches += 1
            assert int(size) <= max(limit.get(fn, 0), 48 * 1024), line
    assert launches == 2 * 2 * 6 + 5 and len(limit) >= 4
