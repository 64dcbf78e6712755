"""The setters' and getters' large copies (csrc/cr_copy.cu) on the CPU, against a
stand-in for the CUDA runtime that keeps its rules on devices: an event belongs
to the device that was current when it was made and can only be recorded on
that device's streams, while a copy may be issued with any device current."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INCLUDE = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")

FAKE = r"""
#include <cuda_runtime.h>
#include <cstdlib>
#include <cstring>
#include "cr_copy.h"
// streams are their device's number + 1, events point to their device's number
static thread_local int g_current = 0;
static int g_fail_host_alloc = 0;
extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = g_current; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { g_current = d; return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  if (g_fail_host_alloc) return cudaErrorMemoryAllocation;
  *p = malloc(n);
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  *e = (cudaEvent_t) new int(g_current);
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete (int*)e; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  return *(int*)e + 1 == (int)(size_t)s ? cudaSuccess : cudaErrorInvalidResourceHandle;
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
  memset(a, 0, sizeof(*a));
  a->type = cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
// a copy in and one out for a context of `device` while `current` is; the device current afterwards
int round_trip(int device, int current, int fail, void* dev, void* out, const void* in, size_t n, int* after) {
  g_current = current;
  g_fail_host_alloc = fail;
  cr::Staging s;
  cudaStream_t st = (cudaStream_t)(size_t)(device + 1);
  int rc = cr::copy_in(s, device, st, dev, in, n);
  if (!rc) rc = cr::copy_out(s, device, st, out, dev, n);
  *after = g_current;
  return rc;
}
}
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    if not os.path.exists(os.path.join(CUDA_INCLUDE, "cuda_runtime.h")):
        pytest.skip("no CUDA headers")
    d = tmp_path_factory.mktemp("copy")
    (d / "fake.cpp").write_text(FAKE)
    src = os.path.join(ROOT, "cudaring_b200", "csrc")
    so = d / "fake.so"
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-pthread", "-Wl,-Bsymbolic", "-I", CUDA_INCLUDE, "-I", src,
                    str(d / "fake.cpp"), "-x", "c++", os.path.join(src, "cr_copy.cu"), "-o", str(so)], check=True)
    lib = C.CDLL(str(so))
    lib.round_trip.argtypes = [C.c_int, C.c_int, C.c_int, C.c_void_p, C.c_void_p, C.c_void_p, C.c_size_t, C.c_void_p]
    return lib


# under the line of 8 MB, at it, and with a short last chunk
@pytest.mark.parametrize("size", [(8 << 20) - 8, 8 << 20, (21 << 20) + 48])
@pytest.mark.parametrize("device,current", [(0, 0), (1, 0), (0, 1)])
@pytest.mark.parametrize("fail", [0, 1])
def test_copies_leave_the_callers_device(fake, size, device, current, fail):
    x = np.random.default_rng(size).integers(0, 256, size, dtype=np.uint8)
    dev, out = np.zeros_like(x), np.zeros_like(x)
    after = C.c_int(-1)
    assert fake.round_trip(device, current, fail, dev.ctypes.data, out.ctypes.data, x.ctypes.data, size,
                           C.byref(after)) == 0
    assert after.value == current
    assert np.array_equal(dev, x) and np.array_equal(out, x)
