"""Context creation reports the calls it depends on: with a launch or a synchronisation that fails it gives an error and
no context, and releases what it holds.  The library's own source with the CUDA calls it makes replaced by fakes (no GPU
is needed: without a driver, a kernel launch is a call that fails)."""
import ctypes
import os
import subprocess

import pytest

from trj_analysis_b200 import build

FAKE = r'''
#pragma once
#include <cuda_runtime.h>
#include <stdlib.h>
#include <string.h>
static int fake_live = 0, fake_fail = 0;  // 1: the launch, 2: the synchronisation, 3: the clear
extern "C" __attribute__((visibility("default"))) int fake_state(int fail) { fake_fail = fail; return fake_live; }
static cudaError_t fake_malloc(void** p, size_t n) { *p = malloc(n); ++fake_live; return cudaSuccess; }
static cudaError_t fake_free(void* p) { free(p); --fake_live; return cudaSuccess; }
static cudaError_t fake_memset(void* p, int v, size_t n) { memset(p, v, n); return fake_fail == 3 ? cudaErrorUnknown : cudaSuccess; }
static cudaError_t fake_count(int* n) { *n = 1; return cudaSuccess; }
static cudaError_t fake_device(int* d) { *d = 0; return cudaSuccess; }
static cudaError_t fake_last() { return fake_fail == 1 ? cudaErrorLaunchFailure : cudaSuccess; }
static cudaError_t fake_sync() { return fake_fail == 2 ? cudaErrorLaunchFailure : cudaSuccess; }
static cudaError_t fake_props(cudaDeviceProp* p, int) {
    memset(p, 0, sizeof(*p)); p->major = 10; p->multiProcessorCount = 148; p->sharedMemPerBlockOptin = 232448; return cudaSuccess;
}
#undef cudaGetDeviceProperties
#define cudaGetDeviceProperties fake_props
#define cudaMalloc(p, n) fake_malloc((void**)(p), n)
#define cudaMallocHost(p, n) fake_malloc((void**)(p), n)
#define cudaFree fake_free
#define cudaFreeHost fake_free
#define cudaMemset fake_memset
#define cudaGetDeviceCount fake_count
#define cudaGetDevice fake_device
#define cudaSetDevice(d) cudaSuccess
#define cudaGetLastError fake_last
#define cudaDeviceSynchronize fake_sync
'''


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("ctx")
    (d / "fake.h").write_text(FAKE)
    out = str(d / "libctx.so")
    flags = [f for f in build.FLAGS if f not in ("-O3", "-lineinfo")]
    subprocess.run([build.NVCC, *flags, "-include", str(d / "fake.h"), "-o", out, os.path.join(build.CSRC, "ctx.cu")],
                   check=True)
    return ctypes.CDLL(out, mode=os.RTLD_LAZY)


@pytest.mark.parametrize("fail", [0, 1, 2, 3])
def test_create_reports_failures(lib, fail):
    before = lib.fake_state(fail)
    ctx = ctypes.c_void_p()
    rc = lib.trj_ctx_create(0, ctypes.byref(ctx))
    if fail == 0:
        assert rc == 0 and ctx.value
        assert lib.trj_ctx_destroy(ctx) == 0
    else:
        assert rc == -2 and not ctx.value
    assert lib.fake_state(0) == before
