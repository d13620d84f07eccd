"""Refused launches, on the CPU: the library's own objects linked with a stand-in for the CUDA runtime whose device
memory is host memory, whose kernels do nothing and whose cluster launches can be told to fail.  What is checked is the
host side: a solver whose cluster kernel a device does not take is not handed out as good."""
import ctypes
import glob
import os
import subprocess

import pytest

from conftest import PKG, ROOT

FAKE = r"""
#include <driver_types.h>
#include <cstdlib>
#include <cstring>
extern "C" {
int fake_refuse = 0, fake_clusters = 0;
static int last = 0;
static char area[1 << 16];
int cudaMalloc(void **p, size_t n) { *p = calloc(1, n + 1); return 0; }
int cudaHostAlloc(void **p, size_t n, unsigned) { *p = calloc(1, n + 1); return 0; }
int cudaFree(void *p) { free(p); return 0; }
int cudaFreeHost(void *p) { free(p); return 0; }
int cudaMemcpy(void *d, const void *s, size_t n, int) { memcpy(d, s, n); return 0; }
int cudaMemcpyAsync(void *d, const void *s, size_t n, int, void *) { memcpy(d, s, n); return 0; }
int cudaMemset(void *d, int v, size_t n) { memset(d, v, n); return 0; }
int cudaMemsetAsync(void *d, int v, size_t n, void *) { memset(d, v, n); return 0; }
int cudaGetSymbolAddress(void **p, const void *) { *p = area; return 0; }
int cudaDeviceGetAttribute(int *v, int a, int) { *v = a == 16 ? 152 : 232448; return 0; }
int cudaGetDevice(int *d) { *d = 0; return 0; }
int cudaGetDeviceCount(int *n) { *n = 1; return 0; }
int cudaStreamCreateWithFlags(void **s, unsigned) { *s = area; return 0; }
int cudaStreamCreateWithPriority(void **s, unsigned, int) { *s = area; return 0; }
int cudaEventCreate(void **e) { *e = area; return 0; }
int cudaEventCreateWithFlags(void **e, unsigned) { *e = area; return 0; }
int cudaEventElapsedTime(float *t, void *, void *) { *t = 1.f; return 0; }
int cudaStreamEndCapture(void *, void **g) { *g = area; return 0; }
int cudaStreamGetCaptureInfo(void *, int *s, void *, void *, const void **d, void *, size_t *n) { *s = 1; *d = 0; *n = 0; return 0; }
int cudaGraphCreate(void **g, unsigned) { *g = area; return 0; }
int cudaGraphInstantiate(void **e, void *, unsigned long long) { *e = area; return 0; }
int cudaGraphConditionalHandleCreate(unsigned long long *h, void *, unsigned, unsigned) { *h = 1; return 0; }
int cudaGraphGetNodes(void *, void *, size_t *n) { *n = 5; return 0; }
static cudaGraph_t body = (cudaGraph_t)area;
int cudaGraphAddNode(void **n, void *, void *, void *, size_t, cudaGraphNodeParams *p) {
    *n = area;
    p->conditional.phGraph_out = &body;
    return 0;
}
int cudaOccupancyMaxActiveClusters(int *n, const void *, void *) { *n = 1; return 0; }
int cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *, int, size_t) { *n = 1; return 0; }
int cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) { *n = 1; return 0; }
int cudaFuncGetAttributes(void *a, const void *) { memset(a, 0, sizeof(cudaFuncAttributes)); return 0; }
const char *cudaGetErrorString(int) { return "refused by the stand-in"; }
int cudaGetLastError() { const int e = last; last = 0; return e; }
int cudaLaunchKernelExC(const void *, const void *, void **) {
    fake_clusters++;
    return fake_refuse ? last = 912 : 0;
}
int cudaGetDriverEntryPointByVersion(...) { return 1; }
void **__cudaRegisterFatBinary(void *) { return (void **)area; }
#define NOP(f) int f(...) { return 0; }
NOP(__cudaRegisterFatBinaryEnd) NOP(__cudaUnregisterFatBinary) NOP(__cudaRegisterFunction) NOP(__cudaRegisterVar)
NOP(__cudaPushCallConfiguration) NOP(__cudaPopCallConfiguration) NOP(__cudaLaunchKernel) NOP(__cudaGetKernel)
NOP(cudaStreamSynchronize) NOP(cudaStreamDestroy) NOP(cudaStreamBeginCapture) NOP(cudaStreamBeginCaptureToGraph)
NOP(cudaStreamWaitEvent) NOP(cudaSetDevice) NOP(cudaGraphLaunch) NOP(cudaGraphExecDestroy) NOP(cudaGraphDestroy)
NOP(cudaFuncSetAttribute) NOP(cudaEventRecord) NOP(cudaEventRecordWithFlags) NOP(cudaEventDestroy)
NOP(cudaEventSynchronize) NOP(cudaMemcpyToSymbol) NOP(cudaLaunchKernel) NOP(cudaGetDeviceProperties)
NOP(cudaDeviceGetStreamPriorityRange)
}
"""


@pytest.fixture(scope="module")
def fake(gb, tmp_path_factory):
    gb.lib()  # built
    objs = sorted(glob.glob(os.path.join(ROOT, PKG, "_build", "*.o")))
    if not objs:
        pytest.skip("the library's object files are not here")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    d = tmp_path_factory.mktemp("fake")
    src, so = str(d / "cudart.cpp"), str(d / "libgbpf_fake.so")
    with open(src, "w") as f:
        f.write(FAKE)
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-w", "-I" + os.path.join(cuda, "include"), src, *objs,
                    "-Wl,-Bsymbolic", "-Wl,-z,defs", "-o", so, "-lpthread"], check=True)
    return ctypes.CDLL(so, mode=ctypes.RTLD_LOCAL)


@pytest.mark.parametrize("nbus,metodo,precision", [(14, 1, "PREC_FP64"), (600, 1, "PREC_FP64"), (236, 0, "PREC_FP64"),
                                                   (14, 0, "PREC_FP32_IR"), (236, 0, "PREC_FP32_IR")])
def test_a_refused_cluster_launch_is_an_error(gb, fake, nbus, metodo, precision):
    grid = ctypes.c_void_p()
    assert fake.gbpf_generate(4, ctypes.c_ulonglong(11), 0, nbus, ctypes.byref(grid)) == 0
    o = gb.Options()
    o.tolerancia, o.no_max_iter, o.lim_inj_reat, o.metodo, o.precision = 1e-8, 10, 0, metodo, getattr(gb, precision)
    launches = ctypes.c_int.in_dll(fake, "fake_clusters")
    for refuse in (0, 1, 0):
        ctypes.c_int.in_dll(fake, "fake_refuse").value = refuse
        launches.value = 0
        s = ctypes.c_void_p()
        st = fake.gbpf_solver_create(grid, ctypes.byref(o._o), 0, ctypes.byref(s))
        assert launches.value > 0
        assert (st != 0) == bool(refuse) and bool(s.value) == (st == 0), (refuse, st)
        if refuse:
            fake.gbpf_last_error.restype = ctypes.c_char_p
            assert b"refused by the stand-in" in fake.gbpf_last_error()
        else:
            fake.gbpf_solver_free(s)
    fake.gbpf_grid_free(grid)
