"""The library's host code on a recording stand-in for the CUDA runtime (no GPU).

api.cu's object is linked with the stand-in instead of libcudart and the kernels: device
memory is host memory, the launchers record what they are asked to launch and where, and
an allocation can be made to fail.  Tests then read the order of launches, copies and
waits, and what each launch is given."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import REPO
from segfault_py_gb300 import _lib, build

CSRC = os.path.join(REPO, "segfault_py_gb300", "csrc")

COMMON = r"""
struct Rec { long long what, cls, kind, stream, n, list, count, split; double rel_load, ms; };
enum { LAUNCH = 1, KERNEL, MEMCPY, SYNC, RECORD, WAIT };
extern std::vector<Rec> fake_log;
extern double fake_q;
inline void put(long long what, const void *st, long long list = 0) { fake_log.push_back({what, -1, -1, (long long)st, 0, list, 0, 0, 0, 0}); }
"""

RUNTIME = r"""
#include <cstdlib>
#include <cstring>
#include <vector>
#include <cuda_runtime_api.h>
#include "fake.h"
std::vector<Rec> fake_log;
double fake_q = 1.0;
static long long fail_in = -1;
extern "C" {
int fake_count() { return (int)fake_log.size(); }
void fake_get(int i, Rec *r) { *r = fake_log[i]; }
void fake_clear() { fake_log.clear(); }
void fake_fail_malloc(long long k) { fail_in = k; }   // the k-th next allocation fails (0: the next)
void fake_q_scale(double s) { fake_q = s; }
cudaError_t cudaMalloc(void **p, size_t n) {
  if (fail_in >= 0 && fail_in-- == 0) { *p = nullptr; return cudaErrorMemoryAllocation; }
  *p = std::calloc(1, n);
  return cudaSuccess;
}
cudaError_t cudaFree(void *p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { put(MEMCPY, 0, (long long)d); std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t st) { put(MEMCPY, st, (long long)d); std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemset(void *d, int v, size_t n) { std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) { std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { *v = 152; return cudaSuccess; }
cudaError_t cudaDeviceGetStreamPriorityRange(int *lo, int *hi) { *lo = 0; *hi = -5; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { put(SYNC, 0); return cudaSuccess; }
static cudaError_t handle(void **p) { static long long next = 0x1000; *p = (void *)next++; return cudaSuccess; }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t *s, unsigned, int) { return handle((void **)s); }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return handle((void **)s); }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return handle((void **)e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return handle((void **)e); }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { put(SYNC, s); return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *s) { *s = cudaStreamCaptureStatusNone; return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) { put(WAIT, s, (long long)e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { put(RECORD, s, (long long)e); return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 1.0f; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "stand-in error"; }
cudaError_t cudaGetSymbolAddress(void **p, const void *) { static std::vector<double> s(8 << 20); *p = s.data(); return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphInstantiateWithFlags(cudaGraphExec_t *, cudaGraph_t, unsigned long long) { return cudaErrorUnknown; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorUnknown; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaErrorUnknown; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *) { return cudaErrorUnknown; }
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *f) { *k = (cudaKernel_t)f; return cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t, dim3, dim3, void **, size_t, cudaStream_t st) { put(KERNEL, st); return cudaSuccess; }
static cudaStream_t call_st;
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, cudaStream_t st) { call_st = st; return 0; }
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *s, void *st) { *g = *b = dim3(1, 1, 1); *s = 0; *(cudaStream_t *)st = call_st; return cudaSuccess; }
char __cudaInitModule(void **) { return 1; }
int sf_fma_peak() { return -3; }      // not in the linked objects
int sf_small_solve() { return -3; }
void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
}
"""

KERNELS = r"""
#include <cmath>
#include <vector>
#include "classes.h"
#include "launch.h"
#include "fake.h"
using namespace sf;
static cudaError_t note(int cls, int kind, const ClassWork *w, int nw, cudaStream_t st) {
  for (int k = 0; k < nw; ++k)
    fake_log.push_back({LAUNCH, cls, kind, (long long)st, w[k].n, (long long)w[k].list, (long long)w[k].count,
                        (long long)w[k].psplit * w[k].wsplit, w[k].rel_load, 0.0});
  return cudaSuccess;
}
namespace sf {
cudaError_t launch_jk_f64(int c, const KParams &, const ClassWork *w, int n, const double *, double *, double *, cudaStream_t s) { return note(c, 0, w, n, s); }
cudaError_t launch_jk_f32(int c, const KParams &, const ClassWork *w, int n, const float *, double *, double *, cudaStream_t s) { return note(c, 1, w, n, s); }
cudaError_t launch_jk_dd(int c, const KParams &, const ClassWork *w, int n, const dd *, double *, double *, cudaStream_t s) { return note(c, 2, w, n, s); }
cudaError_t launch_grad_f64(int c, const KParams &, const ClassWork *w, int n, const double *, double *, cudaStream_t s) { return note(c, 0, w, n, s); }
cudaError_t launch_grad_f32(int c, const KParams &, const ClassWork *w, int n, const float *, double *, cudaStream_t s) { return note(c, 1, w, n, s); }
cudaError_t launch_grad_dd(int c, const KParams &, const ClassWork *w, int n, const dd *, double *, cudaStream_t s) { return note(c, 2, w, n, s); }
cudaError_t launch_jk_persist_f32(int, const KParams &, const PersistWork &, int, const float *, double *, double *, cudaStream_t s) { put(KERNEL, s); return cudaSuccess; }
cudaError_t launch_eri(int, int, const KParams &, const EriWork &, cudaStream_t s) { put(KERNEL, s); return cudaSuccess; }
cudaError_t launch_eri_dd(int, const KParams &, const EriWork &, cudaStream_t s) { put(KERNEL, s); return cudaSuccess; }
cudaError_t launch_md_eri(int, const KParams &, const EriWork &, cudaStream_t s) { put(KERNEL, s); return cudaSuccess; }
cudaError_t launch_md_tc(int, const KParams &, const EriWork &, int, cudaStream_t s) { put(KERNEL, s); return cudaSuccess; }
cudaError_t launch_one_electron(const OneParams &, cudaStream_t s) { put(KERNEL, s); return cudaSuccess; }
cudaError_t launch_one_electron_grad(const OneParams &, const double *, const double *, double *, int, cudaStream_t s) { put(KERNEL, s); return cudaSuccess; }
// bounds that fall off with the distance of the two centres
cudaError_t launch_schwarz(int, const KParams &k, int p0, int n, double *q, cudaStream_t s) {
  for (int i = p0; i < p0 + n; ++i) {
    const int a = k.pr.a[i], b = k.pr.b[i];
    const double x = k.sh.cx[a] - k.sh.cx[b], y = k.sh.cy[a] - k.sh.cy[b], z = k.sh.cz[a] - k.sh.cz[b];
    q[i] = fake_q * std::exp(-0.5 * (x * x + y * y + z * z));
  }
  put(KERNEL, s);
  return cudaSuccess;
}
void md_tc_set_wait_limit(int) {}
cudaError_t persist_blocks_per_sm(int, int *n) { *n = 4; return cudaSuccess; }
int persist_tier_of(int cls) { return cls < 6 ? 0 : -1; }
cudaError_t prepare_eri() { return cudaSuccess; }
cudaError_t prepare_eri_dd() { return cudaSuccess; }
cudaError_t prepare_grad_dd() { return cudaSuccess; }
cudaError_t prepare_grad_f32() { return cudaSuccess; }
cudaError_t prepare_grad_f64() { return cudaSuccess; }
cudaError_t prepare_jk_dd() { return cudaSuccess; }
cudaError_t prepare_jk_f32() { return cudaSuccess; }
cudaError_t prepare_jk_f64() { return cudaSuccess; }
cudaError_t prepare_md() { return cudaSuccess; }
cudaError_t prepare_md_tc() { return cudaSuccess; }
cudaError_t prepare_one_electron() { return cudaSuccess; }
void grad_tables(std::vector<uint2> &t, std::vector<int2> &h) { t.resize(1); h.resize(1); }
}
"""

LAUNCH, KERNEL, MEMCPY, SYNC, RECORD, WAIT = range(1, 7)


class Rec(C.Structure):
    _fields_ = [(k, C.c_longlong) for k in ("what", "cls", "kind", "stream", "n", "list", "count", "split")] + \
               [("rel_load", C.c_double), ("ms", C.c_double)]


def make(out_dir):
    """The stand-in library, its entry points with the argument types of the real one."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    os.makedirs(build.BUILD, exist_ok=True)
    objs = [build._compile(s, False) for s in ("api.cu", "rys_table.cpp")]
    for name, text in (("fake.h", COMMON), ("runtime.cpp", RUNTIME), ("kernels.cu", KERNELS)):
        with open(os.path.join(out_dir, name), "w") as f:
            f.write(text)
    lib = os.path.join(out_dir, "libfake.so")
    inc = ["-I", os.path.join(REPO, "include"), "-I", CSRC, "-I", out_dir]
    subprocess.run([nvcc, "-std=c++17", "--expt-relaxed-constexpr", *build.ARCH, "-Xcompiler", "-fPIC", *inc, "-c",
                    os.path.join(out_dir, "kernels.cu"), "-o", os.path.join(out_dir, "kernels.o")], check=True)
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I", "/usr/local/cuda/include", *inc,
                    os.path.join(out_dir, "runtime.cpp"), os.path.join(out_dir, "kernels.o"), *objs, "-o", lib,
                    "-lpthread"], check=True)
    return Fake(lib)


class Fake:
    def __init__(self, path):
        self.path = path
        real, path0, _lib._lib, _lib.LIB_PATH = _lib._lib, _lib.LIB_PATH, None, path
        try:
            self.L = _lib.lib()   # the argument types
        finally:
            _lib._lib, _lib.LIB_PATH = real, path0
        self.L.fake_q_scale.argtypes = [C.c_double]
        self.L.fake_fail_malloc.argtypes = [C.c_longlong]
        self.L.fake_get.argtypes = [C.c_int, C.c_void_p]

    def handle(self, table, q_scale=1.0):
        from segfault_py_gb300.fock import shell_descs
        arr, keep = shell_descs(table)
        h = C.c_void_p()
        self.ok(self.L.sf_create(C.cast(arr, C.c_void_p), len(arr), C.byref(h)))
        self.L.fake_q_scale(q_scale)
        self.ok(self.L.sf_schwarz(h, None, None))
        self.L.fake_clear()
        n = self.L.sf_nao(h)
        self.mats = [np.eye(n) for _ in range(3)]
        self.grad = np.zeros(3 * (int(max(table["atom"])) + 1))
        return h

    def ok(self, rc):
        assert rc >= 0, self.L.sf_last_error()
        return rc

    def fock(self, h, prec, cut=1e-12, cut32=1e-5, st=0x77):
        D, J, K = (m.ctypes.data for m in self.mats)
        return self.L.sf_fock_jk(h, D, J, K, _lib.PRECISION[prec], cut, cut32, None, st)

    def forces(self, h, prec, cut=1e-12, cut32=1e-5, st=0x77):
        return self.L.sf_grad_jk(h, self.mats[0].ctypes.data, self.grad.ctypes.data, _lib.PRECISION[prec], cut, cut32,
                                 st)

    def log(self, clear=True):
        out = []
        for i in range(self.L.fake_count()):
            r = Rec()
            self.L.fake_get(i, C.byref(r))
            out.append(r)
        if clear:
            self.L.fake_clear()
        return out

    def launches(self, **kw):
        return [r for r in self.log(**kw) if r.what == LAUNCH]
