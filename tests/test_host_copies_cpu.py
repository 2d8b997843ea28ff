"""The host side of the batch calls on a stand-in for the CUDA runtime (no GPU): when a call fails, no copy from or to
its callers' buffers may still be in flight, and a block whose result is out of range leaves every buffer as it was.
The stand-in (preloaded in a child process) keeps asynchronous copies queued until something waits for the stream,
launches nothing, reports the sort as done, and fails the copies it is told to."""
import ctypes
import os
import subprocess
import sys

import pytest

from kolmo_gb300 import build, native

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CTL_CU = r"""
#include <cstddef>
#include <cstdio>
#include "fwd.cuh"
int main() { printf("%zu %zu\n", sizeof(kgb::Ctl), offsetof(kgb::Ctl, done)); }
"""

FAKE = r"""
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <vector>
struct dim3 { unsigned x, y, z; };
namespace {
struct Op { void *dst; const void *src; size_t n; int fill; };
std::vector<Op> ops;                   // queued, not yet done
const char *bad = nullptr;             // copies from or to this buffer fail
const uint32_t *samples = nullptr;     // what the read-back of the sampled indexes gives
size_t nsamples = 0, ctl_size = 0, ctl_done = 0;
int last = 0;
void drain() {
    for (const Op &o : ops) if (o.src) memcpy(o.dst, o.src, o.n); else memset(o.dst, o.fill, o.n);
    for (const Op &o : ops) {
        if (o.src && o.n == ctl_size) *(uint32_t *)((char *)o.dst + ctl_done) = 1;
        if (samples && o.src && o.n == nsamples * 4) memcpy(o.dst, samples, o.n);
    }
    ops.clear();
}
}
extern "C" {
void fake_setup(size_t size, size_t done) { ctl_size = size; ctl_done = done; }
void fake_samples(const uint32_t *v, size_t n) { samples = v; nsamples = n; }
void fake_bad(const void *p) { bad = (const char *)p; }
int fake_pending() { return (int)ops.size(); }
void fake_drain() { drain(); }

int cudaMemcpyAsync(void *d, const void *s, size_t n, int, void *) {
    if (bad && (d == bad || s == bad)) return last = 1;
    ops.push_back({d, s, n, 0});
    return 0;
}
int cudaMemsetAsync(void *d, int v, size_t n, void *) { ops.push_back({d, nullptr, n, v}); return 0; }
int cudaMemcpy(void *d, const void *s, size_t n, int) { drain(); memcpy(d, s, n); return 0; }
int cudaMemset(void *d, int v, size_t n) { drain(); memset(d, v, n); return 0; }
int cudaStreamSynchronize(void *) { drain(); return 0; }
int cudaEventSynchronize(void *) { drain(); return 0; }
int cudaMalloc(void **p, size_t n) { return (*p = calloc(n, 1)) ? 0 : 2; }
int cudaFree(void *p) { free(p); return 0; }
int cudaHostAlloc(void **p, size_t n, unsigned) { return cudaMalloc(p, n); }
int cudaMallocHost(void **p, size_t n) { return cudaMalloc(p, n); }
int cudaFreeHost(void *p) { free(p); return 0; }
int cudaStreamCreateWithFlags(void **s, unsigned) { *s = (void *)64; return 0; }
int cudaStreamDestroy(void *) { return 0; }
int cudaStreamIsCapturing(void *, int *c) { *c = 0; return 0; }
int cudaEventCreate(void **e) { *e = (void *)64; return 0; }
int cudaEventCreateWithFlags(void **e, unsigned) { *e = (void *)64; return 0; }
int cudaEventDestroy(void *) { return 0; }
int cudaEventRecord(void *, void *) { return 0; }
int cudaGetDevice(int *d) { *d = 0; return 0; }
int cudaDeviceGetAttribute(int *v, int, int) { *v = 8; return 0; }
int cudaFuncSetAttribute(const void *, int, int) { return 0; }
int cudaPointerGetAttributes(void *, const void *) { return last = 1; }  // not memory the runtime knows: pageable
int cudaGetLastError() { const int e = last; last = 0; return e; }
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void *) { return 0; }
int __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *m, void **s) {
    *g = *b = dim3{1, 1, 1};
    *m = 0;
    *s = nullptr;
    return 0;
}
int __cudaGetKernel(const void **k, const void *f) { *k = f; return 0; }
int __cudaLaunchKernel(const void *, dim3, dim3, void **, size_t, void *) { return 0; }
}
"""

CHILD = r"""
import ctypes, sys
import numpy as np
from kolmo_gb300 import native
case, fake_path, size, done = sys.argv[1], sys.argv[2], int(sys.argv[3]), int(sys.argv[4])
fake = ctypes.CDLL(fake_path)
fake.fake_setup(ctypes.c_size_t(size), ctypes.c_size_t(done))
L = native.lib()
N, R = 600 << 10, 1 << 19     # two samples a block
T = [np.full(N, 65, np.uint8) for _ in range(2)]
U = [np.full(N, 170, np.uint8) for _ in range(2)]
I = [np.full(2, 5, np.int32) for _ in range(2)]
samples = np.array([5, 6, 5, 6], np.uint32)
fwd = case.startswith("fwd")
if case == "fwd range":
    samples[2] = 0            # block 1: no primary index
if "result" in case:
    fake.fake_bad(ctypes.c_void_p(U[1].ctypes.data))
if "upload" in case:
    fake.fake_bad(ctypes.c_void_p(T[1].ctypes.data))
if fwd:
    fake.fake_samples(ctypes.c_void_p(samples.ctypes.data), ctypes.c_size_t(samples.size))
Job = native.FwdJob if fwd else native.InvJob
jobs = (Job * 2)(*[Job(T[k].ctypes.data, U[k].ctypes.data, N, R, I[k].ctypes.data, 7) for k in range(2)])
call = L.kgbwt_fwd_batch if fwd else L.kgbwt_inv_batch
rc = call(jobs, 2, native.PLAIN)
pending = fake.fake_pending()
fake.fake_drain()
untouched = all((u == 170).all() for u in U)
print(rc, [j.rc for j in jobs], pending, untouched)
if case.endswith("good"):
    assert rc == 0 and all(j.rc == 0 for j in jobs) and not untouched
else:
    assert rc == -2 and all(j.rc == -2 for j in jobs)
    assert untouched or "result" in case
assert pending == 0
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    d = tmp_path_factory.mktemp("fake_runtime")
    (d / "ctl.cu").write_text(CTL_CU)
    (d / "fake.cpp").write_text(FAKE)
    subprocess.run([build.nvcc(), "-std=c++17", "-I", build.INCLUDE, "-I", build.CSRC, "-o", str(d / "ctl"), str(d / "ctl.cu")],
                   check=True)
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-o", str(d / "fake.so"), str(d / "fake.cpp")], check=True)
    size, done = subprocess.run([str(d / "ctl")], check=True, capture_output=True, text=True).stdout.split()
    return str(d / "fake.so"), size, done


@pytest.mark.parametrize("case", ["fwd good", "inv good", "fwd range", "fwd result", "inv result", "fwd upload", "inv upload"])
def test_failed_call_leaves_no_copy_in_flight(fake, case):
    native.lib()  # built
    env = dict(os.environ, LD_PRELOAD=fake[0], PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", CHILD, case, *fake], env=env, capture_output=True, text=True, timeout=120,
                       cwd=ROOT)
    assert r.returncode == 0, r.stdout + r.stderr
