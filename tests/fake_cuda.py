"""Test infrastructure: a stand-in for the CUDA runtime, preloaded into a child process without a GPU. Asynchronous copies
stay queued until something waits for the stream, kernels are not launched, read-backs of the control block say that the
sort is done, copies from or to chosen buffers fail, and waits can be held."""
import os
import subprocess
import sys

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
#include <atomic>
#include <unistd.h>
#include <vector>
struct dim3 { unsigned x, y, z; };
namespace {
struct Op { void *dst; const void *src; size_t n; int fill; };
std::vector<Op> ops;                   // queued, not yet done
const char *bad = nullptr;             // copies from or to this buffer fail
const uint32_t *samples = nullptr;     // what the read-back of the sampled indexes gives
size_t nsamples = 0, npair = 0, ctl_size = 0, ctl_done = 0;
int last = 0, launches = 0;
std::atomic<int> hold{0}, waiting{0};  // held: waits for a stream last until released (10 s at most)
void drain() {
    for (const Op &o : ops) if (o.src) memcpy(o.dst, o.src, o.n); else memset(o.dst, o.fill, o.n);
    for (const Op &o : ops) {
        if (o.src && o.n == ctl_size) *(uint32_t *)((char *)o.dst + ctl_done) = 1;
        if (samples && o.src && (o.n == nsamples * 4 || o.n == npair * 4)) memcpy(o.dst, samples, o.n);
    }
    ops.clear();
}
}
extern "C" {
void fake_setup(size_t size, size_t done) { ctl_size = size; ctl_done = done; }
void fake_samples(const uint32_t *v, size_t n) { samples = v; nsamples = n; }
void fake_pair(const uint32_t *v, size_t n) { samples = v; npair = n; }  // read-backs of this size too
void fake_bad(const void *p) { bad = (const char *)p; }
int fake_pending() { return (int)ops.size(); }
void fake_drain() { drain(); }
int fake_launches() { return launches; }
void fake_hold(int on) { hold = on; }
int fake_waiting() { return waiting; }

int cudaMemcpyAsync(void *d, const void *s, size_t n, int, void *) {
    if (bad && (d == bad || s == bad)) return last = 1;
    ops.push_back({d, s, n, 0});
    return 0;
}
int cudaMemsetAsync(void *d, int v, size_t n, void *) { ops.push_back({d, nullptr, n, v}); return 0; }
int cudaMemcpy(void *d, const void *s, size_t n, int) { drain(); memcpy(d, s, n); return 0; }
int cudaMemset(void *d, int v, size_t n) { drain(); memset(d, v, n); return 0; }
int cudaStreamSynchronize(void *) {
    waiting++;
    for (int i = 0; hold && i < 10000; i++) usleep(1000);
    waiting--;
    drain();
    return 0;
}
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
int __cudaLaunchKernel(const void *, dim3, dim3, void **, size_t, void *) { launches++; return 0; }
}
"""


def compile_fake(d):
    """(path of the stand-in, size of the control block, offset of its `done` word), built in directory d."""
    (d / "ctl.cu").write_text(CTL_CU)
    (d / "fake.cpp").write_text(FAKE)
    subprocess.run([build.nvcc(), "-std=c++17", "-I", build.INCLUDE, "-I", build.CSRC, "-o", str(d / "ctl"), str(d / "ctl.cu")],
                   check=True)
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-o", str(d / "fake.so"), str(d / "fake.cpp")], check=True)
    size, done = subprocess.run([str(d / "ctl")], check=True, capture_output=True, text=True).stdout.split()
    return str(d / "fake.so"), size, done


def run_child(code, fake, *args):
    """Runs `code` (its argv: the stand-in's path, the two numbers, then args) with the stand-in preloaded."""
    native.lib()  # built
    env = dict(os.environ, LD_PRELOAD=fake[0], PYTHONPATH=ROOT)
    return subprocess.run([sys.executable, "-c", code, *fake, *args], env=env, capture_output=True, text=True, timeout=120,
                          cwd=ROOT)
