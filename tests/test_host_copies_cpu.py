"""The host side of the batch calls on a stand-in for the CUDA runtime (no GPU): when a call fails, no copy from or to
its callers' buffers may still be in flight, and a block whose result is out of range leaves every buffer as it was."""
import pytest

import fake_cuda

CHILD = r"""
import ctypes, sys
import numpy as np
from kolmo_gb300 import native
fake_path, size, done, case = sys.argv[1], int(sys.argv[2]), int(sys.argv[3]), sys.argv[4]
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
    return fake_cuda.compile_fake(tmp_path_factory.mktemp("fake_runtime"))


@pytest.mark.parametrize("case", ["fwd good", "inv good", "fwd range", "fwd result", "inv result", "fwd upload", "inv upload"])
def test_failed_call_leaves_no_copy_in_flight(fake, case):
    r = fake_cuda.run_child(CHILD, fake, case)
    assert r.returncode == 0, r.stdout + r.stderr
