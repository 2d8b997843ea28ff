"""Coalesced calls whose combined batch fails, on a stand-in for the CUDA runtime (no GPU). Each call runs again alone, but
an in-place call (T == U) must not once results have been written: its input may be overwritten by then, and the second run
would return the transform of a transform as if it were right."""
import pytest

import fake_cuda

CHILD = r"""
import ctypes, sys, threading, time
import numpy as np
from kolmo_gb300 import codec, native
fake = ctypes.CDLL(sys.argv[1])
fake.fake_setup(ctypes.c_size_t(int(sys.argv[2])), ctypes.c_size_t(int(sys.argv[3])))
fwd, inplace, failing = sys.argv[4] == "fwd", sys.argv[5] == "in place", sys.argv[6]
L = native.lib()
N, R = 600 << 10, 1 << 19     # two samples a block
samples = np.full(4, 5, np.uint32)
class Call(threading.Thread):
    def __init__(self, inplace):
        super().__init__()
        self.T, self.I = np.full(N, 65, np.uint8), np.full(2, 5, np.int32)
        self.U = self.T if inplace else np.full(N, 170, np.uint8)
        self.rc = None
    def run(self):
        Job = native.FwdJob if fwd else native.InvJob
        job = (Job * 1)(Job(self.T.ctypes.data, self.U.ctypes.data, N, R, self.I.ctypes.data, 7))
        self.rc = (L.kgbwt_fwd_batch if fwd else L.kgbwt_inv_batch)(job, 1, native.PLAIN)
def until(f):
    for _ in range(5000):
        if f():
            return
        time.sleep(0.001)
    raise SystemExit("no progress")
calls_of = lambda: codec.dropin_stats()["fwd_calls" if fwd else "inv_calls"]
first, a, b = Call(False), Call(inplace), Call(False)
if fwd:  # calls alone
    fake.fake_samples(ctypes.c_void_p(samples.ctypes.data), ctypes.c_size_t(2))
fake.fake_hold(1)
first.start()
until(fake.fake_waiting)     # the leader waits for its stream: the next two queue behind it
a.start()
until(lambda: calls_of() == 2)
b.start()
until(lambda: calls_of() == 3)
if failing == "result":
    fake.fake_bad(ctypes.c_void_p(b.U.ctypes.data))
else:
    fake.fake_bad(ctypes.c_void_p(b.T.ctypes.data))
if fwd:  # the two together
    fake.fake_pair(ctypes.c_void_p(samples.ctypes.data), ctypes.c_size_t(4))
fake.fake_hold(0)
for c in (first, a, b):
    c.join()
st = codec.dropin_stats()
print(first.rc, a.rc, b.rc, st)
assert st["fwd_largest" if fwd else "inv_largest"] == 2
assert first.rc == 0 and b.rc == -2
assert a.rc == (-2 if inplace and failing == "result" else 0)
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    return fake_cuda.compile_fake(tmp_path_factory.mktemp("fake_runtime"))


@pytest.mark.parametrize("kind", ["fwd", "inv"])
@pytest.mark.parametrize("where", ["in place", "apart"])
@pytest.mark.parametrize("failing", ["result", "upload"])
def test_in_place_calls_do_not_run_on_their_own_output(fake, kind, where, failing):
    r = fake_cuda.run_child(CHILD, fake, kind, where, failing)
    assert r.returncode == 0, r.stdout + r.stderr
