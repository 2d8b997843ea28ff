"""Block lists of the forward engine on a stand-in for the CUDA runtime (no GPU): blocks that overlap are refused before
anything reaches the device (the workspace holds one element per byte of the batch's extent, and the results of two
blocks would share bytes); blocks that only touch, leave gaps or come in another order are taken."""
import pytest

import fake_cuda

CHILD = r"""
import ctypes, sys
import numpy as np
from kolmo_gb300 import native
fake = ctypes.CDLL(sys.argv[1])
fake.fake_setup(ctypes.c_size_t(int(sys.argv[2])), ctypes.c_size_t(int(sys.argv[3])))
L = native.lib()
T, out, I = np.zeros(4096, np.uint8), np.zeros(8192, np.uint8), np.zeros(64, np.int32)
blocks = eval(sys.argv[4])
arr = (native.Block * len(blocks))(*[native.Block(o, n, 1 << 12, k) for k, (o, n) in enumerate(blocks)])
eng = L.kgbwt_engine_create()
rc = L.kgbwt_engine_fwd(eng, T.ctypes.data, out.ctypes.data, I.ctypes.data, None, arr, len(blocks), None, native.PLAIN)
print(rc, fake.fake_launches(), L.kgbwt_last_error())
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    return fake_cuda.compile_fake(tmp_path_factory.mktemp("fake_runtime"))


@pytest.mark.parametrize("blocks,ok", [
    ([(0, 100), (100, 50)], True), ([(100, 50), (0, 100)], True), ([(0, 10), (500, 9), (20, 30)], True),
    ([(0, 100), (99, 50)], False), ([(99, 50), (0, 100)], False), ([(0, 100), (0, 100)], False),
    ([(0, 1000), (2000, 5), (400, 2)], False)])
def test_overlapping_blocks_are_refused(fake, blocks, ok):
    r = fake_cuda.run_child(CHILD, fake, str(blocks))
    assert r.returncode == 0, r.stderr
    rc, launches, err = r.stdout.split(" ", 2)
    if ok:
        assert int(rc) == 0 and int(launches) > 0
    else:
        assert int(rc) == -1 and int(launches) == 0 and "overlap" in err
