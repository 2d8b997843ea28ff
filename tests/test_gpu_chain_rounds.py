"""When rank rounds follow repeat chains: only where at least half of the suffixes that doubling leaves are in groups of
2-8. Texts of a random stretch written 2, 5 or 20 times, with a shorter stretch written twice beside it: the first two
stall in tiny groups and take chains, the third in groups of 20 and takes none. U, sampled indexes and suffix array
against the oracle either way, on the plain path and from the graph."""
import numpy as np
import pytest

import oracle as O
from kolmo_gb300 import codec

pytestmark = pytest.mark.gpu


def _text(copies, seed):
    rng = np.random.default_rng(seed)
    long = rng.integers(97, 101, 3000).astype(np.uint8)
    short = rng.integers(97, 101, 500).astype(np.uint8)
    out = []
    for s in [long] * copies + [short] * 2:  # 16 random bytes end every copy
        out += [s, rng.integers(0, 256, 16).astype(np.uint8)]
    return np.concatenate(out)


@pytest.mark.parametrize("copies,chains", [(2, True), (5, True), (20, False)])
def test_chains_follow_tiny_groups(copies, chains):
    import torch

    t = _text(copies, copies)
    n, r = t.size, 1 << 8
    dT = torch.from_numpy(np.concatenate([t, np.zeros(64, np.uint8)])).cuda()
    dL = torch.zeros(n + 64, dtype=torch.uint8, device="cuda")
    dI = torch.zeros((n - 1) // r + 1, dtype=torch.int32, device="cuda")
    dSA = torch.zeros(n, dtype=torch.int32, device="cuda")
    oU, oI = O.bwt_aux(t, r)[1:]
    oSA = O.suffix_array(t)
    eng = codec.Engine()
    eng.config(lsd_round0=1, lsd_bytes=8, chain_from=1)
    eng.profile(True)
    for plain in (True, False, False):  # the last one runs from the captured graph
        assert eng.fwd(dT, dL, dI, [(0, n, r, 0)], dSA=dSA, plain=plain) == 0
        assert eng.wait()[0] == 0
        if plain:
            assert any(p["kernel"] == "chain" for p in eng.profile_read()) == chains
        I, L = dI.cpu().numpy(), dL.cpu().numpy()[: n + 1]
        p0 = int(I[0])
        assert np.array_equal(I, oI)
        assert np.array_equal(np.concatenate([L[:p0], L[p0 + 1:]]), oU)
        assert np.array_equal(dSA.cpu().numpy(), oSA)
    eng.close()
