"""The workloads this library is measured on: forward and inverse BWT calls through its public entry points.

Two ways in, as programs use them:

* ``host``: the drop-in C entry points (``kolmo_sais_bwt_aux``, ``kolmo_sais_unbwt_aux``) on the caller's own pageable
  buffers, as the block codecs call them; the copies to and from the device are part of the call.
* ``engine``: ``codec.Engine`` on device-resident buffers, one call for a whole batch of blocks, as a server or a
  pipeline that keeps its data on the GPU calls it, with the wait that reports errors.

A case is ``{"name", "dir": "fwd" | "inv", "via", "source", "blocks", "lo", "hi", "sa"}``: `blocks` blocks of
log-uniform lengths in [lo, hi] bytes (a single block has `hi` bytes; equal bounds give equal lengths), `sa` asks the
forward call for the suffix array too. Sampling intervals follow codec 18's rule. Texts come from the package's seeded
generators.
"""
import math
import random
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

from kolmo_gb300 import codec, native
from kolmo_gb300 import workloads as W
from kolmo_gb300.host import codec18_rlog, n_samples

KIB, MIB = 1 << 10, 1 << 20
#: Order-2 Markov bytes, ACGT reads, log lines, word prose with verbatim copies; "mixed": the first three in turn.
TEXTS = ("markov", "acgt", "logs", "prose")
#: Periodic texts (one flipped byte a MiB) and the Fibonacci word: padding, tables of equal records, run-length data.
DEGENERATE = ("periodic-1", "periodic-7", "periodic-4096", "fibonacci")


def _case(name, dir, via, source, blocks, lo, hi, sa=False):
    c = {"dir": dir, "via": via, "source": source, "blocks": blocks, "lo": lo, "hi": hi, "sa": sa}
    return dict(c, name=name) if name else c


def listed():
    return [
        # a small file through the codec: latency and launches
        _case("host fwd logs 20 KB", "fwd", "host", "logs", 1, 20011, 20011),
        _case("host inv logs 20 KB", "inv", "host", "logs", 1, 20011, 20011),
        # one 1 MiB Markov block (the smallest benchmark configuration); the forward with its suffix array
        _case("fwd markov 1 MiB + SA", "fwd", "engine", "markov", 1, MIB, MIB, True),
        _case("inv markov 1 MiB", "inv", "engine", "markov", 1, MIB, MIB),
        # the level-9 planner's trial sorts: consecutive 512 KiB slices of one text, one batch
        _case("fwd prose 64 x 512 KiB", "fwd", "engine", "prose", 64, 512 * KIB, 512 * KIB),
        # a batch of uneven blocks, 16 KiB to 16 MiB: what a server coalesces
        _case("fwd mixed 64 blocks", "fwd", "engine", "mixed", 64, 16 * KIB, 16 * MIB),
        _case("inv mixed 64 blocks", "inv", "engine", "mixed", 64, 16 * KIB, 16 * MIB),
        # one block of a level-8 frame (32 MiB of log lines, less what LZP took out), from and to host memory
        _case("host fwd logs 30 MB", "fwd", "host", "logs", 1, 30146503, 30146503),
        _case("host inv logs 30 MB", "inv", "host", "logs", 1, 30146503, 30146503),
        # the 64 MiB prose block: the headline configuration, both directions
        _case("fwd prose 64 MiB", "fwd", "engine", "prose", 1, 64 * MIB, 64 * MIB),
        _case("inv prose 64 MiB", "inv", "engine", "prose", 1, 64 * MIB, 64 * MIB),
        # the largest and most repetitive block: 4096-byte records repeated over 128 MiB
        _case("fwd periodic-4096 128 MiB", "fwd", "engine", "periodic-4096", 1, 128 * MIB, 128 * MIB),
    ]


def _log_size(rng, lo, hi):
    """A size spread over the logarithm of [lo, hi], mostly odd and ragged, a round one now and then."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if rng.random() < 0.2:
        n = max(lo, n >> 12 << 12)
    return min(hi, max(lo, n))


def draw(rng):
    dir = rng.choice(("fwd", "inv"))
    kind = rng.random()
    if kind < 0.3:  # one block from host memory, as the codecs send it
        n = _log_size(rng, 2 * KIB, 32 * MIB)
        return _case(None, dir, "host", rng.choice(TEXTS), 1, n, n)
    if kind < 0.6:  # one device-resident block
        n = _log_size(rng, 16 * KIB, 64 * MIB)
        return _case(None, dir, "engine", rng.choice(TEXTS), 1, n, n, dir == "fwd" and rng.random() < 0.3)
    if kind < 0.85:  # a batch
        count = _log_size(rng, 2, 96)
        hi = _log_size(rng, 64 * KIB, 16 * MIB)
        lo = hi if rng.random() < 0.25 else _log_size(rng, 16 * KIB, hi)
        hi = max(lo, min(hi, 192 * MIB // count))
        lo = min(lo, hi)
        return _case(None, dir, "engine", rng.choice(TEXTS + ("mixed",)), count, lo, hi,
                     dir == "fwd" and rng.random() < 0.2)
    n = _log_size(rng, 64 * KIB, 64 * MIB)
    return _case(None, dir, "engine", rng.choice(DEGENERATE), 1, n, n)


def _sizes(case):
    """Block lengths: a property of the case, the same for every seed."""
    count, lo, hi = case["blocks"], case["lo"], case["hi"]
    if lo == hi or count == 1:
        return [hi] * count
    rng = random.Random(f"{count}/{lo}/{hi}")
    return [min(hi, max(lo, int(math.exp(rng.uniform(math.log(lo), math.log(hi)))))) for _ in range(count)]


def _text(source, n, seed):
    if source == "prose":  # as many verbatim copies per byte as in the 64 MiB block
        return W.zipf_prose(n, seed, ncopies=max(1, 200 * n // (64 * MIB)))
    if source == "fibonacci":  # every seed another stretch of the word
        skip = seed % 4099
        return np.ascontiguousarray(W.fibonacci(n + skip)[skip:])
    if source.startswith("periodic-"):
        return W.periodic(n, seed, int(source.split("-")[1]))
    return W.source_block(W.SOURCES.index(source), n, seed)


def _texts(case, seed):
    sizes, source = _sizes(case), case["source"]
    if source == "prose" and len(sizes) > 1:  # consecutive stretches of one text
        whole, cuts = _text(source, sum(sizes), seed), np.cumsum(sizes)[:-1]
        return [np.ascontiguousarray(t) for t in np.split(whole, cuts)]
    of = [source if source != "mixed" else W.SOURCES[k % 3] for k in range(len(sizes))]
    with ThreadPoolExecutor(8) as pool:
        return list(pool.map(lambda k: _text(of[k], sizes[k], seed * 1000003 + k), range(len(sizes))))


def _layout(case):
    """(offset, length, sampling interval, first sampled index) of every block of a device batch, and the totals."""
    blocks, off, iout = [], 0, 0
    for n in _sizes(case):
        r = 1 << codec18_rlog(n)
        blocks.append((off, n, r, iout))
        off += (n + 15) // 16 * 16
        iout += n_samples(n, r)
    return blocks, off, iout


def _device_forward(texts, case, sa):
    blocks, end, samples = _layout(case)
    flat = np.zeros(end + 64, np.uint8)
    for t, (off, n, _, _) in zip(texts, blocks):
        flat[off:off + n] = t
    s = {"engine": codec.Engine(), "blocks": blocks, "T": torch.from_numpy(flat).cuda(),
         "L": torch.zeros(end + len(blocks), dtype=torch.uint8, device="cuda"),
         "I": torch.zeros(samples, dtype=torch.int32, device="cuda"),
         "SA": torch.zeros(end, dtype=torch.int32, device="cuda") if sa else None}
    return s


def _checked(rc):
    if rc:
        raise RuntimeError(f"call failed ({rc}): {native.last_error()}")


def _forward(s):
    e = s["engine"]
    _checked(e.fwd(s["T"], s["L"], s["I"], s["blocks"], dSA=s["SA"]))
    _checked(e.wait()[0])


def prepare(case, seed):
    texts = _texts(case, seed)
    if case["via"] == "host" and case["dir"] == "fwd":
        return dict(_host_buffers(texts[0], case), **{"dir": "fwd", "via": "host"})
    s = dict(_device_forward(texts, case, case["sa"]), dir=case["dir"], via=case["via"])
    if case["dir"] == "fwd":
        return s
    # an inverse call's input: the BWT strings (the L columns without their sentinel rows) and the sampled indexes
    _forward(s)
    I = s["I"].cpu().numpy()
    U, iblocks = torch.zeros_like(s["T"]), []
    for b, (off, n, _, iout) in enumerate(s["blocks"]):
        p0 = int(I[iout])
        U[off:off + p0] = s["L"][off + b:off + b + p0]
        U[off + p0:off + n] = s["L"][off + b + p0 + 1:off + b + n + 1]
        iblocks.append((off, n, p0))
    s["engine"].close()
    if case["via"] == "host":
        h = _host_buffers(U[:texts[0].size].cpu().numpy(), case)
        h["I"][:] = I
        return dict(h, dir="inv", via="host")
    return {"engine": codec.Engine(), "blocks": iblocks, "U": U, "out": torch.zeros_like(U), "dir": "inv",
            "via": "engine"}


def _host_buffers(data, case):
    n = int(data.size)
    r = 1 << codec18_rlog(n)
    return {"in": data, "out": np.zeros(n, np.uint8), "A": np.zeros(1, np.int32), "n": n, "r": r,
            "I": np.zeros(n_samples(n, r), np.int32)}


def run(s):
    if s["via"] == "host":
        call = native.lib().kolmo_sais_bwt_aux if s["dir"] == "fwd" else native.lib().kolmo_sais_unbwt_aux
        _checked(call(s["in"].ctypes.data, s["out"].ctypes.data, s["A"].ctypes.data, s["n"], s["r"],
                      s["I"].ctypes.data, 1))
        return {"U": s["out"], "I": s["I"]} if s["dir"] == "fwd" else {"T": s["out"]}
    if s["dir"] == "fwd":
        _forward(s)
        return {k: s[k] for k in ("L", "I", "SA") if s[k] is not None}
    _checked(s["engine"].inv(s["U"], s["out"], s["blocks"]))
    rc, status = s["engine"].wait(len(s["blocks"]))
    _checked(rc)
    return {"T": s["out"], "status": status}


def work(case):
    """Text read and BWT written once (and the reverse), the sampled indexes, the suffix array where asked for."""
    nbytes = sum(2 * n + 4 * n_samples(n, 1 << codec18_rlog(n)) + (4 * n if case["sa"] else 0) for n in _sizes(case))
    return {"bytes": nbytes, "flops": 0}


def _suffix_array(t):
    """Prefix doubling in numpy (the shorter of two equal prefixes sorts first)."""
    n, h = t.size, 1
    rank = t.astype(np.int64) + 1
    while True:
        key = rank * (max(256, n) + 2)
        key[:max(0, n - h)] += rank[h:] if h < n else 0
        sa = np.argsort(key, kind="stable")
        k = key[sa]
        new = np.concatenate([[1], 1 + np.cumsum(k[1:] != k[:-1])])
        rank = np.empty(n, np.int64)
        rank[sa] = new
        if new[-1] == n or h >= n:
            return sa
        h *= 2


def exact(case, seed):
    """The decoded texts of an inverse call; for forward calls of up to 1 MiB, the BWT from a suffix array by numpy."""
    texts = _texts(case, seed)
    blocks, end, samples = _layout(case)
    if case["dir"] == "inv":
        if case["via"] == "host":
            return {"T": texts[0]}
        out = np.zeros(end + 64, np.uint8)
        for t, (off, n, _, _) in zip(texts, blocks):
            out[off:off + n] = t
        return {"T": out, "status": np.zeros(len(blocks), np.int32)}
    if sum(t.size for t in texts) > MIB or case["source"] in DEGENERATE:
        return None
    L, I, SA = np.zeros(end + len(blocks), np.uint8), np.zeros(samples, np.int32), np.zeros(end, np.int32)
    for b, (t, (off, n, r, iout)) in enumerate(zip(texts, blocks)):
        sa = _suffix_array(t)
        SA[off:off + n] = sa
        L[off + b] = t[-1]
        L[off + b + 1:off + b + n + 1] = np.where(sa > 0, t[sa - 1], 0)
        rank = np.empty(n, np.int64)
        rank[sa] = np.arange(n)
        I[iout:iout + n_samples(n, r)] = rank[::r][:n_samples(n, r)] + 1
    if case["via"] == "host":
        p0 = int(I[0])
        n = texts[0].size
        return {"U": np.concatenate([L[:p0], L[p0 + 1:n + 1]]), "I": I}
    return {"L": L, "I": I, "SA": SA} if case["sa"] else {"L": L, "I": I}
