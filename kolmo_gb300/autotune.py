"""Autotuner of the forward sort: times candidate configurations on this GPU for batches of several sizes and writes
the tuning table (JSON, one bucket per batch size) that the library loads (kgbwt_tuning_load, KGBWT_TUNING, or
tuning_gb300.json beside this package). Results never depend on the configuration; only the time does.

    python -m kolmo_gb300.autotune --out kolmo_gb300/tuning_gb300.json [--reps 7] [--quick]

Tuned per bucket: CTAs per SM of the block tile kernel (tile_ctas) and of the bucket passes (msd_ctas), the
counting-sort threshold of the tile kernel (small_group), the warp-level tile path (warp_path), the round-0 path
(lsd_round0: one LSD radix sort of all suffixes, or bucket passes + tiles), the key it sorts (lsd_bytes: 16 or
12 bytes of text, or 8 of an order-preserving code of it) and whether rank rounds follow repeat chains (chain_from: 1 or
0). The tile capacity changes the workspace layout and is left at its default. A bucket's fwd_ms and default_fwd_ms are the
geometric means over its batches.
"""
from __future__ import annotations

import argparse
import itertools
import json
import os
import statistics
import sys

import numpy as np

from . import codec
from . import workloads as W
from .host import codec18_rlog, n_samples

MIB = 1 << 20

# (label, measured batches) per bucket; a bucket covers batches up to twice its measured size. The sources differ in what
# they ask of a configuration, so a bucket is timed on all of them: prose with copied stretches in proportion to its
# length ("prose", 200 in 64 MiB, as the benchmark's block), prose copied over and over ("copies", 200 at every length),
# log lines and Markov bytes.
BUCKETS = [
    ("1 MiB of prose, copies, logs, Markov", [(src, 1 * MIB) for src in ("prose", "copies", "logs", "markov")]),
    ("4 MiB of prose, copies, logs, Markov", [(src, 4 * MIB) for src in ("prose", "copies", "logs", "markov")]),
    ("16 MiB of prose, copies, logs, Markov", [(src, 16 * MIB) for src in ("prose", "copies", "logs", "markov")]),
    ("64 MiB of prose, logs, Markov", [(src, 64 * MIB) for src in ("prose", "logs", "markov")]),
    ("96 mixed blocks, log-uniform 16 KiB-16 MiB", ["mixed96"]),
]

CANDIDATES = {
    "lsd_round0": (1, 0),
    "lsd_bytes": (16, 12, 8),
    "msd_ctas": (8, 4),
    "tile_ctas": (2, 1),
    "small_group": (64, 0),
    "warp_path": (1, 0),
    "chain_from": (1, 0),
}


def _batch(spec, seed):
    if spec == "mixed96":  # the mixed batch's shape (sources and size law) on another seed
        return [t for _, t in W.mixed_batch(96, seed=seed)]
    src, n = spec
    if src in ("prose", "copies"):
        return [W.zipf_prose(n, seed, ncopies=200 if src == "copies" else max(1, 200 * n // (64 * MIB)))]
    return [W.source_block(W.SOURCES.index(src), n, seed)]


def _time_config(texts, cfg, reps):
    """Median forward time (ms, graph path, CUDA events) of the batch under one configuration."""
    import torch

    offs, o = [], 0
    for t in texts:
        offs.append(o)
        o += (t.size + 15) // 16 * 16
    buf = np.zeros(o + 64, np.uint8)
    for t, off in zip(texts, offs):
        buf[off:off + t.size] = t
    blocks, k = [], 0
    for t, off in zip(texts, offs):
        r = 1 << codec18_rlog(int(t.size))
        blocks.append((off, int(t.size), r, k))
        k += n_samples(int(t.size), r)
    dT = torch.from_numpy(buf).cuda()
    dL = torch.zeros(o + len(texts) + 64, dtype=torch.uint8, device="cuda")
    dI = torch.zeros(k, dtype=torch.int32, device="cuda")
    eng = codec.Engine()
    eng.config(0, cfg["tile_ctas"], cfg["msd_ctas"], cfg["small_group"], cfg["warp_path"], cfg["lsd_round0"],
               cfg["lsd_bytes"], cfg["chain_from"])
    s = torch.cuda.Stream()
    times = []
    ref = None
    for it in range(reps + 2):  # call 0 runs plain (a new shape), call 1 captures the graph, the rest are timed
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(s)
        if eng.fwd(dT, dL, dI, blocks, stream=s) or eng.wait()[0]:
            raise RuntimeError("forward failed during tuning")
        e1.record(s)
        s.synchronize()
        if it >= 2:
            times.append(e0.elapsed_time(e1))
        if ref is None:
            ref = dI.cpu().numpy().copy()
    assert np.array_equal(ref, dI.cpu().numpy())  # same result under every configuration
    eng.close()
    return statistics.median(times), ref


def candidate_grid(quick: bool = False) -> list:
    """Every configuration the tuner times (the key only varies on the LSD round 0); quick: the first four."""
    keys = list(CANDIDATES)
    grid = [dict(zip(keys, vals)) for vals in itertools.product(*(CANDIDATES[k] for k in keys))]
    grid = [g for g in grid if g["lsd_round0"] or g["lsd_bytes"] == CANDIDATES["lsd_bytes"][0]]
    return grid[:4] if quick else grid


def default_config() -> dict:
    """The library's defaults: each field's first candidate."""
    return {k: v[0] for k, v in CANDIDATES.items()}


FINALISTS = 8


def tune(reps: int = 7, quick: bool = False, log=print):
    """Per bucket: every candidate timed on each batch, then the FINALISTS best and the default again, in turn, so that
    drift of the GPU's clocks meets all alike. A configuration's figure is the geometric mean over the batches of its
    median times."""
    import torch

    grid = candidate_grid(quick)
    default = default_config()
    buckets = []
    for bi, (name, specs) in enumerate(BUCKETS if not quick else BUCKETS[:2]):
        batches = [_batch(spec, 0x5EED + 97 * bi) for spec in specs]
        refs = [None] * len(batches)

        def timed(cfg, n):
            out = []
            for k, texts in enumerate(batches):
                ms, ref = _time_config(texts, cfg, n)
                refs[k] = ref if refs[k] is None else refs[k]
                assert np.array_equal(refs[k], ref), "configurations disagree"  # results never depend on them
                out.append(ms)
            return out

        first = sorted(((statistics.geometric_mean(timed(c, 3)), i) for i, c in enumerate(grid)))
        final = [grid[i] for _, i in first[:FINALISTS]]
        if default not in final:
            final.append(default)
        rounds = [[timed(c, 5) for c in final] for _ in range(reps)]
        ms = [[statistics.median(r[f][k] for r in rounds) for k in range(len(batches))] for f in range(len(final))]
        mean = [statistics.geometric_mean(m) for m in ms]
        best, dflt = mean.index(min(mean)), final.index(default)
        log(f"{name}: best {final[best]} {mean[best]:.3f} ms (default {mean[dflt]:.3f} ms)")
        for f in sorted(range(len(final)), key=lambda f: mean[f]):
            log(f"    {mean[f]:.4f} ms  " + " ".join(f"{m:.4f}" for m in ms[f]) + f"  {final[f]}")
        buckets.append({"max_bytes": 2 * sum(int(t.size) for t in batches[0]), **final[best],
                        "fwd_ms": round(mean[best], 4), "default_fwd_ms": round(mean[dflt], 4), "workload": name})
    buckets[-1]["max_bytes"] = 1 << 40
    return {"version": 1, "device": torch.cuda.get_device_name(), "generated_by": "kolmo_gb300/autotune.py",
            "reps": reps, "buckets": buckets}


def main(argv=None):
    ap = argparse.ArgumentParser(description=__doc__.splitlines()[0])
    ap.add_argument("--out", default=os.path.join(os.path.dirname(os.path.abspath(__file__)), "tuning_gb300.json"))
    ap.add_argument("--reps", type=int, default=7)
    ap.add_argument("--quick", action="store_true", help="two buckets, four candidates (a smoke run)")
    args = ap.parse_args(argv)
    # measure without any table: every candidate sets all tuned fields explicitly anyway
    codec.tuning_load(None)
    table = tune(args.reps, args.quick)
    with open(args.out, "w") as f:
        json.dump(table, f, indent=1)
    print(f"wrote {args.out} ({len(table['buckets'])} buckets)")
    return 0


if __name__ == "__main__":
    sys.exit(main())
