"""Autotuner for the tile/radix/batch shapes.

Sweeps, on the GPU it runs on:
  - the NTT pass split: levels of the contiguous pass ("r_last") and the most
    levels of a strided column pass ("r_col"), timed on one product per
    scale (the three-prime passes, which serve nn_ntt_mul); and the
    levels of the contiguous pass of batched products ("batch_r_last@s");
  - the batch shapes: the shortest operand sent down the NTT route in a batch
    ("batch_ntt_min", "batch_school_balanced") and the residues a pass item
    covers ("batch_item_words"), timed on the uneven-size workload.
Every candidate's product is checked against the first candidate's (all
choices compute the same exact product).  Writes the best values to
tuning.json beside this file; Context() applies that file at creation
(NN_TUNING=<path> picks another file, NN_TUNING=off none).

    python -m natural_number_gb300.autotune [--n-exps 14,17,20,22,24,26,27] [--batch-scales 13,14,15,16,17] [--jobs 1024]
"""
from __future__ import annotations

import argparse
import json
import os
import time

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
TUNING = os.path.join(HERE, "tuning.json")


def _time(fn, reps: int) -> float:
    import torch
    s = torch.cuda.current_stream()
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    for _ in range(2):  # a batch's second run makes its graph
        fn()
    torch.cuda.synchronize()
    a.record(s)
    for _ in range(reps):
        fn()
    b.record(s)
    torch.cuda.synchronize()
    return a.elapsed_time(b) / reps


def tune_passes(ctx, n_exps) -> tuple[dict, dict]:
    """Per transform scale s = n_exp + 1: the pass split of the three-prime
    2^n_exp x 2^n_exp product (ties keep the default split)."""
    import torch

    from .synth import limbs
    best, log = {}, {}
    for n_exp in n_exps:
        n = 1 << n_exp
        s = n_exp + 1
        a = torch.from_numpy(limbs(11, n)).cuda()
        b = torch.from_numpy(limbs(12, n)).cuda()
        out = torch.empty(2 * n, dtype=torch.uint64, device="cuda")
        ref = None
        results = {}
        reps = max(2, min(20, (1 << 26) // n))
        for r_last in (11, 9, 10, 12):
            for r_col in (9, 8, 7):
                ctx.set_tunable("r_last@%d" % s, r_last)
                ctx.set_tunable("r_col@%d" % s, r_col)
                ms = _time(lambda: ctx.ntt_mul_device(out, a, b, s, 2 * n), reps)
                if ref is None:
                    ref = out.clone()
                elif not torch.equal(ref, out):
                    raise RuntimeError(f"s={s} r_last={r_last} r_col={r_col} changed the product")
                results[f"{r_last},{r_col}"] = ms
        first = min(results.values())
        pick = next(k for k, v in results.items() if v <= first * 1.01)  # default order breaks near-ties
        r_last, r_col = map(int, pick.split(","))
        ctx.set_tunable("r_last@%d" % s, r_last)
        ctx.set_tunable("r_col@%d" % s, r_col)
        best["r_last@%d" % s] = r_last
        best["r_col@%d" % s] = r_col
        log["mul_2^%d_ms" % n_exp] = results
        del a, b, out, ref
    return best, log


def tune_batch_scales(ctx, scales) -> tuple[dict, dict]:
    """Levels of the contiguous pass of two-pass batched transforms (5 to 9),
    timed on a batch of balanced products at each scale, 2^24 transform words
    in all.  The built-in split (0) stays unless another is a tenth faster: its
    tiles are those of the scales beside it, so that a batch of several scales
    has fewer launches (splits 5 % faster here made 70 products of 53 to 19779
    limbs 200 us, 124 with the built-in ones)."""
    import torch

    from .workloads import MulJob
    best, log = {}, {}
    for s in scales:
        n = (1 << (s - 1)) - 1
        count = max(16, (1 << 24) >> s)
        g = torch.Generator(device="cuda")
        g.manual_seed(s)
        a = torch.randint(0, 2**62, (n * count,), dtype=torch.int64, device="cuda", generator=g).view(torch.uint64)
        b = torch.randint(0, 2**62, (n * count,), dtype=torch.int64, device="cuda", generator=g).view(torch.uint64)
        out = torch.zeros(2 * n * count, dtype=torch.uint64, device="cuda")
        jobs = (MulJob * count)()
        for j in range(count):
            jobs[j] = MulJob(a.data_ptr() + 8 * n * j, n, b.data_ptr() + 8 * n * j, n, out.data_ptr() + 16 * n * j)
        sizes = np.full(count, n, dtype=np.uint64)
        results, ref = {}, None
        for r_last in (0, 9, 8, 7, 6, 5):
            if r_last and not 4 <= s - 3 - r_last <= 9:
                continue
            ctx.set_tunable("batch_r_last@%d" % s, r_last)
            plan = ctx.batch(sizes, sizes)
            ms = _time(lambda: plan.run_jobs(jobs), 5)
            ctx.synchronize()
            plan.close()
            if ref is None:
                ref = out.clone()
            elif not torch.equal(ref, out):
                raise RuntimeError(f"s={s} r_last={r_last} changed a product")
            results[str(r_last)] = ms
        pick = int(min(results, key=results.get))
        if results[str(pick)] > 0.9 * results["0"]:
            pick = 0
        ctx.set_tunable("batch_r_last@%d" % s, pick)
        best["batch_r_last@%d" % s] = pick
        log["batch_scale_%d_ms" % s] = results
        del a, b, out, ref
    return best, log


def tune_batch(ctx, jobs: int) -> tuple[dict, dict]:
    """The shortest operand sent down the NTT route and the residues per pass
    item, then the base case of balanced products, on an uneven workload of
    `jobs` products; every setting must give the same products.  (Items of fewer
    than 8192 words are no faster here and double the time to plan a batch.)"""
    import torch

    from .workloads import UnevenProducts
    W = UnevenProducts(jobs, seed=5)
    ref = None

    def ms(settings: dict) -> float:
        nonlocal ref
        for name, value in settings.items():
            ctx.set_tunable(name, value)
        plan = ctx.batch(W.sa, W.sb)
        t = _time(lambda: plan.run_jobs(W.jobs_batch), 3)
        ctx.synchronize()
        plan.close()
        if ref is None:
            ref = W.out_batch.clone()
        elif not torch.equal(ref, W.out_batch):
            raise RuntimeError(f"{settings} changed a product")
        return t

    shapes = {f"{ntt_min},{item}": ms({"batch_ntt_min": ntt_min, "batch_item_words": item})
              for ntt_min in (32, 64, 128, 256) for item in (8192, 16384, 32768)}
    ntt_min, item = map(int, min(shapes, key=shapes.get).split(","))
    best = {"batch_ntt_min": ntt_min, "batch_item_words": item}
    balanced = {str(v): ms({**best, "batch_school_balanced": v}) for v in (0, 56, 112, 224, 448)}
    best["batch_school_balanced"] = int(min(balanced, key=balanced.get))
    for name, value in best.items():
        ctx.set_tunable(name, value)
    return best, {"batch_%d_ms" % jobs: shapes, "batch_%d_balanced_ms" % jobs: balanced}


def main() -> None:
    import torch

    from . import Context
    ap = argparse.ArgumentParser()
    ap.add_argument("--n-exps", default="14,17,20,22,24,26,27")
    ap.add_argument("--batch-scales", default="13,14,15,16,17")
    ap.add_argument("--jobs", type=int, default=1024)
    ap.add_argument("--out", default=TUNING)
    args = ap.parse_args()
    os.environ["NN_TUNING"] = "off"
    ctx = Context(0)
    t0 = time.time()
    best, log = {}, {}
    b, l = tune_passes(ctx, [int(x) for x in args.n_exps.split(",")])
    best.update(b)
    log.update(l)
    b, l = tune_batch(ctx, args.jobs)
    best.update(b)
    log.update(l)
    b, l = tune_batch_scales(ctx, [int(x) for x in args.batch_scales.split(",")])
    best.update(b)
    log.update(l)
    doc = {"tunables": best, "device": torch.cuda.get_device_name(0), "seconds": round(time.time() - t0, 1),
           "timings_ms": log}
    with open(args.out, "w") as f:
        json.dump(doc, f, indent=1)
    print(json.dumps(doc))


def apply(ctx, path: str | None = None) -> dict:
    """Applies tuning.json (or NN_TUNING) to a context; returns what it set."""
    path = path or os.environ.get("NN_TUNING", TUNING)
    if path == "off" or not os.path.exists(path):
        return {}
    with open(path) as f:
        tun = json.load(f).get("tunables", {})
    for k, v in tun.items():
        ctx.set_tunable(k, int(v))
    return tun


if __name__ == "__main__":
    main()
