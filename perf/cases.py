"""The calls whose speed is watched, over the range that a user's program makes.

Products, squares, divisions and decimal conversion go through
natural_number_gb300.Context as a program calls it: one context per process,
operands already where the program keeps them (device memory for the device
calls, page-locked host memory for the host product, as the drop-in natural
keeps its limbs), outputs in buffers that the program owns.  Limbs are uniform
random u64, the values long naturals have.  All results are whole numbers and
compare bit for bit.
"""
import math

import numpy as np
import torch

import natural_number_gb300 as nn

_context = None


def _ctx():
    """The program's one context (its twiddle tables grow with the largest size seen)."""
    global _context
    if _context is None:
        _context = nn.Context(0)
    return _context


def listed():
    return [
        # A pass over many short naturals: the base case, where launches and latency are everything.
        {"name": "mul_64x48", "kind": "mul", "na": 64, "nb": 48},
        # Just above the base case: the smallest transforms, ragged operands.
        {"name": "mul_1500x1201", "kind": "mul", "na": 1500, "nb": 1201},
        # An ordinary product of no special size (1.7 million digits by 1.3 million).
        {"name": "mul_90001x70007", "kind": "mul", "na": 90001, "nb": 70007},
        # The plain product of 2^20 limbs.
        {"name": "mul_1048576", "kind": "mul", "na": 1 << 20, "nb": 1 << 20},
        # The largest: 2^27 limbs (1 GiB) an operand.
        {"name": "mul_134217728", "kind": "mul", "na": 1 << 27, "nb": 1 << 27},
        # A long natural times a short one (a scaling or a partial quotient times a divisor).
        {"name": "mul_3000000x5003", "kind": "mul", "na": 3000000, "nb": 5003},
        # Squaring, as pow does, at an odd length.
        {"name": "sqr_6000001", "kind": "sqr", "na": 6000001},
        # One operand's transform is kept and multiplied again and again (mul_save / mul_load).
        {"name": "cached_100000x140001", "kind": "cached", "na": 100000, "nb": 140001},
        # Thousands of independent products of uneven lengths, planned once, run many times.
        {"name": "batch_4096_uneven", "kind": "batch", "count": 4096, "lo": 1 << 6, "hi": 1 << 18},
        # Quotient and remainder of a 2n- by n-limb division, every step on the device.
        {"name": "div_2800007x1400003", "kind": "div", "na": 2800007, "nb": 1400003},
        # operator* on naturals in host memory: copies in, product, copy out.
        {"name": "host_mul_1048576", "kind": "host_mul", "na": 1 << 20, "nb": 1 << 20},
        # Printing a natural: about 3.8 million decimal digits from host limbs.
        {"name": "to_dec_200003", "kind": "dec", "na": 200003},
    ]


def _log_uniform(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng):
    kind = rng.choice(["mul", "mul", "mul", "unbalanced", "sqr", "cached", "batch", "div", "host_mul", "dec"])
    if kind == "mul":  # lengths of the same order
        na = _log_uniform(rng, 16, 1 << 26)
        return {"kind": "mul", "na": na, "nb": max(8, int(na * rng.uniform(0.5, 1.0)))}
    if kind == "unbalanced":  # any two lengths
        na = _log_uniform(rng, 1 << 10, 1 << 24)
        return {"kind": "mul", "na": na, "nb": _log_uniform(rng, 16, na)}
    if kind == "sqr":
        return {"kind": "sqr", "na": _log_uniform(rng, 16, 1 << 26)}
    if kind == "cached":
        na = _log_uniform(rng, 1 << 10, 1 << 22)
        return {"kind": "cached", "na": na, "nb": max(8, int(na * rng.uniform(0.3, 1.0)))}
    if kind == "batch":
        return {"kind": "batch", "count": _log_uniform(rng, 64, 4096), "lo": _log_uniform(rng, 8, 128),
                "hi": _log_uniform(rng, 1 << 10, 1 << 17)}
    if kind == "div":
        na = _log_uniform(rng, 1 << 9, 1 << 22)
        return {"kind": "div", "na": na, "nb": max(16, int(na * rng.uniform(0.3, 0.7)))}
    if kind == "host_mul":
        na = _log_uniform(rng, 1 << 8, 1 << 22)
        return {"kind": "host_mul", "na": na, "nb": max(16, int(na * rng.uniform(0.5, 1.0)))}
    return {"kind": "dec", "na": _log_uniform(rng, 1 << 10, 1 << 19)}


def _limbs(gen, n):
    """n uniform limbs on the GPU, the top one nonzero, as int64 words."""
    t = torch.randint(-(1 << 63), (1 << 63) - 1, (n,), generator=gen, device="cuda", dtype=torch.int64)
    t[-1] |= 1
    return t


def _inputs(case, seed):
    """The operands of a case as int64 words (a batch: one pool holding all of them)."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    if case["kind"] == "batch":
        na, nb, oa, ob, _, words, _ = _batch_layout(case)
        return (_limbs(gen, words),)
    got = [_limbs(gen, case["na"])]
    if "nb" in case:
        got.append(_limbs(gen, case["nb"]))
    return tuple(got)


def _scale(case):
    """The transform scale of a cached product: 2^s holds its na + nb - 1 coefficients."""
    return max(2, (case["na"] + case["nb"] - 2).bit_length())


def _batch_layout(case):
    """Operand lengths (log-uniform, drawn independently, the same for every seed) and where each operand and product
    starts, 256-byte aligned as an allocator gives them."""
    rng = np.random.default_rng([case["count"], case["lo"], case["hi"]])
    lo, hi = math.log(case["lo"]), math.log(case["hi"] + 1)
    n = np.clip(np.exp(rng.uniform(lo, hi, (2, case["count"]))).astype(np.int64), case["lo"], case["hi"])
    na, nb = n
    up = lambda v: (v + 31) // 32 * 32  # noqa: E731
    starts = np.concatenate([[0], np.cumsum(up(np.concatenate([na, nb])))])
    outs = np.concatenate([[0], np.cumsum(up(na + nb))])
    return na, nb, starts[: na.size], starts[na.size: -1], outs[:-1], int(starts[-1]), int(outs[-1])


def _pinned(words):
    """A page-locked numpy array of u64 limbs holding the given device words."""
    t = torch.empty(words.numel(), dtype=torch.int64, pin_memory=True)
    t.copy_(words)
    return t, t.numpy().view(np.uint64)


def prepare(case, seed):
    ctx = _ctx()
    kind = case["kind"]
    words = _inputs(case, seed)
    u64 = [w.view(torch.uint64) for w in words]
    empty = lambda n: torch.empty(n, dtype=torch.int64, device="cuda")  # noqa: E731
    state = {"ctx": ctx, "kind": kind, "in": u64}
    if kind == "mul":
        state["out"] = empty(case["na"] + case["nb"])
    elif kind == "sqr":
        state["out"] = empty(2 * case["na"])
    elif kind == "cached":
        s = _scale(case)
        state["scale"] = s
        state["kept"] = ctx.transform().forward(u64[0], s)
        state["work"], state["prod"] = ctx.transform(), ctx.transform()
        state["out"] = empty(case["na"] + case["nb"])
    elif kind == "batch":
        na, nb, oa, ob, oo, _, out_words = _batch_layout(case)
        state["out"] = torch.zeros(out_words, dtype=torch.int64, device="cuda")
        a0, o0 = words[0].data_ptr(), state["out"].data_ptr()
        jobs = (nn.MulJob * int(na.size))()
        for k in range(na.size):
            jobs[k] = nn.MulJob(a0 + 8 * int(oa[k]), int(na[k]), a0 + 8 * int(ob[k]), int(nb[k]), o0 + 8 * int(oo[k]))
        state["jobs"], state["plan"] = jobs, ctx.batch(na, nb)
    elif kind == "div":
        state["q"], state["r"] = empty(case["na"] - case["nb"] + 1), empty(case["nb"])
    elif kind == "host_mul":
        state["keep"], state["host"] = zip(*[_pinned(w) for w in words])
        out = torch.empty(case["na"] + case["nb"], dtype=torch.int64, pin_memory=True)
        state["keep"] += (out,)
        state["host_out"] = out.numpy().view(np.uint64)
    else:
        state["host"] = (words[0].cpu().numpy().view(np.uint64),)
    return state


def run(state):
    ctx, kind = state["ctx"], state["kind"]
    if kind == "mul":
        ctx.mul_device(state["out"], state["in"][0], state["in"][1])
        return state["out"]
    if kind == "sqr":
        ctx.sqr_device(state["out"], state["in"][0])
        return state["out"]
    if kind == "cached":
        state["work"].forward(state["in"][1], state["scale"])
        state["prod"].pointwise(state["kept"], state["work"])
        state["prod"].inverse_save(state["out"], state["out"].numel())
        return state["out"]
    if kind == "batch":
        state["plan"].run_jobs(state["jobs"])
        return state["out"]
    if kind == "div":
        ctx.div_device(state["q"], state["r"], state["in"][0], state["in"][1])
        return state["q"], state["r"]
    if kind == "host_mul":
        return ctx.mul(state["host"][0], state["host"][1], out=state["host_out"]).view(np.int64)
    return np.frombuffer(ctx.to_dec_levels(state["host"][0]).encode(), dtype=np.uint8)


def work(case):
    """Bytes of a pass: every operand read once, every result written once."""
    kind = case["kind"]
    if kind == "batch":
        na, nb = _batch_layout(case)[:2]
        return {"bytes": 16 * int(na.sum() + nb.sum()), "flops": 0}
    if kind == "dec":  # 64 log10(2) digits a limb
        return {"bytes": int(8 * case["na"] + 19.27 * case["na"]), "flops": 0}
    if kind == "sqr":
        return {"bytes": 8 * 3 * case["na"], "flops": 0}
    if kind == "div":
        return {"bytes": 8 * (2 * case["na"] + case["nb"] + 1), "flops": 0}
    return {"bytes": 16 * (case["na"] + case["nb"]), "flops": 0}


def _int(words):
    return int.from_bytes(words.cpu().numpy().tobytes(), "little")


def _words(value, n):
    return np.frombuffer(value.to_bytes(8 * n, "little"), dtype=np.int64)


def exact(case, seed):
    """The same from Python's integers, where they take it in a few seconds."""
    kind = case["kind"]
    if kind in ("batch", "dec") or case["na"] > 200000:
        return None
    v = [_int(w) for w in _inputs(case, seed)]
    if kind == "sqr":
        return _words(v[0] * v[0], 2 * case["na"])
    if kind == "div":
        if case["na"] > 20000:  # Python's division is quadratic
            return None
        q, r = divmod(v[0], v[1])
        return _words(q, case["na"] - case["nb"] + 1), _words(r, case["nb"])
    return _words(v[0] * v[1], case["na"] + case["nb"])
