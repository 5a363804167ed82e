"""The work that programs have this library do, as cases that can be timed.

A case is a dict of plain values; `kind` says which public entry point it goes
through:

  mpz       mpz_mul on two host integers (numpy storage): the call a host
            program makes for every multiplication.
  mul, sqr  device.mul / device.sqr on device limbs.
  batch     device.Batch over many uneven pairs, planned once and run.
  spectrum  device.ntt_forward, then device.ntt_reverse, of residues.
  pipeline  mul_host_pipeline over pinned host arrays.
  split     series.binary_split through a multiply service.
  newton    mpd.mpd_reciprocal or mpd.mpd_sqrt, truncated to the working
            precision, through a multiply service (with split, what
            computing pi to many bits consists of).

Limbs are uniform unless the case says "ones" (all 2^64 - 1: the longest
carry chains) or "sparse" (one limb in a hundred nonzero).
"""

from __future__ import annotations

import math
from dataclasses import replace

import numpy as np
import torch

import hypergeometrica_gb300 as H
from hypergeometrica_gb300 import device as D
from hypergeometrica_gb300 import mpd as M
from hypergeometrica_gb300 import series as S

SERIES = {
    "chudnovsky": S.make_chudnovsky_series,
    "e": S.make_e_series,
    "catalan": S.make_catalan_series,
    "apery": S.make_apery_series,
}


def listed():
    return [
        # A product below the schoolbook threshold: what a host program calls most.
        {"name": "mpz 64x48", "kind": "mpz", "nx": 64, "ny": 48, "dist": "uniform"},
        # A host product of a few thousand limbs (the smoke test's sizes).
        {"name": "mpz 3000x2500", "kind": "mpz", "nx": 3000, "ny": 2500, "dist": "uniform"},
        # The single-product configuration: 2^16 x 2^16 limbs, operands on the device.
        {"name": "mul 2^16x2^16", "kind": "mul", "nx": 1 << 16, "ny": 1 << 16, "dist": "uniform"},
        # Operands of no special size, as a computation's intermediate values have them.
        {"name": "mul 1000003x600011", "kind": "mul", "nx": 1000003, "ny": 600011, "dist": "uniform"},
        # The headline product of the balanced sweep.
        {"name": "mul 2^24x2^24", "kind": "mul", "nx": 1 << 24, "ny": 1 << 24, "dist": "uniform"},
        # An unbalanced product: a long number times a short one.
        {"name": "mul 2^24x2^16", "kind": "mul", "nx": 1 << 24, "ny": 1 << 16, "dist": "uniform"},
        # A square (powering, Newton steps): one operand, its own schedule.
        {"name": "sqr 2^20", "kind": "sqr", "nx": 1 << 20, "dist": "uniform"},
        # Binary splitting's leaves: thousands of independent uneven pairs.
        {"name": "batch 4096", "kind": "batch", "count": 4096, "lo_bits": 6, "hi_bits": 14},
        # Both directions of the transform by itself, one prime.
        {"name": "spectrum 2^20", "kind": "spectrum", "log_len": 20, "mod": 0},
        # Products of host data in a row: uploads and downloads beside the work.
        {"name": "pipeline 8 x 2^20", "kind": "pipeline", "count": 8, "nx": 1 << 20, "ny": 1 << 20},
        # Chudnovsky's series for 2^22 bits of pi by binary splitting.
        {"name": "split 2^22 bits", "kind": "split", "series": "chudnovsky", "terms": 89034},
        # The Newton iteration that inverts its result, to the same precision.
        {"name": "reciprocal 2^22 bits", "kind": "newton", "op": "reciprocal", "bits": 1 << 22},
    ]


def _log_int(rng, lo, hi):
    """An integer in [lo, hi], uniform over the logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _dist(rng):
    return rng.choice(["uniform", "uniform", "uniform", "ones", "sparse"])


def draw(rng):
    kind = rng.choice(["mpz", "mul", "mul", "mul", "sqr", "batch", "spectrum", "pipeline", "split", "newton"])
    if kind == "mpz":
        nx = _log_int(rng, 2, 1 << 16)
        return {"kind": kind, "nx": nx, "ny": _log_int(rng, max(2, nx >> 6), nx), "dist": _dist(rng)}
    if kind == "mul":
        nx = _log_int(rng, 1 << 9, 1 << 24)
        return {"kind": kind, "nx": nx, "ny": _log_int(rng, max(101, nx >> 8), nx), "dist": _dist(rng)}
    if kind == "sqr":
        return {"kind": kind, "nx": _log_int(rng, 1 << 9, 1 << 24), "dist": _dist(rng)}
    if kind == "batch":
        lo = rng.randint(4, 9)
        return {"kind": kind, "count": _log_int(rng, 16, 4096), "lo_bits": lo, "hi_bits": rng.randint(lo + 2, 14)}
    if kind == "spectrum":
        return {"kind": kind, "log_len": rng.randint(4, 24), "mod": rng.randint(0, 2)}
    if kind == "pipeline":
        nx = _log_int(rng, 1 << 10, 1 << 20)
        return {"kind": kind, "count": rng.randint(2, 8), "nx": nx, "ny": _log_int(rng, nx >> 3, nx)}
    if kind == "split":
        return {"kind": kind, "series": rng.choice(sorted(SERIES)), "terms": _log_int(rng, 200, 89034)}
    return {"kind": kind, "op": rng.choice(["reciprocal", "sqrt"]), "bits": _log_int(rng, 1 << 14, 1 << 22)}


def _limbs(gen, n, dist, device):
    """n limbs as an int64 tensor, the top one nonzero."""
    if dist == "ones":
        t = torch.full((n,), -1, dtype=torch.int64, device=device)
        t[0] = torch.randint(1, 1 << 62, (1,), generator=gen, device=device)
        return t
    t = torch.randint(-(1 << 63), (1 << 63) - 1, (n,), dtype=torch.int64, generator=gen, device=device)
    if dist == "sparse":
        t = torch.where(torch.rand(n, generator=gen, device=device) < 0.01, t, torch.zeros_like(t))
    t[-1] |= 1
    return t


def _gen(seed, device):
    return torch.Generator(device=device).manual_seed(seed)


def _sizes(case):
    """The operand lengths of a batch's pairs: uniform over their logarithm."""
    rng = np.random.RandomState(case["count"])
    return np.floor(2.0 ** rng.uniform(case["lo_bits"], case["hi_bits"], (case["count"], 2))).astype(np.int64)


def _service(limbs):
    """A multiply service for products of up to `limbs` limbs in all, two slots."""
    n = 1 << max(20, (limbs - 1).bit_length())
    return D.Service(workspace_bytes=2 * 2 * 3 * 8 * n, slots=2)


# Bits that one term adds to a range's partial, as an upper bound (for the service's size).
_TERM_BITS = {"chudnovsky": 110, "e": 20, "catalan": 40, "apery": 110}


def prepare(case, seed):
    H.init()
    kind = case["kind"]
    st = dict(case)
    if kind == "mpz":
        rng = np.random.RandomState(seed % (1 << 32))
        gen = _gen(seed, "cpu")
        for k, n in (("x", case["nx"]), ("y", case["ny"])):
            d = _limbs(gen, n, case["dist"], "cpu").numpy().view(np.uint64)
            st[k] = H.MPZ(int(rng.choice([-1, 1])), d)
    elif kind in ("mul", "sqr"):
        gen = _gen(seed, "cuda")
        st["x"] = _limbs(gen, case["nx"], case["dist"], "cuda")
        if kind == "mul":
            st["y"] = _limbs(gen, case["ny"], case["dist"], "cuda")
        n = case["nx"] + (case["ny"] if kind == "mul" else case["nx"])
        st["out"] = torch.empty(n, dtype=torch.int64, device="cuda")
    elif kind == "batch":
        # Operands and products lie back to back in arenas, as a tree level's partials do.
        sizes = _sizes(case)
        total = int(sizes.sum())
        src = torch.randint(-(1 << 63), (1 << 63) - 1, (total,), dtype=torch.int64, generator=_gen(seed, "cuda"),
                            device="cuda")
        ends = torch.from_numpy(np.cumsum(sizes.reshape(-1)) - 1).cuda()
        src[ends] |= 1
        st["src"], st["out"] = src, torch.empty(total, dtype=torch.int64, device="cuda")
        items, at = [], 0
        for nx, ny in sizes.tolist():
            items.append((src[at: at + nx], src[at + nx: at + nx + ny], st["out"][at: at + nx + ny]))
            at += nx + ny
        st["batch"] = D.Batch(items)
    elif kind == "spectrum":
        p = H.scheme_moduli()[case["mod"]]
        n = 1 << case["log_len"]
        st["a"] = torch.randint(0, p, (n,), dtype=torch.int64, generator=_gen(seed, "cuda"), device="cuda")
        st["fwd"], st["rev"] = torch.empty_like(st["a"]), torch.empty_like(st["a"])
    elif kind == "pipeline":
        gen = _gen(seed, "cpu")
        st["items"] = [(_limbs(gen, case["nx"], "uniform", "cpu").pin_memory(),
                        _limbs(gen, case["ny"], "uniform", "cpu").pin_memory(),
                        torch.empty(case["nx"] + case["ny"], dtype=torch.int64, pin_memory=True))
                       for _ in range(case["count"])]
    elif kind == "split":
        # The series with another constant in its numerators a(k).
        s = SERIES[case["series"]]()
        (coefs, zero), rest, add = s.poly[0], s.poly[1:], seed % 1000003
        st["sum"] = replace(s, a=lambda n, a=s.a: a(n) + add, poly=(((coefs[0] + add,) + coefs[1:], zero),) + rest)
        st["service"] = _service(4 * case["terms"] * _TERM_BITS[case["series"]] // 64)
    else:
        n = -(-case["bits"] // 64) + 2
        t = _limbs(_gen(seed, "cuda"), n, "uniform", "cuda")
        t[-1] = (t[-1] & ((1 << 61) - 1)) | (1 << 61)  # a value in [1/8, 1/4)
        st["a"] = M.MPD(S.DeviceInt(1, t, n), -n)
        st["service"] = _service(4 * n)
    return st


def run(st):
    kind = st["kind"]
    if kind == "mpz":
        r = H.mpz_mul(st["x"], st["y"])
        return {"sign": r.sign, "storage": r.storage}
    if kind == "mul":
        D.mul(st["x"], st["y"], st["out"])
        return st["out"]
    if kind == "sqr":
        D.sqr(st["x"], st["out"])
        return st["out"]
    if kind == "batch":
        st["batch"].run()
        return st["out"]
    if kind == "spectrum":
        st["fwd"].copy_(st["a"])
        D.ntt_forward(st["fwd"], st["mod"])
        st["rev"].copy_(st["fwd"])
        D.ntt_reverse(st["rev"], st["mod"])
        return {"forward": st["fwd"], "reverse": st["rev"]}
    if kind == "pipeline":
        H.mul_host_pipeline(st["items"])
        return [out for _, _, out in st["items"]]
    if kind == "split":
        r = S.binary_split(st["sum"], 0, st["terms"], st["service"])
        return {k: {"sign": v.sign, "limbs": v.t[: v.size]} for k, v in (("p", r.p), ("q", r.q), ("b", r.b), ("r", r.r))}
    newton = M.mpd_reciprocal if st["op"] == "reciprocal" else M.mpd_sqrt
    r = newton(st["a"], st["bits"], st["service"], truncate=True)
    return {"sign": r.mantissa.sign, "limbs": r.mantissa.t[: r.mantissa.size], "exponent": r.exponent}


def work(case):
    """Each input read once and each output written once (8 bytes a limb); the
    arithmetic is on integers."""
    kind = case["kind"]
    if kind in ("mpz", "mul", "pipeline"):
        limbs = 2 * (case["nx"] + case["ny"]) * case.get("count", 1)
    elif kind == "sqr":
        limbs = 3 * case["nx"]
    elif kind == "batch":
        limbs = 2 * int(_sizes(case).sum())
    elif kind == "spectrum":
        limbs = 4 << case["log_len"]
    elif kind == "split":  # the four results
        limbs = 4 * case["terms"] * _TERM_BITS[case["series"]] // 64
    else:
        limbs = 2 * case["bits"] // 64
    return {"bytes": 8.0 * limbs, "flops": 0.0}


def _int(t):
    a = t.cpu().numpy() if isinstance(t, torch.Tensor) else t
    return int.from_bytes(np.ascontiguousarray(a).tobytes(), "little")


def _limbs_of(v, n, kind=np.int64):
    return np.frombuffer(v.to_bytes(8 * n, "little"), dtype=kind).copy()


def exact(case, seed):
    """The product as Python's integers give it, where they are quick enough."""
    kind = case["kind"]
    if kind not in ("mpz", "mul", "sqr"):
        return None
    small = min(case["nx"], case.get("ny", case["nx"]))
    if case["nx"] * small ** 0.585 > float(1 << 16) ** 1.585:
        return None
    if kind == "mpz":
        st = prepare(case, seed)
        v = _int(st["x"].storage) * _int(st["y"].storage)
        return {"sign": st["x"].sign * st["y"].sign, "storage": _limbs_of(v, (v.bit_length() + 63) // 64, np.uint64)}
    st = prepare(case, seed)
    x = _int(st["x"])
    return torch.from_numpy(_limbs_of(x * (x if kind == "sqr" else _int(st["y"])), st["out"].numel()))
