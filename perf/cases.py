"""Workloads of the multiply engine, each through the entry point that a program calls.

A case is a dict of plain values.  ``listed()`` names the fixed ones, ``draw(rng)`` gives more of the same
ranges, ``prepare`` makes what a caller holds before the call (operands, handles, job arrays), ``run`` is one
call, ``work`` the bytes and operations that no implementation of the call can do without.

Kinds:
  mul    one product of device operands (``mul_device``), the drop-in with operands in HBM; ``sqr`` passes one
         operand twice, as the Newton iterations do
  host   the drop-in with host buffers (``mul_mag_ntt``)
  batch  independent products of uneven sizes in one call (``mul_batch``): the lower levels of a product tree
  served requests on device handles, some consuming earlier results, submitted, waited for and read back
  pi     decimal digits of pi from the level-batched Chudnovsky driver (splitting, final assembly and decimal
         conversion)
  bbp    batched hex digits of pi at given positions
"""
import ctypes
import math
import random

import numpy as np
import torch

import pi_gb300 as pm


def listed():
    return [
        # a leaf product of a splitting tree: one call's latency
        {"name": "mul_2e10", "kind": "mul", "la": 16, "lb": 16, "sqr": False},
        # the sweep's balanced sizes: 2^16, 2^20, 2^24 and the headline 2^30 bits
        {"name": "mul_2e16", "kind": "mul", "la": 1 << 10, "lb": 1 << 10, "sqr": False},
        {"name": "mul_2e20", "kind": "mul", "la": 1 << 14, "lb": 1 << 14, "sqr": False},
        {"name": "mul_2e24", "kind": "mul", "la": 1 << 18, "lb": 1 << 18, "sqr": False},
        {"name": "mul_2e30", "kind": "mul", "la": 1 << 24, "lb": 1 << 24, "sqr": False},
        # a long numerator by a short scale, lengths of no particular form
        {"name": "mul_uneven", "kind": "mul", "la": 2500037, "lb": 16411, "sqr": False},
        # a Newton step's square at a length past a power of two
        {"name": "sqr_odd", "kind": "mul", "la": 300007, "lb": 300007, "sqr": True},
        # the plain drop-in on host limbs at the size of a middle splitting level
        {"name": "host_2e21", "kind": "host", "la": 33001, "lb": 32003, "sqr": False},
        # 4096 independent products, operand lengths log-uniform in 2^10 .. 2^22 bits
        {"name": "batch_4096", "kind": "batch", "n": 4096, "lo": 10, "hi": 22},
        # a burst of service requests, 2^12 .. 2^22 bits, 30 % chained, 25 % squares
        {"name": "served_200", "kind": "served", "n": 200, "lo": 12, "hi": 22},
        # 10^8 digits of pi (a few hundred fewer, by the seed)
        {"name": "pi_1e8", "kind": "pi", "digits": 100000000},
        # spot checks of pi's hex digits
        {"name": "bbp_64", "kind": "bbp", "n": 64, "top": 50000000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mul", "mul", "mul", "mul", "sqr", "host", "batch", "served", "pi", "bbp"])
    if kind in ("mul", "sqr"):
        la = _log_int(rng, 8, 1 << 24)
        lb = _log_int(rng, max(8, la // 256), la) if rng.random() < 0.5 else max(8, int(la * rng.uniform(0.5, 1)))
        return {"kind": "mul", "la": la, "lb": la if kind == "sqr" else lb, "sqr": kind == "sqr"}
    if kind == "host":
        la = _log_int(rng, 8192, 1 << 20)
        return {"kind": "host", "la": la, "lb": _log_int(rng, 8192, la) if la > 8192 else la, "sqr": rng.random() < 0.25}
    if kind == "batch":
        lo = rng.randint(8, 14)
        return {"kind": "batch", "n": _log_int(rng, 32, 4096), "lo": lo, "hi": rng.randint(lo + 2, 22)}
    if kind == "served":
        return {"kind": "served", "n": _log_int(rng, 16, 200), "lo": 12, "hi": rng.randint(16, 22)}
    if kind == "pi":
        return {"kind": "pi", "digits": _log_int(rng, 10**5, 10**8)}
    return {"kind": "bbp", "n": _log_int(rng, 4, 64), "top": _log_int(rng, 10**5, 5 * 10**7)}


# ------------------------------------------------------------------ operands


def _limbs(n, seed, salt):
    """n uniform limbs on the GPU (int64 bit patterns), the top one not zero."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 1000003 + salt)
    x = torch.randint(-(1 << 63), (1 << 63) - 1, (n,), generator=g, device="cuda", dtype=torch.int64)
    x[-1] |= 1 << 62
    return x


def _host_limbs(n, seed, salt):
    x = np.random.default_rng([seed, salt]).integers(0, 1 << 64, n, dtype=np.uint64)
    x[-1] |= np.uint64(1 << 62)
    return x


def _shape_rng(case):
    """The sizes inside a batch or a request stream belong to the case, not to the seed."""
    return random.Random("%d %d %d" % (case["n"], case["lo"], case["hi"]))


def _bits_to_limbs(rng, lo, hi):
    return max(1, math.ceil(2 ** rng.uniform(lo, hi) / 64))


def _batch_sizes(case):
    rng = _shape_rng(case)
    return [(_bits_to_limbs(rng, case["lo"], case["hi"]), _bits_to_limbs(rng, case["lo"], case["hi"])) for _ in range(case["n"])]


def _served_plan(case):
    """Requests as (x, y): operands are ("in", limbs) or ("out", earlier request); y None: a square."""
    rng = _shape_rng(case)
    plan, size = [], []
    most = int(2 ** case["hi"] / 64)
    for i in range(case["n"]):
        # results within the size range may be consumed once more
        old = [k for k in range(i) if size[k] <= most]
        if old and rng.random() < 0.3:
            k = rng.choice(old)
            x, nx = ("out", k), size[k]
        else:
            nx = _bits_to_limbs(rng, case["lo"], case["hi"])
            x = ("in", nx)
        if rng.random() < 0.25:
            y, ny = None, nx
        else:
            ny = _bits_to_limbs(rng, case["lo"], case["hi"])
            y = ("in", ny)
        plan.append((x, y))
        size.append(nx + ny)
    return plan, size


def _positions(case, seed):
    return np.sort(np.random.default_rng([seed, 7]).integers(0, case["top"], case["n"], dtype=np.uint64))


class _Handles:
    """Uploaded operands, freed with the state."""

    def __init__(self):
        self.ids = []

    def add(self, limbs):
        h = pm.upload(limbs)
        self.ids.append(h)
        return h

    def __del__(self):
        for h in self.ids:
            try:
                pm.free(h)
            except Exception:  # noqa: BLE001 (interpreter shutdown)
                pass


def prepare(case, seed):
    kind = case["kind"]
    if kind == "mul":
        a = _limbs(case["la"], seed, 1)
        b = a if case["sqr"] else _limbs(case["lb"], seed, 2)
        out = torch.empty(a.numel() + b.numel(), dtype=torch.int64, device="cuda")
        return {"kind": kind, "a": a, "b": b, "out": out}
    if kind == "host":
        a = _host_limbs(case["la"], seed, 1)
        return {"kind": kind, "a": a, "b": a if case["sqr"] else _host_limbs(case["lb"], seed, 2)}
    if kind == "batch":
        sizes = _batch_sizes(case)
        x = _limbs(sum(la + lb for la, lb in sizes), seed, 1)
        out = torch.empty(x.numel(), dtype=torch.int64, device="cuda")
        jobs = (pm.PimulJob * len(sizes))()
        at = 0
        for i, (la, lb) in enumerate(sizes):
            p = x.data_ptr() + 8 * at
            jobs[i] = pm.PimulJob(p, la, p + 8 * la, lb, out.data_ptr() + 8 * at)
            at += la + lb
        return {"kind": kind, "x": x, "out": out, "jobs": jobs}
    if kind == "served":
        plan, _ = _served_plan(case)
        held = _Handles()
        ops = [tuple(o and (("h", held.add(_host_limbs(o[1], seed, 2 * i + k))) if o[0] == "in" else o) for k, o in enumerate(xy))
               for i, xy in enumerate(plan)]
        read = {o[1] for xy in plan for o in xy if o and o[0] == "out"}
        return {"kind": kind, "ops": ops, "held": held, "last": [i for i in range(len(plan)) if i not in read]}
    if kind == "pi":
        # the text of one case has one length: what the seed takes off stays blank
        return {"kind": kind, "digits": case["digits"] - seed % 499, "text": np.full(case["digits"], ord(" "), dtype=np.uint8)}
    return {"kind": kind, "positions": _positions(case, seed)}


def run(state):
    kind = state["kind"]
    if kind == "mul":
        pm.mul_device(state["a"], state["b"], state["out"])
        return state["out"]
    if kind == "host":
        return pm.mul_mag_ntt(state["a"], state["b"])
    if kind == "batch":
        # the C entry point on the caller's own job array, as a native scheduler issues a level
        jobs = state["jobs"]
        rc = pm.lib().pimul_mul_batch(ctypes.cast(jobs, ctypes.c_void_p), len(jobs),
                                      ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc:
            raise pm.PimulError(rc, pm.lib().pimul_last_error().decode())
        return state["out"]
    if kind == "served":
        res, tickets = [], []
        for x, y in state["ops"]:
            hx = x[1] if x[0] == "h" else res[x[1]]
            h, t = pm.submit(hx) if y is None else pm.submit(hx, y[1])
            res.append(h)
            tickets.append(t)
        for t in tickets:
            pm.wait(t)
        out = np.concatenate([pm.download(res[i]) for i in state["last"]])
        for h in res:
            pm.free(h)
        return out
    if kind == "pi":
        digits, _ = pm.pi_chudnovsky_batched(state["digits"])
        state["text"][: len(digits)] = np.frombuffer(digits.encode(), dtype=np.uint8)
        return state["text"]
    return pm.bbp_hex_digits(state["positions"])


# ------------------------------------------------------------------ work


def _product(la, lb, sqr):
    """Operands read and product written once; three (a square: two) transforms of the product's length in
    16-bit coefficients, log2 N / 2 butterflies (a product, a sum, a difference) per point."""
    n = 1 << max(1, (4 * (la + lb) - 2).bit_length())
    flops = (2 if sqr else 3) * 1.5 * n * math.log2(n) + n
    return 8 * ((la if sqr else la + lb) + la + lb), flops


def work(case):
    kind = case["kind"]
    if kind in ("mul", "host"):
        la, lb = case["la"], case["la"] if case["sqr"] else case["lb"]
        b, f = _product(la, lb, case["sqr"])
    elif kind == "batch":
        each = [_product(la, lb, False) for la, lb in _batch_sizes(case)]
        b, f = sum(x[0] for x in each), sum(x[1] for x in each)
    elif kind == "served":
        plan, size = _served_plan(case)
        b = f = 0
        for (x, y), n in zip(plan, size):
            nx = x[1] if x[0] == "in" else size[x[1]]
            p = _product(nx, n - nx, y is None)
            b, f = b + p[0], f + p[1]
    elif kind == "pi":
        # a tree of depth log2(terms) whose levels each hold three numbers of about the result's length, and the
        # digits once out
        limbs = case["digits"] * math.log2(10) / 64
        depth = math.log2(case["digits"] / 14.18)
        p = _product(int(limbs), int(limbs), False)
        b, f = case["digits"] + 8 * limbs, 2 * p[1] * depth / 2
    else:
        # four series, 8k + j for k up to the position: one modular power of about log2(position) squarings and one
        # quotient per term
        terms = 4 * case["n"] * case["top"] / 2
        b, f = 8 * case["n"] + 4 * case["n"], terms * 2 * math.log2(4 * case["top"])
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------ exact values


def _int(limbs):
    return int.from_bytes(np.ascontiguousarray(limbs).astype("<u8").tobytes(), "little")


def _to_limbs(x, n):
    return np.frombuffer(x.to_bytes(8 * n, "little"), dtype="<u8").copy()


def exact(case, seed):
    """Products as Python's integers give them, up to sizes where that takes seconds."""
    if case["kind"] == "mul" and case["la"] + case["lb"] <= 1 << 16:
        a = _limbs(case["la"], seed, 1).cpu().numpy().view(np.uint64)
        b = a if case["sqr"] else _limbs(case["lb"], seed, 2).cpu().numpy().view(np.uint64)
        return torch.from_numpy(_to_limbs(_int(a) * _int(b), a.size + b.size).view(np.int64))
    if case["kind"] == "host" and case["la"] + case["lb"] <= 1 << 17:
        a = _host_limbs(case["la"], seed, 1)
        b = a if case["sqr"] else _host_limbs(case["lb"], seed, 2)
        out = _to_limbs(_int(a) * _int(b), a.size + b.size)
        return out[: int(np.nonzero(out)[0][-1]) + 1]
    return None
