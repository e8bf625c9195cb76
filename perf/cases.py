"""What the framework is timed on: the calls of a silent-OT program, each through the public binding (cuot_b200).

Every case is one pass over data that is already on the GPU, as the protocol code around the engine leaves it there.  A case
is a dict with the `kind` of call and its sizes; the listed ones stand for these uses:

  extension of a Ferret-style COT: GGM MPCOT and primal LPN (d = 10 indices a row).  `role` "both": the two parties of a
      one-GPU deployment (one index computation for both roles' LPN); "send" / "recv": one party of a networked pair.
  extension of an SOT: GGM PPRF of both roles, the quasi-cyclic encode of each role's leaves through a plan of the session's
      polynomial, and the receiver's choice bits.
  dual_lpn: the rate-1/2 encode of 2n noise blocks with a polynomial that is new on every call (no plan).
  transpose: blocks -> 128 bit planes, and 128 planes -> blocks.
  check: the malicious-mode consistency sums over all trees' leaves.
  batch: many extensions of uneven sizes, half SOT and half Ferret-style, as one device program.

All outputs are blocks and bit vectors: they are equal or wrong, so there is no 64-bit reference beside them.
"""
import math

import torch

import cuot_b200
from cuot_b200 import ferret
from cuot_b200.batch import KIND_FERRET, KIND_SOT, Batch, Instance, mixed_shapes

B11, B12, B13 = ferret.FERRET_B11, ferret.FERRET_B12, ferret.FERRET_B13


def listed():
    return [
        # the small single extension: latency and launches
        dict(name="ferret_small", kind="ferret", role="both", t=64, h=10, k=8192),
        # the set-up extension of a session as its receiver runs it: many shallow trees, a tree count that fits nothing
        dict(name="ferret_setup_recv", kind="ferret", role="recv", t=B13.t_pre, h=B13.h_pre, k=B13.k_pre),
        # full-size extensions: both roles on one GPU, and a networked sender with shallower, more numerous trees
        dict(name="ferret_b13", kind="ferret", role="both", t=B13.t, h=B13.h, k=B13.k),
        dict(name="ferret_b11_send", kind="ferret", role="send", t=B11.t, h=B11.h, k=B11.k),
        # SOT from the smallest session requests over the plain configuration to the largest direct size
        dict(name="sot_2e14", kind="sot", t=16, h=10),
        dict(name="sot_2e17", kind="sot", t=64, h=11),
        dict(name="sot_2e20", kind="sot", t=256, h=12),
        dict(name="sot_2e22", kind="sot", t=256, h=14),
        # a one-off encode: the polynomial's own transform is part of the call
        dict(name="dual_lpn_2e18", kind="dual_lpn", e=18),
        # the standalone layout change of a caller that keeps planes
        dict(name="transpose_2e21", kind="transpose", blocks=1 << 21),
        # consistency check of a full-size extension
        dict(name="check_b12", kind="check", t=B12.t, h=B12.h),
        # an engine's batch of mixed sessions
        dict(name="batch_16", kind="batch", count=16, lo=14, hi=20, seed=2024),
    ]


def _between(rng, lo, hi):
    """A whole number, log-uniform over [lo, hi]."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["ferret", "ferret", "ferret", "sot", "sot", "sot", "sot", "dual_lpn", "transpose", "check", "batch"])
    if kind == "ferret":
        h = rng.randint(8, 13)
        t = max(1, _between(rng, 1 << 16, B13.n) >> h)
        n = t << h
        # k in the parameter sets' range of k / n (full size 1/82 .. 1/23, set-up 1/27 .. 1/8)
        return dict(kind=kind, role=rng.choice(["both", "send", "recv"]), t=t, h=h, k=max(1000, int(n / rng.uniform(8, 82))))
    if kind == "sot":
        e = rng.randint(14, 22)
        h = rng.randint(10, min(14, e))
        return dict(kind=kind, t=(1 << e) >> h, h=h)
    if kind == "dual_lpn":
        return dict(kind=kind, e=rng.randint(14, 21))
    if kind == "transpose":
        return dict(kind=kind, blocks=8 * _between(rng, 1 << 9, 1 << 18))
    if kind == "check":
        h = rng.randint(9, 13)
        return dict(kind=kind, t=max(1, _between(rng, 1 << 16, B13.n) >> h), h=h)
    return dict(kind=kind, count=2 * rng.randint(2, 8), lo=14, hi=rng.randint(16, 20), seed=rng.randint(1, 10**6))


def _blocks(count, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randint(0, 256, (count, 16), dtype=torch.uint8, device="cuda", generator=g)


def _shapes(case):
    return mixed_shapes(case["count"], case["seed"], case["lo"], case["hi"])


def _empty(count):
    return torch.empty((count, 16), dtype=torch.uint8, device="cuda")


def prepare(case, seed):
    ctx = cuot_b200.Context(torch.cuda.current_device())
    s = dict(case=case, ctx=ctx)
    kind = case["kind"]
    if kind == "ferret":
        t, h = case["t"], case["h"]
        s["i"] = i = Instance(ctx, KIND_FERRET, t, h, seed, k=case["k"])
        s["lsum"], s["rsum"], s["ss"] = _empty(t * h), _empty(t * h), _empty(t)
        # the receiver holds the messages that the sender's level sums gave it through the OTs
        ctx.ferret_pprf_sender(i.d_roots, h, i.delta, i.v, s["lsum"], s["rsum"], s["ss"])
        s["mc"] = torch.where(i.d_choice[:, None] == 0, s["lsum"], s["rsum"])
    elif kind == "sot":
        t, h = case["t"], case["h"]
        s["i"] = i = Instance(ctx, KIND_SOT, t, h, seed)
        s["m0"], s["m1"] = _empty((h + 1) * t), _empty((h + 1) * t)
        s["plan"] = ctx.qc_plan(i.a, i.n)
    elif kind == "dual_lpn":
        n = 1 << case["e"]
        s["inp"], s["out"] = _blocks(2 * n, seed), _empty(n)
        s["a"] = torch.empty(n // 64, dtype=torch.int64, device="cuda")
        ctx.qc_gen_a(_blocks(1, seed + 1)[0], n, s["a"])
    elif kind == "transpose":
        s["inp"] = _blocks(case["blocks"], seed)
        s["planes"] = torch.empty(16 * case["blocks"], dtype=torch.uint8, device="cuda")
        s["inp_planes"] = _blocks(case["blocks"], seed + 1).view(-1)
        s["out"] = _empty(case["blocks"])
    elif kind == "check":
        s["leaves"], s["seeds"], s["out"] = _blocks(case["t"] << case["h"], seed), _blocks(case["t"], seed + 1), _empty(case["t"])
    else:
        s["insts"] = [Instance(ctx, kd, t, h, seed * 1000 + j, k=k) for j, (kd, t, h, k) in enumerate(_shapes(case))]
        s["batch"] = Batch(ctx, s["insts"])
        s["stream"] = torch.cuda.Stream()
    return s


def run(s):
    case, ctx = s["case"], s["ctx"]
    kind = case["kind"]
    if kind == "ferret":
        i, h, role = s["i"], case["h"], case["role"]
        if role != "recv":
            ctx.ferret_pprf_sender(i.d_roots, h, i.delta, i.v, s["lsum"], s["rsum"], s["ss"])
        if role != "send":
            ctx.ferret_pprf_recver(s["mc"], i.d_choice, s["ss"], h, i.w)
        if role == "both":
            ctx.lpn_primal_dual(i.seed, i.d_kk_s, i.d_kk_r, i.v, i.w, d=i.d)
            return i.v, i.w, s["lsum"], s["rsum"], s["ss"]
        if role == "send":
            ctx.lpn_primal(i.seed, i.d_kk_s, i.v, d=i.d)
            return i.v, s["lsum"], s["rsum"], s["ss"]
        ctx.lpn_primal(i.seed, i.d_kk_r, i.w, d=i.d)
        return i.w
    if kind == "sot":
        i, t, h = s["i"], case["t"], case["h"]
        ctx.sot_pprf_sender(i.d_roots, h, i.delta, i.d_b0, i.d_b1, i.v, s["m0"], s["m1"])
        ctx.sot_pprf_recver(s["m0"], s["m1"], i.d_mc, i.d_choice, t, h, i.w)
        s["plan"].dual_lpn(i.v)
        s["plan"].dual_lpn(i.w)
        ctx.qc_encode_sparse(i.a, i.d_punct, i.n, i.cbits)
        return i.v, i.w, i.cbits, s["m0"], s["m1"]
    if kind == "dual_lpn":
        ctx.sot_dual_lpn_r2(s["a"], s["inp"], 1 << case["e"], s["out"])
        return s["out"]
    if kind == "transpose":
        n = case["blocks"]
        ctx.bit_transpose(s["inp"], n, 16, 0, 128, s["planes"])
        ctx.bit_transpose(s["inp_planes"], 128, n // 8, 0, n, s["out"])
        return s["planes"], s["out"]
    if kind == "check":
        ctx.ferret_chi_sum(s["leaves"], case["h"], s["seeds"], s["out"])
        return s["out"]
    here = torch.cuda.current_stream()
    s["stream"].wait_stream(here)
    s["batch"].run(s["stream"])
    here.wait_stream(s["stream"])
    return [x for i in s["insts"] for x in ((i.v, i.w) if i.kind == KIND_FERRET else (i.v, i.w, i.cbits))]


def _ferret_bytes(t, h, k, roles):
    n = t << h
    # noise and LPN inputs in, correlations out; per tree the root, the level sums (both sides), the choices and a secret sum
    return roles * (16 * n + 16 * k + 16 * t + 33 * t * h + 16 * t)


def _sot_bytes(t, h):
    n = t << h
    # both roles' outputs, the polynomial, the choice bits; per tree roots, base OTs, messages, choices and positions
    return 2 * 16 * n + 2 * n // 8 + t * (16 + 8 + h * (3 * 16 + 1) + (h + 1) * 2 * 16)


def work(case):
    """Bytes that a pass cannot do without.  The arithmetic is AES rounds and GF(2) sums: no floating-point operations."""
    kind = case["kind"]
    if kind == "ferret":
        b = _ferret_bytes(case["t"], case["h"], case["k"], 2 if case["role"] == "both" else 1)
    elif kind == "sot":
        b = _sot_bytes(case["t"], case["h"])
    elif kind == "dual_lpn":
        b = (48 << case["e"]) + (1 << case["e"]) // 8
    elif kind == "transpose":
        b = 2 * 32 * case["blocks"]
    elif kind == "check":
        b = (16 * case["t"] << case["h"]) + 32 * case["t"]
    else:
        b = sum(_sot_bytes(t, h) if kd == KIND_SOT else _ferret_bytes(t, h, k, 2) for kd, t, h, k in _shapes(case))
    return {"bytes": float(b), "flops": 0.0}


def exact(case, seed):
    """Every output is a block or a bit vector (whole bytes): nothing here is a rounded number."""
    return None
