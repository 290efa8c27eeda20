"""Performance cases: what programs built on this framework have it do.

A case is a dict of plain values.  Its ``kind`` names the public entry point:

    prove      one commit + prove through Config.commit_witnesses / Config.prove
    rs_encode  the Reed-Solomon encoder alone (codeword planes left in HBM)
    rs_commit  encoder + leaf hashing + Merkle trees (roots)
    zk         one zero-knowledge commit + prove
    batch      several commits + proves in one captured graph
    served     a burst of mixed requests through the continuous-batching server

Inputs are uniform canonical Goldilocks words, as committed polynomials are;
statements are multilinear evaluations at uniform points.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from whirplonk_b200 import Context, MultilinearExtension, ProtocolParameters, ProverState, cli_domain_separator
from whirplonk_b200.batch import Batch, ProofRequest, Server
from whirplonk_b200.rs import rs_commit_batch, rs_encode
from whirplonk_b200.whir import ENGINE_ID_BLAKE3, ENGINE_ID_SHA2, P, Config
from whirplonk_b200.zk import DeterministicRng, ZkConfig

SECURITY, POW_BITS = 100, 20

_shared = {}


def _ctx() -> Context:
    """One context per process, as a program keeps one per GPU."""
    if "ctx" not in _shared:
        _shared["ctx"] = Context(0)
    return _shared["ctx"]


def _server() -> Server:
    """The process's one server: 24 proofs in flight, half the free memory as its budget."""
    if "server" not in _shared:
        free, _ = torch.cuda.mem_get_info()
        _shared["server"] = Server(_ctx(), hbm_budget=free // 2, max_inflight=24)
    return _shared["server"]


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _prove(name, n, rate, fold=4, batch=1, points=1, sha2=False, field=3, host=False):
    return {"name": name, "kind": "prove", "n": n, "rate": rate, "fold": fold, "batch": batch, "points": points,
            "sha2": sha2, "field": field, "host": host}


def listed():
    return [
        # The smallest proof the benchmark's request mix holds: a chain of small launches.
        _prove("prove_n12_rate2", 12, 1),
        # A small proof at the middle rate.
        _prove("prove_n16_rate4", 16, 2),
        # The command line's default proof, its coefficients in host memory.
        _prove("prove_n18_rate2_host", 18, 1, host=True),
        # Several vectors in one commitment, an odd size, folding 3, SHA-2, two statements.
        _prove("prove_n17_x3_fold3_sha2", 17, 1, fold=3, batch=3, points=2, sha2=True),
        # An ordinary proof at the lowest rate.
        _prove("prove_n20_rate8", 20, 3),
        # The largest proof of the benchmark.
        _prove("prove_n24_rate4", 24, 2),
        # Encoder alone on a few ordinary vectors, as a program with its own hashing calls it.
        {"name": "rs_encode_3x18_exp8", "kind": "rs_encode", "count": 3, "log_len": 18, "log_exp": 3, "depth": 4},
        # Many small columns (a trace) committed at once, expansion 2.
        {"name": "rs_commit_64x16_exp2", "kind": "rs_commit", "count": 64, "log_len": 16, "log_exp": 1, "depth": 4},
        # Few large vectors, expansion 4.
        {"name": "rs_commit_4x22_exp4", "kind": "rs_commit", "count": 4, "log_len": 22, "log_exp": 2, "depth": 4},
        # Zero-knowledge proof of an ordinary polynomial.
        {"name": "zk_n18_rate4", "kind": "zk", "n": 18, "rate": 2, "polys": 1},
        # A prepared batch of small and ordinary proofs, run again and again.
        {"name": "batch16_n14_19", "kind": "batch", "count": 16, "lo": 14, "hi": 19, "mix": 7},
        # A burst of requests of every size on the server.
        {"name": "served24_n12_23", "kind": "served", "count": 24, "lo": 12, "hi": 23, "mix": 3},
    ]


def draw(rng):
    kind = rng.choice(["prove"] * 5 + ["rs_encode"] * 2 + ["rs_commit"] * 2 + ["zk", "batch", "served"])
    if kind == "prove":
        c = _prove("", rng.randint(12, 23), rng.randint(1, 3), fold=rng.choice([4, 4, 4, 2, 3, 5]),
                   batch=rng.choice([1, 1, 1, 2, 3, 5]), points=rng.choice([1, 1, 2, 3]), sha2=rng.random() < 0.2,
                   field=rng.choice([3, 3, 3, 2]), host=rng.random() < 0.3)
        # one vector of 2^23 costs what several smaller ones do
        c["n"] -= max(0, c["n"] - 20) if c["batch"] > 1 else 0
        c["field"] = 3 if c["sha2"] else c["field"]
    elif kind in ("rs_encode", "rs_commit"):
        log_len, log_exp = rng.randint(12, 24), rng.randint(1, 4)
        most = max(0, 26 - log_len - log_exp)
        count = max(1, min(64, int(2 ** rng.uniform(0, most + 0.99))))
        c = {"kind": kind, "count": count, "log_len": log_len, "log_exp": min(log_exp, 27 - log_len),
             "depth": rng.choice([4, 4, 4, 2, 3, 5])}
    elif kind == "zk":
        c = {"kind": kind, "n": rng.randint(12, 22), "rate": rng.randint(1, 3), "polys": rng.choice([1, 1, 2])}
    elif kind == "batch":
        lo = rng.randint(12, 17)
        c = {"kind": kind, "count": rng.randint(2, 24), "lo": lo, "hi": lo + rng.randint(0, 3),
             "mix": rng.randint(0, 10 ** 6)}
    else:
        lo = rng.randint(12, 18)
        c = {"kind": kind, "count": rng.randint(4, 24), "lo": lo, "hi": min(20, lo + rng.randint(0, 4)),
             "mix": rng.randint(0, 10 ** 6)}
    c.pop("name", None)
    return c


def _mix(case):
    """The (num_variables, rate) pairs of a batch or burst: sizes log-uniform."""
    r = random.Random(case["mix"])
    return [(r.randint(case["lo"], case["hi"]), r.randint(1, 3)) for _ in range(case["count"])]


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _words(gen, count):
    """Uniform canonical Goldilocks words on the GPU (as int64 bits)."""
    hi = torch.randint(0, 1 << 32, (count,), generator=gen, device="cuda", dtype=torch.int64)
    lo = torch.randint(0, 1 << 32, (count,), generator=gen, device="cuda", dtype=torch.int64)
    lo.masked_fill_(hi == 0xFFFFFFFF, 0)  # words above p - 1 (one in 2^32)
    return (hi << 32) | lo


def _u64(t):
    return t.cpu().numpy().view(np.uint64)


def _params(rate, fold=4, batch=1, sha2=False):
    return ProtocolParameters(False, rate, fold, fold, SECURITY, POW_BITS, batch,
                              ENGINE_ID_SHA2 if sha2 else ENGINE_ID_BLAKE3)


def _points(gen, count, n, field=3):
    p = _u64(_words(gen, 3 * n * count)).reshape(count, n, 3).copy()
    p[:, :, field:] = 0
    return p


def _requests(case, gen):
    ctx, out, keep = _ctx(), [], []
    for n, rate in _mix(case):
        c = _words(gen, 1 << n)
        pt = _points(gen, 1, n)
        torch.cuda.synchronize()
        ev = np.array(ctx.mle_evaluate(None, pt, on_device_ptr=c.data_ptr()), dtype=np.uint64).reshape(1, 3)
        out.append(ProofRequest(n, _params(rate), c.data_ptr(), pt, ev, on_device=True))
        keep.append(c)
    return out, keep


def _ext2_evaluations(coeffs, points, n):
    """Evaluations at Goldilocks2 points (X^2 = 7): folded in host arithmetic."""
    out = []
    for pt in points:
        v0, v1 = coeffs, np.zeros_like(coeffs)
        for k in range(n):
            h = v0.size // 2
            d0, d1 = _sub(v0[h:], v0[:h]), _sub(v1[h:], v1[:h])
            r0, r1 = pt[k, 0], pt[k, 1]
            a = _add(_mul(d0, r0), _mul(_mul(d1, r1), np.uint64(7)))
            b = _add(_mul(d0, r1), _mul(d1, r0))
            v0, v1 = _add(v0[:h], a), _add(v1[:h], b)
        out.append((int(v0[0]), int(v1[0]), 0))
    return out


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed * 1000003 + 17)
    kind, ctx = case["kind"], _ctx()
    s = {"kind": kind, "case": case}
    if kind == "prove":
        n, nvec = case["n"], case["batch"]
        c = _words(gen, nvec << n)
        pts = _points(gen, case["points"], n, case["field"])
        torch.cuda.synchronize()
        if case["field"] == 2:
            h = _u64(c).reshape(nvec, -1)
            evs = [_ext2_evaluations(h[v], pts[f:f + 1], n)[0] for f in range(case["points"]) for v in range(nvec)]
        else:
            evs = [ctx.mle_evaluate(None, pts[f], on_device_ptr=c.data_ptr() + (8 * v << n))
                   for f in range(case["points"]) for v in range(nvec)]
        params = _params(case["rate"], case["fold"], nvec, case["sha2"])
        s.update(config=Config.from_params(1 << n, params, case["field"]), ds=cli_domain_separator(params),
                 forms=[MultilinearExtension(pts[f]) for f in range(case["points"])], evaluations=evs)
        if case["host"]:
            s["coeffs"] = c.cpu().pin_memory().numpy().view(np.uint64).reshape(nvec, -1)
        else:
            s["device"] = c
    elif kind in ("rs_encode", "rs_commit"):
        s["vectors"] = _words(gen, case["count"] << case["log_len"])
        if kind == "rs_encode":
            words = case["count"] << (case["log_len"] + case["log_exp"])
            s["planes"] = torch.empty(words, dtype=torch.int64, device="cuda")
            s["scratch"] = torch.empty(words, dtype=torch.int64, device="cuda")
    elif kind == "zk":
        n, polys = case["n"], case["polys"]
        params = _params(case["rate"])
        c = _words(gen, polys << n)
        pt = _points(gen, 1, n, field=1)
        torch.cuda.synchronize()
        s.update(config=ZkConfig.from_params(1 << n, params, polys).disable_pow(), ds=cli_domain_separator(params),
                 device=c, forms=[MultilinearExtension(pt[0])], seed=(seed % 256).to_bytes(1, "little") * 32,
                 evaluations=[ctx.mle_evaluate(None, pt, on_device_ptr=c.data_ptr() + (8 * v << n))
                              for v in range(polys)])
    elif kind == "batch":
        reqs, s["keep"] = _requests(case, gen)
        s["batch"] = Batch(ctx, reqs, mode=Batch.GRAPH)
    elif kind == "served":
        s["requests"], s["keep"] = _requests(case, gen)
        s["server"] = _server()
    else:
        raise ValueError(kind)
    torch.cuda.synchronize()
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _bytes(b):
    return np.frombuffer(b, dtype=np.uint8)


def _padded(s, b):
    """The hints, whose length depends on the queries drawn, in the state's fixed
    buffer: zeros behind them, their length in the last 8 bytes."""
    if "hints" not in s:
        s["hints"], s["used"] = np.zeros((s["case"].get("count", 1) << 18) + (1 << 18), dtype=np.uint8), 0
    buf, n = s["hints"], len(b)
    buf[:n] = _bytes(b)
    buf[n:s["used"]] = 0
    buf[-8:] = np.array([n], dtype=np.int64).view(np.uint8)
    s["used"] = n
    return buf


def run(s):
    kind, ctx, case = s["kind"], _ctx(), s["case"]
    if kind == "prove":
        cfg = s["config"]
        ps = ProverState.from_ds(s["ds"], b"", ctx)
        if "device" in s:
            w = cfg.commit(ps, None, on_device_ptr=s["device"].data_ptr())
        else:
            w = cfg.commit(ps, s["coeffs"])
        claim = cfg.prove(ps, None, [w], s["forms"], s["evaluations"])
        narg, hints = ps.proof()
        return {"narg": _bytes(narg), "hints": _padded(s, hints),
                "point": np.array(claim.evaluation_point, dtype=np.uint64).view(np.int64),
                "rlc": np.array(claim.rlc_coefficients, dtype=np.uint64).view(np.int64)}
    if kind == "rs_encode":
        rs_encode(ctx, s["vectors"].data_ptr(), case["count"], case["log_len"], case["log_exp"], case["depth"],
                  s["scratch"].data_ptr(), s["planes"].data_ptr())
        return s["planes"]
    if kind == "rs_commit":
        roots = rs_commit_batch(ctx, None, case["log_exp"], case["depth"], on_device_ptr=s["vectors"].data_ptr(),
                                count=case["count"], log_len=case["log_len"])
        return _bytes(b"".join(roots))
    if kind == "zk":
        cfg = s["config"]
        ps = ProverState.from_ds(s["ds"], b"", ctx)
        rng = DeterministicRng(s["seed"])
        w = cfg.commit(ps, None, rng, on_device_ptr=s["device"].data_ptr())
        claim = cfg.prove(ps, None, w, s["forms"], s["evaluations"], rng)
        narg, hints = ps.proof()
        return {"narg": _bytes(narg), "hints": _padded(s, hints),
                "point": np.array(claim.evaluation_point, dtype=np.uint64).view(np.int64)}
    if kind == "batch":
        s["batch"].run()
        out = [s["batch"].proof(i) for i in range(case["count"])]
    else:
        tickets = [s["server"].submit(r) for r in s["requests"]]
        got = [s["server"].poll(t) for t in tickets]
        assert all(g is not None and g.status == 0 for g in got)
        out = [(g.narg, g.hints) for g in got]
    return {"narg": _bytes(b"".join(a for a, _ in out)), "hints": _padded(s, b"".join(b for _, b in out))}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _commit_work(words, m, N, planes, hash_words):
    """One matrix commitment of `words` message words: (bytes, integer operations).
    The codeword and the tree stay resident, so they are outputs.  A butterfly
    is counted as 3 operations, a hash compression as 700."""
    bfly = planes * (N // 2) * max(0, int(math.log2(max(m, 1))))
    comp = N * -(-8 * hash_words // 64) + N
    return 8 * (words + planes * N) + 64 * N, 3 * bfly + 700 * comp


def _prove_work(n, rate, fold=4, batch=1, field=3, sha2=False):
    sch = Config.from_params(1 << n, _params(rate, fold, batch, sha2), field).schedule
    d = 1 << fold
    b, f = _commit_work(batch << n, (1 << n) // d, sch[1], batch * d, batch * d)
    for r in range(sch[0]):
        vsize, N = sch[6 + 6 * r], sch[7 + 6 * r]
        x, y = _commit_work(field * vsize, vsize // d, N, field * d, field * d)
        b, f = b + x, f + y
    return b, f + 12 * (batch << n)


def work(case):
    kind = case["kind"]
    if kind == "prove":
        b, f = _prove_work(case["n"], case["rate"], case["fold"], case["batch"], case["field"], case["sha2"])
    elif kind in ("rs_encode", "rs_commit"):
        planes = case["count"] << case["depth"]
        m = 1 << (case["log_len"] - case["depth"])
        N = m << case["log_exp"]
        b = 8 * ((case["count"] << case["log_len"]) + (planes * N if kind == "rs_encode" else 0))
        f = 3 * planes * (N // 2) * (case["log_len"] - case["depth"])
        if kind == "rs_commit":
            f += 700 * case["count"] * N * (1 + -(-(8 << case["depth"]) // 64))
    elif kind == "zk":
        b, f = _prove_work(case["n"], case["rate"], field=1)
        b, f = case["polys"] * b, case["polys"] * f
    else:
        b = f = 0
        for n, rate in _mix(case):
            x, y = _prove_work(n, rate)
            b, f = b + x, f + y
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# the encoder's codewords with 64-bit numpy arithmetic
# ---------------------------------------------------------------------------
_M32 = np.uint64(0xFFFFFFFF)
_S32 = np.uint64(32)
_P = np.uint64(P)


def _add(a, b):
    c = a + b
    c = np.where(c < a, c + _M32, c)
    return np.where(c >= _P, c - _P, c)


def _sub(a, b):
    return np.where(a < b, a - b + _P, a - b)


def _mul(a, b):
    """a b mod p from 32-bit limbs: 2^64 = 2^32 - 1 and 2^96 = -1 (mod p)."""
    a0, a1, b0, b1 = a & _M32, a >> _S32, b & _M32, b >> _S32
    p00, p01, p10, p11 = a0 * b0, a0 * b1, a1 * b0, a1 * b1
    mid = (p00 >> _S32) + (p01 & _M32) + (p10 & _M32)
    lo = (p00 & _M32) | (mid << _S32)
    hi = p11 + (p01 >> _S32) + (p10 >> _S32) + (mid >> _S32)
    hl, hh = hi & _M32, hi >> _S32
    t = np.where(lo < hh, lo - hh - _M32, lo - hh)
    u = hl * _M32
    r = t + u
    r = np.where(r < t, r + _M32, r)
    return np.where(r >= _P, r - _P, r)


def exact(case, seed):
    if case["kind"] != "rs_encode" or case["count"] << (case["log_len"] + case["log_exp"]) > 1 << 23:
        return None
    gen = torch.Generator(device="cuda" if torch.cuda.is_available() else "cpu")
    gen.manual_seed(seed * 1000003 + 17)
    v = _u64(_words(gen, case["count"] << case["log_len"]))
    planes = case["count"] << case["depth"]
    m = (1 << case["log_len"]) >> case["depth"]
    N = m << case["log_exp"]
    x = np.zeros((planes, N), dtype=np.uint64)
    x[:, :m] = v.reshape(planes, m)
    # Stockham radix-2, natural order in and out
    w = pow(7, (P - 1) // N, P)
    x, size, s = x.reshape(planes, N, 1), N, 1
    while size > 1:
        half = size // 2
        tw = np.ones(half, dtype=np.uint64)  # powers of the size-th root
        root = np.array([w], dtype=np.uint64)
        k, step = 1, root
        while k < half:
            tw[k:2 * k] = _mul(tw[:k], step)
            step = _mul(step, step)
            k *= 2
        a, b = x[:, :half], x[:, half:]
        x = np.stack([_add(a, b), _mul(_sub(a, b), tw[None, :, None])], axis=2).reshape(planes, half, 2 * s)
        w, size, s = w * w % P, half, 2 * s
    return torch.from_numpy(x.reshape(-1).view(np.int64).copy())
