"""The work that a user of the library has it do, as measurable cases.

A case is a dict of plain values.  `listed()` names the fixed ones, `draw(rng)`
gives another of the same ranges, `prepare(case, seed)` makes what a program
holds before the call (bases, scalars, contexts, tables, a server), `run(state)`
is one pass through the public entry points, `work(case)` its unavoidable
traffic and multiply count, `exact(case, seed)` the result by Python integers
where that takes seconds at most.

Every result is asked for in a canonical form (32-byte encodings or canonical
affine bytes), so it does not depend on the order of the additions.
"""

from __future__ import annotations

import concurrent.futures
import math
import random

import numpy as np
import torch

import helioselene_gb300 as hs
from helioselene_gb300.api import Context, FixedBase, Server

HELIOS, SELENE = hs.HELIOS, hs.SELENE
BOTH = (SELENE, HELIOS)  # the heavier curve first, as the callers of pairs do
FORMATS = {"jacobian51": hs.FMT_JACOBIAN51, "affine51": hs.FMT_AFFINE51, "affine": hs.FMT_AFFINE,
           "compressed": hs.FMT_COMPRESSED}
DEV = "cuda:0"


def listed():
    return [
        # the smallest call: one 16-term MSM from host records, result read back
        # (HeliosPoint::multi_scalar_mul on a handful of points): latency and launches
        {"name": "msm_host_16", "kind": "msm_host", "curve": HELIOS, "n": 16, "format": "jacobian51", "pinned": False},
        # verification of one FCMP++ proof: a Selene MSM of 602 and a Helios MSM of 345
        # terms from ordinary host records, one call after the other
        {"name": "verify_host", "kind": "verify_host", "batch": 1},
        # many verifications at once: 256 MSMs of each size as one launch sequence per curve
        {"name": "verify_batch_256", "kind": "verify_batch", "batch": 1, "count": 256},
        # an ordinary MSM whose bases arrive as 32-byte encodings (wire format): decoding
        # on the device, odd size
        {"name": "msm_encoded_65521", "kind": "msm_host", "curve": SELENE, "n": 65521, "format": "compressed",
         "pinned": False},
        # the headline benchmark: one MSM of 2^20 device-resident terms on each curve, side
        # by side on two streams, 1% edge slices
        {"name": "msm_pair_2p20", "kind": "msm_pair", "n": 1 << 20, "edge": True},
        # the same pair end to end: reference records in pinned host memory, one call per
        # curve from two host threads
        {"name": "msm_pair_host_2p20", "kind": "msm_pair_host", "n": 1 << 20, "pinned": True},
        # the largest single MSM of the size sweep
        {"name": "msm_selene_2p22", "kind": "msm_device", "curve": SELENE, "n": 1 << 22},
        # many MSMs of uneven sizes in one batch per curve, log-uniform in [64, 65536]
        {"name": "batch_1024", "kind": "msm_batch", "count": 1024, "n_min": 64, "n_max": 65536, "sizes_seed": 3},
        # Pedersen commitments r H + sum v_i G_i over a large resident generator set
        {"name": "commit_2p18", "kind": "fixed_base", "curve": HELIOS, "n": 1 << 18, "count": 24, "H": True},
        # one layer of FCMP++ tree hashing: thousands of hashes over few generators
        {"name": "tree_228", "kind": "fixed_base", "curve": SELENE, "n": 228, "count": 8192, "H": False},
        # the server with a queue of requests: the serving mixture of sizes, three quarters
        # of the bases from the resident pool, the others sent along
        {"name": "serve_96", "kind": "serve", "requests": 96, "pool": 1 << 16, "sizes_seed": 4},
        # independent scalar multiplications, affine results
        {"name": "scalar_mul_2p17", "kind": "scalar_mul", "curve": HELIOS, "n": 1 << 17},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["msm_device", "msm_device", "msm_device", "msm_host", "msm_host", "msm_pair", "msm_pair_host",
                       "verify_host", "verify_batch", "msm_batch", "fixed_base", "serve", "scalar_mul"])
    curve = rng.choice([HELIOS, SELENE])
    if kind == "msm_device":
        return {"kind": kind, "curve": curve, "n": _log_uniform(rng, 16, 1 << 22)}
    if kind == "msm_host":
        return {"kind": kind, "curve": curve, "n": _log_uniform(rng, 16, 1 << 20), "format": rng.choice(sorted(FORMATS)),
                "pinned": rng.random() < 0.5}
    if kind == "msm_pair":
        return {"kind": kind, "n": _log_uniform(rng, 1 << 14, 1 << 21), "edge": rng.random() < 0.5}
    if kind == "msm_pair_host":
        return {"kind": kind, "n": _log_uniform(rng, 1 << 14, 1 << 20), "pinned": rng.random() < 0.5}
    if kind == "verify_host":
        # the smallest batch is the listed one
        return {"kind": kind, "batch": rng.randint(2, 64)}
    if kind == "verify_batch":
        return {"kind": kind, "batch": rng.randint(1, 10), "count": _log_uniform(rng, 4, 300)}
    if kind == "msm_batch":
        return {"kind": kind, "count": _log_uniform(rng, 8, 1000), "n_min": 64, "n_max": _log_uniform(rng, 512, 65536),
                "sizes_seed": rng.randrange(1 << 30)}
    if kind == "fixed_base":
        n = _log_uniform(rng, 18, 1 << 18)
        count = min(8192, max(1, int((1 << 22) / n * rng.uniform(0.2, 1.4))))
        return {"kind": kind, "curve": curve, "n": n, "count": count, "H": rng.random() < 0.5}
    if kind == "serve":
        return {"kind": kind, "requests": _log_uniform(rng, 8, 128), "pool": 1 << 16,
                "sizes_seed": rng.randrange(1 << 30)}
    return {"kind": "scalar_mul", "curve": curve, "n": _log_uniform(rng, 64, 1 << 18)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _generator(seed, salt):
    g = torch.Generator(device=DEV)
    g.manual_seed((seed * 1000003 + salt) & 0x7FFFFFFFFFFFFFFF)
    return g


def _field_bytes(seed, salt, n):
    """n 32-byte values, uniform below 2^255 (a value at or above the order or
    the modulus has probability 2^-128)."""
    v = torch.randint(0, 256, (n, 32), dtype=torch.uint8, device=DEV, generator=_generator(seed, salt))
    v[:, 31] &= 0x7F
    return v


def _scalars(seed, curve, n, edge=False):
    s = _field_bytes(seed, 2 * curve, n)
    if edge:  # 1% in total: zero scalars, and scalars with only the top window nonzero
        k = n // 200
        s[:k] = 0
        s[k:2 * k, :30] = 0
    return s


_contexts = {}


def _context(role, curve):
    """The contexts that a program of this kind keeps: one per curve."""
    key = (role, curve)
    if key not in _contexts:
        c = Context(0)
        if role == "pair":  # two MSMs side by side: the Selene stream first, no window split
            c.set_split(0)
            c.set_priority(curve == SELENE)
        _contexts[key] = c
    return _contexts[key]


def _bases(seed, curve, n, edge=False):
    """n affine bases (64 bytes each) on the device: map-to-curve images."""
    u = _field_bytes(seed, 2 * curve + 1, n)
    if edge and n >= 400:  # and one base repeated
        u[-(n // 200):] = u[-1].clone()
    pts = torch.empty(n * 64, dtype=torch.uint8, device=DEV)
    torch.cuda.synchronize()
    _context("single", curve).map_to_curve_device(curve, u.data_ptr(), n, pts.data_ptr())
    torch.cuda.synchronize()
    return pts.view(n, 64)


def _limbs51(x):
    """(n, 32) little-endian bytes -> (n, 5) radix-2^51 limbs (int64)."""
    w = x.contiguous().view(torch.int64).view(-1, 4)
    m = (1 << 51) - 1

    def shr(a, k):  # logical shift
        return (a >> k) & ((1 << (64 - k)) - 1)

    return torch.stack([w[:, 0] & m, (shr(w[:, 0], 51) | (w[:, 1] << 13)) & m, (shr(w[:, 1], 38) | (w[:, 2] << 26)) & m,
                        (shr(w[:, 2], 25) | (w[:, 3] << 39)) & m, shr(w[:, 3], 12) & m], dim=1)


def _records(pts, fmt):
    """Affine bases in one of the input formats (device tensor of bytes)."""
    if fmt == "affine":
        return pts
    if fmt == "compressed":
        enc = pts[:, :32].clone()
        enc[:, 31] |= (pts[:, 32] & 1) << 7
        return enc
    x, y = _limbs51(pts[:, :32]), _limbs51(pts[:, 32:])
    if fmt == "affine51":
        return torch.cat([x, y], dim=1).view(torch.uint8)
    z = torch.zeros_like(x)
    z[:, 0] = 1
    return torch.cat([x, y, z], dim=1).view(torch.uint8)


def _host(t, pinned):
    t = t.reshape(-1)
    h = torch.empty(t.numel(), dtype=torch.uint8, pin_memory=pinned)
    h.copy_(t)
    return h.numpy()


def _host_msm(seed, curve, n, fmt, pinned):
    return {"curve": curve, "scalars": _host(_scalars(seed, curve, n), pinned),
            "points": _host(_records(_bases(seed, curve, n), fmt), pinned), "format": FORMATS[fmt]}


def _verify_sizes(batch):
    return {SELENE: 522 + 80 * batch, HELIOS: 265 + 80 * batch}


def _batch_sizes(case):
    """Sizes per curve of a batch of uneven MSMs (the case's own, the same for every seed)."""
    r = random.Random(case["sizes_seed"])
    sizes = {HELIOS: [], SELENE: []}
    for _ in range(case["count"]):
        sizes[r.choice((HELIOS, SELENE))].append(_log_uniform(r, case["n_min"], case["n_max"]))
    return sizes


def _serve_sizes(case):
    """(curve, points) of each request: 70% of 256..4096 points, 25% of 4096..65536, 5% of 2^18."""
    r = random.Random(case["sizes_seed"])
    out = []
    for i in range(case["requests"]):
        u = r.random()
        n = _log_uniform(r, 256, 4096) if u < 0.70 else _log_uniform(r, 4096, 65536) if u < 0.95 else 1 << 18
        out.append((HELIOS if i % 2 else SELENE, n))
    return out


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "kind": kind}
    if kind == "msm_host":
        s["msm"] = _host_msm(seed, case["curve"], case["n"], case["format"], case["pinned"])
        s["ctx"] = _context("single", case["curve"])
    elif kind == "verify_host":
        s["msms"] = [_host_msm(seed, c, n, "jacobian51", False) for c, n in _verify_sizes(case["batch"]).items()]
        s["ctx"] = _context("single", HELIOS)  # one context for both calls
    elif kind == "msm_pair_host":
        s["msms"] = [_host_msm(seed, c, case["n"], "jacobian51", case["pinned"]) for c in BOTH]
        s["ctxs"] = [_context("single", c) for c in BOTH]
        s["pool"] = concurrent.futures.ThreadPoolExecutor(max_workers=2)
    elif kind == "msm_device":
        c, n = case["curve"], case["n"]
        s.update(ctx=_context("single", c), curve=c, n=n, scalars=_scalars(seed, c, n), points=_bases(seed, c, n),
                 out=torch.zeros(32, dtype=torch.uint8, device=DEV))
    elif kind == "msm_pair":
        n = case["n"]
        s["parts"] = [{"ctx": _context("pair", c), "curve": c, "n": n, "scalars": _scalars(seed, c, n, case["edge"]),
                       "points": _bases(seed, c, n, case["edge"]),
                       "out": torch.zeros(32, dtype=torch.uint8, device=DEV)} for c in BOTH]
    elif kind in ("verify_batch", "msm_batch"):
        if kind == "verify_batch":
            sizes = {c: [n] * case["count"] for c, n in _verify_sizes(case["batch"]).items()}
        else:
            sizes = _batch_sizes(case)
        s["parts"] = [{"ctx": _context("pair", c), "curve": c, "sizes": sizes[c],
                       "scalars": _scalars(seed, c, sum(sizes[c])), "points": _bases(seed, c, sum(sizes[c])),
                       "out": torch.zeros((len(sizes[c]), 32), dtype=torch.uint8, device=DEV)}
                      for c in BOTH if sizes[c]]
    elif kind == "fixed_base":
        c, n = case["curve"], case["n"]
        g = _bases(seed, c, n + 1).cpu().numpy()
        fb = FixedBase(_context("single", c), c, g[:n], H=g[n] if case["H"] else None)
        s.update(fb=fb, count=case["count"], scalars=_scalars(seed, c, case["count"] * (n + (1 if case["H"] else 0))),
                 out=torch.zeros((case["count"], 64), dtype=torch.uint8, device=DEV))
    elif kind == "serve":
        srv = Server(0, slots=8, max_batch_points=1 << 23)
        for c in (HELIOS, SELENE):
            srv.set_pool(c, _bases(seed, c, case["pool"]).cpu().numpy())
        reqs, offs = [], {HELIOS: 0, SELENE: 0}
        sizes = _serve_sizes(case)
        total = {c: sum(n for k, n in sizes if k == c) for c in (HELIOS, SELENE)}
        sc = {c: _host(_scalars(seed + 1, c, max(1, total[c])), True).reshape(-1, 32) for c in total}
        fresh = {c: _host(_bases(seed + 1, c, max(1, total[c])), True).reshape(-1, 64) for c in total}
        idx = np.random.default_rng(seed).integers(0, case["pool"], size=sum(total.values()), dtype=np.uint32)
        at = 0
        for c, n in sizes:
            pooled, o = (3 * n) // 4, offs[c]
            reqs.append((c, sc[c][o:o + n].reshape(-1), idx[at:at + pooled], fresh[c][o:o + n - pooled].reshape(-1)))
            offs[c] += n
            at += n
        s.update(server=srv, requests=reqs)
    else:  # scalar_mul
        c, n = case["curve"], case["n"]
        s.update(ctx=_context("single", c), curve=c, n=n, scalars=_scalars(seed, c, n), points=_bases(seed, c, n),
                 out=torch.zeros((n, 64), dtype=torch.uint8, device=DEV))
    torch.cuda.synchronize()
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _call(ctx, m):
    out = ctx.msm(m["curve"], m["scalars"], m["points"], m["format"], hs.FMT_COMPRESSED)
    return np.frombuffer(out, dtype=np.uint8)


def run(s):
    kind = s["kind"]
    if kind == "msm_host":
        return _call(s["ctx"], s["msm"])
    if kind == "verify_host":
        return [_call(s["ctx"], m) for m in s["msms"]]
    if kind == "msm_pair_host":
        jobs = [s["pool"].submit(_call, c, m) for c, m in zip(s["ctxs"], s["msms"])]
        return [j.result() for j in jobs]
    if kind == "msm_device":
        s["ctx"].msm_device(s["curve"], s["scalars"].data_ptr(), s["points"].data_ptr(), s["n"], s["out"].data_ptr(),
                            hs.FMT_COMPRESSED)
        return s["out"]
    if kind == "msm_pair":
        for p in s["parts"]:
            p["ctx"].msm_device(p["curve"], p["scalars"].data_ptr(), p["points"].data_ptr(), p["n"],
                                p["out"].data_ptr(), hs.FMT_COMPRESSED)
        return [p["out"] for p in s["parts"]]
    if kind in ("verify_batch", "msm_batch"):
        for p in s["parts"]:
            p["ctx"].msm_batch_device(p["curve"], p["sizes"], p["scalars"].data_ptr(), p["points"].data_ptr(),
                                      p["out"].data_ptr(), hs.FMT_COMPRESSED)
        return [p["out"] for p in s["parts"]]
    if kind == "fixed_base":
        s["fb"].commit_device(s["scalars"].data_ptr(), s["count"], s["out"].data_ptr(), hs.FMT_AFFINE)
        return s["out"]
    if kind == "serve":
        srv = s["server"]
        tickets = [srv.submit(c, sc, pool_idx=i, fresh_points=f) for c, sc, i, f in s["requests"]]
        return np.frombuffer(b"".join(srv.wait(t)[0] for t in tickets), dtype=np.uint8)
    s["ctx"].scalar_mul_device(s["curve"], s["scalars"].data_ptr(), s["points"].data_ptr(), s["n"],
                               s["out"].data_ptr(), hs.FMT_AFFINE)
    return s["out"]


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
MUL_OPS = {HELIOS: 2 * 72, SELENE: 2 * 112}  # 32-bit multiply halves of one field product, reduction included
INPUT_BYTES = {"jacobian51": 120, "affine51": 80, "affine": 64, "compressed": 32}


def _msm_products(n):
    """Field products of a Pippenger MSM at its best window width: an affine
    addition (6 products) per point and window, two per bucket, 256 doublings."""
    return min(-(-256 // c) * (6 * n + 12 * (1 << (c - 1))) for c in range(2, 21)) + 256 * 9


def _fixed_products(n):
    return min(-(-256 // c) * 6 * n + 12 * (1 << (c - 1)) for c in range(2, 21))


def work(case):
    kind = case["kind"]
    if kind in ("msm_host", "msm_device"):
        pb = INPUT_BYTES[case.get("format", "affine")]
        products = _msm_products(case["n"])
        if pb == 32:
            products += 300 * case["n"]  # a square root per encoding
        return {"bytes": case["n"] * (32 + pb) + 32, "flops": products * MUL_OPS[case["curve"]]}
    if kind in ("msm_pair", "msm_pair_host"):
        pb = 64 if kind == "msm_pair" else 120
        return {"bytes": 2 * case["n"] * (32 + pb) + 64, "flops": _msm_products(case["n"]) * sum(MUL_OPS.values())}
    if kind in ("verify_host", "verify_batch", "msm_batch"):
        if kind == "msm_batch":
            sizes = _batch_sizes(case)
        else:
            sizes = {c: [n] * case.get("count", 1) for c, n in _verify_sizes(case["batch"]).items()}
        pb = 120 if kind == "verify_host" else 64
        return {"bytes": sum(sum(v) * (32 + pb) + 32 * len(v) for v in sizes.values()),
                "flops": sum(_msm_products(n) * MUL_OPS[c] for c, v in sizes.items() for n in v)}
    if kind == "fixed_base":
        g = case["n"] + (1 if case["H"] else 0)
        return {"bytes": case["count"] * (32 * g + 64) + 64 * g,
                "flops": case["count"] * _fixed_products(g) * MUL_OPS[case["curve"]]}
    if kind == "serve":
        sizes = _serve_sizes(case)
        return {"bytes": sum(n * 32 + (3 * n) // 4 * 4 + (n - (3 * n) // 4) * 64 + 32 for _, n in sizes)
                + 2 * 64 * case["pool"],
                "flops": sum(_msm_products(n) * MUL_OPS[c] for c, n in sizes)}
    # a scalar multiplication: 256 doublings of 9 products and 51 additions of 14
    return {"bytes": case["n"] * (32 + 64 + 64), "flops": case["n"] * (256 * 9 + 51 * 14) * MUL_OPS[case["curve"]]}


# ---------------------------------------------------------------------------
# the result by Python integers (small cases)
# ---------------------------------------------------------------------------
P = 2**255 - 19
Q = 2**255 - 85737960593035654572250192257530476641
FIELD = {HELIOS: P, SELENE: Q}
CURVE_B = {HELIOS: 15789920373731020205926570676277057129217619222203920395806844808978996083412,
           SELENE: 50691664119640283727448954162351551669994268339720539671652090628799494505816}
SWU_Z = {HELIOS: 7, SELENE: -4}
EXACT_MAX_POINTS = 1200


def _sqrt(a, m):
    if m % 8 == 5:
        x = pow(a, (m + 3) // 8, m)
        if x * x % m != a:
            x = x * pow(2, (m - 1) // 4, m) % m
    else:
        x = pow(a, (m + 1) // 4, m)
    return x if x * x % m == a else None


def _swu(u, curve):
    """Simplified SWU map (RFC 9380, 6.6.2) onto y^2 = x^3 - 3x + b."""
    m, b, z = FIELD[curve], CURVE_B[curve], SWU_Z[curve]
    t = z * u * u % m
    den = (t * t + t) % m
    x = (-b * pow(-3, -1, m) * (1 + pow(den, -1, m)) if den else b * pow(-3 * z, -1, m)) % m
    y = _sqrt((x**3 - 3 * x + b) % m, m)
    if y is None:
        x = t * x % m
        y = _sqrt((x**3 - 3 * x + b) % m, m)
    return x, (y if y % 2 == u % m % 2 else (m - y) % m)


def _padd(p, q, m):
    """Affine addition; None is the identity."""
    if p is None or q is None:
        return q if p is None else p
    if p[0] == q[0]:
        if (p[1] + q[1]) % m == 0:
            return None
        lam = (3 * p[0] * p[0] - 3) * pow(2 * p[1], -1, m) % m
    else:
        lam = (q[1] - p[1]) * pow(q[0] - p[0], -1, m) % m
    x = (lam * lam - p[0] - q[0]) % m
    return x, (lam * (p[0] - x) - p[1]) % m


def _msm_exact(seed, curve, n):
    m = FIELD[curve]
    sc = [int.from_bytes(r.tobytes(), "little") for r in _scalars(seed, curve, n).cpu().numpy()]
    us = [int.from_bytes(r.tobytes(), "little") for r in _field_bytes(seed, 2 * curve + 1, n).cpu().numpy()]
    pts = [_swu(u, curve) for u in us]
    c, total = 6, None
    for k in range(-(-256 // c) - 1, -1, -1):
        for _ in range(c):
            total = _padd(total, total, m)
        buckets = [None] * (1 << c)
        for s, p in zip(sc, pts):
            d = (s >> (c * k)) & ((1 << c) - 1)
            buckets[d] = _padd(buckets[d], p, m)
        run = None
        acc = None
        for b in reversed(buckets[1:]):
            run = _padd(run, b, m)
            acc = _padd(acc, run, m)
        total = _padd(total, acc, m)
    if total is None:
        return np.zeros(32, np.uint8)
    return np.frombuffer((total[0] | (total[1] & 1) << 255).to_bytes(32, "little"), dtype=np.uint8)


def exact(case, seed):
    if case["kind"] in ("msm_host", "msm_device") and case["n"] <= EXACT_MAX_POINTS:
        out = _msm_exact(seed, case["curve"], case["n"])
        return out if case["kind"] == "msm_host" else torch.from_numpy(out.copy())
    if case["kind"] == "verify_host" and case["batch"] <= 2:
        return [_msm_exact(seed, c, n) for c, n in _verify_sizes(case["batch"]).items()]
    return None
