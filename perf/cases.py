"""The work that a user of this framework has it do, as cases that can be timed and checked.

Each case is a dict of plain values.  ``prepare`` makes what a program holds before the call (expansions, index and
order arrays, shifts, the operator context or the execution plan), ``run`` is one pass through the public entry
points, ``exact`` computes the same results in FP64 from the defining formulas (solid harmonics and the direct
O(P^4) translation sums) with torch alone.

Expansions are those of unit charges of random sign, uniform in a ball of radius 1/2 around the centre (local inputs:
clouds centred at distance 2 to 4); M2L shifts have a uniform direction and a length in [2, 4], M2M and L2L shifts go
to the corners of an octant cube, as in this repository's benchmark and tests.

Kinds of case:
  device  one batch of translations between device-resident expansions (sfmm_translate_device)
  host    one batch between pinned host arrays (sfmm_translate_host_packed)
  plan    a mixed-order workload of all three operators as an execution plan, built once and replayed
  fmm     a whole uniform-octree pass: P2M at the leaves, M2M up, M2L across, L2L down
  p2x     P2M (regular) or P2L (singular) of the particles of every leaf
  eval    L2P (potential, with or without gradient) or M2P at particles
"""
import math

import numpy as np
import torch

import solidfmm_gb300 as sf
from solidfmm_gb300 import fmm as sf_fmm

PRECISION = {"plain": sf.PLAIN, "split": sf.SPLIT, "split_ff": sf.SPLIT_FF, "tf32x3": sf.TC_TF32,
             "bf16x6": sf.TC_BF16X6}
DEV = "cuda:0"


# ---- the cases ----

def listed():
    return [
        # the coarse levels of a tree, or a small tree: a few hundred translations, where the call's latency counts
        {"name": "m2l_f64_p6_n600", "kind": "device", "op": "m2l", "precision": "plain", "dtype": "f64", "p": 6,
         "n": 600, "share": 8},
        # double precision at the common order 10: an independent batch of 100 000 (the small benchmark workload)
        {"name": "m2l_f64_p10_n100k", "kind": "device", "op": "m2l", "precision": "plain", "dtype": "f64", "p": 10,
         "n": 100_000, "share": 1},
        # double precision at order 16, the precision every user of the C++ interface gets by default
        {"name": "m2l_f64_p16_n500k", "kind": "device", "op": "m2l", "precision": "plain", "dtype": "f64", "p": 16,
         "n": 500_000, "share": 1},
        # the headline workload's precision and order: split precision, a batch far larger than L2
        {"name": "m2l_split_p16_n1m", "kind": "device", "op": "m2l", "precision": "split", "dtype": "f64", "p": 16,
         "n": 1_000_000, "share": 1},
        # the tensor-core mode, for users who need FP32-class accuracy from FP64 expansions
        {"name": "m2l_tf32x3_p16_n300k", "kind": "device", "op": "m2l", "precision": "tf32x3", "dtype": "f64",
         "p": 16, "n": 300_000, "share": 1},
        # single precision throughout, children into parents (eight translations per target)
        {"name": "m2m_f32_p20_n200k", "kind": "device", "op": "m2m", "precision": "plain", "dtype": "f32", "p": 20,
         "n": 200_000, "share": 8},
        # double precision downward pass at a high, odd order: every parent's local into its eight children
        {"name": "l2l_f64_p21_n100k", "kind": "device", "op": "l2l", "precision": "plain", "dtype": "f64", "p": 21,
         "n": 100_000, "share": 8},
        # uneven orders, all three operators, planned once and replayed (adaptive-order codes)
        {"name": "plan_split_p4to24_n150k", "kind": "plan", "precision": "split", "p_lo": 4, "p_hi": 24,
         "n": 150_000},
        # a whole FMM pass: 32 768 leaves of 32 particles at order 12
        {"name": "fmm_split_p12_depth5", "kind": "fmm", "precision": "split", "p": 12, "depth": 5, "per_leaf": 32},
        # leaf expansions from particles, leaves of uneven size (none to about 64 particles)
        {"name": "p2m_p12_32k_leaves", "kind": "p2x", "order": "p2m", "p": 12, "n": 32_768, "per_leaf": 32},
        # potential and gradient of the leaf locals at a million particles
        {"name": "l2p_grad_p12_n1m", "kind": "eval", "order": "l2p", "gradient": True, "p": 12, "n": 1_000_000,
         "per_leaf": 32},
        # a program that keeps its expansions in host memory: the bulk call on pinned arrays, odd order and size
        {"name": "host_m2l_f64_p13_n60k", "kind": "host", "op": "m2l", "precision": "plain", "dtype": "f64", "p": 13,
         "n": 60_001},
    ]


def _spread(rng, lo, hi):
    """An integer spread over the logarithm of [lo, hi]."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["device", "device", "device", "device", "plan", "fmm", "p2x", "eval", "host"])
    if kind in ("device", "host"):
        dtype = rng.choice(["f64", "f64", "f32"])
        precision = "plain" if dtype == "f32" else rng.choice(["plain", "plain", "split", "split_ff", "tf32x3",
                                                               "bf16x6"])
        top = 16 if precision in ("tf32x3", "bf16x6") else (30 if dtype == "f64" and precision == "plain" else 28)
        p = rng.randint(4, top)
        op = rng.choice(["m2l", "m2l", "m2m", "l2l"])
        # at most the work of 300 000 translations at order 16 (host: 60 000), and 2 GB of expansions
        most = int((60_000 if kind == "host" else 300_000) * min(1.0, (16.0 / p) ** 3))
        n = _spread(rng, 1_000 if kind == "host" else 64, most)
        case = {"kind": kind, "op": op, "precision": precision, "dtype": dtype, "p": p, "n": n}
        if kind == "device":
            case["share"] = rng.choice([1, 8])
        return case
    if kind == "plan":
        lo = rng.randint(2, 12)
        return {"kind": "plan", "precision": rng.choice(["plain", "split"]), "p_lo": lo, "p_hi": lo + rng.randint(2, 12),
                "n": _spread(rng, 2_000, 100_000)}
    if kind == "fmm":
        depth = rng.randint(3, 4)
        return {"kind": "fmm", "precision": rng.choice(["plain", "split"]), "p": rng.randint(4, 14), "depth": depth,
                "per_leaf": rng.randint(5, 60)}
    if kind == "p2x":
        return {"kind": "p2x", "order": rng.choice(["p2m", "p2l"]), "p": rng.randint(3, 24), "n": _spread(rng, 64, 20_000),
                "per_leaf": rng.randint(4, 64)}
    order = rng.choice(["l2p", "l2p", "m2p"])
    return {"kind": "eval", "order": order, "gradient": order == "l2p" and rng.random() < 0.6, "p": rng.randint(3, 24),
            "n": _spread(rng, 500, 250_000), "per_leaf": rng.randint(4, 64)}


# ---- solid harmonics in FP64 (rows are coefficients, columns are points) ----
# Layout of an expansion of order P: degree n has its real parts at n(n+1) and its imaginary parts at (n+1)^2.

def _columns(P, x, y, z, singular):
    """(re, im) of R_n^m (or S_n^m), 0 <= m <= n < P, as dicts of column vectors."""
    re, im = {}, {}
    r2 = x * x + y * y + z * z
    zero = torch.zeros_like(x)
    if singular:
        inv = 1.0 / r2
        re[0, 0], im[0, 0] = inv.sqrt(), zero
        for m in range(1, P):
            f = (2 * m - 1) * inv
            a, b = re[m - 1, m - 1], im[m - 1, m - 1]
            re[m, m], im[m, m] = (a * x - b * y) * f, (a * y + b * x) * f
        zi = z * inv
        for m in range(P):
            for n in range(m + 1, P):
                f = (2 * n - 1) * zi
                re[n, m], im[n, m] = f * re[n - 1, m], f * im[n - 1, m]
                if n > m + 1:
                    g = ((n + m - 1) * (n - m - 1)) * inv
                    re[n, m] = re[n, m] - g * re[n - 2, m]
                    im[n, m] = im[n, m] - g * im[n - 2, m]
    else:
        re[0, 0], im[0, 0] = torch.ones_like(x), zero
        for m in range(1, P):
            f = 1.0 / (2 * m)
            a, b = re[m - 1, m - 1], im[m - 1, m - 1]
            re[m, m], im[m, m] = (a * x - b * y) * f, (a * y + b * x) * f
        for m in range(P):
            for n in range(m + 1, P):
                f = 1.0 / ((n + m) * (n - m))
                re[n, m], im[n, m] = (2 * n - 1) * z * re[n - 1, m], (2 * n - 1) * z * im[n - 1, m]
                if n > m + 1:
                    re[n, m] = re[n, m] - r2 * re[n - 2, m]
                    im[n, m] = im[n, m] - r2 * im[n - 2, m]
                re[n, m], im[n, m] = re[n, m] * f, im[n, m] * f
    return re, im


def _full(P, re, im):
    """Complex coefficients C_n^m for every |m| <= n at row n^2 + n + m (C_n^-m = (-1)^m conj C_n^m)."""
    rows = []
    for n in range(P):
        for m in range(-n, n + 1):
            a = abs(m)
            c = torch.complex(re[n, a], im[n, a])
            rows.append(c if m >= 0 else (-1) ** a * c.conj())
    return torch.stack(rows)


def _split_rows(P, e):
    """(re, im) dicts of a (P(P+1), N) coefficient array."""
    re = {(n, m): e[n * (n + 1) + m] for n in range(P) for m in range(n + 1)}
    im = {(n, m): e[(n + 1) * (n + 1) + m] for n in range(P) for m in range(n + 1)}
    return re, im


def _join_rows(P, re, im):
    rows = [None] * (P * (P + 1))
    for n in range(P):
        for m in range(n + 1):
            rows[n * (n + 1) + m] = re[n, m]
            rows[(n + 1) * (n + 1) + m] = im[n, m]
    return torch.stack(rows)


def _translate(op, P, src, shift):
    """The direct translation sums in FP64: src (N, P(P+1)), shift (N, 3) -> (N, P(P+1))."""
    out = torch.empty_like(src)
    PH = 2 * P - 1 if op == "m2l" else P
    step = max(256, int(1.5e9 / (16 * (PH * PH + 3 * P * P))))
    for b in range(0, src.shape[0], step):
        e = src[b:b + step].t()
        x, y, z = (shift[b:b + step, k].contiguous() for k in range(3))
        if op == "m2m":
            x, y, z = -x, -y, -z
        C = _full(P, *_split_rows(P, e))
        H = _full(PH, *_columns(PH, x, y, z, op == "m2l"))
        re, im = {}, {}
        for n in range(P):
            for m in range(n + 1):
                if op == "m2l":    # L_n^m = (-1)^n sum conj(M_k^l) S_{n+k}^{m+l}
                    kl = [(k, l) for k in range(P) for l in range(-k, k + 1)]
                    h = [((n + k) * (n + k) + n + k + m + l) for k, l in kl]
                elif op == "m2m":  # M_n^m = sum_{k <= n} M_k^l R_{n-k}^{m-l}(-r)
                    kl = [(k, l) for k in range(n + 1) for l in range(-k, k + 1) if abs(m - l) <= n - k]
                    h = [((n - k) * (n - k) + n - k + m - l) for k, l in kl]
                else:              # L_n^m = sum_{k >= n} L_k^l conj(R_{k-n}^{l-m})
                    kl = [(k, l) for k in range(n, P) for l in range(-k, k + 1) if abs(l - m) <= k - n]
                    h = [((k - n) * (k - n) + k - n + l - m) for k, l in kl]
                c = C[torch.tensor([k * k + k + l for k, l in kl], device=C.device)]
                g = H[torch.tensor(h, device=C.device)]
                if op == "m2l":
                    v = (c.conj() * g).sum(0) * (-1) ** n
                elif op == "m2m":
                    v = (c * g).sum(0)
                else:
                    v = (c * g.conj()).sum(0)
                re[n, m], im[n, m] = v.real, (v.imag if m else torch.zeros_like(v.real))
        out[b:b + step] = _join_rows(P, re, im).t()
    return out


# ---- inputs ----

def _gen(seed, salt):
    g = torch.Generator(device=DEV)
    g.manual_seed(1_000_003 * int(seed) + salt)
    return g


def _rand(g, *shape):
    return torch.rand(*shape, dtype=torch.float64, device=DEV, generator=g)


def _directions(g, n):
    u = torch.randn(n, 3, dtype=torch.float64, device=DEV, generator=g)
    return u / u.norm(dim=1, keepdim=True)


def _ball(g, n, radius):
    return _directions(g, n) * radius * _rand(g, n, 1) ** (1.0 / 3.0)


def _expansions(g, P, n, local, charges=4):
    """n expansions (n, P(P+1)) of a few unit charges of random sign each, FP64."""
    centre = _directions(g, n) * (2 + 2 * _rand(g, n, 1)) if local else torch.zeros(n, 3, dtype=torch.float64, device=DEV)
    out = None
    for _ in range(charges):
        pos = centre + _ball(g, n, 0.5)
        q = torch.randint(0, 2, (n,), device=DEV, generator=g).to(torch.float64) * 2 - 1
        re, im = _columns(P, *(pos[:, k].contiguous() for k in range(3)), local)
        rows = _join_rows(P, re, im) * q
        out = rows if out is None else out.add_(rows)
    return out.t().contiguous()


def _shifts(g, op, n):
    if op == "m2l":
        return (_directions(g, n) * (2 + 2 * _rand(g, n, 1))).contiguous()
    return 0.5 * (torch.randint(0, 2, (n, 3), device=DEV, generator=g).to(torch.float64) * 2 - 1)


def _batch(case, seed):
    """Sources, shifts and index arrays of a device or host batch.  share = 8: eight translations per source
    (M2L, L2L) or per target (M2M, which accumulates with atomics), listed side by side; share = 1: all distinct."""
    n, P, op, share = case["n"], case["p"], case["op"], case.get("share", 1)
    g = _gen(seed, 11)
    few = (n + share - 1) // share
    ns = n if op == "m2m" else few
    nt = few if op == "m2m" else n
    src = _expansions(g, P, ns, op == "l2l")
    if case["dtype"] == "f32":
        src = src.to(torch.float32)
    i = torch.arange(n, device=DEV)
    near = (i // share).to(torch.int32)
    return {"src": src, "shift": _shifts(g, op, n), "nt": nt,
            "sidx": near if share > 1 and op != "m2m" else None, "tidx": near if share > 1 and op == "m2m" else None}


def _mixed(case, seed):
    """The stages of a mixed-order workload: 40% M2L, 30% M2M, 30% L2L; orders drawn independently per translation,
    sources gathered from a pool, distinct targets."""
    g = _gen(seed, 23)
    n, lo, hi = case["n"], case["p_lo"], case["p_hi"]
    stages = []
    for op, part in (("m2l", 0.4), ("m2m", 0.3), ("l2l", 0.3)):
        m = max(1, int(n * part))
        pool = max(1, m // 4)
        stages.append({"op": op, "n": m, "pool": _expansions(g, hi, pool, op == "l2l"),
                       "sidx": torch.randint(0, pool, (m,), device=DEV, generator=g).to(torch.int32),
                       "pin": torch.randint(lo, hi + 1, (m,), device=DEV, generator=g).to(torch.int32),
                       "pout": torch.randint(lo, hi + 1, (m,), device=DEV, generator=g).to(torch.int32),
                       "shift": _shifts(g, op, m)})
    return stages


def _leaves(case, seed):
    """Leaf centres, ragged leaf ranges and particles around them (P2M, L2P: inside a cube of side 1/32; P2L and
    M2P: at a distance of 2 to 4 leaf sides)."""
    g = _gen(seed, 37)
    per = case["per_leaf"]
    if case["kind"] == "eval":
        nleaf = max(1, case["n"] // per)
        leaf = torch.sort(torch.randint(0, nleaf, (case["n"],), device=DEV, generator=g))[0]
        counts = torch.bincount(leaf, minlength=nleaf)
    else:
        nleaf = case["n"]
        counts = torch.randint(0, 2 * per + 1, (nleaf,), device=DEV, generator=g)
        leaf = torch.repeat_interleave(torch.arange(nleaf, device=DEV), counts)
    k = leaf.numel()
    side = 1.0 / 32
    centre = _rand(g, nleaf, 3)
    if case["order"] in ("p2m", "l2p"):
        off = (_rand(g, k, 3) - 0.5) * side
    else:
        off = _directions(g, k) * (2 + 2 * _rand(g, k, 1)) * side
    offsets = torch.zeros(nleaf + 1, dtype=torch.int64, device=DEV)
    offsets[1:] = torch.cumsum(counts, 0)
    return {"nleaf": nleaf, "leaf": leaf, "centre": centre, "pos": (centre[leaf] + off).contiguous(),
            "charge": _rand(g, k) * 2 - 1, "offsets": offsets.to(torch.int32)}


def _leaf_expansions(case, seed, nleaf):
    """Expansions at leaf scale: locals of charges 2 to 4 leaf sides away, multipoles of charges inside the leaf."""
    g = _gen(seed, 41)
    P, side = case["p"], 1.0 / 32
    local = case["order"] == "l2p"
    out = None
    for _ in range(4):
        d = _directions(g, nleaf) * (2 + 2 * _rand(g, nleaf, 1)) * side if local else (_rand(g, nleaf, 3) - 0.5) * side
        q = _rand(g, nleaf) * 2 - 1
        rows = _join_rows(P, *_columns(P, *(d[:, k].contiguous() for k in range(3)), local)) * q
        out = rows if out is None else out.add_(rows)
    return out.t().contiguous()


def _coords(level):
    """(i, j, k) of the boxes of an octree level, box (i 2^l + j) 2^l + k."""
    i = torch.arange(8 ** level, device=DEV)
    return torch.stack((i // 4 ** level, i // 2 ** level % 2 ** level, i % 2 ** level), 1)


def _particles(case, seed):
    """per_leaf uniform particles in every leaf of the octree, charges in [-1, 1] (leaf by leaf)."""
    g = _gen(seed, 53)
    nleaf = 8 ** case["depth"]
    corner = _coords(case["depth"]).to(torch.float64) / 2 ** case["depth"]
    pos = corner[:, None, :] + _rand(g, nleaf, case["per_leaf"], 3) / 2 ** case["depth"]
    return _rand(g, nleaf, case["per_leaf"]) * 2 - 1, pos.contiguous()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "device":
        b = _batch(case, seed)
        P, n = case["p"], case["n"]
        order = torch.full((n,), P, dtype=torch.int32, device=DEV)
        dst = torch.zeros(b["nt"], P * (P + 1), dtype=b["src"].dtype, device=DEV)
        return {"case": case, "ctx": sf.Context(P, case["dtype"]), "order": order, "dst": dst, **b}
    if kind == "host":
        b = _batch(case, seed)
        P, n = case["p"], case["n"]
        order = np.full(n, P, np.uint32)
        return {"case": case, "ctx": sf.Context(P, case["dtype"]), "order": order, "src": b["src"].cpu().pin_memory(),
                "dst": torch.zeros(n, P * (P + 1), dtype=b["src"].dtype).pin_memory(), "shift": b["shift"].cpu().numpy()}
    if kind == "plan":
        ctx = sf.Context(case["p_hi"], "f64")
        S = case["p_hi"] * (case["p_hi"] + 1)
        plan, stages = sf.Plan(ctx), _mixed(case, seed)
        for s in stages:
            s["dst"] = torch.zeros(s["n"], S, dtype=torch.float64, device=DEV)
            plan.add(s["op"], PRECISION[case["precision"]], s["n"], s["pool"], S, s["pool"].shape[0], s["dst"], S, s["n"],
                     s["pin"], s["pout"], s["shift"], src_index=s["sidx"])
        return {"case": case, "ctx": ctx, "plan": plan.finalize(), "stages": stages}
    if kind == "fmm":
        ctx = sf.Context(case["p"], "f64")
        fmm = sf_fmm.UniformFMM(ctx, case["depth"], PRECISION[case["precision"]], DEV)
        charge, pos = _particles(case, seed)
        return {"case": case, "ctx": ctx, "fmm": fmm, "charge": charge, "pos": pos}
    t = _leaves(case, seed)
    t.update(case=case, ctx=sf.Context(case["p"], "f64"))
    if kind == "p2x":
        t["out"] = torch.zeros(t["nleaf"], case["p"] * (case["p"] + 1), dtype=torch.float64, device=DEV)
        return t
    t["E"] = _leaf_expansions(case, seed, t["nleaf"])
    t["box"] = t["leaf"].to(torch.int32)
    t["pot"] = torch.zeros(case["n"], dtype=torch.float64, device=DEV)
    t["grad"] = torch.zeros(case["n"], 3, dtype=torch.float64, device=DEV) if case["gradient"] else None
    return t


def run(state):
    case, ctx = state["case"], state["ctx"]
    kind = case["kind"]
    if kind == "device":
        src, dst = state["src"], state["dst"]
        ctx.translate_device(case["op"], PRECISION[case["precision"]], case["n"], src, src.shape[1], src.shape[0], dst,
                             dst.shape[1], dst.shape[0], state["order"], state["order"], state["shift"],
                             src_index=state["sidx"], dst_index=state["tidx"], repeat=state["tidx"] is not None)
        return dst
    if kind == "host":
        ctx.translate_host_packed(case["op"], PRECISION[case["precision"]], state["src"], state["dst"], state["order"],
                                  state["order"], state["shift"])
        return state["dst"]
    if kind == "plan":
        state["plan"].run()
        return [s["dst"] for s in state["stages"]]
    if kind == "fmm":
        state["fmm"].run(state["charge"], state["pos"])
        return {"M": state["fmm"].M, "L": state["fmm"].L}
    if kind == "p2x":
        ctx.p2x_ragged(0 if case["order"] == "p2m" else 1, state["nleaf"], state["offsets"], state["charge"], state["pos"],
                       state["centre"], state["out"], state["out"].shape[1])
        return state["out"]
    ctx.evaluate(0 if case["order"] == "l2p" else 1, case["n"], state["pos"], state["E"], state["E"].shape[1],
                 state["nleaf"], state["centre"], state["pot"], gradient=state["grad"], box=state["box"])
    return [state["pot"], state["grad"]] if case["gradient"] else [state["pot"]]


# ---- the work a pass cannot do without ----

def _translation_flops(p_in, p_out):
    """Two rotations of the source and of the result and the z-translation, multiply-adds as two operations."""
    rot = sum(2 * (n + 1) ** 2 for n in range(p_in)) + sum(2 * (n + 1) ** 2 for n in range(p_out))
    zt = sum(4 * (p_in - m) * (p_out - m) for m in range(min(p_in, p_out)))
    return 2.0 * rot + zt + 8 * (p_in * (p_in + 1) + p_out * (p_out + 1))


def work(case):
    kind = case["kind"]
    if kind in ("device", "host"):
        P, n, share = case["p"], case["n"], case.get("share", 1)
        S = P * (P + 1) * (4 if case["dtype"] == "f32" else 8)
        few = (n + share - 1) // share
        ns, nt = (n, few) if case["op"] == "m2m" else (few, n)
        return {"bytes": float(ns * S + 2 * nt * S + n * (24 + 8)), "flops": n * _translation_flops(P, P)}
    if kind == "plan":
        p = range(case["p_lo"], case["p_hi"] + 1)
        S = sum(q * (q + 1) for q in p) / len(p) * 8
        f = sum(_translation_flops(a, b) for a in p for b in p) / len(p) ** 2
        pool = case["n"] / 4
        return {"bytes": float(pool * case["p_hi"] * (case["p_hi"] + 1) * 8 + case["n"] * (2 * S + 24 + 12)),
                "flops": case["n"] * f}
    if kind == "fmm":
        P, depth = case["p"], case["depth"]
        boxes = sum(8 ** l for l in range(2, depth + 1))
        pairs = 0
        for l in range(2, depth + 1):  # interaction pairs: per axis (all, near) counts over the 2^l positions
            every = sum(min(2 ** l, 2 * (i // 2) + 4) - max(0, 2 * (i // 2) - 2) for i in range(2 ** l))
            near = sum(min(2 ** l, i + 2) - max(0, i - 1) for i in range(2 ** l))
            pairs += every ** 3 - near ** 3
        n = pairs + 2 * (boxes - 64)
        particles = 8 ** depth * case["per_leaf"]
        return {"bytes": float(boxes * P * (P + 1) * 8 * 2 + particles * 32),
                "flops": n * _translation_flops(P, P) + particles * P * (P + 1) * 6.0}
    P = case["p"]
    S = P * (P + 1)
    if kind == "p2x":
        k = case["n"] * case["per_leaf"]
        return {"bytes": float(k * 32 + case["n"] * (2 * S * 8 + 28)), "flops": k * S * 6.0}
    nleaf = max(1, case["n"] // case["per_leaf"])
    outs = 4 if case["gradient"] else 1
    return {"bytes": float(nleaf * S * 8 + case["n"] * (28 + 16 * outs)), "flops": case["n"] * S * (6.0 + 2 * outs)}


# ---- the same results in FP64 from the defining formulas ----

def _mask(P, p):
    """(N, P(P+1)) mask of the coefficients of degree below p[i]."""
    degree = torch.tensor([n for n in range(P) for _ in range(2 * (n + 1))], device=DEV)
    return degree[None, :] < p[:, None]


def _exact_fmm(case, seed):
    P, depth = case["p"], case["depth"]
    S = P * (P + 1)
    charge, pos = _particles(case, seed)
    off = [(8 ** l - 1) // 7 for l in range(depth + 2)]  # first box of every level
    M = torch.zeros(off[-1], S, dtype=torch.float64, device=DEV)
    L = torch.zeros_like(M)

    def index(c, l):
        return (c[:, 0] * 2 ** l + c[:, 1]) * 2 ** l + c[:, 2]

    def matrices(op, shifts):  # (K, S, S): row = input coefficient
        K = shifts.shape[0]
        eye = torch.eye(S, dtype=torch.float64, device=DEV)
        for n in range(P):
            eye[(n + 1) * (n + 1)] = 0  # the imaginary part at m = 0 is zero in every expansion
        return _translate(op, P, eye.repeat(K, 1), shifts.repeat_interleave(S, 0)).view(K, S, S)

    centre = (_coords(depth).to(torch.float64) + 0.5) / 2 ** depth
    for j in range(case["per_leaf"]):
        d = pos[:, j] - centre
        rows = _join_rows(P, *_columns(P, *(d[:, k].contiguous() for k in range(3)), False))
        M[off[depth]:] += (rows * charge[:, j]).t()
    octants = torch.tensor([[i, j, k] for i in (0, 1) for j in (0, 1) for k in (0, 1)], device=DEV)
    for l in range(depth, 2, -1):
        c = _coords(l)
        T = matrices("m2m", (0.5 - octants.to(torch.float64)) / 2 ** l)
        for o in range(8):
            at = torch.nonzero((c % 2 == octants[o]).all(1))[:, 0]
            M[off[l - 1] + index(c[at] // 2, l - 1)] += M[off[l] + at] @ T[o]
    r = torch.arange(-3, 4, device=DEV)
    offsets = torch.stack(torch.meshgrid(r, r, r, indexing="ij"), -1).reshape(-1, 3)
    offsets = offsets[offsets.abs().amax(1) >= 2]
    for l in range(2, depth + 1):
        c = _coords(l)
        T = matrices("m2l", -offsets.to(torch.float64) / 2 ** l)
        for o in range(offsets.shape[0]):
            s = c + offsets[o]
            ok = ((s >= 0) & (s < 2 ** l)).all(1) & (((s // 2) - (c // 2)).abs().amax(1) <= 1)
            at = torch.nonzero(ok)[:, 0]
            if at.numel():
                L[off[l] + at] += M[off[l] + index(s[at], l)] @ T[o]
    for l in range(3, depth + 1):
        c = _coords(l)
        T = matrices("l2l", (octants.to(torch.float64) - 0.5) / 2 ** l)
        for o in range(8):
            at = torch.nonzero((c % 2 == octants[o]).all(1))[:, 0]
            L[off[l] + at] += L[off[l - 1] + index(c[at] // 2, l - 1)] @ T[o]
    return {"M": M, "L": L}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("device", "host"):
        b = _batch(case, seed)
        src = b["src"].to(torch.float64)
        if b["sidx"] is not None:
            src = src[b["sidx"].long()]
        out = _translate(case["op"], case["p"], src, b["shift"])
        if b["tidx"] is not None:
            out = torch.zeros(b["nt"], out.shape[1], dtype=out.dtype, device=DEV).index_add_(0, b["tidx"].long(), out)
        return out
    if kind == "plan":
        P = case["p_hi"]
        return [_translate(s["op"], P, s["pool"][s["sidx"].long()] * _mask(P, s["pin"]), s["shift"]) * _mask(P, s["pout"])
                for s in _mixed(case, seed)]
    if kind == "fmm":
        return _exact_fmm(case, seed)
    t = _leaves(case, seed)
    P, leaf = case["p"], t["leaf"]
    singular = case["order"] in ("p2l", "m2p")
    d = t["pos"] - t["centre"][leaf]
    if kind == "p2x":
        out = torch.zeros(t["nleaf"], P * (P + 1), dtype=torch.float64, device=DEV)
        for b in range(0, leaf.numel(), 200_000):
            s = slice(b, b + 200_000)
            re, im = _columns(P, *(d[s, k].contiguous() for k in range(3)), singular)
            out.index_add_(0, leaf[s], (_join_rows(P, re, im) * t["charge"][s]).t())
        return out
    E = _leaf_expansions(case, seed, t["nleaf"])
    pot = torch.zeros(case["n"], dtype=torch.float64, device=DEV)
    grad = torch.zeros(case["n"], 3, dtype=torch.float64, device=DEV)
    for b in range(0, case["n"], 200_000):
        s = slice(b, b + 200_000)
        H = _full(P, *_columns(P, *(d[s, k].contiguous() for k in range(3)), singular))
        er, ei = _split_rows(P, E[leaf[s]].t())
        for n in range(P):
            for m in range(n + 1):
                w = 2.0 if m else 1.0
                c = torch.complex(er[n, m], -ei[n, m]) * w
                pot[s] += (c * H[n * n + n + m]).real
                if case["gradient"] and n > 0:
                    def low(k):
                        return H[(n - 1) * (n - 1) + n - 1 + k] if abs(k) <= n - 1 else torch.zeros_like(c)
                    # d/dx - i d/dy lowers m, d/dx + i d/dy raises it with the other sign, d/dz keeps it
                    grad[s, 0] += (c * (low(m - 1) - low(m + 1))).real * 0.5
                    grad[s, 1] += (c * 1j * (low(m - 1) + low(m + 1))).real * 0.5
                    grad[s, 2] += (c * low(m)).real
    return [pot, grad] if case["gradient"] else [pot]
