"""Timed cases: what programs built on this package ask of it.

Each case is one call (or one forward + backward) through the public entry
points.  Scores come from the benchmark's generator, 3 <e, f> / sqrt(64) with
e, f ~ N(0, 1) in 64 dimensions, at the temperatures its configurations use;
shapes are those of the benchmark, of the tests' rectangular grid, or odd
relatives of them.

kind          what a pass is
value         the value under no_grad: scoring, the smallest call
map           the marginal map under no_grad: inference
train         value and backward into the scores and the learnable parameters
entropy       -value.mean() + 0.01 entropy.mean() and backward into the scores
map_train     the map and backward of a cotangent through it (second order)
plan          forward + adjoint of a packed ragged batch on a kept plan
"""

import math

import numpy as np
import torch
import torch.nn.functional as F

import orihime_b200 as ohm
from orihime_b200 import ragged

AFFINE = ("sw_affine", "nw_affine", "sv_affine")
PLAN_FAMILY = {"sw_affine": "affine", "sw": "linear", "nw": "global", "nw_affine": "global_affine",
               "sv_affine": "saigo_vert"}
D = 64   # embedding dimensions of the score generator


def _case(kind, family, B, L1, L2, T=0.5, ragged_lengths=False, band=0, name=None):
    c = {"kind": kind, "family": family, "B": B, "L1": L1, "L2": L2, "T": T,
         "go": -2.0 if family in AFFINE else -1.0, "ge": -0.5,
         "lengths": ragged_lengths, "band": band}
    if name:
        c["name"] = name
    return c


def _plan_case(family, pairs, lo, hi, seed, cols=0, T=0.5, name=None):
    c = {"kind": "plan", "family": family, "B": pairs, "L1": hi, "L2": hi, "lo": lo, "T": T,
         "go": -2.0 if family in AFFINE else -1.0, "ge": -0.5, "lengths_seed": seed, "cols": cols}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # one short pair scored: launches, the input scan and host work are the time
        _case("value", "sw_affine", 1, 64, 64, name="sw_affine_value_1x64x64"),
        # the plain small batch: the map of eight 128 x 128 pairs, linear gaps
        _case("map", "sw", 8, 128, 128, T=1.0, name="sw_map_8x128x128"),
        # one long pair of odd size (rows not 16-byte aligned): the wavefront's latency
        _case("map", "sw_affine", 1, 1023, 2047, name="sw_affine_map_1x1023x2047"),
        # a training step of the alignment layer with learnable gaps and temperature
        _case("train", "sw_affine", 64, 1024, 1024, name="sw_affine_train_64x1024x1024"),
        # long sequences under a band mask, forward and checkpointed backward
        _case("train", "sw_affine", 4, 8192, 8192, band=1024, name="sw_affine_banded_4x8192x8192"),
        # thousands of pairs of uneven lengths in one packed launch: the benchmark's batch
        _plan_case("sw_affine", 4096, 32, 2048, 3, cols=8, T=1.0, name="sw_affine_plan_4096"),
        # the end-to-end layer's loss: value and entropy, backward into the scores
        _case("entropy", "sw_affine", 256, 512, 512, name="sw_affine_entropy_256x512x512"),
        # a loss on the alignment map itself: forward, adjoint and a Hessian-vector product
        _case("map_train", "sw_affine", 48, 500, 384, name="sw_affine_map_train_48x500x384"),
        # global alignment trained on a padded batch with per-pair lengths
        _case("train", "nw", 64, 512, 512, ragged_lengths=True, name="nw_train_64x512x512_lengths"),
        # a loss on the global alignment map, affine gaps
        _case("map_train", "nw_affine", 16, 512, 384, name="nw_affine_map_train_16x512x384"),
        # Saigo-Vert maps of mid-sized pairs of odd width
        _case("map", "sv_affine", 8, 1000, 701, T=1.0, name="sv_affine_map_8x1000x701"),
        # a packed ragged batch of global alignments
        _plan_case("nw_affine", 1024, 32, 1024, 5, name="nw_affine_plan_1024"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["value", "map", "train", "entropy", "map_train", "plan"])
    T = rng.choice([0.5, 1.0])
    if kind == "plan":
        fam = rng.choice(["sw", "sw_affine", "nw", "nw_affine", "sv_affine"])
        return _plan_case(fam, _log_int(rng, 256, 2048), 32, _log_int(rng, 300, 1500), rng.randrange(1000), T=T)
    fam = rng.choice(["sw", "sw_affine", "nw", "nw_affine", "sv_affine"])
    if kind == "entropy":
        fam = rng.choice(["sw", "sw_affine"])
    L1, L2 = _log_int(rng, 64, 2048), _log_int(rng, 64, 2048)
    most = 16e6 if kind in ("map_train", "entropy") else 64e6   # cells of one padded batch
    B = _log_int(rng, 1, max(1, min(128, int(most / (L1 * L2)))))
    return _case(kind, fam, B, L1, L2, T=T, ragged_lengths=rng.random() < 0.3)


def _plan_lengths(case):
    r = np.random.default_rng(case["lengths_seed"])
    ln = np.exp(r.uniform(math.log(case["lo"]), math.log(case["L1"]), size=(case["B"], 2)))
    return np.rint(ln).astype(np.int64)


def _batch_lengths(case, seed):
    if not case["lengths"]:
        return None
    r = np.random.default_rng(seed)
    top = np.array([case["L1"], case["L2"]])
    ln = np.rint(top * r.uniform(0.4, 1.0, size=(case["B"], 2))).astype(np.int32)
    ln[0] = top
    return torch.from_numpy(ln)


def _inputs(case, seed):
    """Scores (padded batch or packed buffer), lengths, mask and cotangent."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 11)
    if case["kind"] == "plan":
        ln = _plan_lengths(case)
        offsets, ln32 = ragged.layout(ln)
        e = torch.randn(int(ln[:, 0].sum()), D, generator=g, device="cuda")
        f = torch.randn(int(ln[:, 1].sum()), D, generator=g, device="cuda") * (3.0 / D ** 0.5)
        flat = torch.zeros(int(offsets[-1]), device="cuda")
        i = j = 0
        for b, (n, m) in enumerate(ln.tolist()):
            p = ragged.pitch_of(m)
            view = flat[int(offsets[b]):int(offsets[b]) + n * p].view(n, p)
            view[:, :m] = e[i:i + n] @ f[j:j + m].T
            i, j = i + n, j + m
        return {"x": flat, "offsets": offsets, "lengths": ln32}
    B, L1, L2 = case["B"], case["L1"], case["L2"]
    e = torch.randn(B, L1, D, generator=g, device="cuda")
    f = torch.randn(B, L2, D, generator=g, device="cuda") * (3.0 / D ** 0.5)
    s = {"x": torch.bmm(e, f.transpose(1, 2)), "lengths": _batch_lengths(case, seed), "mask": None}
    if s["lengths"] is not None:
        s["lengths"] = s["lengths"].cuda()
    if case["band"]:
        i, j = torch.arange(L1, device="cuda"), torch.arange(L2, device="cuda")
        s["mask"] = ((i[:, None] - j[None, :]).abs() > case["band"]).expand(B, L1, L2).contiguous()
    if case["kind"] == "map_train":
        s["cot"] = torch.randn(B, L1, L2, generator=g, device="cuda")
    return s


def prepare(case, seed):
    s = _inputs(case, seed)
    affine = case["family"] in AFFINE
    if case["kind"] == "plan":
        plan = ragged.Plan(s["lengths"], s["offsets"], family=PLAN_FAMILY[case["family"]], device="cuda",
                           cols_per_lane=case["cols"])
        kw = {"gap_open": case["go"], "gap_ext": case["ge"]} if affine else {"gap": case["go"]}
        return {"kind": "plan", "plan": plan, "x": s["x"], "out": plan.outputs(), "kw": {**kw, "temp": case["T"]}}
    names = (("gap_open_score", case["go"]), ("gap_extend_score", case["ge"])) if affine else (("gap_score", case["go"]),)
    kw = dict(names + (("temperature", case["T"]),))
    learn = []
    if case["kind"] == "train" and not case["band"]:
        kw = {k: torch.tensor(v, device="cuda", requires_grad=True) for k, v in kw.items()}
        learn = list(kw.values())
    if case["kind"] not in ("value", "map"):
        s["x"].requires_grad_(True)
    opt = {"lengths": s["lengths"], "mask": s["mask"]}
    base = case["family"]
    fns = {"map": getattr(ohm, base), "value": getattr(ohm, base + "_value"), "entropy": getattr(ohm, base + "_entropy")}
    return {"kind": case["kind"], "x": s["x"], "cot": s.get("cot"), "kw": {**kw, **opt}, "learn": learn, "fns": fns}


def run(state):
    kind, x, kw = state["kind"], state["x"], state["kw"]
    if kind == "plan":
        r = state["plan"].run(x, out=state["out"], **kw)
        out = {"value": r.value, "map": r.map, "grad_open": r.grad_open, "grad_temp": r.grad_temp}
        if r.grad_ext is not None:
            out["grad_ext"] = r.grad_ext
        return out
    fns = state["fns"]
    if kind in ("value", "map"):
        with torch.no_grad():
            return {kind: fns[kind](x, **kw)}
    if kind == "train":
        v = fns["value"](x, **kw)
        gx, *gp = torch.autograd.grad(-v.mean(), [x] + state["learn"])
        return {"value": v.detach(), "grad_x": gx, "grad_params": list(gp)}
    if kind == "entropy":
        v, h = fns["value"](x, **kw), fns["entropy"](x, **kw)
        (gx,) = torch.autograd.grad(-v.mean() + 0.01 * h.mean(), [x])
        return {"value": v.detach(), "entropy": h.detach(), "grad_x": gx}
    p = fns["map"](x, **kw)
    (gx,) = torch.autograd.grad(p, [x], state["cot"])
    return {"map": p.detach(), "grad_x": gx}


def work(case):
    """Bytes: the scores read once (and the mask or cotangent), every output
    written once.  Flops: the multiply-adds of the recurrence and of its
    adjoint (second order: of their tangents too) per cell."""
    if case["kind"] == "plan":
        cells = int((_plan_lengths(case)[:, 0] * _plan_lengths(case)[:, 1]).sum())
    elif case["lengths"]:
        cells = int(0.49 * case["B"] * case["L1"] * case["L2"])
    else:
        cells = case["B"] * case["L1"] * case["L2"]
    affine = case["family"] in AFFINE
    fwd, adj = (14, 20) if affine else (7, 10)
    n_bytes = {"value": 4, "map": 8, "train": 8 + (1 if case.get("band") else 0), "entropy": 8, "map_train": 16,
               "plan": 8}[case["kind"]]
    flops = {"value": fwd, "map": fwd + adj, "train": fwd + adj, "entropy": 3 * (fwd + adj),
             "map_train": 4 * (fwd + adj), "plan": fwd + adj}[case["kind"]]
    return {"bytes": n_bytes * cells, "flops": flops * cells}


# ---------------------------------------------------------------------------
# the same in 64 bits with plain torch: log-domain dynamic programming along
# anti-diagonals; derivatives of the map come from a complex step
# ---------------------------------------------------------------------------

STEP = 1e-30


NONE = -1e200   # the log of no path: finite, so that complex sums stay free of NaN


def _lse(terms):
    """Elementwise log-sum-exp of equally shaped tensors."""
    if len(terms) == 1:
        return terms[0]
    re = [t.real if t.is_complex() else t for t in terms]
    m = re[0]
    for t in re[1:]:
        m = torch.maximum(m, t)
    return m + torch.log(sum(torch.exp(t - m) for t in terms))


def _skew(x, fill):
    """[B, R, C] -> [R + C - 1, B, R]: element [d, b, i] is x[b, i, d - i]."""
    B, R, C = x.shape
    w = F.pad(x, (0, R), value=fill).reshape(B, R * (C + R))[:, :R * (R + C - 1)]
    return w.reshape(B, R, R + C - 1).permute(2, 0, 1).contiguous()


def _unskew(x, C):
    """The inverse of _skew."""
    n, B, R = x.shape
    w = F.pad(x.permute(1, 2, 0).reshape(B, R * n), (0, R))
    return w.reshape(B, R, n + 1)[:, :, :C]


class _Model:
    """One family: states, the states a match leaves from, gap arcs, ends."""

    def __init__(self, family, go, ge):
        self.linear = family in ("sw", "nw")
        self.local = not family.startswith("nw")
        if self.linear:
            self.states, self.up, self.left = "A", {"A": [("A", go)]}, {"A": [("A", go)]}
            self.ends = "A"
            return
        more = family != "sw_affine"   # D may follow I
        self.states = "MID"
        self.up = {"I": [("M", go), ("I", ge)] + ([("D", go)] if family == "nw_affine" else [])}
        self.left = {"D": [("M", go), ("D", ge)] + ([("I", go)] if more else [])}
        self.ends = "M" if family == "sv_affine" else "MID"


def _solve(model, x, lengths, counts=False):
    """(S [B] over T, map [B, L1, L2], {gap: expected count [B]}) of scores x
    already divided by T (float64 or complex128; NONE where masked)."""
    B, L1, L2 = x.shape
    dev = x.device
    real = torch.float64
    l1 = torch.full((B,), L1, device=dev) if lengths is None else lengths[:, 0].long()
    l2 = torch.full((B,), L2, device=dev) if lengths is None else lengths[:, 1].long()
    re = F.pad(x.real if x.is_complex() else x, (1, 0, 1, 0), value=NONE)   # row and column 0
    sk = _skew(re, NONE)
    if x.is_complex():
        sk = torch.complex(sk, _skew(F.pad(x.imag, (1, 0, 1, 0)), 0.0))
    del re
    n, R = L1 + L2 + 1, L1 + 1
    rows = torch.arange(R, device=dev)[None, :]
    row_ok = rows <= l1[:, None]
    if model.local:
        row_ok = row_ok & (rows >= 1)
    blank = torch.full((B, R), NONE, dtype=x.dtype, device=dev)

    def valid(d):
        j = d - rows
        return row_ok & (j >= (1 if model.local else 0)) & (j <= l2[:, None])

    def down(t):   # the row above: row i holds row i - 1's value
        return torch.cat([blank[:, :1], t[:, :-1]], 1)

    def rise(t):   # the row below
        return torch.cat([t[:, 1:], blank[:, :1]], 1)

    st = model.states
    alpha = {q: torch.empty((n, B, R), dtype=x.dtype, device=dev) for q in (st if counts or model.linear else st[:1])}
    match = torch.empty((n, B, R), dtype=x.dtype, device=dev) if model.linear else None
    p1, p2 = {q: blank for q in st}, {q: blank for q in st}
    zero = torch.zeros_like(blank)
    total = torch.zeros(B, dtype=x.dtype, device=dev) if model.local else None   # the empty alignment
    ends = torch.full((B,), NONE, dtype=x.dtype, device=dev)
    for d in range(n):
        ok = valid(d)
        prev = [down(p2[q]) for q in st] + ([zero] if model.local else [])
        m = sk[d] + _lse(prev)
        cur = {}
        for q in st:
            terms = [m] if q in "AM" else []
            terms += [down(p1[a]) + w for a, w in model.up.get(q, [])]
            terms += [p1[a] + w for a, w in model.left.get(q, [])]
            cur[q] = torch.where(ok, _lse(terms), blank)
        if d == 0 and not model.local:
            cur[st[0]][:, 0] = 0.0
        if match is not None:
            match[d] = torch.where(ok, m, blank)
        for q in alpha:
            alpha[q][d] = cur[q]
        if model.local:
            c = _lse([cur[q] for q in model.ends])
            rowmax = (c.real if c.is_complex() else c).max(1).values
            total = _lse([total, rowmax + torch.log(torch.exp(c - rowmax[:, None]).sum(1))])
        else:
            at = (l1 + l2 == d)
            v = _lse([cur[q] for q in model.ends]).gather(1, l1[:, None])[:, 0]
            ends = torch.where(at, v, ends)
        p2, p1 = p1, cur
    S = total if model.local else ends
    out = torch.zeros((n, B, R), dtype=x.dtype, device=dev)
    num = {}
    b1, b2 = {q: blank for q in st}, {q: blank for q in st}   # beta of diagonals d + 1, d + 2
    s2 = blank   # the match weights of diagonal d + 2
    for d in range(n - 1, -1, -1):
        ok = valid(d)
        stop = ok if model.local else ok & (rows == l1[:, None]) & (d - rows == l2[:, None])
        diag = rise(s2 + b2[st[0]])
        cur = {}
        for q in st:
            terms = [diag]
            if q in model.ends:
                terms.append(torch.where(stop, zero, blank))
            for to, arcs in model.up.items():
                terms += [rise(b1[to]) + w for a, w in arcs if a == q]
            for to, arcs in model.left.items():
                terms += [b1[to] + w for a, w in arcs if a == q]
            cur[q] = torch.where(ok, _lse(terms), blank)
            if counts:
                a0 = alpha[q][d] - S[:, None]
                for arcs, mv in ((model.up, rise), (model.left, lambda t: t)):
                    for to, lst in arcs.items():
                        for a, w in lst:
                            if a == q:
                                key = 0 if model.linear or a != to else 1
                                num[key] = num.get(key, 0.0) + torch.exp(a0 + mv(b1[to]) + w).sum(1)
        first = match[d] if model.linear else alpha["M"][d]
        out[d] = torch.exp(first + cur[st[0]] - S[:, None])
        s2, b2, b1 = (sk[d + 1] if d + 1 < n else blank), b1, cur
    return S, _unskew(out, L2 + 1)[:, 1:, 1:], num


def _with_grads(case, x, lengths):
    """value, map and dS/d(gaps..., T) in float64."""
    T, gaps = case["T"], [case["go"], case["ge"]][:2 if case["family"] in AFFINE else 1]
    S, P, num = _solve(_Model(case["family"], case["go"] / T, case["ge"] / T), x / T, lengths, counts=True)
    g = [num[k] for k in range(len(gaps))]
    sp = (torch.where(x > NONE, x, torch.zeros_like(x)) * P).sum((1, 2))
    return S * T, P, g, S - (sp + sum(c * v for c, v in zip(gaps, g))) / T


def exact(case, seed):
    s = _inputs(case, seed)
    T = case["T"]
    if case["kind"] == "plan":
        ln, off = s["lengths"].astype(np.int64), s["offsets"]
        B = len(ln)
        out = {"map": torch.zeros(int(off[-1]), dtype=torch.float64, device="cuda")}
        names = ["value", "grad_open"] + (["grad_ext"] if case["family"] in AFFINE else []) + ["grad_temp"]
        out.update({k: torch.zeros(B, dtype=torch.float64, device="cuda") for k in names})
        order = np.argsort(-(ln[:, 0] + ln[:, 1]), kind="stable")
        k = 0
        while k < B:   # pairs of like size together, within about 40 GB
            take = order[k:k + 512]
            n1, n2 = np.maximum.accumulate(ln[take, 0]), np.maximum.accumulate(ln[take, 1])
            fits = np.arange(1, len(take) + 1) * (n1 + 1) * (n1 + n2 + 1) * 8 * 6 <= 40e9
            take = take[:max(1, int(fits.sum()))]
            k += len(take)
            n1, n2 = int(ln[take, 0].max()), int(ln[take, 1].max())
            x = torch.full((len(take), n1, n2), NONE, dtype=torch.float64, device="cuda")
            for q, b in enumerate(take.tolist()):
                a, c = int(ln[b, 0]), int(ln[b, 1])
                p = ragged.pitch_of(c)
                x[q, :a, :c] = s["x"][int(off[b]):int(off[b]) + a * p].view(a, p)[:, :c].double()
            idx = torch.from_numpy(take).cuda()
            v, P, g, gT = _with_grads(case, x, torch.from_numpy(ln[take]).cuda())
            for key, t in zip(names, [v] + g + [gT]):
                out[key][idx] = t
            for q, b in enumerate(take.tolist()):
                a, c = int(ln[b, 0]), int(ln[b, 1])
                p = ragged.pitch_of(c)
                out["map"][int(off[b]):int(off[b]) + a * p].view(a, p)[:, :c] = P[q, :a, :c]
            del x, P
        return out
    x, lengths = s["x"].double(), s["lengths"]
    if s["mask"] is not None:
        x = x.masked_fill(s["mask"], NONE)
    B = case["B"]
    plain = _Model(case["family"], case["go"] / T, case["ge"] / T)
    if case["kind"] in ("value", "map"):
        S, P, _ = _solve(plain, x / T, lengths)
        return {"value": S * T} if case["kind"] == "value" else {"map": P}
    if case["kind"] == "train":
        v, P, g, gT = _with_grads(case, x, lengths)
        params = [] if case["band"] else [-t.mean() for t in g + [gT]]
        return {"value": v, "grad_x": -P / B, "grad_params": params}
    if case["kind"] == "entropy":
        t = complex(T, STEP)   # dS/dT and dP/dT from a complex step of the temperature
        S, P, _ = _solve(_Model(case["family"], case["go"] / t, case["ge"] / t), x.to(torch.complex128) / t, lengths)
        S = S * t
        return {"value": S.real, "entropy": S.imag / STEP, "grad_x": (-P.real + 0.01 * P.imag / STEP) / B}
    _, P, _ = _solve(plain, torch.complex(x / T, s["cot"].double() / T * STEP), lengths)
    return {"map": P.real, "grad_x": P.imag / STEP}
