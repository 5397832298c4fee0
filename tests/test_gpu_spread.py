"""Global and Saigo-Vert alignments run in the scaled linear domain and leave
pairs whose values spread too far for it to the log-domain kernels.  Ordinary
pairs against the fp64 oracle; pairs with extreme scores (a clamped score, a
steep ridge, a very low temperature) must give the log-domain call's own bits,
alone and beside ordinary pairs, padded, packed and value-only."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

FAMILIES = {"nw": (("gap",), (-1.0,)), "nw_affine": (("gap_open", "gap_ext"), (-2.0, -0.5)),
            "sv_affine": (("gap_open", "gap_ext"), (-2.0, -0.5))}
PLAN = {"nw": "global", "nw_affine": "global_affine", "sv_affine": "saigo_vert"}


def _run(fam, s, lens, gaps, T, domain=0):
    from orihime_b200 import _lib, _ops

    opt = _lib.Options(domain=domain) if domain else None
    if fam == "nw":
        return _ops.run_linear(s, lens, *gaps, T, options=opt, family="nw")
    return _ops.run_affine(s, lens, *gaps, T, options=opt, family=fam)


def _scores(B, L1, L2, seed, scale=1.5):
    g = torch.Generator().manual_seed(seed)
    return torch.randn(B, L1, L2, generator=g) * scale


@pytest.mark.parametrize("fam", list(FAMILIES))
@pytest.mark.parametrize("shape", [(1, 1), (3, 5), (31, 33), (36, 129), (130, 66), (257, 260)])
def test_ordinary_pairs_against_oracle(fam, shape):
    from oracle import oracle as O

    L1, L2 = shape
    names, gaps = FAMILIES[fam]
    s = _scores(3, L1, L2, L1 * 7 + L2)
    lens = np.array([[L1, L2], [max(L1 - 1, 1), L2], [L1, max(L2 - 2, 1)]], dtype=np.int32)
    v, m, *grads = _run(fam, s.cuda(), torch.from_numpy(lens).cuda(), gaps, 0.7)
    f = {"nw": O.nw, "nw_affine": O.nw_affine, "sv_affine": O.sv}[fam]
    r32, r64 = (f(s.numpy(), lens, *gaps, 0.7, dtype=d) for d in (np.float32, np.float64))
    assert np.abs(v.cpu().numpy() - r64["value"]).max() <= 1e-5 * max(1.0, np.abs(r64["value"]).max())
    err, ref = (np.abs(x - r64["map"]).max() for x in (m.cpu().numpy(), r32["map"]))
    assert err <= max(1e-5, ref)
    keys = [k for k in r64 if k.startswith("grad")]
    for g, k in zip(grads, keys):
        d, ref = np.abs(g.cpu().numpy() - r64[k]).max(), np.abs(r32[k] - r64[k]).max()
        assert d <= max(1e-4 * max(1.0, np.abs(r64[k]).max()), ref), k


@pytest.mark.parametrize("fam", list(FAMILIES))
@pytest.mark.parametrize("kind", ["clamped", "ridge", "cold"])
def test_extreme_pairs_give_the_log_domain_bits(fam, kind):
    from orihime_b200 import _lib, _ops, ragged

    names, gaps = FAMILIES[fam]
    T = 0.03 if kind == "cold" else 0.7
    s = _scores(4, 140, 150, 5)
    if kind == "clamped":
        s[1, 70, 71] = 90.0
    elif kind == "ridge":   # six matches of 2^80 each beside cells that only gaps reach
        for q in range(6):
            s[1, 60 + q, 64 + q] = 39.0
    rows = [1] if kind != "cold" else [0, 1, 2, 3]
    x = s.cuda()
    got = _run(fam, x, None, gaps, T)
    log = _run(fam, x, None, gaps, T, domain=_lib.DOMAIN_LOG)
    for b in rows:
        for g, w in zip(got, log):
            assert torch.equal(g[b], w[b])
    one = _run(fam, x[rows[0]:rows[0] + 1].contiguous(), None, gaps, T)
    assert torch.equal(one[1][0], log[1][rows[0]])
    val = _ops.run_value(fam, x, None, (*gaps, T))
    assert torch.equal(val, got[0])
    flat, off, ln = ragged.pack(list(s))
    plan = ragged.Plan(ln, off, family=PLAN[fam], device="cuda")
    out = plan.run(flat.cuda(), temp=T, **dict(zip(names, gaps)))
    assert plan.status() == 0
    assert torch.equal(out.value, got[0])
    maps = ragged.unpack(out.map, off, ln)
    for b in range(4):
        assert torch.equal(maps[b], got[1][b])
