"""Global alignments of pairs far from square at low temperature: the best path
of such a pair spends most of its steps in gaps, and in its rows lies many
hundreds of bits below other cells.  Packed, against the fp64 oracle: values to
1e-5 of their size (the fp32 outputs' rounding is 6e-8 of it), gradient sums to
1e-4 of theirs or the fp32 oracle's own error, whichever is larger."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

PAIRS = [(318, 38), (372, 32), (860, 35), (207, 40), (40, 300), (33, 700)]


@pytest.mark.parametrize("T", [0.25, 0.35])
@pytest.mark.parametrize("fam,gaps", [("nw", (-1.0,)), ("nw_affine", (-2.0, -0.5))])
def test_thin_pairs_keep_their_best_path(fam, gaps, T):
    from oracle import oracle as O
    from orihime_b200 import ragged

    g = torch.Generator().manual_seed(11)
    pairs = [torch.randn(*s, generator=g) * 1.5 for s in PAIRS]
    flat, off, ln = ragged.pack(pairs)
    plan = ragged.Plan(ln, off, family={"nw": "global", "nw_affine": "global_affine"}[fam], device="cuda")
    kw = {"nw": ("gap",), "nw_affine": ("gap_open", "gap_ext")}[fam]
    out = plan.run(flat.cuda(), temp=T, **dict(zip(kw, gaps)))
    assert plan.status() == 0
    f = {"nw": O.nw, "nw_affine": O.nw_affine}[fam]
    for b, s in enumerate(pairs):
        r32, r64 = (f(s[None].numpy(), None, *gaps, T, dtype=d) for d in (np.float32, np.float64))
        want = float(r64["value"][0])
        assert abs(float(out.value[b]) - want) <= 1e-5 * max(1.0, abs(want))
        want = float(r64["grad_temp"][0])
        ref = abs(float(r32["grad_temp"][0]) - want)
        assert abs(float(out.grad_temp[b]) - want) <= max(1e-4 * max(1.0, abs(want)), ref)


@pytest.mark.parametrize("T", [0.2, 0.25, 0.35])
@pytest.mark.parametrize("cols", [2, 4])
@pytest.mark.parametrize("fam,gaps", [("nw", (-1.0,)), ("nw_affine", (-2.0, -0.5)), ("sv", (-2.0, -0.5))])
def test_temperature_gradient_of_thin_pairs(fam, gaps, cols, T):
    """dS/dT, the small difference of two sums several hundred times its size, to
    1e-4 of its own size whatever the fp32 oracle's error is."""
    from oracle import oracle as O
    from orihime_b200 import ragged

    g = torch.Generator().manual_seed(11)
    pairs = [torch.randn(*s, generator=g) * 1.5 for s in PAIRS]
    flat, off, ln = ragged.pack(pairs)
    plan = ragged.Plan(ln, off, family={"nw": "global", "nw_affine": "global_affine", "sv": "saigo_vert"}[fam],
                       device="cuda", cols_per_lane=cols)
    out = plan.run(flat.cuda(), temp=T, **dict(zip(("gap",) if len(gaps) == 1 else ("gap_open", "gap_ext"), gaps)))
    assert plan.status() == 0
    for b, s in enumerate(pairs):
        want = float(getattr(O, fam)(s[None].numpy(), None, *gaps, T, dtype=np.float64)["grad_temp"][0])
        assert abs(float(out.grad_temp[b]) - want) <= 1e-4 * max(1.0, abs(want)), (b, want)
