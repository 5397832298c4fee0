"""A pair's result does not depend on the batch it is in: padded batches with
few and with many bands, their shards and a packed plan at the columns that
swb_cols_per_lane reports give the same bits, in every padded entry point."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("family", ["affine", "linear"])
@pytest.mark.parametrize("L1,L2,T", [(40, 300, 1.0), (33, 257, 0.25), (20, 64, 1.0)])
def test_large_batch_equals_its_shards_and_a_plan(family, L1, L2, T):
    from orihime_b200 import _lib, _ops, ragged

    B = 800
    g = torch.Generator().manual_seed(L2)
    s = (torch.bmm(torch.randn(B, L1, 64, generator=g), torch.randn(B, 64, L2, generator=g)) * 0.25).contiguous().cuda()
    affine = family == "affine"
    gaps = (-2.0, -0.5) if affine else (-1.0,)
    fam, run = ("sw_affine", _ops.run_affine) if affine else ("sw", _ops.run_linear)
    want = run(s, None, *gaps, T)
    for a, b in ((0, 3), (3, 300), (300, B)):
        for x, y in zip(run(s[a:b].contiguous(), None, *gaps, T), want):
            assert torch.equal(x, y[a:b])
    assert torch.equal(_ops.run_value(fam, s, None, (*gaps, T)), want[0])
    for every in (1, 4):
        got = _ops.run_checkpoint(fam, s, None, (*gaps, T), every)
        if got is None:
            assert T < 0.35
            continue
        for x, y in zip(_ops.run_adjoint(fam, s, None, (*gaps, T), every, got[1]), want):
            assert torch.equal(x, y)
    cols = _lib.load().swb_cols_per_lane(3 if affine else 1, L2, gaps[0], gaps[-1], T)
    flat, off, ln = ragged.pack(list(s.cpu()))
    plan = ragged.Plan(ln, off, family=family, device="cuda", cols_per_lane=cols)
    out = plan.run(flat.cuda(), temp=T, **(dict(gap_open=-2.0, gap_ext=-0.5) if affine else dict(gap=-1.0)))
    assert plan.status() == 0
    assert torch.equal(out.value, want[0]) and torch.equal(out.grad_temp, want[-1])
    maps = ragged.unpack(out.map, off, ln)
    for b in np.linspace(0, B - 1, 40, dtype=int).tolist():
        assert torch.equal(maps[b], want[1][b])
