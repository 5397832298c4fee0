"""Small padded batches (the outside sweep and the band segments) against the
adjoint of whole bands, which a packed plan of the same pairs runs: the same
bits, for pair sizes around the edges of lanes, bands, chunks and segments,
rows aligned to 16 bytes and not, and pairs shorter than the padded shape."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# (padded L1, padded L2, [per-pair lengths])
SHAPES = [
    (1, 65, [(1, 65), (1, 1), (0, 3), (1, 64)]),
    (33, 66, [(33, 66), (32, 65), (31, 2), (5, 66)]),
    (64, 64, [(64, 64), (63, 33), (16, 63), (17, 1)]),
    (131, 129, [(131, 129), (130, 128), (36, 127), (4, 5)]),
    (260, 300, [(260, 300), (257, 256), (33, 257), (128, 4)]),
    (97, 515, [(97, 515), (96, 512), (95, 385), (40, 511)]),
]


@pytest.mark.parametrize("family", ["affine", "linear"])
@pytest.mark.parametrize("shape", SHAPES, ids=[f"{a}x{b}" for a, b, _ in SHAPES])
def test_segments_equal_whole_bands(family, shape):
    from orihime_b200 import _lib, _ops, ragged

    L1, L2, ln = shape
    g = torch.Generator().manual_seed(L1 * 1000 + L2)
    e, f = torch.randn(len(ln), L1, 32, generator=g), torch.randn(len(ln), L2, 32, generator=g)
    s = (torch.bmm(e, f.transpose(1, 2)) * (3.0 / 32 ** 0.5)).contiguous()
    lens = torch.tensor(ln, dtype=torch.int32, device="cuda")
    if family == "affine":
        v, m, *grads = _ops.run_affine(s.cuda(), lens, -2.0, -0.5, 0.7)
        params, code = dict(gap_open=-2.0, gap_ext=-0.5, temp=0.7), 3
    else:
        v, m, *grads = _ops.run_linear(s.cuda(), lens, -1.0, 0.7)
        params, code = dict(gap=-1.0, temp=0.7), 1
    cols = _lib.load().swb_cols_per_lane(code, L2, -2.0, -0.5, 0.7)
    flat, off, lens32 = ragged.pack([s[b, :a, :c] for b, (a, c) in enumerate(ln)])
    plan = ragged.Plan(lens32, off, family=family, device="cuda", cols_per_lane=cols)
    out = plan.run(flat.cuda(), **params)
    assert plan.status() == 0
    assert torch.equal(v, out.value)
    want = [out.grad_open] + ([out.grad_ext] if family == "affine" else []) + [out.grad_temp]
    for a, b in zip(grads, want):
        assert torch.equal(a, b)
    for b, (pm, (a, c)) in enumerate(zip(ragged.unpack(out.map, off, lens32), ln)):
        assert torch.equal(m[b, :a, :c], pm)
        rest = m[b].clone()
        rest[:a, :c] = 0
        assert not np.any(rest.cpu().numpy())


@pytest.mark.parametrize("family", ["affine", "linear"])
@pytest.mark.parametrize("L1,L2", [(1023, 2047), (260, 1500), (64, 700), (33, 1000)])
def test_quiet_stretch_up_to_the_first_rows(family, L1, L2):
    """Whole strips without mass whose chunks reach above row 1: what the
    kernels do there, outside the pair, decides no quiet chunk differently.
    (260 x 1500, linear, seed 1: 192 cells differed, by 3e-35.)  And a
    second run gives the same bits."""
    from orihime_b200 import _ops, ragged

    for seed in (0, 4, 1, 3):
        g = torch.Generator().manual_seed(seed)
        torch.randn(1, L1, L2, generator=g)   # the noted pair follows this draw
        s = (torch.randn(L1, 64, generator=g) @ torch.randn(L2, 64, generator=g).T * 0.75).contiguous()
        kw = dict(gap_open=-2.0, gap_ext=-0.5) if family == "affine" else dict(gap=-1.0)
        run = _ops.run_affine if family == "affine" else _ops.run_linear
        v, m, *grads = run(s[None].cuda(), None, *kw.values(), 1.0)
        flat, off, ln = ragged.pack([s])
        plan = ragged.Plan(ln, off, family=family, device="cuda", cols_per_lane=4)
        for _ in range(2):
            out = plan.run(flat.cuda(), temp=1.0, **kw)
            assert plan.status() == 0
            assert torch.equal(v, out.value) and torch.equal(grads[-1], out.grad_temp)
            assert torch.equal(m[0], ragged.unpack(out.map, off, ln)[0])
