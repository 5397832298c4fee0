"""Local alignments whose scores are large in units of T, where a step gains up
to 115 bits: nothing that the linear domain can hold is lost on its way from
lane to lane or between the forward and the outside recursion.

Against the fp64 oracle: values to 1e-5 of their size; maps to (L1 + L2) 2^-23
(a path's roundings, one of each sign per step); gradients to 1e-4 of their size
or the fp32 oracle's own error, whichever is larger.  Against the log-domain
kernels on many pairs: no map more than 1e-3 off."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

GAPS = {"affine": (-2.0, -0.5), "linear": (-1.0,)}


def _run(family, s, T, **opt):
    from orihime_b200 import _lib, _ops

    run = {"affine": _ops.run_affine, "linear": _ops.run_linear}[family]
    return run(s, None, *GAPS[family], T, options=_lib.Options(**opt))


def _check(family, s, T, cols):
    from oracle import oracle as O

    f = getattr(O, family)
    r32, r64 = (f(s, None, *GAPS[family], T, dtype=d) for d in (np.float32, np.float64))
    out = [x.cpu().numpy().astype(np.float64) for x in _run(family, torch.from_numpy(s).cuda(), T, cols_per_lane=cols)]
    names = ["value", "map"] + (["grad_open", "grad_ext"] if family == "affine" else ["grad_gap"]) + ["grad_temp"]
    for name, got in zip(names, out):
        want = r64[name]
        err = np.abs(got - want).max()
        if name == "value":
            tol = 1e-5 * max(1.0, np.abs(want).max())
        elif name == "map":
            tol = (s.shape[1] + s.shape[2]) * 2.0 ** -23
        else:
            tol = max(1e-4 * max(1.0, np.abs(want).max()), np.abs(r32[name] - want).max())
        assert err <= tol, (name, err, tol)


def _matches(L1, L2, seed):
    r = np.random.default_rng(seed)
    return (r.normal(size=(L1, 64)) @ r.normal(size=(L2, 64)).T * 0.375)[None].astype(np.float32)


@pytest.mark.parametrize("family", ["affine", "linear"])
def test_value_just_below_the_row_survives_the_hand_over(family):
    s = np.full((1, 5, 4), -5.0, np.float32)
    s[0, 0, 2], s[0, 1, 3], s[0, 2, 1], s[0, 3, 2] = 12.0, 79.0, 79.0, 79.0
    _check(family, s, 1.0, 2)


@pytest.mark.parametrize("family", ["affine", "linear"])
@pytest.mark.parametrize("cols,T", [(2, 0.25), (2, 0.35), (4, 0.35), (8, 0.5)])
@pytest.mark.parametrize("shape", [(860, 35), (318, 38), (593, 172), (172, 593), (500, 384)],
                         ids=lambda s: f"{s[0]}x{s[1]}")
def test_thin_pairs(family, cols, T, shape):
    _check(family, _matches(*shape, seed=shape[0]), T, cols)


@pytest.mark.parametrize("family", ["affine", "linear"])
@pytest.mark.parametrize("cols,T,shape", [(2, 0.2, (200, 200)), (2, 0.25, (600, 172)), (4, 0.35, (600, 172))])
def test_maps_of_many_pairs_equal_the_log_domain(family, cols, T, shape):
    from orihime_b200 import _lib

    g = torch.Generator().manual_seed(5)
    B = 256
    s = torch.bmm(torch.randn(B, shape[0], 64, generator=g), torch.randn(B, 64, shape[1], generator=g)) * 0.375
    s = s[s.abs().amax((1, 2)) / T <= 80].contiguous().cuda()
    lin = _run(family, s, T, cols_per_lane=cols, domain=_lib.DOMAIN_LINEAR)
    log = _run(family, s, T, cols_per_lane=4, domain=_lib.DOMAIN_LOG)
    assert all(torch.isfinite(x).all() for x in lin)
    assert float((lin[1] - log[1]).abs().max()) < 1e-3


@pytest.mark.parametrize("family", ["affine", "linear"])
def test_public_route_keeps_the_paths_of_many_pairs(family):
    """The padded entry points' own columns at T = 0.25: map, value alone and the
    value op's gradient."""
    import orihime_b200 as ohm
    from orihime_b200 import _lib

    g = torch.Generator().manual_seed(6)
    s = (torch.bmm(torch.randn(256, 600, 64, generator=g), torch.randn(256, 64, 172, generator=g)) * 0.375)
    s = s[s.abs().amax((1, 2)) / 0.25 <= 80].contiguous().cuda()
    log = _run(family, s, 0.25, cols_per_lane=4, domain=_lib.DOMAIN_LOG)
    kw = (dict(gap_open_score=-2.0, gap_extend_score=-0.5) if family == "affine" else dict(gap_score=-1.0))
    fn, fv = (ohm.sw_affine, ohm.sw_affine_value) if family == "affine" else (ohm.sw, ohm.sw_value)
    assert float((fn(s, temperature=0.25, **kw) - log[1]).abs().max()) < 1e-3
    torch.testing.assert_close(fv(s, temperature=0.25, **kw), log[0], rtol=1e-5, atol=1e-3)
    x = s.clone().requires_grad_(True)
    fv(x, temperature=0.25, **kw).sum().backward()
    assert float((x.grad - log[1]).abs().max()) < 1e-3
