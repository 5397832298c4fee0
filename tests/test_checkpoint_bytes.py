"""What the value op keeps between its forward and its backward: host logic, on CPU."""

import pytest
import torch


@pytest.mark.parametrize("fam", ["sw_affine", "sw"])
@pytest.mark.parametrize("shape", [(64, 1024, 1024), (4, 16384, 16384), (1, 16384, 16384), (2, 8192, 8192),
                                   (16, 1024, 1024), (1, 4096, 4096)])
def test_stride_4_keeps_below_half_of_the_map(fam, shape):
    from orihime_b200 import _ops

    B, L1, L2 = shape
    assert _ops.checkpoint_bytes(fam, B, L1, L2, 4) < 2.0 * B * L1 * L2


@pytest.mark.parametrize("fam", ["sw_affine", "sw"])
@pytest.mark.parametrize("shape", [(1, 64, 64), (8, 128, 128), (64, 1024, 1024), (1, 16384, 16384), (150, 256, 65),
                                   (5000, 256, 65), (4, 8192, 8192), (6, 8192, 8192), (4, 16384, 16384),
                                   (3, 1, 7), (2, 0, 5)])
def test_dense_checkpoints_only_within_the_limits(fam, shape):
    from orihime_b200 import _ops, operator

    every = operator._checkpoint_every(fam, torch.empty(shape, device="meta"))
    dense = _ops.checkpoint_bytes(fam, *shape, 1)
    small = dense <= operator.SMALL_CHECKPOINT_BYTES
    fits = dense <= operator.DENSE_CHECKPOINT_BYTES and dense <= 4 * shape[0] * shape[1] * shape[2]
    assert every == (1 if small or fits else operator.CHECKPOINT_EVERY)
    assert operator._checkpoint_every("sw_affine", torch.empty(64, 1024, 1024, device="meta")) == 1
    assert operator._checkpoint_every("sw_affine", torch.empty(5000, 256, 65, device="meta")) == 4
