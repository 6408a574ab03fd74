"""GPU: the autotuner where a reprojection's scratch (max(n_mets, null_dim) doubles) is too long for the
256-thread configuration of 6657 to 7680 reactions, first in the process and after a model of the
same length whose scratch does fit was tuned."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_large_configs import _block_model

pytestmark = pytest.mark.gpu


def _long_scratch_model(pkg, blocks=2222, constrained=100):
    """Block model of which only the first blocks are constrained: null dimension above 6144."""
    full, _, _ = _block_model(pkg, blocks, seed=1)
    b = np.arange(constrained)
    row = np.concatenate([2 * b, 2 * b, 2 * b + 1, 2 * b + 1])
    col = np.concatenate([3 * b, 3 * b + 1, 3 * b + 1, 3 * b + 2])
    val = np.concatenate([np.ones(constrained), -np.ones(constrained), np.ones(constrained), -np.ones(constrained)])
    n = 3 * blocks
    model = pkg.HostModel(n, 2 * constrained, row, col, val, full.lb, full.ub)
    free = np.arange(3 * constrained, n)
    N = np.zeros((n, constrained + len(free)))
    N[3 * b, b] = N[3 * b + 1, b] = N[3 * b + 2, b] = 1.0 / np.sqrt(3.0)
    N[free, constrained + np.arange(len(free))] = 1.0
    rng = np.random.default_rng(2)
    t = rng.uniform(-4.0, 4.0, (N.shape[1], 16))
    t[:constrained] *= np.sqrt(3.0)
    return model, N, N @ t


def test_autotune_with_a_long_scratch(pkg):
    model, N, warm = _long_scratch_model(pkg)
    assert N.shape[1] > 6144
    other, No, wo = _block_model(pkg, 2222, seed=3)
    for first in (False, True):
        if first:
            with pkg.Sampler(other, wo) as s:  # the same padded length, scratch of 4444
                s.set_null_space(No)
                assert s.autotune() in (256, 384, 512)
        with pkg.Sampler(model, warm, reproject_form=1) as s:
            s.set_null_space(N)
            want, _ = s.sample(3, 2, seed=4)
            assert s.autotune() in (384, 512)
            got, _ = s.sample(3, 2, seed=4)
        assert np.array_equal(got, want)
