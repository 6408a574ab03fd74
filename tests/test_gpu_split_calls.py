"""GPU: chains split over calls on both sides of the line of 2e7 (chains x n_rxns x null_dim).  With the form
of the reprojection named, the parts are the whole call's columns bit for bit; left to the library
(reproject_form 0), which takes the size of the call into account, they agree to rounding."""
from __future__ import annotations

import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", [0, 1, 3])
def test_parts_equal_the_whole(pkg, small_model, golden, form):
    sharding = importlib.import_module("achr_gb300.sharding")
    N, T, world = golden["N"], 21, 3
    total = int(np.ceil(2.2e7 / N.size))  # deferred by choice as a whole, not in parts
    with pkg.Sampler(small_model, golden["warmup"], reproject_form=form) as s:
        s.set_null_space(N)
        whole, st = s.sample(total, T, seed=8)
        parts, segments = [], []
        for rank in range(world):
            off, count = sharding.split_chains(rank, world, total)
            pts, pst = s.sample(count, T, seed=8, chain_offset=off)
            parts.append(pts)
            segments.append(pst["segments"] > 0)
    got = np.concatenate(parts, axis=1)
    assert st["reprojections"] > 0 and (st["segments"] > 0) == (form != 1) and all(v == (form == 3) for v in segments)
    if form:
        assert np.array_equal(got, whole)
    else:
        assert np.abs(got - whole).max() <= 1e-9 * max(1.0, np.abs(whole).max())
