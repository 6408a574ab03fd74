"""GPU: the chain kernel at the edges of its configuration ladder (odd lengths, one reaction past a
configuration, the largest of each) against the oracle, with bounds that FP32 holds exactly and with
bounds it does not, and along hit-and-run directions.

The models are the block-diagonal ones of test_gpu_large_configs.py, whose null space is known."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_large_configs import _block_model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [126, 129, 255, 387, 513, 768, 771, 1026, 1281, 1539, 2049, 2562, 3072, 3075, 3840, 4095,
                               4608, 5121])
@pytest.mark.parametrize("form", ["exact bounds", "rounded bounds", "directions"])
def test_ladder_edges_match_oracle(pkg, oracle_mod, n, form):
    if form != "exact bounds" and n > 2600 and n % 2 == 0:
        pytest.skip("covered by the odd lengths")
    model, N, warm = _block_model(pkg, n // 3, seed=n)
    if form != "rounded bounds":
        model.lb, model.ub = np.floor(model.lb), np.ceil(model.ub)
    P, T = 12, 25
    kw = {}
    with pkg.Sampler(model, warm) as s:
        s.set_null_space(N)
        cols = warm
        if form == "directions":
            cols = N @ np.random.default_rng(n).standard_normal((N.shape[1], 40))
            s.set_directions(cols)
            kw = {"centre_point": s.centre()}
        pts, st = s.sample(P, T, seed=n)
    prob = oracle_mod.Problem(model, cols, N, **kw)
    ref, rst = prob.sample(n, P, T, hit_and_run=form == "directions")
    assert np.abs(pts - ref).max() <= 1e-10 * max(1.0, np.abs(ref).max())
    for k in ("accepted", "rejected", "checks", "reprojections"):
        assert st[k] == rst[k], k
