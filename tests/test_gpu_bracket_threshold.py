"""GPU: a large u_tol, for which the box bounds the candidacy threshold too loosely for brackets formed with
the direction: the FP64 evaluations stay about those of the separate bracket pass, the points are the same."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_large_configs import _block_model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [96, 1059, 3741])
@pytest.mark.parametrize("u_tol", [1e-9, 1e-6, 1e-5, 1e-4, 1e-3])
def test_exact_evaluations(pkg, n, u_tol):
    model, N, warm = _block_model(pkg, n // 3, seed=n)
    pts, evals = [], []
    for bracket_pass in (0, 1):
        with pkg.Sampler(model, warm, u_tol=u_tol, bracket_pass=bracket_pass) as s:
            s.set_null_space(N)
            x, st = s.sample(40, 25, seed=2)
        pts.append(x)
        evals.append(st["exact_evals"])
    assert np.array_equal(pts[0], pts[1])
    assert evals[1] <= evals[0] <= 2 * evals[1]
