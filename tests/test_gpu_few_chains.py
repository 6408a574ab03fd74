"""GPU: a chain's points are the same in a launch of few chains, which takes more threads per chain, and in one of
many, bit for bit: reprojecting through the residual (whose z takes the same turns in either)."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_large_configs import _block_model
from test_zz_no_alloc import _device_model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [96, 258, 1020, 1059, 2562, 5001, 7440])
def test_residual_form(pkg, n):
    model, N, warm = _block_model(pkg, n // 3, seed=n)
    warm = warm + 1e-7 * np.random.default_rng(n).standard_normal(warm.shape)  # every check reprojects
    with pkg.Sampler(model, warm, reproject_form=2) as s:
        s.set_null_space(N)
        many, st = s.sample(2600, 12, seed=3)
        assert st["reprojections"] > 0
        for P in (1, 150, 300, 1000):
            assert np.array_equal(s.sample(P, 12, seed=3)[0], many[:, :P]), P


@pytest.mark.parametrize("n", [96, 1059, 2562, 5001])
def test_without_allocation(pkg, native, n):
    torch = pytest.importorskip("torch")
    model, N, warm = _block_model(pkg, n // 3, seed=n)
    warm = warm + 1e-7 * np.random.default_rng(n).standard_normal(warm.shape)
    keep = {}
    dm = _device_model(pkg, torch, model, warm, N, keep)
    got = {}
    for P in (3, 150, 2600):
        x = torch.empty((n, P), dtype=torch.float64, device="cuda")
        st = pkg.sample_noalloc(dm, P, 12, x.data_ptr(), P, torch.cuda.current_stream().cuda_stream, seed=3)
        assert st["reprojections"] > 0
        got[P] = x.cpu().numpy()
    for P in (3, 150):
        assert np.array_equal(got[P], got[2600][:, :P]), P
