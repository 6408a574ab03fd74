"""GPU: runs whose checks do reproject give the same points in every configuration (few chains per SM
or many, an explicit thread count, the long scratch of 6657 to 7680 reactions).  The block models'
own warmup points satisfy S x = 0 exactly and never reproject; here they are moved off null(S)."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_autotune_scratch import _long_scratch_model
from test_gpu_large_configs import _block_model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [96, 126, 129, 255, 510, 771, 1059, 1281, 2562, 3840, 6657, 7440, 7680])
def test_points_and_accumulators(pkg, n):
    torch = pytest.importorskip("torch")
    model, N, warm = _block_model(pkg, n // 3, seed=n)
    warm = warm + 1e-7 * np.random.default_rng(n).standard_normal(warm.shape)

    def run(s, P):
        x = torch.empty((n, P), dtype=torch.float64, device="cuda")
        A = torch.empty_like(x)
        st = [s.sample_resume(P, step0, steps, step0 > 0, x.data_ptr(), A.data_ptr(), P, seed=n, with_stats=True)
              for step0, steps in ((0, 7), (7, 5))]
        # 12 steps have two checks, both of points off null(S) by about 1e-7
        assert all(q["reprojections"] > 0 and q["segments"] == 0 for q in st)
        return x[:, :40].cpu().numpy(), A[:, :40].cpu().numpy()

    with pkg.Sampler(model, warm, reproject_form=1) as s:
        s.set_null_space(N)
        base = run(s, 40)
        others = [run(s, P) for P in (300, 1200)]
    with pkg.Sampler(model, warm, reproject_form=1, threads_per_chain=512) as s:
        s.set_null_space(N)
        others.append(run(s, 40))
    for x, A in others:
        assert np.array_equal(base[0], x) and np.array_equal(base[1], A)


def test_long_scratch(pkg, oracle_mod):
    model, N, warm = _long_scratch_model(pkg)
    warm = warm + 1e-7 * np.random.default_rng(6).standard_normal(warm.shape)
    pts = []
    for threads in (0, 512):
        with pkg.Sampler(model, warm, reproject_form=1, threads_per_chain=threads) as s:
            s.set_null_space(N)
            pts.append(s.sample(3, 4, seed=5))
    (x0, st0), (x1, st1) = pts
    ref, rst = oracle_mod.sample(model, warm, N, 5, 3, 4)
    assert np.array_equal(x0, x1)
    assert st0["reprojections"] == st1["reprojections"] == rst["reprojections"] > 0
    assert np.abs(x0 - ref).max() <= 1e-10 * max(1.0, np.abs(ref).max())
