"""GPU: the points of a chain do not depend on the configuration a launch takes: few chains per SM
(more threads per chain) or many, an explicit thread count, or the accumulator kept partly in
registers (6657 to 7680 reactions), there also where the reprojection's scratch is too long for it.
Every coordinate is computed by the same operations in each, so the results are compared bit for bit.

The models are the block-diagonal ones of test_gpu_large_configs.py, whose null space is known."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_large_configs import _block_model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [96, 126, 129, 255, 510, 771, 1059, 1281, 2562, 3840, 6657, 7440, 7680])
def test_points_independent_of_configuration(pkg, n):
    torch = pytest.importorskip("torch")
    model, N, warm = _block_model(pkg, n // 3, seed=n)
    T = 12

    def run(s, P):
        x = torch.empty((n, P), dtype=torch.float64, device="cuda")
        A = torch.empty_like(x)
        for step0 in (0, 7):
            s.sample_resume(P, step0, 7 if step0 == 0 else T - 7, step0 > 0, x.data_ptr(), A.data_ptr(), P, seed=n)
        torch.cuda.synchronize()
        return x[:, :40].cpu().numpy(), A[:, :40].cpu().numpy()

    with pkg.Sampler(model, warm, residual_tol=1e-15) as s:  # a reprojection at nearly every check
        s.set_null_space(N)
        base = run(s, 40)
        others = [run(s, P) for P in (300, 600, 1200, 2500)]
    with pkg.Sampler(model, warm, residual_tol=1e-15, threads_per_chain=512) as s:
        s.set_null_space(N)
        others.append(run(s, 40))
    for x, A in others:
        assert np.array_equal(base[0], x) and np.array_equal(base[1], A)


def test_long_scratch_takes_another_configuration(pkg):
    n, blocks, constrained = 6666, 2222, 100
    full, _, _ = _block_model(pkg, blocks, seed=1)
    b = np.arange(constrained)
    row = np.concatenate([2 * b, 2 * b, 2 * b + 1, 2 * b + 1])
    col = np.concatenate([3 * b, 3 * b + 1, 3 * b + 1, 3 * b + 2])
    val = np.concatenate([np.ones(constrained), -np.ones(constrained), np.ones(constrained), -np.ones(constrained)])
    model = pkg.HostModel(n, 2 * constrained, row, col, val, full.lb, full.ub)
    free = np.arange(3 * constrained, n)
    d = constrained + len(free)
    assert d > 6144  # the accumulator's share of shared memory, the reprojection's scratch
    N = np.zeros((n, d))
    N[3 * b, b] = N[3 * b + 1, b] = N[3 * b + 2, b] = 1.0 / np.sqrt(3.0)
    N[free, constrained + np.arange(len(free))] = 1.0
    rng = np.random.default_rng(2)
    t = rng.uniform(-4.0, 4.0, (d, 16))
    t[:constrained] *= np.sqrt(3.0)
    warm = N @ t
    pts = []
    for threads in (0, 512):
        with pkg.Sampler(model, warm, residual_tol=0.0, reproject_form=1, threads_per_chain=threads) as s:
            s.set_null_space(N)
            pts.append(s.sample(3, 4, seed=5))
    (x0, st0), (x1, st1) = pts
    assert np.array_equal(x0, x1)
    assert st0["reprojections"] == st1["reprojections"]


@pytest.mark.parametrize("n", [1059, 3072, 6000, 7440])  # the larger: z takes turns beside the residual
@pytest.mark.parametrize("form", [1, 2])
def test_reprojection_independent_of_configuration(pkg, oracle_mod, n, form):
    model, N, warm = _block_model(pkg, n // 3, seed=n)
    warm = warm + 1e-7 * np.random.default_rng(n).standard_normal(warm.shape)  # every check reprojects
    T = 22
    with pkg.Sampler(model, warm, reproject_form=form) as s:
        s.set_null_space(N)
        base, st = s.sample(16, T, seed=9)
        for P in (200, 700):
            assert np.array_equal(s.sample(P, T, seed=9)[0][:, :16], base)
    ref, rst = oracle_mod.sample(model, warm, N, 9, 16, T)
    assert st["reprojections"] == rst["reprojections"] > 0
    assert np.abs(base - ref).max() <= 1e-10 * max(1.0, np.abs(ref).max())
