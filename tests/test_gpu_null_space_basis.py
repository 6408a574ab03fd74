"""GPU: reprojections go onto the basis the caller set (achr_set_null_space), on both sides of the line
from which runs on %f warmup points are deferred: the deferred form and the residual form are built
from S, so a basis that does not span null(S) (a subspace, all of the space) stays with N (N^T x)."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_large_configs import _block_model

pytestmark = pytest.mark.gpu
LINE = 2.0e7  # chains x n_rxns x null_dim from which a run is deferred


def _narrower(pkg, blocks, dropped, seed):
    """Block model, its basis less some blocks' columns, and warmup points in that span up to 1e-6."""
    model, N, _ = _block_model(pkg, blocks, seed)
    rng = np.random.default_rng(seed + 1)
    N = np.ascontiguousarray(N[:, dropped:])
    warm = N @ (rng.uniform(-0.9, 0.9, (N.shape[1], 64)) * 5.0 * np.sqrt(3.0))
    return model, N, warm + rng.uniform(-1e-6, 1e-6, warm.shape)


@pytest.mark.parametrize("work", [0.98, 1.02])
def test_narrower_basis_is_kept(pkg, oracle_mod, work):
    model, N, warm = _narrower(pkg, 40, 5, seed=11)
    P, T, some = int(np.ceil(work * LINE / N.size)), 21, 64
    with pkg.Sampler(model, warm) as s, pkg.Sampler(model, warm, reproject_form=1) as ref:
        for q in (s, ref):
            q.set_null_space(N)
        pts, st = s.sample(P, T, seed=5)
        want, rst = ref.sample(P, T, seed=5)
    got, gst = oracle_mod.sample(model, warm, N, 5, some, T)
    assert gst["reprojections"] > 0
    assert np.abs(pts[:, :some] - got).max() <= 1e-10 * max(1.0, np.abs(got).max())
    assert st["segments"] == 0 and st["reprojections"] == rst["reprojections"] > 0
    assert np.array_equal(pts, want)


@pytest.mark.parametrize("work", [0.98, 1.02])
def test_basis_of_the_null_space_may_be_deferred(pkg, small_model, golden, work):
    """Another orthonormal basis of the same space, a rotation of the golden one, and others in between."""
    Q = np.linalg.qr(np.random.default_rng(3).standard_normal((golden["N"].shape[1],) * 2))[0]
    N = golden["N"] @ Q
    P = int(np.ceil(work * LINE / N.size))
    with pkg.Sampler(small_model, golden["warmup"]) as s:
        for basis, whole in ((N, True), (N[:, 1:], False), (2.0 * N, False), (N, True)):
            s.set_null_space(basis)
            st = s.sample(P + P // 10 if not whole else P, 2, seed=5)[1]
            assert (st["segments"] > 0) == (whole and work > 1.0)


def test_keep_all_basis_is_the_identity(pkg):
    """S of full column rank: the reference's rule keeps all n columns, N (N^T x) = x, on a run above the line."""
    n, m = 48, 48
    rng = np.random.default_rng(7)
    S = rng.choice([-2.0, -1.0, 1.0, 2.0], (m, n)) * (rng.random((m, n)) < 0.1)
    S[np.arange(n), np.arange(n)] = 9.0
    row, col = np.nonzero(S)
    model = pkg.HostModel(n, m, row, col, S[row, col], np.full(n, -10.0), np.full(n, 10.0))
    warm = rng.uniform(-5.0, 5.0, (n, 2 * n))
    P = int(np.ceil(1.1 * LINE / (n * n)))
    with pkg.Sampler(model, warm) as s, pkg.Sampler(model, warm, reproject_form=1) as ref:
        assert s.null_dim == n
        pts, st = s.sample(P, 12, seed=2)
        want, rst = ref.sample(P, 12, seed=2)
    assert rst["reprojections"] > 0
    # N is orthonormal to rounding only: each of two reprojections moves a point by a few units in the last place
    assert np.abs(want).max() > 1.0 and st["segments"] == 0 and st["reprojections"] == rst["reprojections"]
    assert np.array_equal(pts, want)


@pytest.mark.parametrize("fixed", [False, True])
def test_residual_form_leaves_a_narrower_basis_to_the_kernel(pkg, fixed):
    """n d >= 4e6, where the automatic choice is the residual form (built from S): a caller's narrower
    basis, and ACHR_NULL_FIXED with blocked reactions, keep N (N^T x)."""
    blocks, dropped = 1200, 40
    model, N, warm = _narrower(pkg, blocks, dropped, seed=4)
    assert N.size >= 4.0e6
    opts = {}
    if fixed:
        lb, ub = np.array(model.lb), np.array(model.ub)
        lb[:3 * dropped:3] = ub[:3 * dropped:3] = 0.0  # one reaction of each dropped block
        warm[:3 * dropped:3] = 0.0
        model = pkg.HostModel(model.n_rxns, model.n_mets, model.row, model.col, model.val, lb, ub)
        opts = {"null_space": pkg.NULL_FIXED}
    pts = []
    for form in (0, 1):
        with pkg.Sampler(model, warm, reproject_form=form, **opts) as s:
            if not fixed:
                s.set_null_space(N)
            assert s.null_dim == blocks - dropped
            p, st = s.sample(4, 11, seed=3)
            assert st["segments"] == 0 and st["reprojections"] > 0
            pts.append(p)
    assert np.array_equal(pts[0], pts[1])
