"""GPU: the preconditioner's loss and gradients at the edges of its kernels' tiles (the 128 x 128
products, their split contractions and 16-byte loads; the 64 x 64 blocks of the inverse) against the
FP64 oracle, with the tolerance of test_loss_grad_matches_fp64_oracle."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("d,r,B,pad", [(1, 1, 1, 0), (5, 8, 3, 0), (9, 4, 4096, 0), (64, 64, 64, 1), (130, 65, 129, 2),
                                       (257, 129, 67, 0), (100, 33, 5001, 3), (300, 200, 256, 0), (1030, 256, 300, 1)])
def test_loss_grad_at_tile_edges(pkg, d, r, B, pad):
    from oracle import precond
    rng = np.random.default_rng(d + r)
    s = (0.3 * rng.standard_normal(d)).astype(np.float32)
    U = (0.8 / np.sqrt(r) * rng.standard_normal((d, r))).astype(np.float32)
    Y = (rng.standard_normal((d, B + pad)) * np.exp(rng.uniform(-1, 1, (d, 1)))).astype(np.float32)
    ds, dU, dY = (torch.from_numpy(v).cuda() for v in (s, U, Y))
    gs, gU = torch.full_like(ds, np.nan), torch.full_like(dU, np.nan)
    loss = pkg.precond_loss_grad(d, r, B, ds.data_ptr(), dU.data_ptr(), dY.data_ptr(), B + pad, gs.data_ptr(),
                                 gU.data_ptr())
    val, gs_ref, gU_ref = precond.loss_grad(s, U, Y[:, :B])
    assert abs(loss - val) <= 1e-4 * max(1.0, abs(val))
    assert np.abs(gs.cpu().numpy() - gs_ref).max() <= 2e-4 * max(1.0, np.abs(gs_ref).max())
    assert np.abs(gU.cpu().numpy() - gU_ref).max() <= 2e-4 * max(1.0, np.abs(gU_ref).max())


def test_indefinite_parameters_are_refused(pkg):
    d, r, B = 70, 66, 32
    z = torch.zeros(d, device="cuda")
    U = torch.full((d, r), float("nan"), device="cuda")
    Y = torch.ones((d, B), device="cuda")
    with pytest.raises(pkg.AchrError) as err:
        pkg.precond_loss_grad(d, r, B, z.data_ptr(), U.data_ptr(), Y.data_ptr(), B, z.clone().data_ptr(),
                              U.clone().data_ptr())
    assert err.value.status == 6  # ACHR_ERR_NUMERIC
