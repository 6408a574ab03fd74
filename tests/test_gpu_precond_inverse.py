"""GPU: the preconditioner's inverse at the ranks where its kernels change path (the triangle in
shared memory, to 304, or not), where a last block is ragged, and at the largest, against the FP64 oracle
with the tolerance of test_loss_grad_matches_fp64_oracle."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("d,r", [(40, 31), (40, 32), (40, 33), (300, 37), (300, 66), (64, 304), (64, 305), (64, 320),
                                 (64, 321), (40, 1001), (40, 1024)])
def test_inverse_at_path_edges(pkg, d, r):
    from oracle import precond
    B = 96
    rng = np.random.default_rng(d + r)
    s = (0.3 * rng.standard_normal(d)).astype(np.float32)
    U = (0.8 / np.sqrt(r) * rng.standard_normal((d, r))).astype(np.float32)
    Y = rng.standard_normal((d, B)).astype(np.float32)
    ds, dU, dY = (torch.from_numpy(v).cuda() for v in (s, U, Y))
    gs, gU = torch.full_like(ds, np.nan), torch.full_like(dU, np.nan)
    loss = pkg.precond_loss_grad(d, r, B, ds.data_ptr(), dU.data_ptr(), dY.data_ptr(), B, gs.data_ptr(), gU.data_ptr())
    val, gs_ref, gU_ref = precond.loss_grad(s, U, Y)
    assert abs(loss - val) <= 1e-4 * max(1.0, abs(val))
    assert np.abs(gs.cpu().numpy() - gs_ref).max() <= 2e-4 * max(1.0, np.abs(gs_ref).max())
    assert np.abs(gU.cpu().numpy() - gU_ref).max() <= 2e-4 * max(1.0, np.abs(gU_ref).max())
