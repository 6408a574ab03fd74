"""GPU: deferred runs of one context queued on several streams, with nothing between them, give the points
of runs one after another (they share the context's buffers, so each waits for the last)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("form,P", [(3, 3000), (0, 10000)])
def test_runs_on_two_streams(pkg, small_model, golden, form, P):
    n, T = small_model.n_rxns, 25
    with pkg.Sampler(small_model, golden["warmup"], reproject_form=form) as s:
        s.set_null_space(golden["N"])
        want = []
        for k in range(4):
            pts, st = s.sample(P, T, seed=k)
            assert st["segments"] > 0 and st["reprojections"] > 0
            want.append(pts)
    with pkg.Sampler(small_model, golden["warmup"], reproject_form=form) as s:  # buffers made on the first of them
        s.set_null_space(golden["N"])
        streams = [torch.cuda.Stream() for _ in range(2)]
        outs = [torch.zeros((n, P), dtype=torch.float64, device="cuda") for _ in range(4)]
        torch.cuda.synchronize()
        for k, out in enumerate(outs):
            s.sample_device(P, T, out.data_ptr(), P, stream=streams[k % 2].cuda_stream, seed=k)
        torch.cuda.synchronize()
        for k, out in enumerate(outs):
            assert np.array_equal(out.cpu().numpy(), want[k])
