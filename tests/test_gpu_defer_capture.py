"""GPU: captured runs.  Where deferral is a choice (n d < 2.5e5) a captured run reprojects in the chain kernel
whatever ran before it; where it was asked for, the graph's buffers outlive larger runs after the capture."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _capture(s, P, T, out, seed):
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        s.sample_device(P, T, out.data_ptr(), P, stream=torch.cuda.current_stream().cuda_stream, seed=seed)
    return g


@pytest.mark.parametrize("form", [0, 3])
def test_replay_after_a_larger_run(pkg, small_model, golden, form):
    N = golden["N"]
    P, T = int(np.ceil(2.2e7 / N.size)), 11
    out = torch.zeros((small_model.n_rxns, P), dtype=torch.float64, device="cuda")
    with pkg.Sampler(small_model, golden["warmup"], reproject_form=form) as s, \
            pkg.Sampler(small_model, golden["warmup"], reproject_form=3 if form == 3 else 1) as ref:
        for q in (s, ref):
            q.set_null_space(N)
        assert s.sample(P, T, seed=1)[1]["segments"] > 0  # deferred, its buffers there
        g = _capture(s, P, T, out, seed=9)
        assert s.sample(2 * P, 8 * T, seed=2)[1]["segments"] > 0  # more chains and more segments
        other = torch.randn(1 << 26, device="cuda")  # (memory given back would be here)
        g.replay()
        torch.cuda.synchronize()
        want, _ = ref.sample(P, T, seed=9)
        assert torch.isfinite(other).all()
    assert np.array_equal(out.cpu().numpy(), want)
