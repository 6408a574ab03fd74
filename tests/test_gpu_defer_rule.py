"""GPU: which runs defer their reprojections on their own (chains x n_rxns x null_dim >= 2e7 on %f
warmup points), and that both sides of the line give the same chains: points within 1e-10 of the
in-kernel FP64 form with equal counts, the run cut into segments included."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
KEYS = ("accepted", "rejected", "checks", "reprojections", "stuck_chains")


@pytest.mark.parametrize("work,deferred", [(0.98, False), (1.02, True)])
def test_line_between_the_forms(pkg, small_model, golden, work, deferred):
    N = golden["N"]
    P = int(np.ceil(work * 2.0e7 / (small_model.n_rxns * N.shape[1])))
    with pkg.Sampler(small_model, golden["warmup"]) as s, \
            pkg.Sampler(small_model, golden["warmup"], reproject_form=1) as ref:
        for q in (s, ref):
            q.set_null_space(N)
        a, st = s.sample(P, 12, seed=5)
        b, rst = ref.sample(P, 12, seed=5)
        assert (st["segments"] > 0) == deferred and rst["segments"] == 0
        assert st["reprojections"] > 0
        x = torch.zeros((small_model.n_rxns, P), dtype=torch.float64, device="cuda")
        A = torch.zeros_like(x)
        s.sample_resume(P, 0, 5, False, x.data_ptr(), A.data_ptr(), P, seed=5)
        s.sample_resume(P, 5, 7, True, x.data_ptr(), A.data_ptr(), P, seed=5)
        torch.cuda.synchronize()
    assert np.abs(a - b).max() <= 1e-10 * max(1.0, np.abs(b).max())
    assert np.abs(x.cpu().numpy() - b).max() <= 1e-10 * max(1.0, np.abs(b).max())
    for k in KEYS:
        assert st[k] == rst[k], k


def test_capture_before_the_buffers_exist_stays_in_the_kernel(pkg, small_model, golden):
    """A captured run of a fresh context cannot allocate: it reprojects in the chain kernel, and the
    graph gives the points of the in-kernel form."""
    N = golden["N"]
    P = int(np.ceil(2.2e7 / (small_model.n_rxns * N.shape[1])))
    out = torch.zeros((small_model.n_rxns, P), dtype=torch.float64, device="cuda")
    with pkg.Sampler(small_model, golden["warmup"]) as s, \
            pkg.Sampler(small_model, golden["warmup"], reproject_form=1) as ref:
        for q in (s, ref):
            q.set_null_space(N)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            s.sample_device(P, 11, out.data_ptr(), P, stream=torch.cuda.current_stream().cuda_stream, seed=9)
        g.replay()
        torch.cuda.synchronize()
        want, _ = ref.sample(P, 11, seed=9)
    assert np.array_equal(out.cpu().numpy(), want)
