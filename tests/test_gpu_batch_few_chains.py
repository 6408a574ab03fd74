"""GPU: a batch of few chains runs its models with more threads per chain (its work queues are then those of other
configurations); the points are those of the models' own runs, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_large_configs import _block_model

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("chains", [(1, 2, 1, 3), (40, 30, 50, 60), (200, 0, 300, 250), (1000, 900, 700, 800)])
def test_points_of_a_batch(pkg, chains):
    models = [_block_model(pkg, n // 3, seed=n) for n in (96, 510, 1059, 2562)]
    samplers = [pkg.Sampler(m, w) for m, _, w in models]
    outs = [torch.zeros((s.n, P), dtype=torch.float64, device="cuda") for s, P in zip(samplers, chains)]
    for s, (_, N, _) in zip(samplers, models):
        s.set_null_space(N)
    pkg.sample_batch(samplers, list(chains), 25, [o.data_ptr() for o in outs], [max(P, 1) for P in chains], seed=6)
    torch.cuda.synchronize()
    off = 0
    for s, P, out in zip(samplers, chains, outs):
        if P:
            assert np.array_equal(out.cpu().numpy(), s.sample(P, 25, seed=6, chain_offset=off)[0])
        off += P
        s.close()
