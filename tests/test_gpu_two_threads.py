"""GPU: two host threads, each with its own context and stream, whose models take the same kernels with
different amounts of shared memory: a residual-form reprojection beside none, deferred passes of two sizes."""
from __future__ import annotations

import threading

import numpy as np
import pytest

from test_gpu_large_configs import _block_model

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("sizes,threads_per_chain,calls", [
    (((1000, 2), (1001, 1)), 512, 2000),  # 512 x 8, z beside the residual or none
    (((150, 3), (250, 3)), 128, 300),     # the passes of 450 and of 750 reactions
], ids=["chain_kernel", "deferred_passes"])
def test_shared_memory_of_concurrent_launches(pkg, sizes, threads_per_chain, calls):
    runs = []
    for blocks, form in sizes:
        model, N, warm = _block_model(pkg, blocks, seed=form)
        warm = warm + 1e-7 * np.random.default_rng(blocks).standard_normal(warm.shape)
        s = pkg.Sampler(model, warm, reproject_form=form, threads_per_chain=threads_per_chain)
        s.set_null_space(N)
        want, st = s.sample(2, 2, seed=1)
        assert st["reprojections"] > 0
        runs.append((s, want, torch.cuda.Stream(), torch.zeros(want.shape, dtype=torch.float64, device="cuda"), []))
    go = threading.Barrier(2)

    def work(s, want, stream, out, errors):
        go.wait()
        for _ in range(calls):
            try:
                s.sample_device(2, 2, out.data_ptr(), 2, stream=stream.cuda_stream, seed=1)
            except pkg.AchrError as e:
                errors.append(str(e))
                return

    threads = [threading.Thread(target=work, args=r) for r in runs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for s, want, _, out, errors in runs:
        assert not errors, errors[0]
        assert np.array_equal(out.cpu().numpy(), want)
        s.close()
