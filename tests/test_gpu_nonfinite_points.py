"""GPU: a NaN or an infinity among a block of points stays one: the chain's null-space coordinates are
NaN, the batched reprojection leaves NaN in every reaction the bad value's metabolites reach, and the
other chains are untouched."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import dense_S

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

# the quiet NaN of arithmetic, one of the other sign, and one with every fraction bit set (rounding it
# as an integer would carry into the sign)
BAD = [0x7FF8000000000000, 0xFFF8000000000000, 0x7FFFFFFFFFFFFFFF, 0x7FF0000000000000, 0xFFF0000000000000]


@pytest.fixture(scope="module")
def sampler(pkg, small_model, golden):
    with pkg.Sampler(small_model, golden["warmup"]) as s:
        s.set_null_space(golden["N"])
        yield s


def _points(sampler, P, bits, chain, reaction):
    good, _ = sampler.sample(P, 12, seed=4)
    bad = good.copy()
    bad[reaction, chain] = np.array([bits], np.uint64).view(np.float64)[0]
    return torch.from_numpy(good).cuda(), torch.from_numpy(bad).cuda()


@pytest.mark.parametrize("centred", [False, True])
@pytest.mark.parametrize("bits", BAD, ids=[f"{b:x}" for b in BAD])
def test_null_space_coordinates(sampler, bits, centred):
    P, chain = 40, 33
    good, bad = _points(sampler, P, bits, chain, 17)
    mu = good.mean(1).contiguous()
    out = []
    for x in (good, bad):
        Y = torch.zeros((sampler.precond_dim()[0], P), device="cuda")
        sampler.null_coords(P, x.data_ptr(), P, Y.data_ptr(), P, d_mu=mu.data_ptr() if centred else 0)
        out.append(Y)
    assert torch.isfinite(out[0]).all()
    assert torch.isnan(out[1][:, chain]).all()
    rest = [p for p in range(P) if p != chain]
    assert torch.equal(out[0][:, rest], out[1][:, rest])


@pytest.mark.parametrize("bits", BAD, ids=[f"{b:x}" for b in BAD])
def test_batched_reprojection(sampler, small_model, bits):
    P, chain = 40, 33
    S = dense_S(small_model)
    reaction = int(np.argmax((S != 0).sum(axis=0)))
    good, bad = _points(sampler, P, bits, chain, reaction)
    good += 1e-6 * torch.randn_like(good)  # (something to reproject in every chain)
    bad[:, [p for p in range(P) if p != chain]] = good[:, [p for p in range(P) if p != chain]]
    for x in (good, bad):
        sampler.reproject(P, x.data_ptr(), P, max_rounds=1, with_stats=False)
    touched = np.flatnonzero((S != 0).any(axis=0))  # every z of the chain is NaN
    assert torch.isfinite(good).all()
    assert torch.isnan(bad[touched.tolist(), chain]).all()
    rest = [p for p in range(P) if p != chain]
    assert torch.equal(good[:, rest], bad[:, rest])
