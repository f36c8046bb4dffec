"""Ensemble.predict's float64 arithmetic on the device (needs a GPU): the bits of the same formulas in
numpy, from the members' own outputs."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("members", [1, 3])
@pytest.mark.parametrize("rows", [1, 37, 129, 65537])  # the last: one row beyond a chunk
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_predict_equals_numpy(members, rows, dtype):
    from tissuemc_b200 import surrogate as S

    ens = S.Ensemble(members=members, batch=256, seed=4)
    rng = np.random.default_rng(rows)
    ens.norm = S.Norm(rng.normal(size=13), rng.uniform(0.5, 2.0, 13), rng.normal(size=66), rng.uniform(0.1, 1.0, 66))
    X = rng.normal(size=(rows, 13)).astype(dtype)
    Xn = np.zeros((rows, S.K_IN), np.float32)
    Xn[:, :13] = (X - ens.norm.x_mean) / ens.norm.x_std
    Xd = torch.from_numpy(Xn).cuda().bfloat16()
    assert torch.equal(ens._x(X), Xd)
    ref = np.empty((members, rows, S.N_OUT))
    stream = torch.cuda.current_stream().cuda_stream
    for i, m in enumerate(ens.members):
        S._ensure_rows(m, rows)
        Z = torch.empty(rows, S.N_OUT_PAD, device="cuda")
        ref[i] = m.forward(Xd, rows, stream, Z_out=Z)[:, :S.N_OUT].cpu().numpy() * ens.norm.y_std + ens.norm.y_mean
    assert np.array_equal(ens.predict_members(X), ref)
    assert np.array_equal(ens.predict(X), ref.mean(0))
