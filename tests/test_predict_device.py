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


@pytest.mark.parametrize("form", ["float32 statistics", "statistics that broadcast", "a list of rows", "mixed statistics"])
def test_predict_of_other_forms_equals_numpy(form):
    from tissuemc_b200 import surrogate as S

    ens = S.Ensemble(members=2, batch=256, seed=4)
    rng = np.random.default_rng(5)
    norm = [rng.normal(size=13), rng.uniform(0.5, 2.0, 13), rng.normal(size=66), rng.uniform(0.1, 1.0, 66)]
    X = rng.normal(size=(300, 13)).astype(np.float32)
    if form == "float32 statistics":
        norm = [v.astype(np.float32) for v in norm]
    elif form == "statistics that broadcast":
        norm = [norm[0][:1], norm[1][None], norm[2][None], norm[3][:1]]
    elif form == "mixed statistics":
        norm = [norm[0].astype(np.float32), norm[1], norm[2], norm[3].astype(np.float32)]
    ens.norm = S.Norm(*norm)
    Xn = np.zeros((300, S.K_IN), np.float32)
    Xn[:, :13] = (X - ens.norm.x_mean) / ens.norm.x_std
    Xd = torch.from_numpy(Xn).cuda().bfloat16()
    given = X.tolist() if form == "a list of rows" else X
    if form == "a list of rows":  # numpy reads a list in float64
        Xn[:, :13] = (np.array(given) - ens.norm.x_mean) / ens.norm.x_std
        Xd = torch.from_numpy(Xn).cuda().bfloat16()
    ref = np.empty((2, 300, S.N_OUT))
    stream = torch.cuda.current_stream().cuda_stream
    for i, m in enumerate(ens.members):
        S._ensure_rows(m, 300)
        Z = torch.empty(300, S.N_OUT_PAD, device="cuda")
        ref[i] = m.forward(Xd, 300, stream, Z_out=Z)[:, :S.N_OUT].cpu().numpy() * ens.norm.y_std + ens.norm.y_mean
    assert np.array_equal(ens.predict_members(given), ref)
    assert np.array_equal(ens.predict(given), ref.mean(0))
