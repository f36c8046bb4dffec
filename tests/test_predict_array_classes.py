"""Which arrays Ensemble.predict's device arithmetic takes: those whose numpy arithmetic is plain float64. A masked
array's operations leave its hidden elements as they are, so it stays with numpy."""

from __future__ import annotations

import numpy as np
import pytest

from tissuemc_b200 import surrogate as S


def _forms(tmp_path):
    rng = np.random.default_rng(2)
    X, mean, std = rng.normal(size=(40, 13)), rng.normal(size=13), rng.uniform(0.5, 2.0, 13)
    on_disk = np.memmap(tmp_path / "x", dtype=np.float64, mode="w+", shape=X.shape)
    on_disk[:] = X
    masked = np.ma.masked_array(X, mask=rng.random(X.shape) < 0.3)
    return [("plain", X, mean, std, True), ("on disk", on_disk, mean, std, True), ("rows", X.tolist(), mean, std, True),
            ("masked", masked, mean, std, False), ("matrix", np.asmatrix(X), mean, std, False),
            ("masked mean", X, np.ma.masked_array(mean), std, False), ("masked std", X, mean, np.ma.masked_array(std), False)]


def test_only_plain_float64_arrays_go_to_the_device(tmp_path):
    for name, X, mean, std, plain in _forms(tmp_path):
        assert S._float64_vectors(13, X, mean, std) == plain, name


@pytest.mark.gpu
def test_network_inputs_of_every_array_class_are_numpys(tmp_path):
    torch = pytest.importorskip("torch")
    ens = S.Ensemble(members=1, batch=256, seed=4)
    for name, X, mean, std, _ in _forms(tmp_path):
        ens.norm = S.Norm(mean, std, np.zeros(66), np.ones(66))
        Xn = np.zeros((40, S.K_IN), np.float32)
        Xn[:, :13] = (X - mean) / std
        assert torch.equal(ens._x(X), torch.from_numpy(Xn).cuda().bfloat16()), name


@pytest.mark.gpu
def test_predict_members_of_no_members_is_empty():
    ens = S.Ensemble(members=0, batch=256)
    ens.norm = S.Norm(np.zeros(13), np.ones(13), np.zeros(66), np.ones(66))
    assert ens.predict_members(np.zeros((5, 13))).shape == (0, 5, S.N_OUT)
