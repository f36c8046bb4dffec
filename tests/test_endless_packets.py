"""A tissue that the validation accepts but that float32 cannot hold (mua = 1e-46, d = 1e39): every score is no
number until the step cap ends the packet. A run whose packets are walked alone must count as one whose
lanes walk them (needs a GPU)."""

from __future__ import annotations

import numpy as np
import pytest

import tissuemc_b200 as tmc

pytestmark = pytest.mark.gpu

MANY = 4_194_305  # more than 16 photons to each of the resident lanes: not walked alone


@pytest.mark.parametrize("cap", [13, 20, 23])
def test_scores_that_are_no_numbers(cap):
    spec = tmc.RunSpec(layers=[(1.0, 1e-46, 0.0, 0.0, 1e39)], dz=0.01, dr=0.01, nz=4, nr=3, na=2)
    few, many = (tmc.run(spec, tmc.options(seed=1, batches=1, photons=n, step_cap=cap)) for n in (7, MANY))
    # a photon's part of the absorbed weight and of A(r,z), modulo 2^64: 2^63 for every step (or 0)
    assert int(few.anomalies.sum()) % 7 == 0 and int(many.anomalies.sum()) == int(few.anomalies.sum()) // 7 * MANY
    per_photon = (cap % 2) << 63
    for r, n in ((few, 7), (many, MANY)):
        assert int(r.raw[4]) == (n * per_photon) % (1 << 64)
        assert int(r.raw[5:].sum(dtype=np.uint64)) == (n * per_photon) % (1 << 64)
