"""The walk's autotuner times the kernel that the whole run will take, whatever the size of its sample (needs
a GPU)."""

from __future__ import annotations

import pytest

import tissuemc_b200 as tmc

pytestmark = pytest.mark.gpu


def test_the_sample_runs_the_whole_runs_kernel():
    """A run of 200,000 photons walks its last packets alone and ends in two thirds of the time (3.0 against
    4.4 ms) of a sample of as many photons of a long run, whose kernel does not."""
    spec = tmc.workload("skin5")
    small = min(tmc.run(spec, photons=200_000, batches=10, seed=1).kernel_seconds for _ in range(5))
    _, _, sample, _ = tmc.autotune(spec, tmc.options(seed=1, batches=10, photons=100_000_000), sample_photons=200_000)
    assert sample > 1.15 * small
    _, _, whole, _ = tmc.autotune(spec, tmc.options(seed=1, batches=10, photons=200_000), sample_photons=200_000)
    assert whole < 1.15 * small
