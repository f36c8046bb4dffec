"""How a walk's launch spreads its photons (needs a GPU): small runs leave lanes of their warps idle, so
every size around the places where the grid and the lanes change must give the tallies of the same run
cut into shards and of other block sizes, bit for bit."""

from __future__ import annotations

import numpy as np
import pytest

import tissuemc_b200 as tmc

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

# 148 SMs x 256 threads = 37,888 photons fill one block per SM; 4 such blocks are resident
SIZES = [1, 2, 31, 33, 1183, 1185, 2369, 37887, 37889, 75777, 151551, 151553, 400001]


@pytest.mark.parametrize("photons", SIZES)
def test_tallies_do_not_depend_on_the_spread(photons):
    spec = tmc.workload("slab_n14")
    batches = min(7, photons)
    opt = tmc.options(seed=5, batches=batches, photons=photons)
    ref = tmc.run(spec, opt)
    assert int(ref.photons.sum()) == photons and not ref.anomalies.any()
    for threads in (32, 96, 192):
        o = tmc.options(seed=5, batches=batches, photons=photons, threads_per_block=threads)
        assert np.array_equal(tmc.run(spec, o).raw, ref.raw), threads
    sz = tmc.query_sizes(spec, opt)
    buf = torch.zeros(int(sz.device_words), dtype=torch.int64, device="cuda")
    total = torch.zeros_like(buf)
    stream = torch.cuda.current_stream().cuda_stream
    for rank in range(min(3, photons)):
        first, count = tmc.shard_range(photons, rank, min(3, photons))
        tmc.run_device_range(spec, opt, first, count, buf.data_ptr(), stream)
        total += buf
    words = int(sz.tally_words)
    assert np.array_equal(total[:words].cpu().numpy().view(np.uint64), ref.raw)


def _shards_equal_whole(spec, photons, parts, **kw):
    """The whole run (a size that ends in its lanes) against the sum of its shards (sizes that walk their
    last packets alone)."""
    opt = tmc.options(seed=9, batches=10, photons=photons, **kw)
    whole = tmc.run(spec, opt)
    sz = tmc.query_sizes(spec, opt)
    buf = torch.zeros(int(sz.device_words), dtype=torch.int64, device="cuda")
    total = torch.zeros_like(buf)
    for rank in range(parts):
        first, count = tmc.shard_range(photons, rank, parts)
        tmc.run_device_range(spec, opt, first, count, buf.data_ptr(), torch.cuda.current_stream().cuda_stream)
        total += buf
    words = int(sz.tally_words)
    assert np.array_equal(total[:words].cpu().numpy().view(np.uint64), whole.raw)
    return whole


# mismatched indices, an isotropic layer, a thick weakly absorbing slab (long photons, many layers of
# roulette), a layer so thin that most steps meet a boundary
TISSUES = {
    "slab": [(1.4, 5.0, 95.0, 0.8, 0.05)],
    "mixed": [(1.37, 1.0, 100.0, 0.9, 0.1), (1.5, 1.0, 10.0, 0.0, 0.002), (1.33, 2.0, 10.0, -0.3, 0.2)],
    "thick": [(1.5, 0.5, 200.0, 0.9, 0.3)],
}


@pytest.mark.parametrize("tissue", sorted(TISSUES))
@pytest.mark.parametrize("step_cap", [0, 1, 13, 40])
def test_packets_walked_alone_give_the_same_tallies(tissue, step_cap):
    spec = tmc.RunSpec(layers=TISSUES[tissue], dz=0.005, dr=0.01, nz=21, nr=33, na=7)
    r = _shards_equal_whole(spec, 2_600_000, 2, step_cap=step_cap)  # 2.42e6 is the last size walked alone
    assert bool(r.anomalies.any()) == (step_cap in (1, 13, 40))


def test_packets_walked_alone_in_exact_math_and_without_profiles():
    spec = tmc.RunSpec(layers=TISSUES["mixed"], dz=0.005, dr=0.01, nz=21, nr=33, na=7)
    _shards_equal_whole(spec, 90_000, 3, fast_math=False)  # 75,776 is the last size in exact math
    _shards_equal_whole(spec, 2_600_000, 2, profiles=False, rung=6)


@pytest.mark.parametrize("fast", [1, 0])
@pytest.mark.parametrize("photons", [1, 40, 3000])
def test_small_sweeps_equal_single_runs(photons, fast):
    """Sweeps of few photons: blocks that switch configuration before their lanes are full, grids larger
    than a block's tile, one photon per configuration."""
    cfgs = tmc.sweep_sample(3, 37)
    for c in cfgs:
        c.photons = photons
    for nz, nr in ((64, 64), (5, 3), (130, 90)):
        opt = tmc.sweep_options(nz=nz, nr=nr, fast_math=fast, batches=1)
        res = tmc.sweep_run(cfgs, opt, raw=True)
        loop = tmc.sweep_run_loop(cfgs, opt, raw=True)
        assert np.array_equal(res.raw, loop.raw)
