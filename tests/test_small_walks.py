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
