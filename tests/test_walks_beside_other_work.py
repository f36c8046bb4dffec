"""Walks too small to fill their warps' lanes, launched while other kernels hold part of the GPU (needs a
GPU): their blocks then start at different times, and the tallies must still be those of the run alone."""

from __future__ import annotations

import numpy as np
import pytest

import tissuemc_b200 as tmc

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


# 3 to 16 lanes a warp in 148 blocks of 8 warps in fast math, 2 to 8 in exact math: more than a block walks alone
# from the start, but few enough for one warp's lanes alone to be below the limit (16 packets a block, 8)
@pytest.mark.parametrize("fast, photons", [(True, 2500), (True, 3552), (True, 5000), (True, 10_000), (True, 18_944),
                                           (False, 1500), (False, 2369), (False, 9000)])
def test_small_walk_beside_a_large_one(fast, photons):
    spec = tmc.workload("slab_n14")
    opt = tmc.options(seed=3, batches=10, photons=photons, fast_math=fast)
    alone = tmc.run(spec, opt)
    launched = photons * (1.0 - alone.specular)
    assert abs(float(alone.rd.sum() + alone.tt.sum() + alone.absorbed.sum()) - launched) < 1e-3 * photons  # roulette
    sz = tmc.query_sizes(spec, opt)
    words = int(sz.tally_words)
    large = tmc.options(seed=1, batches=10, photons=400_000)
    large_buf = torch.zeros(int(tmc.query_sizes(spec, large).device_words), dtype=torch.int64, device="cuda")
    bufs = [torch.zeros(int(sz.device_words), dtype=torch.int64, device="cuda") for _ in range(12)]
    here, beside = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    for buf in bufs:  # small launches keep arriving while the large ones come and go
        tmc.run_device(spec, large, large_buf.data_ptr(), beside.cuda_stream)
        tmc.run_device(spec, opt, buf.data_ptr(), here.cuda_stream)
    torch.cuda.synchronize()
    for buf in bufs:
        assert np.array_equal(buf[:words].cpu().numpy().view(np.uint64), alone.raw)
