"""The two forms of the fused ensemble kernel (needs a GPU): a tile's members one after another on one
SM, or one member per CTA of a cluster. Both must give the same bits: the rows of a large call (whole
rounds of tiles, then a partial round) against the same rows asked for in small calls."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _server(members, seed):
    from tissuemc_b200 import surrogate as S

    ens = S.Ensemble(members=members, batch=256, seed=seed)
    rng = np.random.default_rng(seed)
    for m in ens.members:
        for b in m.b:
            b.copy_(torch.from_numpy(rng.normal(0, 0.05, b.shape[0]).astype(np.float32)))
    y_mean = np.concatenate([np.full(S.N_RD, -2.0), [0.05, 0.6]])
    y_std = np.concatenate([np.full(S.N_RD, 0.3), [0.02, 0.1]])
    ens.norm = S.Norm(np.zeros(S.N_FEAT), np.ones(S.N_FEAT), y_mean, y_std)
    return S.FusedServer(ens), rng


# 20,000 rows: one tile on every SM of a B200 and 9 tiles left over for the clusters; 5,000: clusters
# that walk more than one tile; 1 and 129: a partial tile
@pytest.mark.parametrize("members", [1, 2, 3, 4, 8])
@pytest.mark.parametrize("n", [1, 129, 5000, 20000])
def test_rows_do_not_depend_on_the_form(members, n):
    server, rng = _server(members, 11 + members)
    X = rng.normal(size=(n, 13)).astype(np.float32)
    spreads: list = []
    y, rd, route = server(X, spreads)
    for a in sorted({0, max(0, n - 300), n // 2}):
        b = min(n, a + 300)
        part: list = []
        y2, rd2, route2 = server(X[a:b], part)
        assert np.array_equal(y[a:b], y2) and np.array_equal(rd[a:b], rd2) and np.array_equal(route[a:b], route2)
        assert np.array_equal(spreads[0][a:b], part[0])
    pm = server.ens.predict_members(X)  # through the per-layer kernels
    # activations round to BF16 in both; an FP32 sum's last bit can move one to its neighbour
    assert np.abs(y - pm.mean(0)).max() <= 1e-2 * np.abs(pm.mean(0)).max()


@pytest.mark.parametrize("n_out,nbins", [(1, 0), (17, 16), (33, 33), (64, 64), (97, 64), (128, 40)])
@pytest.mark.parametrize("n", [200, 19200])
def test_output_counts(n_out, nbins, n):
    """Outputs and bins that end inside a warp's columns, in both forms: against the 128-output call's
    first columns and the definition of R_d."""
    import ctypes

    from tissuemc_b200 import surrogate as S

    server, rng = _server(3, 5)
    g = torch.Generator(device="cuda").manual_seed(3)
    for m in server.ens.members:  # all 128 outputs of the last layer in use
        m.Wb[-1].copy_(torch.randn(128, 512, device="cuda", generator=g) * 0.03)
    server = S.FusedServer(server.ens)
    X = torch.from_numpy(rng.normal(size=(n, 13)).astype(np.float32)).cuda()
    mean = torch.linspace(-2.5, -1.5, 128, device="cuda")
    std = torch.linspace(0.2, 0.3, 128, device="cuda")
    areas = torch.linspace(0.5, 1.5, 64, device="cuda")

    def call(no, nb, members=3):
        out = torch.full((n * no + 8,), -7.0, device="cuda")
        rd = torch.empty(n, device="cuda")
        S._call("tmc_b200_nn_ensemble_infer", S._p(server.packed), S._p(server.bias), members, S._p(X), n, 13,
                S._p(server.x_mean), S._p(server.x_std), no, S._p(mean), S._p(std), S._p(areas), nb,
                ctypes.c_float(0.01), S._p(out), S._p(rd), S._p(None), S._p(None),
                ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert bool((out[n * no:] == -7.0).all())
        return out[:n * no].view(n, no), rd

    full, _ = call(128, 64)
    out, rd = call(n_out, nbins)
    assert torch.equal(out, full[:, :n_out])
    # one member's R_d is the sum over its own outputs: float32 sums of positive terms, 10^y to 2 ulp
    one, rd1 = call(n_out, nbins, members=1)
    ref = (10.0 ** one[:, :nbins].double() * areas[:nbins].double()).sum(1)
    assert bool(((rd1.double() - ref).abs() <= 64 * 2.0 ** -22 * ref + 1e-30).all())
