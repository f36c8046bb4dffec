"""The work whose speed is measured: what programs that use this package have it do, through its
public entry points, from the smallest calls to the largest.

Six kinds of case, one for each path a user's program calls:

  walk     ``tmc.run``: one Monte Carlo run of a layered tissue, tallies back on the host
  sweep    ``tmc.sweep_run``: many tissues in one launch, as a parameter study or the surrogate's
           training data need them
  grad     ``surrogate.Member.forward`` and ``backward``: the loss and every gradient of one network
           on one batch, as a training loop of the user's own calls them
  train    ``surrogate.Ensemble.train``: the ensemble's own training loop
  predict  ``surrogate.Ensemble.predict``: the forward pass an inverse fit makes at every iteration
  serve    ``surrogate.FusedServer``: gated queries, from host arrays (the whole call) or between
           device buffers (``launch``)

Every input comes from the seed alone.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import tissuemc_b200 as tmc
from tissuemc_b200 import surrogate as sg

DEV = "cuda:0"

# (n, mua, mus, g, d) per layer, the grid, the mean interactions and boundary steps of a photon
TISSUES = {
    # the bundled homogeneous slab, n = 1.4 in air
    "slab": dict(layers=[(1.4, 5.0, 95.0, 0.8, 0.05)], dz=0.0025, dr=0.005, nz=20, nr=50, na=30, steps=(19.71, 2.03)),
    # the three-layer tissue of the MCML manual's tables 6.6 and 6.7 (one isotropic layer, n = 1.37
    # in air), on an odd grid with exit angles
    "three": dict(layers=[(1.37, 1.0, 100.0, 0.9, 0.1), (1.37, 1.0, 10.0, 0.0, 0.1), (1.37, 2.0, 10.0, 0.7, 0.2)],
                  dz=0.01, dr=0.01, nz=41, nr=53, na=11, steps=(60.31, 5.84)),
    # the bundled five-layer skin stack, whose tallies are larger than shared memory
    "skin5": dict(layers=[(1.4, 4.0, 400.0, 0.8, 0.01), (1.4, 2.0, 300.0, 0.85, 0.02), (1.4, 1.0, 200.0, 0.9, 0.1),
                          (1.4, 0.5, 150.0, 0.9, 0.2), (1.4, 0.3, 100.0, 0.9, 1.0)],
                  dz=0.001, dr=0.002, nz=400, nr=500, na=30, steps=(604.20, 14.30)),
}
SWEEP_STEPS = (141.1, 3.8)  # the sweep distribution, weighted by photons
# operations of one interaction and one boundary step (float32 and special functions)
STEP_OPS = (61 + 12, 25 + 3)
IN, HIDDEN, OUT, OUT_PAD = 13, 512, 66, 128
DIMS = [(64, HIDDEN), (HIDDEN, HIDDEN), (HIDDEN, HIDDEN), (HIDDEN, HIDDEN), (HIDDEN, OUT_PAD)]  # (in, out)
MACS = IN * HIDDEN + 3 * HIDDEN * HIDDEN + HIDDEN * OUT  # multiply-adds of one member for one query
MEMBERS = 4
WEIGHTS = sum(k * n + n for k, n in DIMS)


def listed():
    return [
        # a first look at a tissue: few photons, the call's fixed costs and one photon's latency
        dict(name="walk_slab_1e4", kind="walk", tissue="slab", photons=10_000, batches=10, fast=True),
        # the bundled slab as its .mci asks for it
        dict(name="walk_slab_1e6", kind="walk", tissue="slab", photons=1_000_000, batches=10, fast=True),
        # a layered tissue in exact math, an odd number of photons, uneven batches
        dict(name="walk_three_exact", kind="walk", tissue="three", photons=300_007, batches=16, fast=False),
        # the bundled skin stack as its .mci asks for it: the longest single run
        dict(name="walk_skin5_1e8", kind="walk", tissue="skin5", photons=100_000_000, batches=100, fast=True),
        # the Monte Carlo solves that verify a few fits, with their whole tallies
        dict(name="sweep_97", kind="sweep", configs=97, photons=100_000, raw=True),
        # the parameter study: 4096 tissues, 1e4 to 1e6 photons each
        dict(name="sweep_4096", kind="sweep", configs=4096, photons=0, raw=False),
        # one network's gradients on the training batch
        dict(name="grad_4096", kind="grad", batch=4096),
        # a short training of the ensemble (16 batches an epoch)
        dict(name="train_65536", kind="train", rows=65536, epochs=25, batch=4096),
        # one iteration of 1000 inverse fits in four parameters: 8 perturbed inputs a fit
        dict(name="predict_8000", kind="predict", rows=8000),
        # a handful of queries from an interactive client, host to host
        dict(name="serve_100", kind="serve", rows=100, device=False),
        # one serving batch whose inputs and outputs stay on the device
        dict(name="serve_65536_device", kind="serve", rows=65536, device=True),
        # the serving run: a million queries from pinned host memory, all results on the host
        dict(name="serve_1e6", kind="serve", rows=1_000_000, device=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["walk", "walk", "sweep", "grad", "train", "predict", "serve", "serve"])
    if kind == "walk":
        tissue = rng.choice(sorted(TISSUES))
        fast = rng.random() < 0.75
        top = {"slab": 1e8, "three": 1e8, "skin5": 6e7}[tissue] if fast else 2e7
        return dict(kind=kind, tissue=tissue, photons=_log(rng, 1e4, top), batches=rng.choice([1, 7, 10, 64, 100]),
                    fast=fast)
    if kind == "sweep":
        n = _log(rng, 16, 3000)
        return dict(kind=kind, configs=n, photons=rng.choice([0, _log(rng, 1e4, 2e5)]), raw=n <= 512 and rng.random() < 0.5)
    if kind == "grad":
        return dict(kind=kind, batch=64 * _log(rng, 4, 128))
    if kind == "train":
        return dict(kind=kind, rows=rng.randint(16384, 65536), epochs=rng.randint(2, 25), batch=rng.choice([1024, 2048, 4096]))
    if kind == "predict":
        return dict(kind=kind, rows=_log(rng, 64, 65536))
    return dict(kind=kind, rows=_log(rng, 16, 1_000_000), device=rng.random() < 0.5)


# ------------------------------------------------------------------------------ inputs
def _features(seed, n):
    """Raw features of n tissues of the sweep distribution (1 to 3 layers), float64 (n, 13)."""
    r = np.random.default_rng(seed)
    x = np.zeros((n, IN))
    layers = r.integers(1, 4, n)
    for l in range(3):
        there = layers > l
        x[:, 4 * l + 0] = np.where(there, r.uniform(-2.0, 1.0, n), 0.0)               # log10 mua
        x[:, 4 * l + 1] = np.where(there, r.uniform(0.0, math.log10(50.0), n), 0.0)   # log10 mus'
        x[:, 4 * l + 2] = np.where(there, r.uniform(0.7, 0.95, n), 0.0)               # g
        x[:, 4 * l + 3] = np.where(there, r.uniform(-2.0, 0.0, n), -3.0)              # log10 d (-3: absent)
    x[:, 12] = r.uniform(1.33, 1.5, n)
    return x


def _norm():
    """Means and standard deviations of the inputs and of log10 R_d(r), T_t, A."""
    x = _features(12345, 4096)
    return (x.mean(0), x.std(0), np.concatenate([np.linspace(1.0, -3.2, 64), [0.2, 0.5]]),
            np.concatenate([np.linspace(0.6, 1.0, 64), [0.25, 0.25]]))


def _weights(seed, members):
    """Float32 weights and biases of an ensemble whose members agree to about a percent, as members
    trained on the same data do."""
    g = torch.Generator(device="cpu").manual_seed(seed)
    base = []
    for i, (k, n) in enumerate(DIMS):
        w = torch.randn(n, k, generator=g) * math.sqrt(2.0 / (IN if i == 0 else k))
        b = torch.randn(n, generator=g) * 0.05
        if i == 0:
            w[:, IN:] = 0.0
        if i == len(DIMS) - 1:
            w, b = 0.5 * w, 0.5 * b
            w[OUT:] = 0.0
            b[OUT:] = 0.0
        base.append((w, b))
    if members == 1:
        return [base]
    return [[(w * (1.0 + 0.004 * torch.randn(w.shape, generator=g)), b) for w, b in base] for _ in range(members)]


def _load(member, weights):
    for i, (w, b) in enumerate(weights):
        member.W[i].copy_(w)
        member.b[i].copy_(b)
        member.Wb[i].copy_(member.W[i])
        member.WT[i].copy_(member.W[i].t())


def _ensemble(seed, batch):
    ens = sg.Ensemble(members=MEMBERS, batch=batch, seed=seed % 1000, device=DEV)
    for m, w in zip(ens.members, _weights(seed, MEMBERS), strict=True):
        _load(m, w)
    ens.norm = sg.Norm(*_norm())
    return ens


def _targets(x, seed):
    """Smooth targets with a little noise, in the units of the network's outputs."""
    r = np.random.default_rng(seed + 1)
    xm, xs, ym, ys = _norm()
    h = np.tanh((x - xm) / xs @ r.standard_normal((IN, 32)) * 0.3)
    return (h @ r.standard_normal((32, OUT)) / math.sqrt(16.0) + 0.02 * r.standard_normal((len(x), OUT))) * ys + ym


def prepare(case, seed):
    kind = case["kind"]
    if kind == "walk":
        t = TISSUES[case["tissue"]]
        spec = tmc.RunSpec(layers=t["layers"], photons=case["photons"], dz=t["dz"], dr=t["dr"], nz=t["nz"], nr=t["nr"],
                           na=t["na"])
        return dict(kind=kind, spec=spec, opt=tmc.options(seed=seed, batches=case["batches"], fast_math=case["fast"]))
    if kind == "sweep":
        cfgs = tmc.sweep_sample(seed, case["configs"])
        if case["photons"]:
            for c in cfgs:
                c.photons = case["photons"]
        return dict(kind=kind, cfgs=cfgs, opt=tmc.sweep_options(), raw=case["raw"])
    if kind == "grad":
        b = case["batch"]
        m = sg.Member(b, seed % 1000, DEV)
        _load(m, _weights(seed, 1)[0])
        x, y = _grad_batch(case, seed)
        return dict(kind=kind, m=m, x=x.to(DEV).to(torch.bfloat16), y=y.to(DEV), scale=1.0 / (b * OUT))
    if kind == "train":
        x = _features(seed, case["rows"])
        return dict(kind=kind, ens=_ensemble(seed, case["batch"]), x=x, y=_targets(x, seed), epochs=case["epochs"])
    if kind == "predict":
        return dict(kind=kind, ens=_ensemble(seed, 256), x=_features(seed, case["rows"]))
    n = case["rows"]
    s = dict(kind=kind, server=sg.FusedServer(_ensemble(seed, 256)), device=case["device"], n=n)
    x = torch.from_numpy(_features(seed, n).astype(np.float32))
    if case["device"]:
        f32 = dict(dtype=torch.float32, device=DEV)
        s.update(x=x.to(DEV), out=torch.empty(n, OUT, **f32), rd=torch.empty(n, **f32), spread=torch.empty(n, **f32),
                 route=torch.empty(n, dtype=torch.uint8, device=DEV))
    else:
        s["x"] = x.pin_memory()
    return s


def _grad_batch(case, seed):
    """Normalised inputs (padded to 64 columns) and targets of one batch, float32 on the host."""
    xm, xs, ym, ys = _norm()
    raw = _features(seed, case["batch"])
    x = torch.zeros(case["batch"], 64)
    x[:, :IN] = torch.from_numpy((raw - xm) / xs)
    return x, torch.from_numpy((_targets(raw, seed) - ym) / ys).float()


# ------------------------------------------------------------------------------ one pass
def run(state):
    kind = state["kind"]
    if kind == "walk":
        r = tmc.run(state["spec"], state["opt"])
        return dict(rd=r.rd, tt=r.tt, absorbed=r.absorbed, events=r.events.view(np.int64),
                    anomalies=r.anomalies.view(np.int64), a_z=r.a_z, rd_r=r.rd_r, tt_r=r.tt_r, a_rz=r.a_rz, rd_ra=r.rd_ra,
                    tt_ra=r.tt_ra, raw=r.raw.view(np.int64), specular=r.specular)
    if kind == "sweep":
        r = tmc.sweep_run(state["cfgs"], state["opt"], raw=state["raw"])
        return dict(summary=r.summary, raw=r.raw.view(np.int64) if r.raw is not None else None)
    if kind == "grad":
        m, s = state["m"], torch.cuda.current_stream().cuda_stream
        m.forward(state["x"], m.B, s)
        m.backward(state["x"], state["y"], s, state["scale"])
        return dict(z=m.Z[-1], loss=m.loss, gw=m.gW, gb=m.gb)
    if kind == "train":
        ens = state["ens"]
        ens.train(state["x"], state["y"], epochs=state["epochs"], ema=0.999)
        return dict(loss=np.array(ens.history[-state["epochs"]:]), w=[m.W for m in ens.members], b=[m.b for m in ens.members])
    if kind == "predict":
        return state["ens"].predict(state["x"])
    if state["device"]:
        state["server"].launch(state["x"], state["n"], state["out"], state["rd"], state["spread"], state["route"],
                               torch.cuda.current_stream().cuda_stream)
        return dict(y=state["out"], rd=state["rd"], spread=state["spread"], route=state["route"])
    y, rd, route = state["server"](state["x"], copy=False)
    return dict(y=y, rd=rd, route=route)


# ------------------------------------------------------------------------------ the least a pass does
def work(case):
    kind = case["kind"]
    if kind == "walk":
        t = TISSUES[case["tissue"]]
        words = case["batches"] * (4 + len(t["layers"])) + t["nr"] * t["nz"] + 2 * t["nr"] * t["na"]
        return dict(bytes=8 * words, flops=case["photons"] * sum(a * b for a, b in zip(t["steps"], STEP_OPS, strict=True)))
    if kind == "sweep":
        mean = case["photons"] or (1e6 - 1e4) / math.log(100.0)
        words = (10 * 7 + 64 * 64 + 2 * 64) if case["raw"] else 67
        return dict(bytes=case["configs"] * 8 * words,
                    flops=case["configs"] * mean * sum(a * b for a, b in zip(SWEEP_STEPS, STEP_OPS, strict=True)))
    if kind == "grad":  # forward, gradients of the weights, gradients of the activations but the inputs'
        b = case["batch"]
        return dict(bytes=b * (2 * IN + 4 * OUT + 4 * OUT_PAD) + WEIGHTS * (2 + 4), flops=2 * b * (3 * MACS - IN * HIDDEN))
    if kind == "train":  # a step reads and writes weights, moments and averages
        steps = case["epochs"] * (case["rows"] // case["batch"])
        return dict(bytes=steps * MEMBERS * (case["batch"] * (2 * IN + 4 * OUT) + WEIGHTS * 32),
                    flops=2 * steps * MEMBERS * case["batch"] * (3 * MACS - IN * HIDDEN))
    out = 8 * OUT if kind == "predict" else 4 * OUT + 5
    return dict(bytes=case["rows"] * (4 * IN + out) + MEMBERS * 2 * WEIGHTS, flops=2 * case["rows"] * MEMBERS * MACS)


# ------------------------------------------------------------------------------ in 64 bits
def _gelu(x):
    return 0.5 * x * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (x + 0.044715 * x ** 3)))


def _outputs(x, weights):
    """One member's 128 output columns for float64 inputs (rows, 64)."""
    for i, (w, b) in enumerate(weights):
        x = x @ w.to(x).t() + b.to(x)
        if i < len(weights) - 1:
            x = _gelu(x)
    return x


def exact(case, seed):
    kind = case["kind"]
    if kind in ("walk", "sweep", "train"):
        return None  # random walks have no exact value; a training follows the roundings of all its steps
    if kind == "grad":
        x, y = (t.double().to(DEV) for t in _grad_batch(case, seed))
        ws = [tuple(t.double().to(DEV).requires_grad_() for t in p) for p in _weights(seed, 1)[0]]
        z = _outputs(x, ws)
        loss = ((z[:, :OUT] - y) ** 2).sum() / (case["batch"] * OUT)
        loss.backward()
        return dict(z=z.detach(), loss=loss.detach().reshape(1), gw=[w.grad for w, _ in ws], gb=[b.grad for _, b in ws])
    xm, xs, ym, ys = (torch.from_numpy(v).to(DEV) for v in _norm())
    raw = _features(seed, case["rows"])
    x = torch.zeros(case["rows"], 64, dtype=torch.float64, device=DEV)
    given = raw if kind == "predict" else raw.astype(np.float32)
    x[:, :IN] = (torch.from_numpy(given).to(DEV).double() - xm) / xs
    mean, rds = 0.0, []
    r = torch.arange(64, dtype=torch.float64, device=DEV)
    areas = math.pi * ((r + 1) ** 2 - r ** 2) * 0.01 * 0.01
    for w in _weights(seed, MEMBERS):
        ws = [(a.to(DEV), b.to(DEV)) for a, b in w]
        y = torch.cat([_outputs(c, ws)[:, :OUT] for c in x.split(65536)]) * ys + ym
        mean = mean + y / MEMBERS
        rds.append((10.0 ** y[:, :64] * areas).sum(1))
    if kind == "predict":
        return mean
    rd = torch.stack(rds)
    # members this close differ by their bfloat16 roundings too: the spread and the route have no exact value
    whole = dict(y=mean, rd=rd.mean(0), route=None)
    return dict(whole, spread=None) if case["device"] else whole
