"""The work that users of this library have it do, as measurable cases.

A case is one call (or one training step) through a public entry point:

    plan       a captured FBME plan replayed on new observations
               (``make_stable_plan`` / ``make_fastest_plan``)
    uneven     a captured plan over scenes of different shapes
    learned    the plan with the learned warm start and its fallback
    certified  a captured ``certified_hybrid_uamp`` plan
    cg         ``sbl_2d`` with ``mode="cg"``
    dense      ``sbl_2d`` in its default mode at a small sample count
               (resolves to the exact dense posterior)
    train      one training step of the warm-start network

``listed`` gives the fixed cases, ``draw`` further ones of the same ranges.
``exact`` restates the paths in 64-bit torch, written from the equations,
for those that have a 64-bit value: not for cg (a Hutchinson estimate from
a PCG iteration stopped at a tolerance) and not for the learned plan (the
BF16 network decides where the solve starts).
"""

import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fbme-sbl_b200"))

from fbme_b200.learned import WarmStartNet, make_learned_plan  # noqa: E402
from fbme_b200.uneven import make_uneven_plan  # noqa: E402
from torch_sbl import SBLConfig, make_cuda_graph_sbl_plan, sbl_2d  # noqa: E402
from torch_sbl_fastest_stable import make_fastest_plan, make_stable_plan  # noqa: E402

EPS = float(np.finfo(np.float32).eps)    # the solver's FP32 constants: loading,
TINY = float(np.finfo(np.float32).tiny)  # gate margin and floors are defined by them
K = 32                                   # active-set size of the locked profiles
EXCHANGE = 12                            # FBME-Stable's exchange candidates


def _plan(name, profile, scenes, grid, prefix, scene="points", snr=15.0, masked=False):
    return dict(name=name, path="plan", profile=profile, scenes=scenes, n1=grid[0], n2=grid[1], m1=prefix[0],
                m2=prefix[1], scene=scene, snr=snr, masked=masked)


def listed():
    return [
        # the published single-scene example: the smallest replay, pure latency
        _plan("stable-1x40x32", "stable", 1, (40, 32), (20, 16), snr=10.0),
        # one scene at a time in a real-time loop, the minimum-latency profile
        _plan("fast-1x256x256", "fast", 1, (256, 256), (128, 128)),
        # a batch on a grid that is no FFT length, odd prefix
        _plan("fast-24x200x180", "fast", 24, (200, 180), (101, 77)),
        # missing samples: one observation mask shared by the batch
        _plan("stable-masked-16x256x256", "stable", 16, (256, 256), (128, 128), masked=True),
        # the throughput workload: a large batch of equal scenes
        _plan("stable-512x256x256", "stable", 512, (256, 256), (128, 128)),
        # the largest grid: clustered scatterers, rectangular prefix
        _plan("stable-32x512x512", "stable", 32, (512, 512), (256, 192), scene="clusters", snr=20.0),
        # scenes of many shapes in one plan
        dict(name="uneven-64", path="uneven", profile="stable", scenes=64, shapes=0),
        # the learned warm start with its on-device fallback
        dict(name="learned-512x256x256", path="learned", scenes=512, n1=256, n2=256, m1=128, m2=128),
        # certified solves: whole-grid evidence certificate and one repair
        dict(name="certified-64x256x256", path="certified", scenes=64, n1=256, n2=256, m1=128, m2=128, snr=15.0),
        # the matrix-free EM solver at a sample count above the dense limit
        dict(name="cg-8x256x256", path="cg", scenes=8, n1=256, n2=256, m1=128, m2=128, iters=6),
        # the default call on a small scene
        dict(name="dense-1x64x64", path="dense", scenes=1, n1=64, n2=64, m1=32, m2=32, iters=30),
        # training the warm-start network: features, forward, backward, Adam
        dict(name="train-16x256x256", path="train", batch=16, n1=256, n2=256),
    ]


_FFT_LENGTHS = (32, 48, 64, 96, 128, 192, 256, 384, 512)
_UNEVEN_GRIDS = ((128, 128), (192, 256), (256, 256), (384, 256))


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _prefix(rng, n):
    return max(8, int(round(rng.uniform(0.3, 0.7) * n)))


def draw(rng: random.Random):
    path = rng.choices(("plan", "uneven", "learned", "certified", "cg", "dense", "train"),
                       (12, 2, 2, 1, 1, 1, 1))[0]
    if path == "plan":
        if rng.random() < 0.75:
            n1, n2 = rng.choice(_FFT_LENGTHS), rng.choice(_FFT_LENGTHS)
        else:  # any length
            n1, n2 = _log_int(rng, 32, 400), _log_int(rng, 32, 400)
        most = max(1, min(512, 512 * 65536 // (4 * n1 * n2)))
        return dict(path="plan", profile=rng.choice(("stable", "fast")), scenes=_log_int(rng, 1, most), n1=n1, n2=n2,
                    m1=_prefix(rng, n1), m2=_prefix(rng, n2), scene=rng.choice(("points", "clusters")),
                    snr=round(rng.uniform(5.0, 25.0), 1), masked=rng.random() < 0.15)
    if path == "uneven":
        return dict(path="uneven", profile=rng.choice(("stable", "fast")), scenes=_log_int(rng, 4, 64),
                    shapes=rng.randrange(1, 1 << 20))
    if path == "learned":
        return dict(path="learned", scenes=_log_int(rng, 16, 512), n1=256, n2=256, m1=128, m2=128)
    if path == "certified":
        n1, n2 = rng.choice(_FFT_LENGTHS[2:7]), rng.choice(_FFT_LENGTHS[2:7])
        return dict(path="certified", scenes=_log_int(rng, 1, 64), n1=n1, n2=n2, m1=_prefix(rng, n1),
                    m2=_prefix(rng, n2), snr=round(rng.uniform(5.0, 25.0), 1))
    if path == "cg":
        n1, n2 = rng.choice((96, 128, 192, 256)), rng.choice((96, 128, 192, 256))
        return dict(path="cg", scenes=rng.randint(2, 8), n1=n1, n2=n2, m1=max(48, _prefix(rng, n1)),
                    m2=max(48, _prefix(rng, n2)), iters=rng.randint(3, 6))
    if path == "dense":
        n1, n2 = rng.choice((32, 48, 64)), rng.choice((32, 48, 64))
        return dict(path="dense", scenes=1, n1=n1, n2=n2, m1=n1 // 2 - rng.randint(0, 3), m2=n2 // 2 - rng.randint(0, 3),
                    iters=rng.randint(8, 30))
    n1, n2 = rng.choice((128, 192, 256)), rng.choice((128, 192, 256))
    return dict(path="train", batch=rng.randint(4, 16), n1=n1, n2=n2)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _randn_c(g, *shape):
    return torch.complex(torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64),
                         torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64))


def _scenes(seed, b, n1, n2, kind="points", points=None):
    """Sparse images [b, n1, n2] complex128: points with Rayleigh magnitudes
    and uniform phases at random pixels (their number K, or K ~ U{lo..hi} per
    scene), or clusters of log-normal points around random centres."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = n1 * n2
    if kind == "points":
        lo, hi = points or (max(20, n // 330),) * 2
        idx = torch.randint(0, n, (b, hi), generator=g, device="cuda")
        count = torch.randint(lo, hi + 1, (b, 1), generator=g, device="cuda")
        a = _randn_c(g, b, hi) * (torch.arange(hi, device="cuda") < count)
    else:
        per, iso = max(1, n // 350), max(1, n // 5000)
        c1 = torch.rand(b, 10, 1, generator=g, device="cuda") * n1
        c2 = torch.rand(b, 10, 1, generator=g, device="cuda") * n2
        o1 = 6.0 * torch.randn(b, 10, per // 10 + 1, generator=g, device="cuda")
        o2 = 6.0 * torch.randn(b, 10, per // 10 + 1, generator=g, device="cuda")
        i1, i2 = (c1 + o1).round().long() % n1, (c2 + o2).round().long() % n2
        idx = torch.cat([(i1 * n2 + i2).reshape(b, -1), torch.randint(0, n, (b, iso), generator=g, device="cuda")], 1)
        mag = torch.randn(idx.shape, generator=g, device="cuda", dtype=torch.float64).exp()
        phase = 2.0 * math.pi * torch.rand(idx.shape, generator=g, device="cuda", dtype=torch.float64)
        a = torch.polar(mag, phase)
    idx = idx.sort(1).values  # one amplitude a pixel, whatever order the sums run in
    again = torch.zeros_like(idx, dtype=torch.bool)
    again[:, 1:] = idx[:, 1:] == idx[:, :-1]
    x = torch.zeros(b, n, dtype=torch.complex128, device="cuda")
    return x.scatter_add(1, idx, a.masked_fill(again, 0.0)).view(b, n1, n2), g


def _observe(x, g, m1, m2, snr_db):
    """Noisy complex64 prefix block of the unnormalised 2-D DFT of ``x``."""
    clean = torch.fft.fft2(x)[:, :m1, :m2]
    power = clean.abs().square().mean((1, 2), keepdim=True)
    noise = (power / (10.0 ** (snr_db / 10.0)) / 2.0).sqrt() * _randn_c(g, *clean.shape)
    return (clean + noise).to(torch.complex64).contiguous()


def _observations(case, seed):
    b, n1, n2, m1, m2 = (case[k] for k in ("scenes", "n1", "n2", "m1", "m2"))
    points = (100, 400) if case["path"] == "learned" else None
    parts, step = [], max(1, (1 << 25) // (n1 * n2))
    for i, b0 in enumerate(range(0, b, step)):
        x, g = _scenes(seed * 1009 + i, min(step, b - b0), n1, n2, case.get("scene", "points"), points)
        snr = case.get("snr")
        if snr is None:  # a spread of noise levels
            snr = 5.0 + 20.0 * torch.rand(x.shape[0], 1, 1, generator=g, device="cuda", dtype=torch.float64)
        parts.append(_observe(x, g, m1, m2, snr))
    return torch.cat(parts)


def _mask(case):
    """The plan's observation mask: a random 70 % of the samples."""
    if not case.get("masked"):
        return None
    g = torch.Generator(device="cuda").manual_seed(17)
    return torch.rand(case["m1"], case["m2"], generator=g, device="cuda") < 0.7


def _uneven_shapes(case):
    rng = random.Random(case["shapes"])
    grids = [_UNEVEN_GRIDS[rng.randrange(len(_UNEVEN_GRIDS))] for _ in range(case["scenes"])]
    return [(g, (_prefix(rng, g[0]), _prefix(rng, g[1]))) for g in grids]


def _uneven_observations(case, seed):
    rng = random.Random(seed)
    ys = []
    for i, ((n1, n2), (m1, m2)) in enumerate(_uneven_shapes(case)):
        count = max(1, int(round(rng.uniform(0.01, 0.03) * n1 * n2)))
        x, g = _scenes(seed * 1009 + i, 1, n1, n2, "points", (count, count))
        ys.append(_observe(x, g, m1, m2, rng.uniform(5.0, 25.0))[0])
    return ys


def _training_batch(case, seed):
    """Backprojections of half-prefix observations and the log-power targets."""
    b, n1, n2 = case["batch"], case["n1"], case["n2"]
    x, g = _scenes(seed * 1009, b, n1, n2, "points", (100, 400))
    y = _observe(x, g, n1 // 2, n2 // 2, 15.0)
    field = torch.zeros(b, n1, n2, dtype=torch.complex64, device="cuda")
    field[:, : n1 // 2, : n2 // 2] = y
    bp = (torch.fft.ifft2(field) * (n1 * n2)).reshape(b, -1).contiguous()
    dp = y.abs().square().mean((1, 2)).double()[:, None]
    target = torch.log(x.reshape(b, -1).abs().square() / (dp / (n1 * n2)) + 1e-3).clamp(-20.0, 20.0)
    return bp, target.float().contiguous()


def prepare(case, seed):
    path = case["path"]
    if path == "train":
        bp, target = _training_batch(case, seed)
        return dict(case=case, bp=bp, target=target, net=WarmStartNet(torch.device("cuda", 0), seed=3))
    if path == "uneven":
        ys = _uneven_observations(case, seed)
        plan = make_uneven_plan(ys, [g for g, _ in _uneven_shapes(case)], profile=case["profile"])
        return dict(case=case, y=ys, plan=plan)
    y = _observations(case, seed)
    grid = (case["n1"], case["n2"])
    if path == "plan":
        make = make_stable_plan if case["profile"] == "stable" else make_fastest_plan
        return dict(case=case, y=y, plan=make(y, grid, observation_mask=_mask(case)))
    if path == "learned":
        return dict(case=case, y=y, plan=make_learned_plan(y, grid))
    if path == "certified":
        return dict(case=case, y=y, plan=make_cuda_graph_sbl_plan(
            y, grid, config=SBLConfig.certified_hybrid_uamp(device="cuda")))
    if path == "cg":
        return dict(case=case, y=y, config=SBLConfig(mode="cg", active_set=False, max_iter=case["iters"]))
    return dict(case=case, y=y[0], config=SBLConfig(max_iter=case["iters"]))


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
_FIELDS = ("x", "posterior_variance", "precision", "noise_variance", "effective_dof")
_PLAN_FIELDS = _FIELDS + ("negative_log_evidence", "evidence_trace", "support_mask", "support_exchanges_accepted",
                          "status")
_CERT_FIELDS = _FIELDS + ("negative_log_evidence", "evidence_trace", "support_exchanges_accepted",
                          "inactive_max_evidence_ratio", "inactive_best_index", "inactive_evidence_gain",
                          "inactive_optimal_variance", "active_max_evidence_gain", "active_best_index",
                          "coordinate_stationary", "status")


def _take(res, names):
    return {k: getattr(res, k) for k in names if getattr(res, k) is not None}


def run(state):
    case = state["case"]
    path = case["path"]
    if path == "train":
        net, b, n1, n2 = state["net"], case["batch"], case["n1"], case["n2"]
        net.features(state["bp"], n1, n2)
        out = net.forward(b, n1, n2)
        loss = net.backward(state["target"], b, n1, n2)
        net.adam(1e-3)
        return {"out": out, "loss": loss, "grad": net.grad, "params": net.params}
    if path in ("plan", "learned"):
        return _take(state["plan"].replay(state["y"]), _PLAN_FIELDS)
    if path == "uneven":
        res = state["plan"].replay(state["y"])
        out = {k: torch.cat([getattr(r, k).reshape(-1) for r in res]) for k in ("noise_variance",
                                                                             "negative_log_evidence", "status")}
        # the dense results of all scenes are slices of the engine's packed buffers
        packed = state["plan"].engine.out
        return {**out, **{k: packed[k] for k in ("x", "posterior_variance", "precision", "support_mask")}}
    if path == "certified":
        return _take(state["plan"].replay(state["y"]), _CERT_FIELDS)
    return _take(sbl_2d(state["y"], (case["n1"], case["n2"]), config=state["config"]), _FIELDS)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _sweeps(n, m, certified=False):
    """UAMP sweep budget of the presets."""
    if certified:
        return max(3, math.ceil(1.0 + n / m))
    return max(3, math.ceil(0.8 * n / m))


def _transform_flops(n1, n2, m1, m2):
    """One prefix transform as two passes of row FFTs."""
    return 5.0 * m1 * n2 * math.log2(n2) + 5.0 * n2 * n1 * math.log2(n1)


def _solve_work(b, n1, n2, m1, m2, profile):
    n, m = n1 * n2, m1 * m2
    t = _sweeps(n, m, profile == "certified")
    evals = {"stable": 3, "fast": 2}.get(profile, 5)
    flops = (2 * t + 1) * _transform_flops(n1, n2, m1, m2) + 30.0 * n * (t + 1) + evals * 8.0 * K**3
    if profile == "stable":
        flops += 8.0 * K * n  # the exchange's residual correlations
    if profile == "certified":
        flops += 2 * n * (8 * (K + K * (K - 1) // 2) + 6 * K + 8)
    return dict(bytes=b * (8.0 * m + 17.0 * n), flops=b * flops)


def work(case):
    path = case["path"]
    if path == "uneven":
        w = [_solve_work(1, *g, *s, case["profile"]) for g, s in _uneven_shapes(case)]
        return {k: sum(v[k] for v in w) for k in ("bytes", "flops")}
    if path == "train":
        n = case["batch"] * case["n1"] * case["n2"]
        return dict(bytes=16.0 * n, flops=3 * 2.0 * 792 * n)
    b, n1, n2, m1, m2 = (case[k] for k in ("scenes", "n1", "n2", "m1", "m2"))
    if path == "plan":
        return _solve_work(b, n1, n2, m1, m2, case["profile"])
    if path == "learned":
        w = _solve_work(b, n1, n2, m1, m2, "stable")
        return dict(bytes=w["bytes"], flops=w["flops"] - b * 4 * _transform_flops(n1, n2, m1, m2)
                    + b * 2.0 * 792 * n1 * n2)
    if path == "certified":
        return _solve_work(b, n1, n2, m1, m2, "certified")
    if path == "cg":  # at least one restart interval (8) per solve, 16 probes and the data
        its = 8.0 * (case["iters"] + 1) * 17 * b
        return dict(bytes=b * (8.0 * m1 * m2 + 16.0 * n1 * n2),
                    flops=its * 2 * _transform_flops(n1, n2, m1, m2))
    m = m1 * m2
    return dict(bytes=8.0 * m + 16.0 * n1 * n2, flops=(case["iters"] + 1) * 8.0 * m**3)


# ---------------------------------------------------------------------------
# 64-bit values
# ---------------------------------------------------------------------------
def _abs2(z):
    return z.real.square() + z.imag.square()


class _Op:
    """The prefix operator in complex128 (masked: unobserved samples zero)."""

    def __init__(self, n1, n2, m1, m2, mask=None):
        self.n1, self.n2, self.m1, self.m2 = n1, n2, m1, m2
        self.mask = None if mask is None else mask.to(torch.float64)
        self.m = m1 * m2 if mask is None else int(mask.sum())

    def data(self, y):
        return y if self.mask is None else y * self.mask

    def forward(self, x):
        b = x.shape[0]
        return self.data(torch.fft.fft2(x.view(b, self.n1, self.n2))[:, : self.m1, : self.m2])

    def adjoint(self, d):
        b = d.shape[0]
        return (torch.fft.ifft2(self.data(d), s=(self.n1, self.n2)) * (self.n1 * self.n2)).reshape(b, -1)

    def gram(self, active):
        """A_S^H A_S of the atoms ``active`` [b, k] (flat grid indices)."""
        w = torch.ones(self.m1, self.m2, dtype=torch.float64, device="cuda") if self.mask is None else self.mask
        table = torch.fft.ifft2(w.to(torch.complex128), s=(self.n1, self.n2)) * (self.n1 * self.n2)
        a1, a2 = active // self.n2, active % self.n2
        d1 = (a1[:, :, None] - a1[:, None, :]) % self.n1
        d2 = (a2[:, :, None] - a2[:, None, :]) % self.n2
        return table[d1, d2]


def _posterior(gram, gamma, nu, c, energy, m):
    """Reduced exact posterior and negative log evidence, with the solver's
    deterministic loading of the equilibrated system."""
    k = gamma.shape[1]
    eye = torch.eye(k, dtype=torch.complex128, device="cuda")
    s = gram / nu[:, None, None] + torch.diag_embed(1.0 / gamma).to(torch.complex128)
    d = s.diagonal(dim1=1, dim2=2).real.sqrt()
    e = s / d[:, :, None] / d[:, None, :]
    load = 8.0 * EPS * e.diagonal(dim1=1, dim2=2).real.abs().mean(1)
    chol = torch.linalg.cholesky(e + load[:, None, None] * eye)
    rhs = c / nu[:, None]
    mean = torch.cholesky_solve((rhs / d)[:, :, None], chol)[:, :, 0] / d
    inv = torch.linalg.solve_triangular(chol, eye.expand_as(chol), upper=False)
    pv = _abs2(inv).sum(1) / d.square()
    dd = ((gamma - pv) / gamma.square()).clamp_min(0.0)
    logdet = (m * nu.log() + gamma.log().sum(1)
              + 2.0 * (chol.diagonal(dim1=1, dim2=2).real.log().sum(1) + d.log().sum(1)))
    quad = (energy / nu - (rhs.conj() * mean).real.sum(1)).clamp_min(0.0)
    return mean, pv, dd, logdet + quad


def _solve64(y, n1, n2, profile, mask=None):
    """FBME-Fast / FBME-Stable in 64 bits: UAMP sweeps, top-K, polish."""
    y = y.to(torch.complex128)
    b, m1, m2 = y.shape
    op = _Op(n1, n2, m1, m2, mask)
    y = op.data(y)
    n, m = n1 * n2, op.m
    energy = _abs2(y).sum((1, 2))
    dp = (energy / m).clamp_min(EPS)
    floor = (dp * 1e-12).clamp_min(TINY)
    bp = op.adjoint(y)
    e = _abs2(bp)
    prior = 0.1 * e / e.sum(1, keepdim=True).clamp_min(EPS) * dp[:, None] + 0.9 * dp[:, None] / n
    prior = torch.maximum(prior, floor[:, None])
    nu = torch.maximum(1e-2 * dp, floor)
    d = 0.05
    mean, var = torch.zeros_like(bp), prior.clone()
    msg, pred = torch.zeros_like(y), torch.zeros_like(y)
    dv = prior.sum(1)
    sweeps = _sweeps(n, m)
    for it in range(sweeps + 1):
        dvc = dv.clamp_min(TINY)
        cand = (y - (pred - dvc[:, None, None] * msg)) / (dvc + nu)[:, None, None]
        msg = op.data(d * msg + (1.0 - d) * cand)
        pv = ((dvc + nu) / m).clamp_min(TINY)[:, None]
        den = (prior + pv).clamp_min(TINY)
        mean = d * mean + (1.0 - d) * (prior / den) * (mean + pv * op.adjoint(msg))
        var = (d * var.clamp_min(TINY) + (1.0 - d) * prior * pv / den).clamp_min(TINY)
        if it == sweeps:  # the last pass is the E-step alone
            break
        dof = (1.0 - var / prior.clamp_min(TINY)).clamp(0.0, 1.0).sum(1).clamp_max(m * (1.0 - 10.0 * EPS))
        dv = var.sum(1)
        pred = op.forward(mean)
        res = _abs2(y - pred).sum((1, 2))
        nu = torch.maximum(0.15 * nu + 0.85 * torch.maximum((res + nu * dof) / m, floor), floor)
        second = (_abs2(mean) + var).clamp_max(1e12)
        prior = torch.maximum(0.15 * prior + 0.85 * torch.maximum(second, floor[:, None]), floor[:, None])
    score = _abs2(mean) + var
    k = min(K, n)
    active = torch.topk(score, k, dim=1).indices
    gamma = torch.maximum(score.gather(1, active), floor[:, None])
    evals = 3 if profile == "stable" else 2
    exchanges = torch.zeros(b, dtype=torch.int64, device="cuda")
    best, pending, trace = None, None, []
    for p in range(evals):
        c = bp.gather(1, active)
        mu, pv, dd, nle = _posterior(op.gram(active), gamma, nu, c, energy, m)
        cand = dict(active=active, mu=mu, pv=pv, dd=dd, gamma=gamma, nu=nu, nle=nle)
        if best is None:
            best = cand
        else:
            ok = nle <= best["nle"] - 64.0 * EPS * (1.0 + nle.abs() + best["nle"].abs())
            if pending is not None:
                exchanges, pending = exchanges + (ok & pending), None
            best = {q: torch.where(ok.view(-1, *[1] * (v.ndim - 1)), cand[q], v) for q, v in best.items()}
        trace.append(best["nle"])
        if p + 1 == evals:
            break
        active, mu, pv, g0, nu0 = (best[q] for q in ("active", "mu", "pv", "gamma", "nu"))
        x = torch.zeros(b, n, dtype=torch.complex128, device="cuda").scatter(1, active, mu)
        resid = y - op.forward(x)
        dof = (1.0 - pv / g0.clamp_min(TINY)).clamp(0.0, 1.0).sum(1)
        nu = torch.maximum((_abs2(resid).sum((1, 2)) + nu0 * dof) / m, floor)
        gamma = torch.maximum(_abs2(mu) + pv, floor[:, None]).clamp_max(1e12)
        ex = min(EXCHANGE, k - 1, n - k) if profile == "stable" else 0
        if ex > 0 and p == 0:
            rs = _abs2(op.adjoint(resid)).scatter(1, active, -math.inf)
            add_e, add_i = torch.topk(rs, ex, dim=1)
            down = (pv / g0).clamp(TINY, 1.0)
            delete = -down.log() - _abs2(mu) / g0 / down
            del_g, pos = torch.topk(delete, ex, dim=1)
            ratio = add_e / (nu0 * m).clamp_min(TINY)[:, None]
            add_g = torch.where(ratio > 1.0, ratio - 1.0 - ratio.clamp_min(TINY).log(), 0.0)
            swap = add_g + del_g > 0.0
            new_g = ((add_e - (nu0 * m)[:, None]).clamp_min(0.0) / float(m) ** 2)
            new_g = torch.maximum(new_g, floor[:, None]).clamp_max(1e12)
            gamma = gamma.scatter(1, pos, torch.where(swap, new_g, gamma.gather(1, pos)))
            active = active.scatter(1, pos, torch.where(swap, add_i, active.gather(1, pos)))
            pending = swap.any(1)
    f = best
    x = torch.zeros(b, n, dtype=torch.complex128, device="cuda").scatter(1, f["active"], f["mu"])
    var = floor[:, None].expand(b, n).scatter(1, f["active"], f["pv"])
    prior = floor[:, None].expand(b, n).scatter(1, f["active"], f["gamma"])
    rel = (f["gamma"] * f["dd"]).clamp(0.0, 1.0)
    dof = rel.sum(1) * (m * (1.0 - 10.0 * EPS) / rel.sum(1).clamp_min(EPS)).clamp_max(1.0)
    return dict(x=x.view(b, n1, n2), posterior_variance=var.view(b, n1, n2),
                precision=(1.0 / prior).view(b, n1, n2), noise_variance=f["nu"], effective_dof=dof,
                negative_log_evidence=f["nle"], evidence_trace=torch.stack(trace, 1))


def _dense64(y, n1, n2, iters):
    """The exact-posterior EM loop through the data covariance, in 64 bits."""
    y = y.to(torch.complex128)
    m1, m2 = y.shape
    n, m = n1 * n2, m1 * m2
    op = _Op(n1, n2, m1, m2)
    flat = y.reshape(-1)
    eps64 = float(np.finfo(np.float64).eps)
    i1 = torch.arange(m, device="cuda") // m2
    i2 = torch.arange(m, device="cuda") % m2
    lag = ((i1[:, None] - i1[None, :]) % n1) * n2 + (i2[:, None] - i2[None, :]) % n2
    dp = _abs2(flat).mean().clamp_min(EPS)
    floor = (dp * 1e-12).clamp_min(TINY)
    e = _abs2(op.adjoint(y[None])[0])
    prior = torch.maximum(0.1 * e / e.sum().clamp_min(EPS) * dp + 0.9 * dp / n, floor)
    nu = torch.maximum(1e-2 * dp, floor)
    eye = torch.eye(m, dtype=torch.complex128, device="cuda")

    def posterior(prior, nu):
        q = torch.fft.fft2(prior.view(n1, n2).to(torch.complex128)).reshape(-1)[lag] + nu * eye
        q = q + 8.0 * eps64 * q.diagonal().real.abs().mean() * eye
        chol = torch.linalg.cholesky(q)
        qi = torch.cholesky_inverse(chol)
        z = (qi @ flat[:, None])[:, 0]
        sums = torch.zeros(n, 2, dtype=torch.float64, device="cuda").index_add(
            0, lag.reshape(-1), torch.view_as_real(qi).reshape(-1, 2))
        dd = (torch.fft.ifft2(torch.view_as_complex(sums).view(n1, n2)) * n).real.reshape(-1)
        mean = prior * op.adjoint(z.view(1, m1, m2))[0]
        return mean, (prior - prior.square() * dd).clamp_min(0.0), dd

    def relevance(prior, dd):
        rel = (prior * dd).clamp(0.0, 1.0)
        return rel * (m * (1.0 - 10.0 * EPS) / rel.sum().clamp_min(EPS)).clamp_max(1.0)

    for _ in range(iters):
        mean, pv, dd = posterior(prior, nu)
        rel = relevance(prior, dd)
        prec = ((rel + 1e-8) / (_abs2(mean) + 1e-8)).clamp(1e-12, 1e12)
        res = _abs2(y - op.forward(mean[None])[0]).sum()
        new_nu = torch.maximum((res + nu * rel.sum() + 1e-8) / (m + 1e-8), floor)
        prior = torch.maximum(0.15 * prior + 0.85 / prec, floor)
        nu = 0.15 * nu + 0.85 * new_nu
    mean, pv, dd = posterior(prior, nu)
    return dict(x=mean.view(n1, n2), posterior_variance=pv.view(n1, n2), precision=(1.0 / prior).view(n1, n2),
                noise_variance=nu, effective_dof=relevance(prior, dd).sum())


def _train64(case, seed):
    """The network's output, loss and gradient in 64 bits."""
    b, n1, n2 = case["batch"], case["n1"], case["n2"]
    bp, target = _training_batch(case, seed)
    flat = WarmStartNet(torch.device("cuda", 0), seed=3).params.double().requires_grad_(True)
    e = _abs2(bp.to(torch.complex128))
    f0 = torch.log(e / e.mean(1, keepdim=True).clamp_min(1e-30) + 1e-3)
    x = torch.stack([f0, f0.mean(1, keepdim=True).expand_as(f0)], 1).view(b, 2, n1, n2)
    at = 0
    for ci, co in ((2, 8), (8, 8), (8, 1)):
        w = flat[at: at + 9 * ci * co].view(3, 3, ci, co).permute(3, 2, 0, 1)
        at += 9 * ci * co
        x = torch.nn.functional.conv2d(x, w, flat[at: at + co], padding=1)
        at += co
        if co > 1:
            x = torch.relu(x)
    out = x.reshape(b, -1)
    loss = (out - target.double()).square().mean()
    grad, = torch.autograd.grad(loss, flat)
    return dict(out=out.detach(), loss=loss.detach(), grad=grad)


def exact(case, seed):
    path = case["path"]
    if path == "plan":
        y = _observations(case, seed)
        step = max(1, (1 << 24) // (case["n1"] * case["n2"]))  # scenes at a time
        parts = [_solve64(y[i: i + step], case["n1"], case["n2"], case["profile"], _mask(case))
                 for i in range(0, y.shape[0], step)]
        return {k: torch.cat([p[k] for p in parts]) for k in parts[0]}
    if path == "uneven":
        parts = [_solve64(y[None], *g, case["profile"])
                 for y, (g, _) in zip(_uneven_observations(case, seed), _uneven_shapes(case))]
        return {k: torch.cat([p[k].reshape(-1) for p in parts])
                for k in ("x", "posterior_variance", "precision", "noise_variance", "negative_log_evidence")}
    if path == "dense":
        return _dense64(_observations(case, seed)[0], case["n1"], case["n2"], case["iters"])
    if path == "train":
        return _train64(case, seed)
    return None  # cg, learned, certified (its decisions hang on FP32 ratios): see above
