#!/usr/bin/env python
"""FBME plan-replay throughput on B200: scenes/s and % of the HBM roofline.

Workload: FBME-Stable replay of 256x256-grid / 128x128-prefix scenes
(200 Rayleigh point scatterers, 15 dB, polish_size 32), a batch of
``--batch`` scenes per step solved by one captured plan.  Synthetic scenes
stand in for recorded data (seeded, shapes and value laws as named).

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

N > 1 runs one process per GPU (torchrun); every rank solves its own batch
(weak scaling, no collective on the data path); timing is the max over ranks.
``--impl reference`` times the CPU restatement of the reference algorithm on
the host cores (the reference ships no compiled code).
"""

from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import tempfile
import time
from pathlib import Path

REPO = Path(__file__).resolve().parent
for _p in (str(REPO), str(REPO / "fbme-sbl_b200")):
    if _p not in sys.path:
        sys.path.insert(0, _p)

METRIC = "scenes/s at equal NMSE: plain vs learned+batched FBME on 1 B200; % roofline"
UNIT = "scenes/s"
GRID, PREFIX = (256, 256), (128, 128)
DFT_FORMS = {0: "FP32 FFT stages (two-pass register FFT)",
             3: "tcgen05 split-BF16 3-term, FP32 accumulation",
             6: "tcgen05 split-BF16 6-term, FP32 accumulation"}
WORKLOAD = ("FBME-Stable replay, 256x256 grid / 128x128 prefix, 200 Rayleigh points, 15 dB, "
            "polish_size=32")


def _args() -> argparse.Namespace:
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=100)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", choices=("ours", "reference"), default="ours")
    ap.add_argument("--batch", type=int, default=512, help="scenes per step per GPU")
    ap.add_argument("--profile", choices=("stable", "fast"), default="stable")
    ap.add_argument("--cpu-rounds", type=int, default=2,
                    help="rounds of one scene per host core in the CPU baseline sample")
    ap.add_argument("--no-cg", action="store_true", help="skip the mode='cg' section")
    ap.add_argument("--no-cpu", action="store_true")
    ap.add_argument("--no-certificate", action="store_true", help="skip the global-certificate section")
    ap.add_argument("--no-learned", action="store_true", help="skip the learned-vs-plain section")
    ap.add_argument("--no-uneven", action="store_true", help="skip the batched-uneven section")
    ap.add_argument("--no-precision", action="store_true", help="skip the precision-workload section")
    return ap.parse_args()


def _scenes(n: int, seed0: int):
    from fbme_b200 import scenes

    return [scenes.config_scene("c2", seed0 + i) for i in range(n)]


# ---------------------------------------------------------------- ranks
def shard_seeds(rank: int, batch: int) -> range:
    """Scene seeds of one rank: ranks solve disjoint scenes (weak scaling,
    no data-path collective)."""
    return range(rank * batch, (rank + 1) * batch)


def max_over_ranks(v: float, dist=None, device=None) -> float:
    """The job's time: the maximum of the ranks' device times."""
    if dist is None:
        return v
    import torch

    t = torch.tensor([v], device=device, dtype=torch.float64)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def job_rate(scenes_per_rank: int, steps: int, world: int, job_ms: float) -> float:
    """Whole-job scenes/s: every rank's scenes over the slowest rank's time."""
    return scenes_per_rank * steps * world / (job_ms / 1000.0)


def learned_section(device, steps: int, batch: int = 256) -> dict:
    """Plain vs learned+batched FBME on held-out scenes of the learned
    distribution (256x256 / 128x128, K ~ U{100..400}, SNR ~ U[5, 25] dB,
    seeds 2*10^6 ...): scenes/s of the warm-started plan (1 UAMP sweep,
    check and plain fallback in a device graph, nothing read on the host):
    pipelined (each replay's fallback overlaps the next replay's warm solve;
    the headline) and stream-ordered; of the plain Stable plan on the same
    batch, and of the plain plan solving one scene per replay; raw NMSE of
    each."""
    import numpy as np
    import torch

    from fbme_b200 import scenes
    from fbme_b200.learned import make_learned_plan
    from torch_sbl_fastest_stable import make_stable_plan

    # 1024 held-out seeds (the evaluation set of the learned workload), in
    # batches of `batch`; rates are timed on the first batch
    n_eval = max(1024, batch)
    sc = [scenes.learned_scene(2_000_000 + i) for i in range(n_eval)]
    ys = [torch.from_numpy(np.stack([s.y for s in sc[k:k + batch]])).to(device)
          for k in range(0, n_eval - batch + 1, batch)]
    xts = [np.stack([s.x.reshape(-1) for s in sc[k:k + batch]]) for k in range(0, n_eval - batch + 1, batch)]
    y = ys[0]

    def nmse_of(plan, **kw):
        """Mean raw NMSE (dB) of `plan` over every evaluation batch."""
        vals = []
        for yb, xt in zip(ys, xts):
            xh = plan.replay(yb, synchronize=True, **kw).x.cpu().numpy().reshape(len(xt), -1)
            vals.append(10 * np.log10(np.sum(np.abs(xh - xt) ** 2, 1) / np.sum(np.abs(xt) ** 2, 1)))
        return float(np.mean(np.concatenate(vals)))

    def rate(fn, n_scenes, reps, join=None):
        for _ in range(3):
            fn()
        torch.cuda.synchronize(device)
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(reps):
            fn()
        if join is not None:
            join()  # the last replay's fallback is inside the timed region
        e1.record()
        torch.cuda.synchronize(device)
        return n_scenes * reps / (e0.elapsed_time(e1) / 1000.0)

    learned = make_learned_plan(y, GRID, warmup=1, pipelined=True)
    plain = make_stable_plan(y, GRID, warmup=1)
    r_learned = rate(lambda: learned.replay(y), batch, steps, learned.join)
    fallbacks = learned.fallbacks
    overflow = int(learned.overflows.item())  # replays (warm-up included) beyond the device capacity
    ordered = make_learned_plan(y, GRID, warmup=1)
    r_ordered = rate(lambda: ordered.replay(y), batch, steps)
    r_warm = rate(lambda: ordered.replay(y, fallback=False), batch, steps)
    del ordered
    n_learned = nmse_of(learned)
    fallbacks_eval = 0
    for yb in ys:  # fallbacks over the evaluation set (each read synchronises)
        learned.replay(yb)
        fallbacks_eval += learned.fallbacks
    r_plain = rate(lambda: plain.replay(y), batch, steps)
    n_plain = nmse_of(plain)
    single = make_stable_plan(y[:1], GRID, warmup=1)
    r_single = rate(lambda: single.replay(y[:1]), 1, max(steps, 50))
    # plain FBME at larger sweep budgets: the cheapest one that reaches the
    # learned plan's NMSE is the equal-NMSE comparison
    from fbme_b200.learned import plain_config
    from fbme_b200.plans import CUDAGraphSBLPlan

    budgets = {}
    equal = None
    for sweeps in (6, 8, 12, 16):
        p = CUDAGraphSBLPlan(y, GRID, config=plain_config(sweeps), warmup=1)
        n_p = nmse_of(p)
        r_p = rate(lambda: p.replay(y), batch, steps)
        budgets[str(sweeps)] = {"scenes_per_s": r_p, "nmse_db": n_p}
        if equal is None and n_p <= n_learned:
            equal = {"plain_sweeps": sweeps, "plain_scenes_per_s": r_p, "learned_vs_plain": r_learned / r_p}
        del p
    return {
        "workload": "held-out learned-distribution scenes, 256x256 / 128x128, K~U{100..400}, "
                    f"SNR~U[5,25] dB, batch {batch}; NMSE and fallbacks over {n_eval} held-out seeds",
        "learned_batched_scenes_per_s": r_learned,
        "learned_batched_stream_ordered_scenes_per_s": r_ordered,
        "fallback": f"device graph: check, compaction into {learned.capacity} slots, plain re-solve, "
                    "scatter; pipelined with the next replay's warm solve on a high-priority stream",
        "fallback_overflow_replays": overflow,
        "warm_solve_alone_scenes_per_s": r_warm,  # the same plan without its fallback check (not a result)
        "plain_batched_scenes_per_s": r_plain,
        "plain_single_scene_scenes_per_s": r_single,
        "learned_batched_vs_plain_single": r_learned / r_single,
        "learned_vs_plain_batched": r_learned / r_plain,
        "nmse_db": {"plain": n_plain, "learned": n_learned},
        "fallbacks_per_replay": fallbacks,
        "fallbacks_on_eval_set": fallbacks_eval,
        "learned_sweeps": 1, "plain_sweeps": 4,
        "plain_budgets": budgets,
        "equal_nmse": equal if equal is not None else
        "no plain budget up to 16 sweeps reaches the learned NMSE",
    }


# Published single-scene replay latencies of the reference (RTX 4090, 40x32
# grid, 20x16 prefix, 21 targets, 10 dB; device P50 over 20 repeats of
# resident input copy + warm solve): FBME-Fast 0.6415 ms, FBME-Stable
# 1.0988 ms.
PUBLISHED_MS = {"fast": 0.6415, "stable": 1.0988}


def published_shape_section(device, repeats: int = 20) -> dict:
    """The same protocol on the B200 with a seeded synthetic scene of the
    archived shape (its generator and arrays were not released): device
    P50 and max over `repeats` replays, each timed with CUDA events around
    the resident input copy and the replay."""
    import torch

    from fbme_b200 import scenes
    from torch_sbl_fastest_stable import make_fastest_plan, make_stable_plan

    sc = scenes.point_scene((40, 32), (20, 16), 21, 10.0, 200, "cn")
    y = torch.from_numpy(sc.y).to(device)
    out = {"workload": "one 40x32 / 20x16 scene, 21 CN(0,1) points, 10 dB, seed 200"}
    for name, make in (("fast", make_fastest_plan), ("stable", make_stable_plan)):
        plan = make(y, (40, 32), warmup=3)
        times = []
        for _ in range(repeats + 3):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            plan.replay(y)
            e1.record()
            torch.cuda.synchronize(device)
            times.append(e0.elapsed_time(e1))
        t = sorted(times[3:])
        p50 = 0.5 * (t[len(t) // 2 - 1] + t[len(t) // 2])
        out[name] = {"device_p50_ms": p50, "device_max_ms": t[-1],
                     "published_rtx4090_p50_ms": PUBLISHED_MS[name],
                     "speedup_vs_published": PUBLISHED_MS[name] / p50}
    return out


def uneven_section(device, steps: int, n_scenes: int = 64) -> dict:
    """The batched-uneven workload: 64 scenes with grids from {128x128,
    192x256, 256x256, 384x256}, prefix ratio per axis U[0.3, 0.7],
    sparsity 1-3 %, SNR U[5, 25] dB (every scene its own shape).  Scenes/s
    of one captured uneven plan, and of one single-scene plan per scene
    replayed in turn (the only way to solve such a batch with equal-shape
    plans); the two give bit-identical results.  For scale, the rate of
    one equal-shape plan of 64 scenes of the headline shape."""
    import numpy as np
    import torch

    from fbme_b200 import scenes
    from fbme_b200.uneven import make_uneven_plan
    from torch_sbl_fastest_stable import make_stable_plan

    sc = scenes.uneven_batch(0, n_scenes)
    ys = [torch.from_numpy(s.y).to(device) for s in sc]
    grids = [s.grid for s in sc]

    def rate(fn, reps):
        for _ in range(3):
            fn()
        torch.cuda.synchronize(device)
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(reps):
            fn()
        e1.record()
        torch.cuda.synchronize(device)
        return n_scenes * reps / (e0.elapsed_time(e1) / 1000.0)

    plan = make_uneven_plan(ys, grids, warmup=1)
    r_uneven = rate(lambda: plan.replay(), steps)
    singles = [make_stable_plan(y, g, warmup=1) for y, g in zip(ys, grids)]

    def one_by_one():
        for q in singles:
            q.replay()

    r_single = rate(one_by_one, max(2, steps // 10))
    # for scale: one equal-shape plan of 64 scenes of the headline shape
    # (256x256 / 128x128)
    eq = [scenes.config_scene("c2", 5_000_000 + i) for i in range(n_scenes)]
    y_eq = torch.from_numpy(np.stack([s.y for s in eq])).to(device)
    eq_plan = make_stable_plan(y_eq, GRID, warmup=1)
    r_equal = rate(lambda: eq_plan.replay(y_eq), steps)
    return {
        "workload": f"{n_scenes} uneven scenes, grids from {{128x128, 192x256, 256x256, 384x256}}, "
                    "prefix ratio U[0.3,0.7] per axis, 1-3 % CN(0,1) points, SNR U[5,25] dB",
        "distinct_shapes": len({(s.grid, s.y.shape) for s in sc}),
        "uneven_plan_scenes_per_s": r_uneven,
        "single_scene_plans_scenes_per_s": r_single,
        "uneven_vs_single_scene_plans": r_uneven / r_single,
        "equal_shape_plan_scenes_per_s": r_equal,
        "equal_shape_workload": f"{n_scenes} scenes of 256x256 / 128x128 in one equal-shape plan",
        "uneven_vs_equal_shape": r_uneven / r_equal,
        "dft_form": "FP32 FFT stages" if int(plan.engine.native_cfg.dft_terms) == 0
                    else "split-BF16 tensor-core stages",
    }


def precision_section(device, steps: int, y_main=None, batch: int = 32) -> dict:
    """The precision workload (512x512 grid, 256x192 prefix, clustered
    log-normal scatterers, 20 dB) under the three operator modes: 3- and
    6-term split-BF16 tensor-core products and FP32 FFTs (dft_terms 0).
    Per mode: scenes/s of one captured FBME-Stable plan over `batch` scenes,
    its NMSE against the ground truth, and the relative L2 error of A x and
    A^H y against an FP64 FFT on one random complex input.  With `y_main`
    (the headline batch), the headline workload is also replayed with the
    3-term products and with FP32 FFTs, with the per-stage table of each."""
    import numpy as np
    import torch

    from fbme_b200 import scenes
    from fbme_b200.config import SBLConfig, fbme_profile_config
    from fbme_b200.engine import FBMEEngine
    from fbme_b200.plans import CUDAGraphSBLPlan

    grid, prefix = (512, 512), (256, 192)
    sc = [scenes.config_scene("c3", 4_000_000 + i) for i in range(batch)]
    y = torch.from_numpy(np.stack([s.y for s in sc])).to(device)
    truth = np.stack([s.x for s in sc])
    rng = np.random.default_rng(11)
    xr = (rng.standard_normal(grid) + 1j * rng.standard_normal(grid)).astype(np.complex64)
    yr = (rng.standard_normal(prefix) + 1j * rng.standard_normal(prefix)).astype(np.complex64)
    ref_f = np.fft.fft2(xr.astype(np.complex128))[:prefix[0], :prefix[1]]
    ref_a = np.fft.ifft2(yr.astype(np.complex128), s=grid) * (grid[0] * grid[1])

    def rel(a, b):
        return float(np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel()))

    out = {"workload": f"{batch} precision-workload scenes per replay, 512x512 grid / 256x192 prefix, "
                       "800 clustered + 50 isolated log-normal scatterers, 20 dB; FBME-Stable"}
    for name, terms in (("bf16x3", 3), ("bf16x6", 6), ("fp32_fft", 0)):
        eng = FBMEEngine(1, grid, prefix, SBLConfig.paper_hybrid_uamp(uamp_polish_size=32, dft_terms=terms),
                         device)
        fx = eng.dft_forward(torch.from_numpy(xr.reshape(1, -1)).to(device)).cpu().numpy().reshape(prefix)
        ay = eng.dft_adjoint(torch.from_numpy(yr.reshape(1, -1)).to(device)).cpu().numpy().reshape(grid)
        cfg = fbme_profile_config("stable")
        cfg.dft_terms = terms
        plan = CUDAGraphSBLPlan(y, grid, config=cfg, warmup=1)
        for _ in range(3):
            plan.replay(y)
        torch.cuda.synchronize(device)
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(steps):
            res = plan.replay(y)
        e1.record()
        torch.cuda.synchronize(device)
        ms = e0.elapsed_time(e1) / steps
        x_hat = res.x.cpu().numpy()
        out[name] = {"dft_terms": terms, "scenes_per_s": batch / (ms / 1000.0), "ms_per_replay": ms,
                     "nmse_db": float(np.mean([scenes.nmse_db(x_hat[i], truth[i]) for i in range(batch)])),
                     "forward_rel_l2_vs_fp64": rel(fx, ref_f), "adjoint_rel_l2_vs_fp64": rel(ay, ref_a)}
        del plan, eng
    if y_main is not None:
        B = y_main.shape[0]
        main = {"workload": WORKLOAD + f", batch {B}"}
        for name, terms in (("bf16x3", 3), ("fp32_fft", 0)):
            cfg = fbme_profile_config("stable")
            cfg.dft_terms = terms
            plan = CUDAGraphSBLPlan(y_main, GRID, config=cfg, warmup=1)
            for _ in range(3):
                plan.replay(y_main)
            torch.cuda.synchronize(device)
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            for _ in range(steps):
                plan.replay(y_main)
            e1.record()
            torch.cuda.synchronize(device)
            ms = e0.elapsed_time(e1) / steps
            prof = plan._engine.profile(plan.input_buffer.view(B, -1))
            main[name] = {"scenes_per_s": B / (ms / 1000.0), "ms_per_replay": ms,
                          "stages": stages_table(prof, B, GRID, PREFIX, _peaks(), terms)}
            del plan
        out["headline_workload"] = main
    return out


# mode="cg" workloads: sbl_2d's default cg path (active_set off) with the EM
# loop capped at a fixed iteration count, as the reference's CPU sbl_2d is
# timed at 256x256 (its uncapped C1 run takes 200 iterations).
CG_CASES = (("c1", (64, 64), 20, 64), ("c2", (256, 256), 6, 8))  # (config, grid, EM iterations, GPU batch)


def cg_section(device) -> dict:
    """Scenes/s of the native cg solve (fbme_cg_solve through CGEngine,
    including its host reads at the PCG and convergence checks) at C1 and
    C2, EM iterations capped as CG_CASES states."""
    import numpy as np
    import torch

    from fbme_b200 import scenes
    from fbme_b200.cg import CGEngine
    from fbme_b200.config import SBLConfig

    out = {}
    for name, grid, iters, batch in CG_CASES:
        sc = [scenes.config_scene(name, 3_000_000 + i) for i in range(batch)]
        y = torch.from_numpy(np.stack([s.y.reshape(-1) for s in sc])).to(device)
        cfg = SBLConfig(mode="cg", active_set=False, max_iter=iters)
        eng = CGEngine(batch, grid, sc[0].y.shape, cfg, device)
        probes = eng.default_probes()
        eng.solve(y, probes)
        torch.cuda.synchronize(device)
        reps = 3
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(reps):
            res = eng.solve(y, probes)
        e1.record()
        torch.cuda.synchronize(device)
        ms = e0.elapsed_time(e1) / reps
        hist = res.history.get("cg_iterations") if res.history else None
        out[name] = {"grid": list(grid), "scenes_per_solve": batch, "em_iterations": res.iterations,
                     "ms_per_solve": ms, "scenes_per_s": batch / (ms / 1000.0),
                     "status_nonzero": int((res.status != 0).sum().item()),
                     "pcg_iterations": hist}
        eng.close()
    return out


def certificate_flops_per_atom(k: int) -> int:
    """FP32 FLOPs of one grid atom in the certificate scan: K complex
    multiply-adds for q_j and K(K-1)/2 for the forward substitution (8 each),
    K complex scalings and squared norms (6 each), the ratio (about 8)."""
    return 8 * (k + k * (k - 1) // 2) + 6 * k + 8


def certificate_section(device, steps: int, batch: int = 64) -> dict:
    """certified_hybrid_uamp (global certificate, one support repair) against
    the same solve without it (fast_hybrid_uamp with 4 polish iterations) on
    256^2/128^2 scenes: scenes/s of each, and the certificate kernel's time
    and FP32 rate (1 + repairs grid scans per replay) against the nominal
    FP32 FMA peak (148 SMs x 128 lanes x 2 FLOP x 1.965 GHz)."""
    import numpy as np
    import torch

    from fbme_b200 import scenes
    from fbme_b200.config import SBLConfig
    from fbme_b200.engine import FBMEEngine

    sc = [scenes.config_scene("c2", 6_000_000 + i) for i in range(batch)]
    y = torch.from_numpy(np.stack([v.y.reshape(-1) for v in sc])).to(device)
    grid, sample = sc[0].grid, sc[0].y.shape
    out = {"grid": list(grid), "scenes": batch}
    for name, cfg in (("certified", SBLConfig.certified_hybrid_uamp(device="cuda")),
                      ("uncertified", SBLConfig.fast_hybrid_uamp(device="cuda", uamp_polish_iterations=4))):
        eng = FBMEEngine(batch, grid, sample, cfg, device)
        for _ in range(3):
            eng.run(y)
        torch.cuda.synchronize(device)
        reps = max(steps, 5)
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(reps):
            eng.run(y)
        e1.record()
        torch.cuda.synchronize(device)
        ms = e0.elapsed_time(e1) / reps
        out[name] = {"ms_per_replay": ms, "scenes_per_s": batch / (ms / 1000.0)}
        if name == "certified":
            prof = eng.profile(y)
            cms = prof.get("certificate", (0.0, 0))[0]
            scans = 1 + cfg.uamp_polish_support_repairs
            flops = scans * batch * grid[0] * grid[1] * certificate_flops_per_atom(cfg.uamp_polish_size)
            peak = 148 * 128 * 2 * 1.965e9
            out[name].update(certificate_kernel_ms=cms, grid_scans=scans,
                             fp32_tflops=flops / (cms * 1e-3) / 1e12 if cms else None,
                             fp32_frac_of_nominal=flops / (cms * 1e-3) / peak if cms else None,
                             repairs_kept=int(eng.cert["support_repairs_accepted"].sum()))
        eng.close()
    out["certified_vs_uncertified"] = out["certified"]["scenes_per_s"] / out["uncertified"]["scenes_per_s"]
    return out


# ---------------------------------------------------------------- CPU side
def _oracle_solve(args):
    y, grid, profile = args
    from oracle import fbme_oracle as O

    return O.fbme_solve(y, grid, profile)["x"]


def _oracle_cg_solve(args):
    y, grid, iters = args
    import numpy as np

    from oracle import fbme_oracle as O

    return O.fast_sbl_cg(y[None].astype(np.complex64), grid,
                         O.OracleConfig(mode="cg", active_set=False, max_iter=iters))["x"]


def _pool_rate(fn, work, rounds: int) -> float:
    """Items per second of ``fn`` over ``work`` on a spawn pool of one
    process per host core (one thread each), after one warm-up round."""
    import multiprocessing as mp

    ctx = mp.get_context("spawn")  # the parent has a CUDA context: never fork
    with ctx.Pool(len(work), initializer=_limit_threads) as pool:
        pool.map(fn, work)
        t0 = time.perf_counter()
        for _ in range(rounds):
            pool.map(fn, work)
        dt = time.perf_counter() - t0
    return len(work) * rounds / dt


def cpu_baseline(profile: str, rounds: int = 2) -> dict:
    """The oracle port (numpy restatement of the reference) on every host
    core: one process per core, each solving its own scene of the plan
    workload; plus the C1 cg-mode leg standing in for the reference's CPU
    sbl_2d (EM loop capped, CG_CASES)."""
    from fbme_b200 import scenes

    cores = os.cpu_count() or 1
    sc = _scenes(cores, 1_000_000)
    value = _pool_rate(_oracle_solve, [(s.y, s.grid, profile) for s in sc], rounds)
    _, grid, iters, _ = CG_CASES[0]
    c1 = [scenes.config_scene("c1", 1_000_000 + i) for i in range(cores)]
    cg_rate = _pool_rate(_oracle_cg_solve, [(s.y, s.grid, iters) for s in c1], 1)
    return {"value": value, "unit": UNIT, "cores": cores, "kind": "port",
            "sample": f"{cores * rounds} scenes of the same workload ({rounds} rounds of one scene per core), "
                      "numpy oracle, one single-threaded process per host core",
            "c1_cg": {"value": cg_rate, "unit": UNIT, "cores": cores,
                      "sample": f"{cores} 64x64 / 32x32 scenes, oracle mode='cg' (sbl_2d's default path, "
                                f"active_set off), {iters} EM iterations, one per core"}}


def run_reference(a: argparse.Namespace) -> None:
    """Reference arm: the CPU restatement with every host core (spawn pool)."""
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    import multiprocessing as mp

    cores = os.cpu_count() or 1
    sc = _scenes(cores, 2_000_000)
    work = [(s.y, s.grid, a.profile) for s in sc]
    ctx = mp.get_context("spawn")
    with ctx.Pool(cores, initializer=_limit_threads) as pool:
        for _ in range(a.warmup):
            pool.map(_oracle_solve, work)
        t0 = time.perf_counter()
        for _ in range(a.steps):
            pool.map(_oracle_solve, work)
        dt = time.perf_counter() - t0
    value = cores * a.steps / dt
    line = {
        "metric": METRIC, "value": value, "unit": UNIT, "impl": "reference", "n_gpus": a.gpus,
        "steps": a.steps, "warmup": a.warmup, "ms_per_step": 1000.0 * dt / a.steps,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "c64",
        "data": "synthetic",
        "config": {"workload": WORKLOAD, "scenes_per_step": cores, "profile": a.profile},
        "cpu_baseline": {"value": value, "unit": UNIT, "cores": cores, "kind": "port",
                         "sample": f"{cores} scenes per step, one per host core (spawn pool)"},
        "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


def _limit_threads() -> None:
    os.environ["OMP_NUM_THREADS"] = "1"


# ---------------------------------------------------------------- clocks
class Clocks:
    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_id: str | None) -> None:
        self.file = tempfile.NamedTemporaryFile("w+", suffix=".csv", delete=False)
        cmd = ["nvidia-smi", f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits",
               "-lms", "100"]
        if gpu_id:
            cmd += ["-i", gpu_id]
        try:
            self.proc = subprocess.Popen(cmd, stdout=self.file, stderr=subprocess.DEVNULL)
        except OSError:
            self.proc = None

    def stop(self) -> dict:
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        self.file.flush()
        self.file.seek(0)
        sm, mx, reasons = [], [], set()
        names = ("hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap")
        for line in self.file.read().splitlines():
            parts = [p.strip() for p in line.split(",")]
            if len(parts) < 9:
                continue
            try:
                sm.append(float(parts[1]))
                mx.append(float(parts[2]))
            except ValueError:
                continue
            for name, val in zip(names, parts[5:9]):
                if val.lower() == "active":
                    reasons.add(name)
        os.unlink(self.file.name)
        return {"sm_mhz": statistics.median(sm) if sm else None,
                "sm_max_mhz": max(mx) if mx else None, "reasons": sorted(reasons),
                "samples": len(sm)}


# ---------------------------------------------------------------- roofline
def _peaks() -> dict:
    """Roofline denominators: MEASURED_PEAKS.json when the run has it, else
    the earlier measurement on this GPU type (6650 GB/s copy, 1590 TFLOP/s
    dense BF16 burst)."""
    p = REPO / "MEASURED_PEAKS.json"
    if p.exists():
        d = json.loads(p.read_text())
        return {"hbm": float(d["hbm_gbs"]), "bf16": float(d.get("bf16_tflops", 1590.0)),
                "source": "measured: MEASURED_PEAKS.json hbm_gbs / bf16_tflops"}
    return {"hbm": 6650.0, "bf16": 1590.0,
            "source": "fallback: 6650 GB/s copy and 1590 TFLOP/s BF16 (MEASURED_PEAKS.json absent)"}


def algorithmic_bytes(group: str, n: int, m: int) -> int:
    """Algorithmic HBM bytes of one scene for one launch of a kernel group
    (intermediates of the two-stage DFT are not counted)."""
    table = {
        "adjoint_denoise": 32 * n,    # read gamma, mu, v; write mu', v', gamma' (or keys)
        "message": 24 * m,            # read y, m; write m'
        "forward_1": 8 * n,           # read mu
        "forward_residual": 16 * m,   # read y; write prediction
        "sweep1_denoise": 24 * n + 16 * m,
    }
    return table.get(group, 0)


def physical_bytes(group: str, grid, prefix, fused_denoise: bool = False) -> int:
    """Bytes one scene moves to and from HBM in one launch of a kernel group,
    intermediates included (each array read or written once).  With
    `fused_denoise` (the FP32 FFT stages) adjoint stage 2 runs the denoiser
    in its epilogue: the group reads U instead of the lift A^H m; and adjoint
    stage 1 forms the message it transforms."""
    n1, n2 = grid
    m1, m2 = prefix
    n, m = n1 * n2, m1 * m2
    t_fwd, t_adj = 8 * m2 * n1, 8 * n2 * m1  # the two-stage intermediates T, U
    table = {
        # read lift 8 (fused: U), mu 8, gamma 4, v 4; write mu 8, v 4, gamma 4
        "adjoint_denoise": (t_adj + 32 * n) if fused_denoise else 40 * n,
        "message": 32 * m,                    # read y, prediction, message; write message
        # read message (fused: y, prediction, message; write message); write U
        "adjoint_1": (32 if fused_denoise else 8) * m + t_adj,
        "adjoint_2": t_adj + 8 * n,           # read U; write lift
        "forward_1": 8 * n + t_fwd,           # read mu; write T
        "forward_residual": t_fwd + 16 * m,   # read T, y; write prediction
    }
    return table.get(group, 0)


def stage_flops(group: str, grid, prefix, terms: int = 3, n_tile: int = 256) -> int:
    """Tensor-core FLOPs one scene executes in one launch of a DFT stage:
    the real GEMM [rows, 2K] x [2K, 2C] padded to the tile (128 rows, 64-wide
    K chunks, n_tile columns), once per split-BF16 product."""
    n1, n2 = grid
    m1, m2 = prefix
    rkc = {"forward_1": (n1, n2, m2), "forward_residual": (m2, n1, m1),
           "adjoint_1": (m1, m2, n2), "adjoint_2": (n2, m1, n1)}.get(group)
    if rkc is None:
        return 0
    r, k, c = rkc
    up = lambda v, q: -(-v // q) * q  # noqa: E731
    return 2 * up(r, 128) * up(2 * k, 64) * up(2 * c, n_tile) * terms


def scene_bytes(n: int, m: int, t_u: int, p: int) -> int:
    """Algorithmic bytes of one Stable solve: (T_u+1) sweeps of 32N+24M,
    8M+8N initialisation, 12N top-K read, P re-reads of y, 17N outputs."""
    return (t_u + 1) * (32 * n + 24 * m) + 8 * m + 8 * n + 12 * n + p * 8 * m + 17 * n


def stages_table(prof: dict, batch: int, grid, prefix, peaks: dict, terms: int = 3, n_tile: int = 256) -> dict:
    """Per kernel group of one replay: launches, time per launch, the bytes
    it must move (physical_bytes) against HBM, and for the DFT stages the
    executed tensor FLOPs against dense BF16."""
    out = {}
    for g, (ms, cnt) in prof.items():
        pb = physical_bytes(g, grid, prefix, terms == 0) * batch
        fl = stage_flops(g, grid, prefix, terms, n_tile) * batch
        if not (pb or fl) or cnt == 0:
            continue
        per_s = ms / cnt / 1000.0
        row = {"launches": cnt, "ms_per_launch": round(ms / cnt, 5), "bytes_per_launch": pb,
               "hbm_gbs": round(pb / per_s / 1e9, 1), "hbm_frac": round(pb / per_s / 1e9 / peaks["hbm"], 4)}
        if fl:
            row["tensor_tflops"] = round(fl / per_s / 1e12, 1)
            row["tensor_frac"] = round(fl / per_s / 1e12 / peaks["bf16"], 4)
            row["flops_per_launch"] = fl
        out[g] = row
    return out


# ---------------------------------------------------------------- our arm
def run_ours(a: argparse.Namespace) -> None:
    import numpy as np
    import torch

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    dist = None
    if world > 1:
        import datetime

        import torch.distributed as dist_mod

        dist = dist_mod
        torch.cuda.set_device(local)
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120))
    device = torch.device("cuda", local if world > 1 else 0)
    torch.cuda.set_device(device)

    from torch_sbl_fastest_stable import make_fastest_plan, make_stable_plan

    B = a.batch
    seeds = shard_seeds(rank, B)
    sc = _scenes(len(seeds), seeds.start)
    y_np = np.stack([s.y for s in sc])
    x_true = np.stack([s.x for s in sc]).astype(np.complex64)
    y_host = torch.from_numpy(y_np).pin_memory()
    y_dev = y_host.to(device)
    make = make_stable_plan if a.profile == "stable" else make_fastest_plan
    plan = make(y_dev, GRID, polish_size=32, warmup=1)

    def barrier():
        if dist is not None:
            dist.barrier()
        torch.cuda.synchronize(device)

    def job_ms(v: float) -> float:
        return max_over_ranks(v, dist, device)

    gpu_id = None
    try:
        gpu_id = "GPU-" + str(torch.cuda.get_device_properties(device).uuid)
    except Exception:
        pass
    clocks = Clocks(gpu_id)
    stream = torch.cuda.current_stream(device)
    for _ in range(max(a.warmup, 3)):
        plan.replay(y_dev)
    barrier()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    for _ in range(a.steps):
        plan.replay(y_dev)
    e1.record(stream)
    barrier()
    clk = clocks.stop()
    ms = job_ms(e0.elapsed_time(e1))
    value = job_rate(B, a.steps, world, ms)

    # end to end through the public API (fbme_b200.streaming.HostPipeline):
    # every step copies its observations from pinned host memory and its
    # result back to pinned host memory, overlapped with the neighbouring
    # steps' solves.  Headline: the compact result (active indices and x
    # values -- x is zero elsewhere -- noise variance, evidence, status);
    # e2e_dense reads the dense x back instead.
    from fbme_b200.streaming import HostPipeline

    res = plan.result

    def run_pipeline(dense: bool):
        pipe = HostPipeline(plan, dense=dense)
        outs = [pipe.host_result(), pipe.host_result()]
        for i in range(2):
            pipe.submit(y_host, outs[i % 2])
        pipe.synchronize()
        barrier()
        e0.record(stream)
        for i in range(a.steps):
            pipe.submit(y_host, outs[i % 2])
        pipe.join()
        e1.record(stream)
        barrier()
        t = job_ms(e0.elapsed_time(e1))
        last = outs[(a.steps - 1) % 2]
        d2h = sum(getattr(last, f).numel() * getattr(last, f).element_size()
                  for f in ("noise_variance", "negative_log_evidence", "status", "active_indices",
                            "active_values", "x") if getattr(last, f) is not None)
        return job_rate(B, a.steps, world, t), last, d2h

    e2e, host_res, e2e_d2h = run_pipeline(False)
    e2e_dense, _, e2e_dense_d2h = run_pipeline(True)

    # quality of this batch (raw NMSE, no gain alignment), from the host result
    x_hat = host_res.dense_x(GRID).numpy().reshape(B, -1)
    assert np.array_equal(x_hat, res.x.cpu().numpy().reshape(B, -1))
    num = np.sum(np.abs(x_hat - x_true.reshape(B, -1)) ** 2, axis=1)
    den = np.sum(np.abs(x_true.reshape(B, -1)) ** 2, axis=1)
    nmse_db = float(10.0 * np.log10(np.mean(num / den)))
    status_bad = int((res.status != 0).sum().item())

    # live per-kernel timing (one eagerly launched replay with CUDA events)
    prof = plan._engine.profile(plan.input_buffer.view(B, -1))
    n, m = GRID[0] * GRID[1], PREFIX[0] * PREFIX[1]
    launches = sum(c for _, c in prof.values())
    dom = max(prof.items(), key=lambda kv: kv[1][0])
    dom_name, (dom_ms, dom_cnt) = dom
    per_launch_s = dom_ms / max(dom_cnt, 1) / 1000.0
    alg = algorithmic_bytes(dom_name, n, m) * B
    peaks = _peaks()
    peak = peaks["hbm"]
    achieved = alg / per_launch_s / 1e9 if alg else None
    fft_stages = int(plan._engine.native_cfg.dft_terms) == 0
    stages = stages_table(prof, B, GRID, PREFIX, peaks, int(plan._engine.native_cfg.dft_terms))
    t_u = plan._engine.native_cfg.uamp_iterations
    p_iters = plan._engine.native_cfg.polish_iterations
    step_bytes = scene_bytes(n, m, t_u, p_iters) * B
    step_gbs = step_bytes / (ms / a.steps / 1000.0) / 1e9

    cpu = None
    if rank == 0 and world == 1 and not a.no_cpu:
        cpu = cpu_baseline(a.profile, a.cpu_rounds)
    cg = cg_section(device) if world == 1 and not a.no_cg else None
    certificate = certificate_section(device, a.steps) if world == 1 and not a.no_certificate else None
    learned = None
    if world == 1 and not a.no_learned:
        learned = learned_section(device, min(a.steps, 20), a.batch)
    uneven = None
    if world == 1 and not a.no_uneven:
        uneven = uneven_section(device, min(a.steps, 20))
    published = published_shape_section(device) if world == 1 and not a.no_uneven else None
    precision = None
    if world == 1 and not a.no_precision:
        precision = precision_section(device, min(a.steps, 20), y_dev)

    if rank == 0:
        line = {
            "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": a.steps,
            "warmup": a.warmup, "ms_per_step": ms / a.steps, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "c64", "data": "synthetic",
            "config": {
                "workload": WORKLOAD, "profile": a.profile, "scenes_per_step_per_gpu": B,
                "parallelism": f"scene-sharded x{world}", "l2": "inputs larger than L2 "
                f"(resident state {step_bytes / 1e6:.0f} MB algorithmic traffic per step)",
                "dft": DFT_FORMS[int(plan._engine.native_cfg.dft_terms)],
                "nmse_db": nmse_db, "scenes_with_status": status_bad,
            },
            "e2e": {"value": e2e, "unit": UNIT, "h2d_bytes_per_step": int(y_host.numel() * 8),
                    "d2h_bytes_per_step": int(e2e_d2h),
                    "api": "fbme_b200.streaming.HostPipeline (pinned host batches, copies overlapped with "
                           "the neighbouring solves); result: active indices + x values (x is zero "
                           "elsewhere), noise variance, evidence, status",
                    "dense": {"value": e2e_dense, "d2h_bytes_per_step": int(e2e_dense_d2h)}},
            "roofline": {
                "bound": "hbm", "kernel": dom_name,
                "achieved": achieved, "peak": peak, "unit": "GB/s",
                "frac": (achieved / peak) if achieved else None,
                "traffic": physical_bytes(dom_name, GRID, PREFIX, fft_stages) * B or None,
                "traffic_source": ("the kernel's own byte accounting (bench.physical_bytes: adjoint "
                                   "stage 2 with the denoiser in its epilogue reads the intermediate U, "
                                   "8 N2 M1 B per scene beyond the algorithmic 32 B/px)" if fft_stages else
                                   "the kernel's own byte accounting (bench.physical_bytes: the lift "
                                   "A^H m that adjoint stage 2 writes is read back, 8 B/px beyond the "
                                   "algorithmic 32 B/px)") + "; ncu DRAM counters agree in profiles/",
                "algorithmic_bytes_per_launch": alg, "launch_ms": per_launch_s * 1000.0,
                "peak_source": peaks["source"],
                "step_algorithmic_gbs": step_gbs, "step_frac": step_gbs / peak,
                "stages": stages,
            },
            "kernel_ms_per_replay": {k: round(v[0], 4) for k, v in prof.items()},
            "gpu_launches": launches * a.steps,
            "launches_per_step": launches,
            "clocks": clk,
        }
        if cpu is not None:
            line["cpu_baseline"] = cpu
        if learned is not None:
            line["learned"] = learned
        if uneven is not None:
            line["uneven"] = uneven
        if cg is not None:
            line["cg"] = cg
        if certificate is not None:
            line["certificate"] = certificate
        if published is not None:
            line["published_shape"] = published
        if precision is not None:
            line["precision"] = precision
        print(json.dumps(line), flush=True)
    del plan
    if dist is not None:
        dist.barrier()
        dist.destroy_process_group()


def main() -> None:
    a = _args()
    if a.impl == "reference":
        run_reference(a)
    else:
        run_ours(a)


if __name__ == "__main__":
    main()
