"""Batched ensembles over many uneven envs, in all three modes: one launch per
stage over every env's tiles (staged), one persistent launch per step, and
the envs' own kernels as branches of one graph."""
from __future__ import annotations

import math
import time

import numpy as np
import pytest

from conftest import log_uniform
from oracle.oracle import face_mask_all

pytestmark = pytest.mark.gpu
MODES = {"persistent": 0, "staged": 1, "graph": 2}  # BFB_BATCH_MODE_*


def make_instance(bfb, rng, edge_lo, edge_hi, n_agents_max, prec, dt):
    shape = tuple(int(v) for v in rng.integers(edge_lo, edge_hi + 1, 3))
    S = int(rng.integers(1, 7))
    D, lam = log_uniform(rng, 1e2, 1e5, S), log_uniform(rng, 1e-3, 1.0, S)
    rho0 = rng.random((*shape, S))
    fm = np.zeros((6, S), np.uint8)
    fm[0, 0] = fm[1, 0] = 1  # 38.0 on the x-faces for substrate 0, as the 200^3 agents workload has
    act = np.zeros(S, np.uint8)
    act[0] = 1
    na = int(rng.integers(0, n_agents_max + 1))
    box = np.array(shape) * 20.0
    pos = rng.random((na, 3)) * box
    vol = np.full(na, 4.0 / 3.0 * math.pi * 125.0)
    sec, upt, sat = log_uniform(rng, 1e-2, 10.0, (3, na, S))
    spec = dict(shape=shape, S=S, D=D, lam=lam, rho0=rho0, fm=fm, act=act, pos=pos, vol=vol, sec=sec, upt=upt,
                sat=sat, box=(0, 0, 0, *box))
    return spec, build(bfb, spec, prec, dt)


def build(bfb, spec, prec, dt):
    env = bfb.Env(spec["shape"], spec["S"], dx=20.0, precision=prec)
    env.set_coefficients(spec["D"], spec["lam"])
    env.set_field(spec["rho0"])
    env.set_dirichlet_uniform(spec["act"], np.full(spec["S"], 38.0), face_mask=spec["fm"])
    if len(spec["pos"]):
        env.set_agents(spec["pos"], spec["vol"], spec["sec"], spec["upt"], spec["sat"], dt)
    return env


def oracle_run(oracle, spec, dt, steps):
    rho = spec["rho0"]
    vals = np.full_like(rho, 38.0)
    fm = spec["fm"] * spec["act"][None, :]
    if len(spec["pos"]):
        vox = oracle.bin_agents(spec["pos"], spec["box"], 20.0, spec["shape"])
        vox = np.where(vox < 0, 0, vox)
        t1, t2 = oracle.agent_constants(dt, 20.0, spec["vol"], spec["sec"], spec["upt"], spec["sat"])
    for _ in range(steps):
        rho = oracle.lod_steps(rho, dt, 20.0, spec["D"], spec["lam"], 1, vals, fm)
        if len(spec["pos"]):
            rho = oracle.cells_step(rho, vox, t1, t2)
    return rho


@pytest.mark.parametrize("mode", ["staged", "persistent", "graph"])
@pytest.mark.parametrize("warps", [1, 2])
def test_batch_small_fp64_bitexact(bfb, oracle, warps, mode):
    rng = np.random.default_rng(404)
    dt, steps = 0.01, 4
    specs, envs = zip(*[make_instance(bfb, rng, 2, 24, 300, bfb.FP64, dt) for _ in range(12)])
    batch = bfb.Batch(envs)
    batch.set_mode(MODES[mode])
    batch.set_warps(warps)
    batch.simulate(dt, steps, bfb.STEP_DIFFUSION | bfb.STEP_CELLS)
    batch.synchronize()
    for spec, env in zip(specs, envs):
        assert np.array_equal(env.get_field(), oracle_run(oracle, spec, dt, steps)), spec["shape"]


def make_aligned_instance(bfb, rng, prec, dt, n_agents=400):
    """Shapes whose row pitches suit TMA on every axis (edges multiples of 8,
    S in {2, 4}), so every stage of the persistent kernel runs TMA tiles."""
    shape = tuple(int(v) * 8 for v in rng.integers(2, 7, 3))
    S = int(rng.choice([2, 4]))
    D, lam = log_uniform(rng, 1e2, 1e5, S), log_uniform(rng, 1e-3, 1.0, S)
    rho0 = rng.random((*shape, S))
    fm = np.zeros((6, S), np.uint8)
    fm[:, 0] = [1, 1, 0, 1, 1, 0]
    act = np.zeros(S, np.uint8)
    act[0] = 1
    box = np.array(shape) * 20.0
    pos = rng.random((n_agents, 3)) * box
    vol = np.full(n_agents, 4.0 / 3.0 * math.pi * 125.0)
    sec, upt, sat = log_uniform(rng, 1e-2, 10.0, (3, n_agents, S))
    spec = dict(shape=shape, S=S, D=D, lam=lam, rho0=rho0, fm=fm, act=act, pos=pos, vol=vol, sec=sec, upt=upt,
                sat=sat, box=(0, 0, 0, *box))
    return spec, build(bfb, spec, prec, dt)


@pytest.mark.parametrize("mode,warps,tiles", [("persistent", 1, 1), ("persistent", 2, 3), ("persistent", 4, 8),
                                              ("persistent", 1, 64), ("staged", 1, 2), ("staged", 4, 2),
                                              ("graph", 1, 2)])
def test_batch_tma_items_fp64_bitexact(bfb, oracle, mode, warps, tiles):
    rng = np.random.default_rng(900 + warps * 10 + tiles)
    dt, steps = 0.01, 3
    specs, envs = zip(*[make_aligned_instance(bfb, rng, bfb.FP64, dt) for _ in range(6)])
    batch = bfb.Batch(envs)
    batch.set_mode(MODES[mode])
    assert batch.mode == MODES[mode]
    batch.set_warps(warps)
    batch.set_tiles_per_item(tiles)
    batch.simulate(dt, steps, bfb.STEP_DIFFUSION | bfb.STEP_CELLS)
    batch.synchronize()
    for spec, env in zip(specs, envs):
        assert np.array_equal(env.get_field(), oracle_run(oracle, spec, dt, steps)), spec["shape"]


@pytest.mark.parametrize("warps", [1, 2, 4])
@pytest.mark.parametrize("steps", [3, 9])
def test_batch_many_small_and_one_large_fp64_bitexact(bfb, oracle, warps, steps):
    """More envs than the staged mode steps by their own kernels: small ones share stage launches
    while one larger env (over 1 MB) runs its own chain beside them; bit for bit."""
    dt = 0.01
    rng = np.random.default_rng(77)
    made = [make_instance(bfb, rng, 1, 14, 60, bfb.FP64, dt) for _ in range(39)]
    made.append(make_instance(bfb, rng, 52, 56, 500, bfb.FP64, dt))
    specs, envs = zip(*made)
    batch = bfb.Batch(envs)
    batch.set_warps(warps)
    batch.simulate(dt, steps, bfb.STEP_DIFFUSION | bfb.STEP_CELLS)
    batch.synchronize()
    for spec, env in zip(specs, envs):
        assert np.array_equal(env.get_field(), oracle_run(oracle, spec, dt, steps))


@pytest.mark.parametrize("mode", ["staged", "persistent", "graph"])
def test_batch_wide_substrates_fp64_bitexact(bfb, oracle, mode):
    """Envs with more than 32 substrates (a lane solves several z lines) next
    to ordinary ones in one batch."""
    rng = np.random.default_rng(77)
    dt, steps = 0.01, 3
    specs, envs = [], []
    for shape, S in (((6, 5, 7), 40), ((9, 4, 6), 33), ((8, 8, 8), 3)):
        D, lam = log_uniform(rng, 1e2, 1e5, S), log_uniform(rng, 1e-3, 1.0, S)
        fm = np.zeros((6, S), np.uint8)
        fm[0, 0] = fm[1, 0] = 1
        act = np.zeros(S, np.uint8)
        act[0] = 1
        spec = dict(shape=shape, S=S, D=D, lam=lam, rho0=rng.random((*shape, S)), fm=fm, act=act,
                    pos=np.zeros((0, 3)), vol=np.zeros(0), sec=None, upt=None, sat=None, box=None)
        specs.append(spec)
        envs.append(build(bfb, spec, bfb.FP64, dt))
    batch = bfb.Batch(envs)
    batch.set_mode(MODES[mode])
    batch.simulate(dt, steps, bfb.STEP_DIFFUSION)
    batch.synchronize()
    for spec, env in zip(specs, envs):
        assert np.array_equal(env.get_field(), oracle_run(oracle, spec, dt, steps)), (spec["shape"], spec["S"])


def test_batch_autotune_restores_fields(bfb, oracle):
    rng = np.random.default_rng(31)
    dt, steps = 0.01, 2
    specs, envs = zip(*[make_aligned_instance(bfb, rng, bfb.FP64, dt) for _ in range(5)])
    batch = bfb.Batch(envs)
    before = [e.get_field_raw() for e in envs]
    (w, t), ms = batch.autotune(dt, bfb.STEP_DIFFUSION | bfb.STEP_CELLS, trials=1)
    assert w in (1, 2, 4) and t in (1, 2, 4, 8) and ms > 0
    assert batch.mode in (bfb.BATCH_MODE_STAGED, bfb.BATCH_MODE_PERSISTENT, bfb.BATCH_MODE_GRAPH)
    for e, b0 in zip(envs, before):
        assert np.array_equal(e.get_field_raw(), b0)
    batch.simulate(dt, steps, bfb.STEP_DIFFUSION | bfb.STEP_CELLS)
    batch.synchronize()
    for spec, env in zip(specs, envs):
        assert np.array_equal(env.get_field(), oracle_run(oracle, spec, dt, steps))


@pytest.mark.parametrize("mode", ["staged", "persistent", "graph"])
def test_batch_fp32_equals_per_instance_loop(bfb, mode):
    rng = np.random.default_rng(405)
    dt, steps = 0.01, 5
    made = [make_instance(bfb, rng, 3, 40, 800, bfb.FP32, dt) for _ in range(10)]
    specs = [m[0] for m in made]
    envs_b = [m[1] for m in made]
    envs_l = [build(bfb, sp, bfb.FP32, dt) for sp in specs]
    b = bfb.Batch(envs_b)
    b.set_mode(MODES[mode])
    b.simulate(dt, steps, bfb.STEP_DIFFUSION | bfb.STEP_CELLS)
    b.synchronize()
    lp = bfb.Batch(envs_l)
    lp.simulate_loop(dt, steps, bfb.STEP_DIFFUSION | bfb.STEP_CELLS)
    for eb, el in zip(envs_b, envs_l):
        assert np.array_equal(eb.get_field_raw(), el.get_field_raw())


def test_ensemble_256_batch_vs_loop_and_fp64_check(bfb):
    """Uneven ensemble: 256 envs, edges U{32..160} per axis, 1-6 substrates, 0-20k
    agents each, 200 steps in FP32; FP64 check on 8 sampled envs; the batch
    (staged launches, and one persistent launch per step) against the
    per-instance launch loop."""
    rng = np.random.default_rng(4)
    dt, steps = 0.01, 200
    made = [make_instance(bfb, rng, 32, 160, 20_000, bfb.FP32, dt) for _ in range(256)]
    specs = [m[0] for m in made]
    envs = [m[1] for m in made]
    vs = sum(int(np.prod(sp["shape"])) * sp["S"] for sp in specs)
    flags = bfb.STEP_DIFFUSION | bfb.STEP_CELLS
    batch = bfb.Batch(envs)

    def timed(n):
        batch.simulate(dt, 2, flags)  # warm-up (graph capture)
        batch.synchronize()
        t0 = time.perf_counter()
        batch.simulate(dt, n, flags)
        batch.synchronize()
        return (time.perf_counter() - t0) / n

    batch.set_mode(bfb.BATCH_MODE_PERSISTENT)
    batch.set_warps(1)
    batch.set_tiles_per_item(4)
    t_pers = timed(20)
    batch.set_mode(bfb.BATCH_MODE_STAGED)
    t_staged = timed(20)
    batch.set_mode(bfb.BATCH_MODE_GRAPH)
    t_graph = timed(20)
    tuned, _ = batch.autotune(dt, flags, trials=2)  # mode, warps per CTA and tiles per item
    mode = {v: k for k, v in MODES.items()}[batch.mode]
    t_batch = timed(steps - 66)  # 202 steps in all (4 x 2 warm + 3 x 20 + 134), as the FP64 check below
    # per-instance launch loop over fresh copies of the same envs
    loop_envs = [build(bfb, sp, bfb.FP32, dt) for sp in specs]
    loop = bfb.Batch(loop_envs)
    loop.simulate_loop(dt, 2, flags)
    t0 = time.perf_counter()
    loop.simulate_loop(dt, steps, flags)
    t_loop = (time.perf_counter() - t0) / steps
    # FP64 check on 8 sampled envs (same 202 steps)
    pick = rng.choice(len(specs), 8, replace=False)
    errs = []
    for q in pick:
        e64 = build(bfb, specs[q], bfb.FP64, dt)
        e64.simulate(dt, steps + 2, flags)
        e64.synchronize()
        errs.append(envs[q].compare(e64)[0])
        e64.close()
    print(f"\nuneven ensemble (256 envs, {vs / 1e6:.0f} M voxel*substrates, 200 steps): batch, autotuned "
          f"({mode}, warps, tiles per item = {tuned}) {t_batch * 1e3:.3f} ms/step ({vs / t_batch:.3e} vox*sub/s); "
          f"staged (1 warp) {t_staged * 1e3:.3f}, persistent (1 warp, 4 tiles) {t_pers * 1e3:.3f}, "
          f"graph {t_graph * 1e3:.3f}; "
          f"per-instance loop {t_loop * 1e3:.3f} ms/step ({vs / t_loop:.3e}); "
          f"FP32 vs FP64 rel Linf on 8 envs: max {max(errs):.2e}")
    assert max(errs) <= 1e-5


def shared_stage_envs(bfb, kind, prec, dt, n=36):
    """More envs than a batch steps by their own kernels, each under 1 MB, so that all share the
    staged mode's launches: ragged shapes, shapes whose rows suit TMA on every axis, some with
    more than 32 substrates, or some without bulk copies (the cp.async tiles of both widths)."""
    rng = np.random.default_rng(sum(map(ord, kind)))
    made = []
    for k in range(n):
        if kind == "aligned":
            shape, S = tuple(int(v) * 8 for v in rng.integers(1, 4, 3)), int(rng.choice([2, 4]))
        elif kind == "wide" and k % 3 == 0:
            shape, S = tuple(int(v) for v in rng.integers(2, 9, 3)), int(rng.choice([33, 40]))
        else:
            shape, S = tuple(int(v) for v in rng.integers(1, 25, 3)), int(rng.integers(1, 7))
        na = int(rng.integers(0, 200))
        sec, upt, sat = log_uniform(rng, 1e-2, 10.0, (3, na, S))
        fm = np.zeros((6, S), np.uint8)
        fm[:, 0] = [1, 1, 0, 1, 1, 0]
        act = np.zeros(S, np.uint8)
        act[0] = 1
        box = np.array(shape) * 20.0
        spec = dict(shape=shape, S=S, D=log_uniform(rng, 1e2, 1e5, S), lam=log_uniform(rng, 1e-3, 1.0, S),
                    rho0=rng.random((*shape, S)), fm=fm, act=act, pos=rng.random((na, 3)) * box,
                    vol=np.full(na, 500.0), sec=sec, upt=upt, sat=sat, box=(0, 0, 0, *box))
        env = build(bfb, spec, prec, dt)
        if kind == "plain" and k % 2:
            env.set_option(bfb.OPT_USE_TMA, 0)
        made.append((spec, env))
    return tuple(zip(*made))


@pytest.mark.parametrize("kind", ["ragged", "aligned", "wide", "plain"])
@pytest.mark.parametrize("warps", [1, 2, 4])
def test_shared_stages_fp64_bitexact(bfb, oracle, kind, warps):
    """The staged mode's shared launches on every kind of tile: FP64 against the oracle."""
    dt, steps = 0.01, 3
    specs, envs = shared_stage_envs(bfb, kind, bfb.FP64, dt)
    batch = bfb.Batch(envs)
    batch.set_mode(bfb.BATCH_MODE_STAGED)
    batch.set_warps(warps)
    batch.simulate(dt, steps, bfb.STEP_DIFFUSION | bfb.STEP_CELLS)
    batch.synchronize()
    for spec, env in zip(specs, envs):
        assert np.array_equal(env.get_field(), oracle_run(oracle, spec, dt, steps)), (spec["shape"], spec["S"])


@pytest.mark.parametrize("kind", ["ragged", "aligned", "wide", "plain"])
@pytest.mark.parametrize("warps", [1, 4])
def test_shared_stages_fp32_equal_the_loop(bfb, kind, warps):
    """The same in FP32, bit for bit against one env at a time; nine steps (both graphs)."""
    dt, steps = 0.01, 9
    _, envs = shared_stage_envs(bfb, kind, bfb.FP32, dt)
    _, alone = shared_stage_envs(bfb, kind, bfb.FP32, dt)
    batch = bfb.Batch(envs)
    batch.set_mode(bfb.BATCH_MODE_STAGED)
    batch.set_warps(warps)
    batch.simulate(dt, steps, bfb.STEP_DIFFUSION | bfb.STEP_CELLS)
    batch.synchronize()
    for eb, el in zip(envs, alone):
        el.simulate(dt, steps, bfb.STEP_DIFFUSION | bfb.STEP_CELLS)
        el.synchronize()
        assert np.array_equal(eb.get_field_raw(), el.get_field_raw()), eb.shape


def test_batch_autotune_of_own_kernels_keeps_the_warps(bfb):
    """Where every env is stepped by its own kernels the staged mode has one shape: the autotuner
    does not choose among equal ones, so a staged choice keeps the setting that has no effect."""
    rng = np.random.default_rng(32)
    dt = 0.01
    _, envs = zip(*[make_aligned_instance(bfb, rng, bfb.FP32, dt, 50) for _ in range(3)])
    batch = bfb.Batch(envs)
    for _ in range(8):
        batch.set_warps(3)
        batch.set_mode(bfb.BATCH_MODE_STAGED)
        (w, _), _ = batch.autotune(dt, bfb.STEP_DIFFUSION | bfb.STEP_CELLS, trials=1)
        assert batch.mode != bfb.BATCH_MODE_STAGED or w == 3


@pytest.mark.parametrize("mode", ["staged", "persistent", "graph"])
@pytest.mark.parametrize("n_envs", [5, 40])
def test_settings_change_while_the_batch_runs(bfb, oracle, mode, n_envs):
    """Agents (fewer, more, none), coefficients and faces set anew on a batch's envs right after a
    call that has not been waited for, and the autotuner on steps in flight: every call uses the
    settings of its own time; bit for bit."""
    dt = 0.01
    rng = np.random.default_rng(500 + n_envs)
    made = [make_instance(bfb, rng, 10, 30 if n_envs < 10 else 14, 200, bfb.FP64, dt) for _ in range(n_envs)]
    specs, envs = (list(v) for v in zip(*made))
    batch = bfb.Batch(envs)
    batch.set_mode(MODES[mode])
    want = [sp["rho0"] for sp in specs]
    flags = bfb.STEP_DIFFUSION | bfb.STEP_CELLS
    for q, (steps, n_agents) in enumerate([(40, None), (24, 30), (9, 700), (17, 0), (8, 100)]):
        if n_agents is not None:
            for k in range(0, n_envs, 2):
                sp = specs[k]
                sp["pos"] = rng.random((n_agents, 3)) * np.array(sp["shape"]) * 20.0
                sp["vol"] = np.full(n_agents, 500.0)
                sp["sec"], sp["upt"], sp["sat"] = log_uniform(rng, 1e-2, 10.0, (3, n_agents, sp["S"]))
                envs[k].set_agents(sp["pos"], sp["vol"], sp["sec"], sp["upt"], sp["sat"], dt)
            for k in range(1, n_envs, 2):
                sp = specs[k]
                if q % 2:
                    sp["D"] = log_uniform(rng, 1e2, 1e5, sp["S"])
                    envs[k].set_coefficients(sp["D"], sp["lam"])
                else:
                    sp["fm"] = np.zeros((6, sp["S"]), np.uint8)
                    sp["fm"][q, 0] = 1
                    envs[k].set_dirichlet_uniform(sp["act"], np.full(sp["S"], 38.0), face_mask=sp["fm"])
        batch.simulate(dt, steps, flags)
        for k, sp in enumerate(specs):
            want[k] = oracle_run(oracle, dict(sp, rho0=want[k]), dt, steps)
    batch.autotune(dt, flags, trials=1)  # its copies wait for the steps above
    for sp, env, w in zip(specs, envs, want):
        assert np.array_equal(env.get_field(), w), sp["shape"]
