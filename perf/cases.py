"""Performance cases: the calls that programs built on this library make.

A case is a dict of plain values. ``prepare`` builds what the program has in
hand before the call, ``run`` is one pass through the Python binding, ``work``
the bytes and operations the pass cannot do without, and ``exact`` the same
outputs from plain torch in FP64.

Kinds of case:
  host     one bfb_step_host call on a pinned host field: the drop-in call that
           an unmodified BioFVM driver makes once per time step
  steps    bfb_simulate on a device-resident field: the main loop (diffusion,
           with bulk terms, Dirichlet faces and agents where the model has them)
  cycle    one mechanics time step: the agents have moved (bfb_set_agents),
           diffusion steps with secretion / uptake, then the gradient vectors
           that chemotaxis reads
  gradients  the gradient vectors alone
  batch    an ensemble of uneven grids stepped together
  inverse  one training step of an inverse problem: forward, then backward with
           the gradients of the initial field, D, lambda and the agents' rates
"""
import importlib.util
import math
import random
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parents[1]
DX, DT = 20.0, 0.01
FACE_VALUE = 38.0
CELL_VOLUME = 4.0 / 3.0 * math.pi * 125.0


def _package():
    if "biofvm_b_b200" in sys.modules:
        return sys.modules["biofvm_b_b200"]
    pkg = ROOT / "biofvm-b_b200"
    spec = importlib.util.spec_from_file_location("biofvm_b_b200", pkg / "__init__.py",
                                                  submodule_search_locations=[str(pkg)])
    mod = importlib.util.module_from_spec(spec)
    sys.modules["biofvm_b_b200"] = mod
    spec.loader.exec_module(mod)
    return mod


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------
def _grid(kind, name, nx, ny, nz, S, bits, steps, **more):
    c = {"name": name, "kind": kind, "nx": nx, "ny": ny, "nz": nz, "S": S, "bits": bits, "steps": steps,
         "faces": "none", "agents": 0, "bulk": False}
    c.update(more)
    return c


def listed():
    return [
        # the smallest call: a tissue patch, one drop-in solver call on host data per time step
        _grid("host", "host_32x30x28_s2_fp64", 32, 30, 28, 2, 64, 1, faces="all"),
        # a small vessel-fed domain, every face held, one substrate, one row in four 16-byte aligned
        _grid("steps", "cube75_s1_fp64", 75, 75, 75, 1, 64, 10, faces="all"),
        # a ragged box with bulk sources (every voxel supplied and consumed) and held x faces
        _grid("steps", "ragged_s5_fp64_bulk", 101, 103, 99, 5, 64, 5, faces="x", bulk=True),
        # a mid-size tumour with three substrates on a grid that is a whole number of nothing
        _grid("steps", "ragged_s3_fp32_agents", 129, 127, 126, 3, 32, 10, faces="x", agents=20_000),
        # the reference's tumour example: 200^3 x 8, 100k cells
        _grid("steps", "tumor200_s8_fp32_agents", 200, 200, 200, 8, 32, 10, faces="x", agents=100_000),
        # the headline grid of the benchmark in both precisions
        _grid("steps", "cube256_s8_fp32", 256, 256, 256, 8, 32, 10),
        _grid("steps", "cube256_s8_fp64", 256, 256, 256, 8, 64, 4),
        # the largest grid
        _grid("steps", "cube512_s4_fp32", 512, 512, 512, 4, 32, 4),
        # the mechanics time step of an agent-based model
        _grid("cycle", "cycle_120x110x100_s4_fp32", 120, 110, 100, 4, 32, 10, faces="x", agents=40_000),
        # chemotaxis on the headline grid
        _grid("gradients", "gradients256_s8_fp32", 256, 256, 256, 8, 32, 0),
        # a parameter sweep: uneven grids with agents, stepped together
        {"name": "batch48_fp32", "kind": "batch", "envs": 48, "lo": 32, "hi": 160, "agents": 20_000, "mix": 20240,
         "bits": 32, "steps": 8},
        # fitting secretion rates, diffusion and decay to a target field
        _grid("inverse", "inverse128_s2_fp32", 128, 128, 128, 2, 32, 20, agents=10_000, every=5),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["host", "steps", "steps", "steps", "steps", "cycle", "gradients", "batch", "inverse"])
    bits = rng.choice([32, 64])
    if kind == "batch":
        return {"kind": "batch", "envs": rng.randint(4, 56), "lo": rng.randint(24, 48), "hi": rng.randint(80, 160),
                "agents": rng.choice([0, 5_000, 20_000]), "mix": rng.randrange(1 << 20), "bits": bits,
                "steps": rng.randint(2, 8)}
    top = {"host": 160, "steps": 320, "cycle": 200, "gradients": 256, "inverse": 128}[kind]
    edge = _log_int(rng, 20, top)
    nx, ny, nz = (max(8, int(edge * rng.uniform(0.75, 1.25))) for _ in range(3))
    S = rng.randint(1, 8)
    most = {"host": 6e7, "steps": 1.2e9, "cycle": 3e8, "gradients": 1.2e9, "inverse": 4e7}[kind]
    while nx * ny * nz * S * bits // 8 > most:
        if S > 1:
            S -= 1
        else:
            nx = nx * 3 // 4
    agents = _log_int(rng, 200, 100_000) if kind in ("steps", "cycle", "inverse") else 0
    agents = min(agents, nx * ny * nz // 8)
    if kind == "steps" and rng.random() < 0.4:
        agents = 0
    steps = {"host": 1, "gradients": 0, "inverse": rng.randint(4, 20)}.get(kind, rng.randint(1, 10))
    while steps > 1 and steps * nx * ny * nz * S * bits // 8 > 4e9:
        steps -= 1
    more = {"faces": rng.choice(["none", "x", "all"]), "agents": agents,
            "bulk": kind == "steps" and nx * ny * nz * S < 6e6 and rng.random() < 0.4}
    if kind == "inverse":
        more["every"] = rng.randint(2, steps)
    c = _grid(kind, "", nx, ny, nz, S, bits, steps, **more)
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# Inputs (from the seed alone)
# ---------------------------------------------------------------------------
def _mix_shapes(case):
    """(nx, ny, nz, S, agents) of every instance of a batch: part of the case, not of the seed."""
    r = random.Random(case["mix"])
    return [(r.randint(case["lo"], case["hi"]), r.randint(case["lo"], case["hi"]), r.randint(case["lo"], case["hi"]),
             r.randint(1, 6), r.randint(0, case["agents"])) for _ in range(case["envs"])]


def _log_uniform(rng, lo, hi, size):
    return np.exp(rng.uniform(np.log(lo), np.log(hi), size))


def _model(shape, S, faces, agents, bulk, seed):
    """One grid's inputs: coefficients, field (device FP64), faces, agents, bulk terms."""
    rng = np.random.default_rng([seed & 0x7FFFFFFF, *shape, S])
    nx, ny, nz = shape
    m = {"shape": shape, "S": S, "D": _log_uniform(rng, 1e2, 1e5, S), "lam": _log_uniform(rng, 1e-3, 1.0, S)}
    gen = torch.Generator(device="cuda").manual_seed(int(rng.integers(1 << 31)))
    m["rho0"] = torch.rand((nx, ny, nz, S), generator=gen, device="cuda", dtype=torch.float64)
    m["mask"] = np.zeros((6, S), np.uint8)
    m["act"] = np.zeros(S, np.uint8)
    if faces == "x":  # the first substrate enters through the x faces
        m["mask"][0:2, 0] = 1
        m["act"][0] = 1
    elif faces == "all":
        m["mask"][:] = 1
        m["act"][:] = 1
    m["value"] = np.full(S, FACE_VALUE) / (1.0 + np.arange(S))
    if agents:  # a ball of cells in the middle of the domain
        u = rng.normal(size=(agents, 3))
        u /= np.linalg.norm(u, axis=1, keepdims=True)
        u *= rng.random((agents, 1)) ** (1.0 / 3.0)
        box = np.array(shape) * DX
        m["pos"] = box / 2 + u * (0.45 * box)
        m["vol"] = np.full(agents, CELL_VOLUME)
        m["sec"], m["upt"], m["sat"] = _log_uniform(rng, 1e-2, 10.0, (3, agents, S))
    if bulk:
        m["bulk"] = [rng.random((nx, ny, nz, S)) * s for s in (0.5, FACE_VALUE, 0.2)]  # supply, target, uptake
    return m


class _FieldView:
    """The env's device field for torch, rows at the env's pitch; keeps the env alive."""

    def __init__(self, env):
        e = 8 if env.precision == 0 else 4
        nx, ny, nz, S = env.shape
        pitch = env.field_pitch() * e
        self.env = env
        self.__cuda_array_interface__ = {"shape": (nx, ny, nz, S), "typestr": "<f8" if e == 8 else "<f4",
                                         "strides": (ny * pitch, pitch, S * e, e),
                                         "data": (env.field_device_ptr(), False), "version": 3, "stream": None}


def _env(bfb, m, bits, with_field=True):
    env = bfb.Env(m["shape"], m["S"], dx=DX, precision=bfb.FP64 if bits == 64 else bfb.FP32)
    env.set_coefficients(m["D"], m["lam"])
    if m["act"].any():
        env.set_dirichlet_uniform(m["act"], m["value"], face_mask=m["mask"])
    if with_field:
        torch.cuda.synchronize()  # the field is made on torch's stream, the env copies on its own
        env.set_field_device(m["rho0"].data_ptr(), bfb.FP64)
    return env


def _set_agents(env, m):
    env.set_agents(m["pos"], m["vol"], m["sec"], m["upt"], m["sat"], DT)


def _case_model(case, seed):
    return _model((case["nx"], case["ny"], case["nz"]), case["S"], case["faces"], case["agents"], case["bulk"], seed)


def prepare(case, seed):
    bfb = _package()
    kind, bits = case["kind"], case["bits"]
    dtype = torch.float64 if bits == 64 else torch.float32
    st = {"kind": kind, "steps": case["steps"], "flags": bfb.STEP_DIFFUSION}
    if kind == "batch":
        envs = []
        for q, (nx, ny, nz, S, na) in enumerate(_mix_shapes(case)):
            m = _model((nx, ny, nz), S, "x", na, False, seed * 1009 + q)
            env = _env(bfb, m, bits)
            if na:
                _set_agents(env, m)
            envs.append(env)
        st["flags"] |= bfb.STEP_CELLS
        st["batch"] = bfb.Batch(envs)
        st["fields"] = [torch.as_tensor(_FieldView(e), device="cuda") for e in envs]
        return st
    m = _case_model(case, seed)
    if kind == "host":
        st["env"] = _env(bfb, m, bits, with_field=False)
        st["host"] = torch.empty(m["rho0"].shape, dtype=torch.float64, pin_memory=True)
        st["host"].copy_(m["rho0"])
        return st
    if kind == "inverse":
        from biofvm_b_b200 import autograd
        st["env"] = _env(bfb, m, bits, with_field=False)
        st["simulate"] = autograd.simulate
        st["every"] = case["every"]
        st["rho0"] = m["rho0"].to(dtype).requires_grad_()
        st["target"] = (0.5 * m["rho0"]).to(dtype)
        for k in ("D", "lam"):
            st[k] = torch.tensor(m[k], requires_grad=True)
        st["agents"] = None
        if case["agents"]:
            st["agents"] = {"pos": m["pos"], "volume": m["vol"], "dt": DT}
            for k in ("sec", "upt", "sat"):
                st[k] = torch.tensor(m[k], requires_grad=True)
        return st
    env = st["env"] = _env(bfb, m, bits)
    st["field"] = torch.as_tensor(_FieldView(env), device="cuda")
    if kind in ("cycle", "gradients"):
        st["grad"] = torch.empty((*m["shape"], m["S"], 3), device="cuda", dtype=dtype)
    if kind == "cycle":
        st["agents"] = m if case["agents"] else None
        st["flags"] |= bfb.STEP_CELLS
    elif case["agents"]:
        _set_agents(env, m)
        st["flags"] |= bfb.STEP_CELLS
    if case["bulk"]:
        env.set_bulk(*m["bulk"])
        st["flags"] |= bfb.STEP_BULK
    return st


def run(st):
    kind, steps, flags = st["kind"], st["steps"], st["flags"]
    if kind == "steps":
        st["env"].simulate(DT, steps, flags)
        return st["field"]
    if kind == "host":
        st["env"].step_host_ptr(st["host"].data_ptr(), DT, steps)
        return st["host"]
    if kind == "gradients":
        st["env"].compute_gradients_device(st["grad"].data_ptr())
        return st["grad"]
    if kind == "batch":
        st["batch"].simulate(DT, steps, flags)
        return st["fields"]
    if kind == "cycle":
        env = st["env"]
        out = {"field": st["field"], "gradients": st["grad"]}
        if st["agents"] is not None:
            _set_agents(env, st["agents"])
            out["voxels"] = env.agent_voxels()
        env.simulate(DT, steps, flags)
        env.compute_gradients_device(st["grad"].data_ptr())
        return out
    # inverse: L = 0.5 * ||u - target||^2
    rates = [st["sec"], st["upt"], st["sat"]] if st["agents"] else [None] * 3
    u = st["simulate"](st["env"], st["rho0"], st["D"], st["lam"], DT, steps, st["every"], st["agents"], *rates)
    wrt = [st["rho0"], st["D"], st["lam"]] + (rates if st["agents"] else [])
    return [u.detach(), *torch.autograd.grad(u, wrt, u.detach() - st["target"])]


# ---------------------------------------------------------------------------
# What a pass cannot do without: per diffusion step the field read and written
# once (a step couples every voxel with every other, so the steps of a pass do
# not merge), the agents' constants and the bulk terms read, the gradient
# vectors written. Operations: multiply-adds of the two substitutions per axis
# (counted as 2 each, 3 per voxel, substrate and axis).
# ---------------------------------------------------------------------------
def _work_grid(c, V, S, agents):
    e, N, steps = c["bits"] // 8, V * S, c["steps"]
    kind = c["kind"]
    step = 2 * N * e + 2 * agents * S * e + (2 * N * e if c.get("bulk") else 0)
    flops = steps * (18 * N + 2 * agents * S)
    if kind == "host":
        return 2 * N * 8, flops
    if kind == "gradients":
        return 4 * N * e, 6 * N
    if kind == "cycle":
        return steps * step + 4 * N * e + agents * (4 + 3 * S) * 8, flops + 6 * N
    if kind == "inverse":  # forward and reverse; the sums for D and lambda read each sweep's result and adjoint
        return 2 * steps * step + steps * 6 * N * e + agents * (4 + 6 * S) * 8, 2 * flops + steps * 18 * N
    return steps * step, flops


def work(case):
    if case["kind"] == "batch":
        got = [_work_grid(case, nx * ny * nz, S, na) for nx, ny, nz, S, na in _mix_shapes(case)]
        return {"bytes": sum(b for b, _ in got), "flops": sum(f for _, f in got)}
    b, f = _work_grid(case, case["nx"] * case["ny"] * case["nz"], case["S"], case["agents"])
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# The same in FP64 with plain torch
# ---------------------------------------------------------------------------
class _Exact:
    def __init__(self, m):
        self.m = m
        self.shape, self.S = m["shape"], m["S"]
        dev = "cuda"
        c1 = m["D"] * DT / DX / DX
        c2 = m["lam"] * DT / 3.0
        self.c1, self.c2 = (torch.tensor(v, device=dev) for v in (c1, c2))
        self.den, self.c = [], []
        for n in self.shape:
            den = np.tile(1.0 + 2.0 * c1 + c2, (n, 1))
            den[0] = den[-1] = 1.0 + c1 + c2
            if n == 1:
                den[0] = 1.0 + c2
            c = np.zeros_like(den)
            c[0] = -c1 / den[0]
            for q in range(1, n):
                den[q] += c1 * c[q - 1]
                c[q] = -c1 / den[q]
            self.den.append(torch.tensor(den, device=dev))
            self.c.append(torch.tensor(c, device=dev))
        self.value = torch.tensor(m["value"], device=dev)
        self.on = m["mask"].astype(bool) & m["act"].astype(bool)[None, :]

    def faces(self, u, value):
        for f in range(6):
            for d in np.flatnonzero(self.on[f]):
                u.select(f // 2, 0 if f % 2 == 0 else -1)[..., d] = value[d]
        return u

    def solve(self, u, axis):
        """A_axis^-1 u"""
        perm = [axis] + [q for q in range(4) if q != axis]
        v = u.permute(perm).contiguous()
        if axis == 0:
            v = v.clone()
        den, c, n = self.den[axis], self.c[axis], self.shape[axis]
        v[0].div_(den[0])
        for q in range(1, n):
            v[q].addcmul_(v[q - 1], self.c1).div_(den[q])
        for q in range(n - 2, -1, -1):
            v[q].addcmul_(v[q + 1], -c[q])
        return v.permute([perm.index(q) for q in range(4)]).contiguous()

    def agents(self):
        """Rounds of (agents, voxel, t1, t2): at most one agent of a voxel per round, in list order."""
        m = self.m
        nx, ny, nz = self.shape
        q = np.minimum(np.floor(m["pos"] / DX).astype(np.int64), np.array(self.shape) - 1)
        vox = (q[:, 0] * ny + q[:, 1]) * nz + q[:, 2]
        order = np.argsort(vox, kind="stable")
        s = vox[order]
        start = np.concatenate([[True], s[1:] != s[:-1]]) if len(s) else np.zeros(0, bool)
        first = np.maximum.accumulate(np.where(start, np.arange(len(s)), 0))
        rank = np.empty(len(s), np.int64)
        rank[order] = np.arange(len(s)) - first
        c = (DT * m["vol"] / DX**3)[:, None]
        t1, t2 = m["sec"] * m["sat"] * c, 1.0 + c * m["sec"] + c * m["upt"]
        rounds = []
        for r in range(int(rank.max()) + 1 if len(s) else 0):
            a = np.flatnonzero(rank == r)
            rounds.append([torch.tensor(x, device="cuda") for x in (a, vox[a], t1[a], t2[a])])
        return vox.astype(np.int32), rounds

    def step(self, u, bulk=None, rounds=(), keep=None):
        if bulk is not None:
            u = (u + DT * bulk[0]) / (bulk[1] * DT + 1.0)
        u = u.clone()
        for axis in range(3):
            y = self.solve(self.faces(u, self.value), axis)
            if keep is not None:
                keep.append(y)
            u = y.clone() if keep is not None else y
        u = self.faces(u, self.value).contiguous()
        flat = u.view(-1, self.S)
        for _, v, t1, t2 in rounds:
            if keep is not None:
                keep.append(flat[v])
            flat[v] = (flat[v] + t1) / t2
        return u

    def gradients(self, u):
        out = torch.zeros((*u.shape, 3), device=u.device, dtype=u.dtype)
        for a in range(3):
            n = u.shape[a]
            if n == 1:
                continue
            g = out[..., a]
            g.narrow(a, 1, n - 2).copy_((u.narrow(a, 2, n - 2) - u.narrow(a, 0, n - 2)) / (2 * DX))
            g.select(a, 0).copy_((u.select(a, 1) - u.select(a, 0)) / DX)
            g.select(a, n - 1).copy_((u.select(a, n - 1) - u.select(a, n - 2)) / DX)
        return out


def _rounded(u, bits):
    return u if bits == 64 else u.float().double()


def exact(case, seed):
    kind, bits, steps = case["kind"], case["bits"], case["steps"]
    if kind == "batch":
        outs = []
        for q, (nx, ny, nz, S, na) in enumerate(_mix_shapes(case)):
            m = _model((nx, ny, nz), S, "x", na, False, seed * 1009 + q)
            x = _Exact(m)
            u, rounds = _rounded(m["rho0"], bits), x.agents()[1] if na else ()
            for _ in range(steps):
                u = x.step(u, None, rounds)
            outs.append(u)
        return outs
    m = _case_model(case, seed)
    x = _Exact(m)
    u = _rounded(m["rho0"], bits)
    if kind == "gradients":
        return x.gradients(u)
    vox, rounds = x.agents() if case["agents"] else (None, ())
    bulk = None
    if case["bulk"]:
        s, t, k = (torch.tensor(b, device="cuda") for b in m["bulk"])
        bulk = (s * t, k + s)
    if kind != "inverse":
        for _ in range(steps):
            u = x.step(u, bulk, rounds)
        if kind == "cycle":
            out = {"field": u, "gradients": x.gradients(u)}
            if case["agents"]:
                out["voxels"] = vox
            return out
        return u
    # inverse: the transposed step, latest first
    kept = []
    for _ in range(steps):
        kept.append([])
        u = x.step(u, None, rounds, kept[-1])
    lam = u - _rounded(0.5 * m["rho0"], bits)
    zero = torch.zeros(x.S, device="cuda", dtype=torch.float64)
    g1, g2 = zero.clone(), zero.clone()  # dL/dc1, dL/dc2
    na = case["agents"]
    gt1, gt2 = (torch.zeros((na, x.S), device="cuda", dtype=torch.float64) for _ in range(2))
    for k in reversed(kept):
        lam = lam.clone()
        flat = lam.view(-1, x.S)
        for (a, v, t1, t2), before in zip(reversed(rounds), reversed(k[3:])):
            g = flat[v] / t2
            gt1[a] += g
            gt2[a] -= g * (before + t1) / t2
            flat[v] = g
        for axis in (2, 1, 0):
            mu = x.solve(x.faces(lam, zero), axis)
            y, n = k[axis], x.shape[axis]
            d = lambda t: t.narrow(axis, 0, n - 1) - t.narrow(axis, 1, n - 1)  # noqa: E731
            g1 -= (d(mu) * d(y)).sum((0, 1, 2))
            g2 -= (mu * y).sum((0, 1, 2))
            lam = mu
        lam = x.faces(lam.clone(), zero).contiguous()
    out = [u, lam, (g1 * DT / DX**2).cpu(), (g2 * DT / 3.0).cpu()]
    if na:
        c = torch.tensor(DT * m["vol"] / DX**3, device="cuda")[:, None]
        sec, sat = (torch.tensor(m[q], device="cuda") for q in ("sec", "sat"))
        out += [(gt1 * sat * c + gt2 * c).cpu(), (gt2 * c).cpu(), (gt1 * sec * c).cpu()]
    return out
