"""Performance cases: what users of the lattice update run, through its public entry points.

A pass of a flow case advances the simulation by a number of time steps and then reads the
whole state back into pinned host memory, as a run between two outputs does.  The families:

  sphere   flow past a sphere (``updateGrid`` per step): single-level or with a 2:1 refinement
           block, every storage form, with or without the learned subgrid closure, free-slip or
           velocity walls, a uniform or a per-cell Smagorinsky constant, and, where ``drag`` is
           set, the drag of every step queued into pinned memory as the reference driver reads it
  box      decaying turbulence in a periodic box (streaming, both periodic copies, update)
  channel  the customised update: body force, a moving wall, a fixed wall, forced-velocity cells
  scalar   scalar transport in a channel with a prescribed inlet concentration
  batch    many single-level sphere cases advanced together from a CUDA graph
  train    Adam steps of the learned closure, then its loss and gradient over a held-out range

Sizes of the listed cases come from the repository's own configurations (the 512x256x256 refined
sphere and its half-scale form, the 128x64x64 sphere, the 256^3 turbulence box, the 64-case batch,
the 65,536-sample training batch) or lie between them.
"""
import ctypes
import math
from dataclasses import replace

import numpy as np
import torch

from periodicshiftlbm_b200 import (GridStruct, InfoStruct, SphereConfig, applyBCPeriodicX, applyBCPeriodicY,
                                   applyLocalCellUpdate, applyStreaming, config2, fillEquilibriumFromFunction,
                                   getSphereForceAsync, make_sphere_grids, setBodyForce, updateGrid)
from periodicshiftlbm_b200._lib import CELL_FLUID, CELL_SOLID, call
from periodicshiftlbm_b200.batch import Batch, batch_configs, make_batch_grids
from periodicshiftlbm_b200.grid import MARKER_FORCED_VELOCITY, MARKER_MOVING_WALL
from periodicshiftlbm_b200.sgs import Trainer, load_params, set_sgs_mlp
from periodicshiftlbm_b200.turbulence import box_grid, fill_from_velocity, step as box_step

ELEMENT = {"f32": 4, "f16": 2, "bf16": 2}


def _sphere(name, nx, ny, nz, storage="f32", steps=100, refined=False, closure=0, walls=0, sponge=False, drag=False):
    return {"name": name, "family": "sphere", "nx": nx, "ny": ny, "nz": nz, "storage": storage, "steps": steps,
            "refined": refined, "closure": closure, "walls": walls, "sponge": sponge, "drag": drag}


def listed():
    return [
        # the smallest grid of the batched study on its own: launches and latency
        _sphere("sphere64_f32", 64, 32, 32, steps=400),
        # the reference driver's loop on the 128x64x64 validation case: one step, its drag, the next
        _sphere("sphere128_drag_f32", 128, 64, 64, steps=400, drag=True),
        # a user's own domain: odd extents, velocity walls and an outlet sponge, BF16 storage
        _sphere("sphere_odd_bf16", 251, 117, 125, storage="bf16", steps=400, walls=1, sponge=True),
        # the refined sphere at half scale (the precision study's size), FP16 storage
        _sphere("sphere256_refined_f16", 256, 128, 128, storage="f16", steps=300, refined=True),
        # the headline: the refined 512x256x256 sphere, FP32
        _sphere("sphere512_refined_f32", 512, 256, 256, steps=200, refined=True),
        # its second form: FP16 storage with the learned closure on every 4th update
        _sphere("sphere512_refined_f16_closure", 512, 256, 256, storage="f16", steps=200, refined=True, closure=4),
        # the turbulence study's coarse box, Smagorinsky, FP32
        {"name": "box256_f32", "family": "box", "M": 256, "storage": "f32", "closure": 0, "steps": 200},
        # a box of the reduced study with the closure on every update, FP16 storage
        {"name": "box128_f16_closure", "family": "box", "M": 128, "storage": "f16", "closure": 1, "steps": 300},
        # the customised update of the rotating-machinery cases
        {"name": "channel_f32", "family": "channel", "nx": 256, "ny": 98, "nz": 128, "storage": "f32", "steps": 400},
        # scalar transport on a medium channel
        {"name": "scalar_f32", "family": "scalar", "nx": 192, "ny": 98, "nz": 96, "storage": "f32", "steps": 400},
        # the batched study: 64 uneven cases per step
        {"name": "batch64_f32", "family": "batch", "count": 64, "draw": 2024, "storage": "f32", "steps": 200},
        # training of the closure at the study's batch size
        {"name": "train_65536", "family": "train", "samples": 524288, "batch": 65536, "steps": 50},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    family = rng.choice(["sphere", "sphere", "sphere", "box", "channel", "scalar", "batch", "train"])
    storage = rng.choice(["f32", "f16", "bf16"])
    if family == "sphere":
        nx = log_int(48, 400)
        ny, nz = (max(24, int(nx * rng.uniform(0.4, 0.55))) for _ in range(2))
        refined = nx >= 96 and rng.random() < 0.5
        closure = rng.choice([0, 1, 4]) if storage != "f32" else 0
        return {k: v for k, v in _sphere("", nx, ny, nz, storage=storage, steps=rng.randint(100, 200), refined=refined,
                                         closure=closure, walls=rng.choice([0, 0, 1]),
                                         sponge=closure == 0 and rng.random() < 0.3,
                                         drag=rng.random() < 0.3).items() if k != "name"}
    if family == "box":
        return {"family": "box", "M": 2 * log_int(24, 150), "storage": storage,
                "closure": rng.choice([0, 1, 4]) if storage != "f32" else rng.choice([0, 1]),
                "steps": rng.randint(100, 200)}
    if family in ("channel", "scalar"):
        nx = log_int(48, 320)
        ny, nz = (max(16, int(nx * rng.uniform(0.3, 0.6))) for _ in range(2))
        return {"family": family, "nx": nx, "ny": ny, "nz": nz, "storage": storage, "steps": rng.randint(100, 200)}
    if family == "batch":
        return {"family": "batch", "count": log_int(4, 64), "draw": rng.randint(1, 9999), "storage": storage, "steps": rng.randint(100, 200)}
    return {"family": "train", "samples": log_int(20000, 1000000), "batch": log_int(4096, 262144),
            "steps": rng.randint(20, 60)}


# ---- inputs ------------------------------------------------------------------------------
def _pinned_state(grids, rows=27):
    return [torch.empty((rows, g.cellCount), dtype=torch.float32, pin_memory=True) for g in grids]


def _sphere_config(case, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if case["refined"] and (nx, ny, nz) in ((512, 256, 256), (256, 128, 128)):
        return config2(scale=nx / 512, wall_mode=case["walls"], cs_mode=int(case["sponge"]), seed=seed)
    radius = min(ny, nz) / 10.0
    refine = None
    if case["refined"]:  # the same proportions as the 512x256x256 case
        refine = ((5 * nx // 32, 5 * ny // 16, 5 * nz // 16), (13 * nx // 32, 11 * ny // 16, 11 * nz // 16))
    les = case["refined"] or case["sponge"] or nx > 200
    return SphereConfig(name="sphere", nx=nx, ny=ny, nz=nz, sphere=(nx / 4.0, ny / 2.0, nz / 2.0), radius=radius,
                        u_in=0.05, nu=0.05 * 2 * radius / (1e5 if les else 100.0), smagorinsky=0.1 if les else 0.0,
                        wall_mode=case["walls"], seed=seed, refine=refine, cs_mode=int(case["sponge"]))


def _velocity(M, seed, u_rms=0.04, k0=4.0):
    """A seeded divergence-free random-phase velocity with E(k) ~ k^4 exp(-2 (k / k0)^2), [3, z, y, x]."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    a = torch.fft.rfftn(torch.randn((3, M, M, M), device="cuda", generator=gen), dim=(1, 2, 3))
    k = [torch.fft.fftfreq(M, 1.0 / M, device="cuda")[:, None, None], torch.fft.fftfreq(M, 1.0 / M, device="cuda")[None, :, None],
         torch.fft.rfftfreq(M, 1.0 / M, device="cuda")[None, None, :]]
    k2 = k[0] ** 2 + k[1] ** 2 + k[2] ** 2
    along = (a[0] * k[2] + a[1] * k[1] + a[2] * k[0]) / k2.clamp(min=1.0)
    a = torch.stack([a[0] - k[2] * along, a[1] - k[1] * along, a[2] - k[0] * along])
    u = torch.fft.irfftn(a * torch.sqrt(k2) * torch.exp(-k2 / k0 ** 2), s=(M, M, M), dim=(1, 2, 3))
    return (u * (u_rms / u.square().mean().sqrt())).cpu().numpy()


def _channel_start(case, seed):
    """rho, u of the channel's start as four planes [4][N]: a profile along x with a seeded perturbation."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    r = np.random.default_rng(seed)
    y = (np.arange(ny, dtype=np.float64) / (ny - 1))[None, :, None]
    phase = r.uniform(0.0, 2.0 * np.pi, (3, 4))
    x = (2.0 * np.pi * np.arange(nx) / (nx - 1))[None, None, :]
    z = (2.0 * np.pi * np.arange(nz) / nz)[:, None, None]
    out = np.empty((4, nz, ny, nx), dtype=np.float32)
    out[0] = 1.0
    for c in range(3):
        u = 0.0
        for m in range(4):
            u = u + np.cos((m + 1) * x + phase[c, m]) * np.cos((m + 1) * z + 2.0 * phase[c, m]) / (m + 1)
        out[1 + c] = (0.16 * y * (1.0 - y) if c == 0 else 0.0) + 0.01 * np.sin(np.pi * y) * u
    return np.ascontiguousarray(out.reshape(4, -1))


def _channel_parts(case):
    """(markers, given) of the channel: a fixed wall at j = 0, a wall moving along x at j = Ny - 1, a block of
    forced-velocity cells; and (markers, inlet concentration) of the scalar form."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    m = np.full((nz, ny, nx), CELL_FLUID, dtype=np.uint8)
    m[:, 0] = CELL_SOLID
    if case["family"] == "channel":
        m[:, ny - 1] = MARKER_MOVING_WALL
        m[nz // 3:nz // 2, ny // 3:ny // 2, nx // 3:nx // 2] = MARKER_FORCED_VELOCITY
        given = np.zeros((nz, ny, nx, 4), dtype=np.float32)
        given[..., 0] = 1.0
        given[:, ny - 1, :, 1] = 0.03
        given[nz // 3:nz // 2, ny // 3:ny // 2, nx // 3:nx // 2, 1:] = (0.05, 0.01, -0.01)
        return m.reshape(-1), np.ascontiguousarray(given.reshape(-1, 4))
    m[:, ny - 1] = CELL_SOLID
    conc = np.full((nz, ny, nx), np.nan, dtype=np.float32)
    conc[:, :ny // 2, 0] = 1.0
    conc[:, ny // 2:, 0] = 0.0
    conc[:, :, nx - 1] = 0.0
    return m.reshape(-1), conc.reshape(-1)


CHANNEL_NU, CHANNEL_FORCE, SCALAR_TAU = 0.005, (2e-6, 0.0, 0.0), 0.6
BOX_NU, BOX_CS = 1e-5, 0.1


def _samples(case, seed):
    """Closure features and eddy viscosities like the filtered turbulence samples."""
    r = np.random.default_rng(seed)
    n = case["samples"]
    p = load_params()
    x = (np.asarray(p["in_shift"]) + r.standard_normal((n, 10)) / np.asarray(p["in_scale"])).astype(np.float32)
    x[:, 7] = np.sqrt(np.square(x[:, :3]).sum(1) + 2.0 * np.square(x[:, 3:6]).sum(1))
    x[:, 9] = 1.0
    t = float(p["out_scale"]) * np.abs(x[:, 7] / x[:, 7].mean()) * r.exponential(1.0, n)
    return x, t.astype(np.float32)


def _start_params(case, seed):
    r = np.random.default_rng(seed + 1)
    p = load_params()
    return {"w1": r.normal(0.0, math.sqrt(0.2), (32, 10)), "b1": r.normal(0.0, 0.1, 32),
            "w2": r.normal(0.0, 0.25, (32, 32)), "b2": r.normal(0.0, 0.1, 32), "w3": r.normal(0.0, 0.18, 32),
            "b3": np.float64(0.1), "in_shift": p["in_shift"], "in_scale": p["in_scale"], "out_scale": p["out_scale"]}


def prepare(case, seed):
    family = case["family"]
    if family == "sphere":
        cfg = _sphere_config(case, seed)
        grids, sc = make_sphere_grids(cfg, storage=case["storage"])
        if case["closure"]:
            for g in grids:
                set_sgs_mlp(g, load_params(), g.Info.res / grids[0].Info.res, interval=case["closure"])
        state = {"grids": grids, "case": sc, "out": _pinned_state(grids)}
        if case["drag"]:
            state["drag"] = torch.zeros((case["steps"], 3), dtype=torch.float64, pin_memory=True)
    elif family == "box":
        g = box_grid(case["M"], BOX_NU, storage=case["storage"], cs=BOX_CS)
        if case["closure"]:
            set_sgs_mlp(g, load_params(), 1.0, interval=case["closure"] if case["storage"] != "f32" else None)
        fill_from_velocity(g, _velocity(case["M"], seed))
        state = {"grids": [g], "out": _pinned_state([g])}
    elif family in ("channel", "scalar"):
        g = GridStruct(InfoStruct(cellCountX=case["nx"], cellCountY=case["ny"], cellCountZ=case["nz"], nu=CHANNEL_NU),
                       storage=case["storage"])
        markers, field = _channel_parts(case)
        g.markers = markers
        start = _channel_start(case, seed)
        call("psl_fill_equilibrium_field", g.handle, start.ctypes.data)
        state = {"grids": [g], "out": _pinned_state([g])}
        if family == "channel":
            call("psl_set_given_field", g.handle, field.ctypes.data)
            setBodyForce(g, *CHANNEL_FORCE)
        else:
            g.enableScalarTransport(SCALAR_TAU)
            g.setScalarGiven(field)
            state["scalar"] = torch.empty((27, g.cellCount), dtype=torch.float32, pin_memory=True)
    elif family == "batch":
        configs = [replace(c, seed=c.seed + seed) for c in batch_configs(case["count"], case["draw"])]
        grids, _ = make_batch_grids(configs, storage=case["storage"])
        n = sum(g.cellCount for g in grids)
        batch = Batch(grids)
        batch.autotune(2)  # as the batched study does before its run; does not advance the grids
        state = {"grids": grids, "batch": batch, "out": [torch.empty(27 * n, dtype=torch.float32, pin_memory=True)]}
    else:
        t = Trainer(case["samples"])
        t.add_samples(*_samples(case, seed))
        t.params = _start_params(case, seed)
        state = {"trainer": t, "held": min(case["samples"], 65536)}
    return dict(state, plan=dict(case), seed=seed % 1000)


# ---- one pass ----------------------------------------------------------------------------
def run(state):
    case = state["plan"]
    family, steps = case["family"], case.get("steps")
    if family == "train":
        t = state["trainer"]
        held_loss, grad = t.gradient(0, state["held"])
        last = t.train(steps, case["batch"], 1e-3, state["seed"])
        p = t.params
        return {"held_loss": held_loss, "grad": grad, "last_loss": last, "params": {k: p[k] for k in ("w1", "b1", "w2", "b2", "w3", "b3")}}
    grids, out = state["grids"], state["out"]
    if family == "batch":
        state["batch"].run(steps)
        at, flat = 0, out[0].numpy()
        for g in grids:
            g.read_populations(flat[at:at + 27 * g.cellCount])
            at += 27 * g.cellCount
        return out[0]
    if family == "sphere":
        drag = state.get("drag")
        for s in range(steps):
            updateGrid(grids, 0)
            if drag is not None:
                getSphereForceAsync(grids[-1], state["case"], drag.data_ptr() + 24 * s)
    elif family == "box":
        for _ in range(steps):
            box_step(grids[0])
    else:
        for _ in range(steps):
            applyStreaming(grids[0])
            applyBCPeriodicX(grids[0])
            applyLocalCellUpdate(grids[0])
    for g, h in zip(grids, out):
        g.read_populations(h.numpy())
    result = {"f": out}
    if "drag" in state:
        result["drag"] = state["drag"]
    if family == "scalar":
        call("psl_get_scalar_populations", grids[0].handle, ctypes.c_void_p(state["scalar"].data_ptr()))
        result["T"] = state["scalar"]
    return result


# ---- the work of a pass ------------------------------------------------------------------
FLOPS_PER_UPDATE = 600.0  # additions and multiplications of one cell's cumulant collision


def work(case):
    """Each step reads and writes every updated cell's 27 populations once; the final state is read once."""
    if case["family"] == "train":
        # forward 2 x 1376, backward twice that, per sample
        return {"bytes": 44.0 * (case["steps"] * case["batch"] + min(case["samples"], 65536)),
                "flops": 3.0 * 2.0 * 1376.0 * (case["steps"] * case["batch"] + min(case["samples"], 65536))}
    per = 54.0 * ELEMENT[case["storage"]]
    if case["family"] == "sphere":
        cfg = _sphere_config(case, 0)
        updates = cfg.updates_per_step()
        cells = sum(i.cellCount for i in cfg.infos())
    elif case["family"] == "box":
        updates = cells = (case["M"] + 1) ** 2 * case["M"]
    elif case["family"] == "batch":
        updates = cells = sum(c.nx * c.ny * c.nz for c in batch_configs(case["count"], case["draw"]))
    else:
        updates = cells = case["nx"] * case["ny"] * case["nz"]
    if case["family"] == "scalar":
        per, cells = per + 216.0, 2 * cells
    return {"bytes": case["steps"] * per * updates + 108.0 * cells, "flops": case["steps"] * FLOPS_PER_UPDATE * updates}


# ---- the same in 64 bits -----------------------------------------------------------------
# The D3Q27 directions in the order in which the populations come back, and their weights.
CX = (0, 1, -1, 0, 0, 0, 0, 1, -1, 1, -1, -1, 1, 0, 0, -1, 1, 0, 0, -1, 1, -1, 1, 1, -1, -1, 1)
CY = (0, 0, 0, 0, 0, -1, 1, 0, 0, 0, 0, -1, 1, 1, -1, 1, -1, 1, -1, 1, -1, -1, 1, -1, 1, -1, 1)
CZ = (0, 0, 0, -1, 1, 0, 0, -1, 1, 1, -1, 0, 0, -1, 1, 0, 0, 1, -1, -1, 1, 1, -1, -1, 1, -1, 1)
WEIGHT = tuple((8 / 27, 2 / 27, 1 / 54, 1 / 216)[abs(a) + abs(b) + abs(c)] for a, b, c in zip(CX, CY, CZ))


def _equilibrium(rho_u):
    rho, u = rho_u[0], rho_u[1:]
    u2 = (u * u).sum(0)
    out = []
    for q in range(27):
        cu = CX[q] * u[0] + CY[q] * u[1] + CZ[q] * u[2]
        out.append(rho * WEIGHT[q] * (1.0 + 3.0 * cu + 4.5 * cu * cu - 1.5 * u2))
    return torch.stack(out)


def _collide(f, nu, cs, force=None):
    """The cumulant collision with every relaxation rate but the shear rate at 1 and a Smagorinsky shear rate,
    in central moments about the (half-force shifted) velocity."""
    m = {}
    c = (CX, CY, CZ)
    rho = f.sum(0)
    j = [sum((c[a][q] * f[q] for q in range(27) if c[a][q]), torch.zeros_like(rho)) for a in range(3)]
    for a in range(3):
        for b in range(a, 3):
            m[a, b] = sum((c[a][q] * c[b][q] * f[q] for q in range(27) if c[a][q] * c[b][q]), torch.zeros_like(rho))
    u = [(j[a] + 0.5 * force[a]) / rho if force is not None else j[a] / rho for a in range(3)]
    k = {ab: m[ab] - u[ab[0]] * j[ab[1]] - u[ab[1]] * j[ab[0]] + rho * u[ab[0]] * u[ab[1]] for ab in m}
    first = [rho * u[a] - j[a] for a in range(3)]  # the first central moments change sign
    tau = 3.0 * nu + 0.5
    if cs:
        dev = sum((k[a, a] - rho / 3.0) ** 2 for a in range(3)) + 2.0 * (k[0, 1] ** 2 + k[0, 2] ** 2 + k[1, 2] ** 2)
        w = 1.0 / (0.5 * tau + 0.5 * torch.sqrt(tau * tau + 18.0 * cs * torch.sqrt(dev) / rho))
    else:
        w = torch.full_like(rho, 1.0 / tau)
    xx, yy, zz = k[0, 0], k[1, 1], k[2, 2]
    dxu = -0.5 * w / rho * (2.0 * xx - yy - zz) - 0.5 / rho * (xx + yy + zz - rho)
    dyv = dxu + 1.5 * w / rho * (xx - yy)
    dzw = dxu + 1.5 * w / rho * (xx - zz)
    g = 3.0 * rho * (1.0 - 0.5 * w)
    ea = (1.0 - w) * (xx - yy) - g * (u[0] ** 2 * dxu - u[1] ** 2 * dyv)
    eb = (1.0 - w) * (xx - zz) - g * (u[0] ** 2 * dxu - u[2] ** 2 * dzw)
    ec = rho - 1.5 * rho * (u[0] ** 2 * dxu + u[1] ** 2 * dyv + u[2] ** 2 * dzw)
    xx, yy, zz = (ea + eb + ec) / 3.0, (eb - 2.0 * ea + ec) / 3.0, (ea - 2.0 * eb + ec) / 3.0
    xy, xz, yz = (1.0 - w) * k[0, 1], (1.0 - w) * k[0, 2], (1.0 - w) * k[1, 2]
    K = {(0, 0, 0): rho, (1, 0, 0): first[0], (0, 1, 0): first[1], (0, 0, 1): first[2], (2, 0, 0): xx, (0, 2, 0): yy,
         (0, 0, 2): zz, (1, 1, 0): xy, (1, 0, 1): xz, (0, 1, 1): yz, (2, 1, 1): (xx * yz + 2.0 * xz * xy) / rho,
         (1, 2, 1): (yy * xz + 2.0 * xy * yz) / rho, (1, 1, 2): (zz * xy + 2.0 * xz * yz) / rho,
         (2, 2, 0): (xx * yy + 2.0 * xy * xy) / rho, (0, 2, 2): (yy * zz + 2.0 * yz * yz) / rho,
         (2, 0, 2): (xx * zz + 2.0 * xz * xz) / rho}
    K[2, 2, 2] = ((xx * K[0, 2, 2] + yy * K[2, 0, 2] + zz * K[2, 2, 0] + 4.0 * (yz * K[2, 1, 1] + xz * K[1, 2, 1] + xy * K[1, 1, 2])) / rho
                  - (16.0 * xy * xz * yz + 4.0 * (xz * xz * yy + yz * yz * xx + xy * xy * zz) + 2.0 * xx * yy * zz) / (rho * rho))
    for a in range(3):  # back to populations, one axis at a time: orders 0, 1, 2 -> velocities -1, 0, 1
        v, new = u[a], {}
        for rest in {key[:a] + key[a + 1:] for key in K}:
            m0, m1, m2 = (K.get(rest[:a] + (o,) + rest[a:]) for o in range(3))
            s0, s1, s2 = [], [], []
            if m0 is not None:
                s0.append(0.5 * (v * v - v) * m0), s1.append((1.0 - v * v) * m0), s2.append(0.5 * (v * v + v) * m0)
            if m1 is not None:
                s0.append((v - 0.5) * m1), s1.append(-2.0 * v * m1), s2.append((v + 0.5) * m1)
            if m2 is not None:
                s0.append(0.5 * m2), s1.append(-m2), s2.append(0.5 * m2)
            for o, s in enumerate((s0, s1, s2)):
                new[rest[:a] + (o,) + rest[a:]] = sum(s[1:], s[0])
        K = new
    return torch.stack([K[CX[q] + 1, CY[q] + 1, CZ[q] + 1] for q in range(27)])


def _stream(f, nx, ny):
    for q in range(27):
        f[q] = torch.roll(f[q], CX[q] + nx * CY[q] + nx * ny * CZ[q])


def _periodic(f, shape, axis):
    nz, ny, nx = shape
    for q in range(27):
        c, g = (CX, CY)[axis][q], f[q].view(nz, ny, nx)
        left, right = (g[:, :, 0], g[:, :, nx - 1]) if axis == 0 else (g[:, 0], g[:, ny - 1])
        if c > 0:
            left.copy_(right)
        elif c < 0:
            right.copy_(left)


def _opposite(q):
    return q if q == 0 else (q + 1 if q % 2 else q - 1)


def _scalar_collision(f, T):
    rho = f.sum(0)
    c = torch.tensor([CX, CY, CZ], dtype=torch.float64, device=f.device)
    u = torch.einsum("aq,qn->an", c, f) / rho
    mean = (f * T).sum(0) / rho
    s = torch.einsum("aq,qn->an", c, f * (T - mean))
    us = (u * s).sum(0)
    a = (1.0 - 1.0 / SCALAR_TAU) * 3.0 / rho
    return mean + a * (torch.einsum("aq,an->qn", c, s) - us)


def _exact_flow(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    family = case["family"]
    if family == "box":
        M = case["M"]
        nx, ny, nz, nu, cs = M + 1, M + 1, M, float(np.float32(BOX_NU)), float(np.float32(BOX_CS))
        u, ix = torch.from_numpy(_velocity(M, seed)).to(dev), torch.arange(M + 1, device=dev) % M
        rho_u = torch.ones((4, M, M + 1, M + 1), dtype=torch.float64, device=dev)
        rho_u[1:] = u[:, :, ix][:, :, :, ix]
        f = _equilibrium(rho_u.reshape(4, -1))
    else:
        nx, ny, nz, nu, cs = case["nx"], case["ny"], case["nz"], float(np.float32(CHANNEL_NU)), 0.0
        f = _equilibrium(torch.from_numpy(_channel_start(case, seed)).to(dev).double())
        markers, field = (torch.from_numpy(v).to(dev) for v in _channel_parts(case))
        solid = (markers & 7) == CELL_SOLID
        swap = [_opposite(q) for q in range(27)]
    if family == "channel":
        forced, u_given = (markers == MARKER_FORCED_VELOCITY), field.double()[:, 1:].T
        wall = torch.stack([6.0 * WEIGHT[q] * (CX[q] * u_given[0] + CY[q] * u_given[1] + CZ[q] * u_given[2]) for q in range(27)])
        wall = wall * (markers == MARKER_MOVING_WALL)
        body = torch.tensor([float(np.float32(v)) for v in CHANNEL_FORCE], dtype=torch.float64, device=dev)[:, None]
        c = torch.tensor([CX, CY, CZ], dtype=torch.float64, device=dev)
    if family == "scalar":
        T, given = torch.zeros_like(f), ~torch.isnan(field) & ~solid
        conc = field.double()
    for _ in range(case["steps"]):
        _stream(f, nx, ny)
        _periodic(f, (nz, ny, nx), 0)
        if family == "box":
            _periodic(f, (nz, ny, nx), 1)
            f = _collide(f, nu, cs)
            continue
        force = None
        if family == "channel":
            force = body + torch.where(forced, f.sum(0) * u_given - torch.einsum("aq,qn->an", c, f), 0.0)
        post = _collide(f, nu, cs, force)
        if family == "scalar":
            _stream(T, nx, ny)
            Tg = torch.where(given, conc, T)
            T = torch.where(solid, T[swap], _scalar_collision(post, Tg))
        back = f[swap] + wall if family == "channel" else f[swap]
        f = torch.where(solid, back, post)
    out = {"f": [f.cpu()]}
    if family == "scalar":
        out["T"] = T.cpu()
    return out


def _exact_train(case, seed):
    """The held-out loss and gradient at the start parameters; the trained parameters follow random batches."""
    x, t = (torch.from_numpy(v).double() for v in _samples(case, seed))
    n = min(case["samples"], 65536)
    p = {k: torch.tensor(np.asarray(v, dtype=np.float32), dtype=torch.float64, requires_grad=k[0] in "wb")
         for k, v in _start_params(case, seed).items()}
    xn = (x[:n] - p["in_shift"]) * p["in_scale"]
    h = torch.relu(torch.relu(xn @ p["w1"].T + p["b1"]) @ p["w2"].T + p["b2"])
    loss = torch.mean((torch.nn.functional.softplus(h @ p["w3"] + p["b3"]) - t[:n] / p["out_scale"]) ** 2)
    loss.backward()
    keys = ("w1", "b1", "w2", "b2", "w3", "b3")
    return {"held_loss": loss.item(), "grad": {k: p[k].grad.numpy() for k in keys}, "last_loss": None,
            "params": {k: None for k in keys}}


def exact(case, seed):
    """The flows without moment-based boundary conditions and without the closure, and the closure's gradient; the
    others would take a second solver (inflow, outflow, refinement) or minutes."""
    if case["family"] == "train":
        return _exact_train(case, seed)
    if case["family"] in ("channel", "scalar") or (case["family"] == "box" and not case["closure"]):
        return _exact_flow(case, seed)
    return None
