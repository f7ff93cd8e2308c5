"""The scalar update's staged populations: grids around a block of 128 cells, every cell kind
that touches T (solid, free-slip, prescribed, fluid), FP32 and 16-bit flow storage, against
the same update evaluated in FP64 from the populations read before it."""
import numpy as np
import pytest

from periodicshiftlbm_b200 import GridStruct, InfoStruct, _lib, applyLocalCellUpdate, applyStreaming, fillEquilibriumFromFunction

pytestmark = pytest.mark.gpu

CX = np.array([0, 1, -1, 0, 0, 0, 0, 1, -1, 1, -1, -1, 1, 0, 0, -1, 1, 0, 0, -1, 1, -1, 1, 1, -1, -1, 1])
CY = np.array([0, 0, 0, 0, 0, -1, 1, 0, 0, 0, 0, -1, 1, 1, -1, 1, -1, 1, -1, 1, -1, -1, 1, -1, 1, -1, 1])
CZ = np.array([0, 0, 0, -1, 1, 0, 0, -1, 1, 1, -1, 0, 0, -1, 1, 0, 0, 1, -1, -1, 1, 1, -1, -1, 1, -1, 1])


@pytest.mark.parametrize("dims", [(8, 4, 4), (43, 3, 1), (32, 3, 4), (19, 7, 5)])
@pytest.mark.parametrize("storage", ["f32", "f16"])
def test_scalar_update_of_every_cell_kind(dims, storage):
    tau = 0.7
    g = GridStruct(InfoStruct(cellCountX=dims[0], cellCountY=dims[1], cellCountZ=dims[2], nu=0.02), storage=storage)
    n = g.cellCount
    rng = np.random.default_rng(n)
    kind = rng.choice(4, n, p=[0.4, 0.2, 0.2, 0.2])  # fluid, solid, free-slip (outer normal -y), prescribed fluid
    markers = np.full(n, _lib.CELL_FLUID, dtype=np.uint8)
    markers[kind == 1] = _lib.CELL_SOLID
    markers[kind == 2] = _lib.CELL_MIRROR | (((0 + 1) * 9 + (-1 + 1) * 3 + (0 + 1)) << 3)
    g.markers = markers
    fillEquilibriumFromFunction(g, rho=1.0, u=(0.03, -0.02, 0.01))
    g.enableScalarTransport(tau)
    given = np.where(kind == 3, rng.uniform(0.0, 1.0, n), np.nan).astype(np.float32)
    g.setScalarGiven(given)
    g.TArray = rng.uniform(0.0, 1.0, (27, n)).astype(np.float32)
    applyStreaming(g)
    T0 = g.TArray.astype(np.float64)
    applyLocalCellUpdate(g)
    f, T1 = g.fArray.astype(np.float64), g.TArray
    opposite = np.array([0] + [q + 1 if q % 2 else q - 1 for q in range(1, 27)])
    index = {(a, b, c): q for q, (a, b, c) in enumerate(zip(CX, CY, CZ))}
    reflect = np.array([index[a, -b, c] for a, b, c in zip(CX, CY, CZ)])
    for c in range(n):
        if kind[c] == 1:
            assert np.array_equal(T1[:, c], T0[opposite, c].astype(np.float32))
            continue
        T = T0[:, c].copy()
        if kind[c] == 2:  # populations leaving the outer wall (c_y = +1 for normal -y) take their reflections
            T = np.where(CY > 0, T[reflect], T)
        if kind[c] == 3:
            T[:] = given[c]
        rho = f[:, c].sum()
        u = np.array([(k * f[:, c]).sum() for k in (CX, CY, CZ)]) / rho
        mean = (f[:, c] * T).sum() / rho
        s = np.array([(k * f[:, c] * (T - mean)).sum() for k in (CX, CY, CZ)])
        want = mean + (1.0 - 1.0 / tau) * 3.0 / rho * ((CX - u[0]) * s[0] + (CY - u[1]) * s[1] + (CZ - u[2]) * s[2])
        # 16-bit flow: the collision uses the unrounded populations, f read back is rounded to 2^-11 of f - w
        assert np.max(np.abs(T1[:, c] - want)) < (2e-6 if storage == "f32" else 2e-3), (c, kind[c])
    g.close()


@pytest.mark.parametrize("dims", [(5, 3, 2), (64, 64, 63), (64, 64, 64)])  # below, just below and at 1 MiB per row
def test_scalar_populations_through_pinned_and_pageable_memory(dims):
    import ctypes

    import torch

    from periodicshiftlbm_b200._lib import call

    g = GridStruct(InfoStruct(cellCountX=dims[0], cellCountY=dims[1], cellCountZ=dims[2], nu=0.02))
    n = g.cellCount
    g.enableScalarTransport(0.7)
    g.shifter = (np.arange(27) * 7919 % n).astype(np.int32)
    want = np.random.default_rng(n).uniform(0.0, 1.0, (27, n)).astype(np.float32)
    pinned = torch.from_numpy(want.copy()).pin_memory()
    back = torch.zeros((27, n), dtype=torch.float32, pin_memory=True)
    for write_pinned in (True, False):
        g.TArray = np.zeros((27, n), np.float32)
        if write_pinned:
            call("psl_set_scalar_populations", g.handle, ctypes.c_void_p(pinned.data_ptr()))
        else:
            g.TArray = want
        assert np.array_equal(g.TArray, want)
        back.zero_()
        call("psl_get_scalar_populations", g.handle, ctypes.c_void_p(back.data_ptr()))
        assert np.array_equal(back.numpy(), want)
    g.close()


W = np.array([8 / 27] + [2 / 27] * 6 + [1 / 54] * 12 + [1 / 216] * 8)
STORE = {"f32": 2.0 ** -24, "f16": 2.0 ** -11, "bf16": 2.0 ** -8}  # rounding of a stored f - w (f32: of f)


@pytest.mark.parametrize("dims", [(8, 4, 4), (43, 3, 1), (32, 3, 4), (19, 7, 5)])
@pytest.mark.parametrize("storage", ["f32", "f16", "bf16"])
def test_scalar_update_flow_and_overrides(orc, dims, storage):
    """f and T after the update against the oracle's collision of the populations before it: solid,
    free-slip and fluid cells, each with and without a prescribed concentration (which solid cells
    ignore and free-slip cells take after mirroring)."""
    tau, nu = 0.7, 0.02
    g = GridStruct(InfoStruct(cellCountX=dims[0], cellCountY=dims[1], cellCountZ=dims[2], nu=nu), storage=storage)
    n = g.cellCount
    rng = np.random.default_rng(n + 1)
    kind = rng.choice(3, n, p=[0.4, 0.3, 0.3])  # fluid, solid, free-slip (outer normal -y)
    given = np.where(rng.random(n) < 0.4, rng.uniform(0.0, 1.0, n), np.nan).astype(np.float32)
    markers = np.full(n, _lib.CELL_FLUID, dtype=np.uint8)
    markers[kind == 1] = _lib.CELL_SOLID
    markers[kind == 2] = _lib.CELL_MIRROR | (((0 + 1) * 9 + (-1 + 1) * 3 + (0 + 1)) << 3)
    g.markers = markers
    fillEquilibriumFromFunction(g, rho=1.0, u=(0.03, -0.02, 0.01))
    g.fArray = g.fArray * (1.0 + rng.uniform(-1e-2, 1e-2, (27, n))).astype(np.float32)
    g.enableScalarTransport(tau)
    g.setScalarGiven(given)
    g.TArray = rng.uniform(0.0, 1.0, (27, n)).astype(np.float32)
    applyStreaming(g)
    f0, T0 = g.fArray, g.TArray
    applyLocalCellUpdate(g)
    f1, T1 = g.fArray, g.TArray
    opposite = np.array([0] + [q + 1 if q % 2 else q - 1 for q in range(1, 27)])
    index = {(a, b, c): q for q, (a, b, c) in enumerate(zip(CX, CY, CZ))}
    reflect = np.array([index[a, -b, c] for a, b, c in zip(CX, CY, CZ)])
    for c in range(n):
        if kind[c] == 1:
            assert np.array_equal(f1[:, c], f0[opposite, c]) and np.array_equal(T1[:, c], T0[opposite, c])
            continue
        f, T = f0[:, c].astype(np.float64), T0[:, c].astype(np.float64)
        if kind[c] == 2:
            f, T = np.where(CY > 0, f[reflect], f), np.where(CY > 0, T[reflect], T)
        if given[c] == given[c]:
            T[:] = given[c]
        f = orc.collision(f, float(np.float32(nu)), 0.0, dtype=np.float64)
        # the collision's FP32 arithmetic (5e-6 relative), then the storage rounding
        assert np.all(np.abs(f1[:, c] - f) <= 5e-6 * f + STORE[storage] * (f if storage == "f32" else np.abs(f - W)) + 1e-7), c
        rho = f.sum()
        u = np.array([(k * f).sum() for k in (CX, CY, CZ)]) / rho
        mean = (f * T).sum() / rho
        s = np.array([(k * f * (T - mean)).sum() for k in (CX, CY, CZ)])
        want = mean + (1.0 - 1.0 / tau) * 3.0 / rho * ((CX - u[0]) * s[0] + (CY - u[1]) * s[1] + (CZ - u[2]) * s[2])
        # FP32 sums of 27 terms of T in [0, 1] (27 x 2^-24 each) over f good to 5e-6, whatever f is stored as
        assert np.max(np.abs(T1[:, c] - want)) < 1e-5, (c, kind[c])
    g.close()
