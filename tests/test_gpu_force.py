"""The one-launch force reduction at its edges: one block, a ragged last block, every block of
the fixed scratch (boxes beyond 512 x 256 cells), against the FP64 sum over the read-back
populations; and the destinations a queued force can be written to."""
import numpy as np
import pytest

from periodicshiftlbm_b200 import getSphereForce, getSphereForceAsync, make_sphere_grids, updateGrid
from periodicshiftlbm_b200._lib import CELL_SOLID
from periodicshiftlbm_b200.cases import SphereConfig

pytestmark = pytest.mark.gpu

CX = np.array([0, 1, -1, 0, 0, 0, 0, 1, -1, 1, -1, -1, 1, 0, 0, -1, 1, 0, 0, -1, 1, -1, 1, 1, -1, -1, 1])
CY = np.array([0, 0, 0, 0, 0, -1, 1, 0, 0, 0, 0, -1, 1, 1, -1, 1, -1, 1, -1, 1, -1, -1, 1, -1, 1, -1, 1])
CZ = np.array([0, 0, 0, -1, 1, 0, 0, -1, 1, 1, -1, 0, 0, -1, 1, 0, 0, 1, -1, -1, 1, 1, -1, -1, 1, -1, 1])


def sphere(n, radius):
    cfg = SphereConfig(name="force", nx=n, ny=n, nz=n, sphere=(n / 2, n / 2, n / 2), radius=radius, u_in=0.05, nu=0.01)
    grids, case = make_sphere_grids(cfg)
    for _ in range(2):
        updateGrid(grids, 0)
    return grids[0], case


@pytest.mark.parametrize("n,radius", [(16, 1.5), (16, 2.6), (32, 9.0), (64, 27.0)])
def test_force_against_read_back_populations(n, radius):
    g, case = sphere(n, radius)
    f = g.fArray.astype(np.float64)
    solid = (g.markers & 7) == CELL_SOLID
    terms = [2.0 * (c[:, None] * f[:, solid]).sum(0) for c in (CX, CY, CZ)]
    got = getSphereForce(g, case)
    for t, v in zip(terms, got):
        # FP64 sums in another order: 2^-53 per addition of the magnitudes, some 1e5 of them
        assert abs(v - t.sum()) <= 1e-11 * np.abs(t).sum()
    g.close()


def test_queued_force_destinations():
    import torch

    g, case = sphere(32, 9.0)
    want = getSphereForce(g, case)
    pinned = torch.zeros(3, dtype=torch.float64).pin_memory()
    device = torch.zeros(3, dtype=torch.float64, device="cuda")
    pageable = np.zeros(3)
    odd = torch.zeros(40, dtype=torch.uint8).pin_memory()  # 4 bytes off: no aligned doubles
    for ptr in (pinned.data_ptr(), device.data_ptr(), pageable.ctypes.data, odd.data_ptr() + 4):
        getSphereForceAsync(g, case, ptr)
    g.synchronize()
    torch.cuda.synchronize()
    assert np.array_equal(pinned.numpy(), want)
    assert np.array_equal(device.cpu().numpy(), want)
    assert np.array_equal(pageable, want)
    assert np.array_equal(odd.numpy()[4:28].copy().view(np.float64), want)
    g.close()


def test_queued_force_at_the_end_of_its_range():
    """The last three doubles of a registered range and of a device allocation."""
    import torch

    g, case = sphere(32, 9.0)
    want = getSphereForce(g, case)
    page = 4096
    raw = np.zeros(3 * page, dtype=np.uint8)
    start = -raw.ctypes.data % page  # one page of it registered, pageable memory behind
    host = raw[start:start + page]
    cudart = torch.cuda.cudart()
    assert int(cudart.cudaHostRegister(host.ctypes.data, page, 0)) == 0
    try:
        device = torch.zeros(1 << 20, dtype=torch.float64, device="cuda")
        getSphereForceAsync(g, case, host.ctypes.data + page - 24)
        getSphereForceAsync(g, case, device.data_ptr() + 8 * ((1 << 20) - 3))
        g.synchronize()
        torch.cuda.synchronize()
        assert np.array_equal(host[-24:].copy().view(np.float64), want)
        assert np.array_equal(device[-3:].cpu().numpy(), want)
        assert not host[:-24].any() and not raw[start + page:].any()
    finally:
        assert int(cudart.cudaHostUnregister(host.ctypes.data)) == 0
    g.close()


def test_replayed_captures_and_direct_calls_interleaved():
    """Captured force calls over two boxes (a few blocks, and all 512 of the scratch) replayed with
    direct calls in between: every result is the direct call's, bit for bit."""
    import copy

    import torch

    g, small = sphere(64, 5.0)
    large = copy.copy(small)
    large.radius = 27.0  # the same solid cells inside a box of 55^3 cells
    want = {"small": getSphereForce(g, small), "large": getSphereForce(g, large)}
    got = {k: torch.zeros(3, dtype=torch.float64, pin_memory=True) for k in ("small", "large", "direct")}
    stream = torch.cuda.Stream()
    g.synchronize()
    g.set_stream(stream.cuda_stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        getSphereForceAsync(g, small, got["small"].data_ptr())
        getSphereForceAsync(g, large, got["large"].data_ptr())
        getSphereForceAsync(g, small, got["small"].data_ptr())
    for round_ in range(4):
        for k in got:
            got[k].fill_(float("nan"))
        with torch.cuda.stream(stream):
            graph.replay()
            getSphereForceAsync(g, large if round_ % 2 else small, got["direct"].data_ptr())
            graph.replay()
        stream.synchronize()
        for k in ("small", "large"):
            assert np.array_equal(got[k].numpy(), want[k]), (round_, k)
        assert np.array_equal(got["direct"].numpy(), want["large" if round_ % 2 else "small"]), round_
    del graph
    g.set_stream(0)
    g.close()
