"""The training kernel's tiling at its edges: batches around one 32-sample warp tile, around
one tile per block (148 blocks) and around one tile per warp (148 blocks of 14 warps), against
the FP64 oracle's gradient."""
import numpy as np
import pytest

from oracle import mlp_oracle as mo
from periodicshiftlbm_b200.sgs import Trainer

pytestmark = pytest.mark.gpu

SAMPLES = 80_000


@pytest.mark.parametrize("count", [1, 31, 32, 33, 148 * 32, 148 * 32 + 1, 148 * 14 * 32, 148 * 14 * 32 + 1])
def test_gradient_at_tile_edges(count):
    rng = np.random.default_rng(11)
    x = rng.normal(0.0, 1.0, (SAMPLES, 10)).astype(np.float32)
    t = rng.uniform(0.0, 0.02, SAMPLES).astype(np.float32)
    p = mo.random_params(5)
    tr = Trainer(SAMPLES)
    tr.add_samples(x, t)
    tr.params = p
    first = SAMPLES - count
    loss, g = tr.gradient(first, count)
    p32 = {k: np.asarray(v, dtype=np.float32).astype(np.float64) for k, v in p.items()}
    want_loss, want = mo.loss_and_grad64(p32, x[first:], t[first:])
    # FP32 chains of at most 64 products per accumulator, 32 per pre-activation (2^-24 each),
    # summed over warps and blocks: a few 1e-6 of the norm, with room for the cells whose
    # pre-activation is within rounding of zero
    assert abs(loss - want_loss) <= 1e-5 * abs(want_loss)
    for k in want:
        a, b = np.asarray(g[k], np.float64).ravel(), np.asarray(want[k], np.float64).ravel()
        assert np.linalg.norm(a - b) <= 2e-5 * np.linalg.norm(b) + 1e-12, k
    tr.close()
