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


PIECE = 148 * 14 * 4 * 32  # samples of one launch: four tiles per warp
CHAIN = (128 + 14) * 2.0 ** -24  # relative error bound of 128 FP32 additions per warp and 14 warps


def equal_samples(n):
    """A trainer of n equal samples: the mean gradient over any number of them is one sample's."""
    rng = np.random.default_rng(3)
    x, t = rng.normal(0.0, 1.0, (1, 10)).astype(np.float32), np.float32([0.004])
    tr = Trainer(n)
    tr.add_samples(np.repeat(x, n, 0), np.repeat(t, n))
    tr.params = mo.random_params(5)
    return tr


@pytest.mark.parametrize("log2", [15, 18, 20, 22])
def test_long_sums_keep_their_accuracy(log2):
    tr = equal_samples(1 << log2)
    loss1, one = tr.gradient(0, 1)
    loss, g = tr.gradient(0, 1 << log2)  # a power of two: 1/count scales every term exactly
    assert abs(loss - loss1) <= CHAIN * loss1
    for k in one:
        assert np.all(np.abs(np.asarray(g[k]) - np.asarray(one[k])) <= CHAIN * np.abs(one[k])), k
    tr.close()


@pytest.mark.parametrize("count", [PIECE - 1, PIECE, PIECE + 1, 2 * PIECE + 33])
def test_gradient_at_piece_edges(count):
    rng = np.random.default_rng(12)
    n = 2 * PIECE + 64
    x = rng.normal(0.0, 1.0, (n, 10)).astype(np.float32)
    t = rng.uniform(0.0, 0.02, n).astype(np.float32)
    p = mo.random_params(5)
    tr = Trainer(n)
    tr.add_samples(x, t)
    tr.params = p
    first = n - count
    loss, g = tr.gradient(first, count)
    p32 = {k: np.asarray(v, dtype=np.float32).astype(np.float64) for k, v in p.items()}
    want_loss, want = mo.loss_and_grad64(p32, x[first:], t[first:])
    assert abs(loss - want_loss) <= 1e-5 * abs(want_loss)
    for k in want:
        a, b = np.asarray(g[k], np.float64).ravel(), np.asarray(want[k], np.float64).ravel()
        assert np.linalg.norm(a - b) <= 2e-5 * np.linalg.norm(b) + 1e-12, k
    tr.close()


def test_training_step_over_several_pieces():
    """One Adam step on equal samples: whatever rows the batch draws, the parameters move as with a
    batch of one (the update of a gradient g is lr g / (|g| + 1e-8), so a relative error of g moves
    it by no more than that part of lr)."""
    n, lr = 4096, 1e-3
    tr = equal_samples(n)
    start = tr.params
    last1 = tr.train(1, 1, lr, 7)
    one = tr.params
    tr.params = start
    last = tr.train(1, 2 * PIECE + 4 * 32, lr, 7)
    many = tr.params
    assert abs(last - last1) <= 2.0 * CHAIN * last1
    for k in ("w1", "b1", "w2", "b2", "w3", "b3"):
        a, b = np.asarray(many[k]), np.asarray(one[k])
        # 2 CHAIN: the sums, and 1/count rounded; FP32 rounding of the parameter and the update
        assert np.all(np.abs(a - b) <= lr * (2.0 * CHAIN + 2.0 ** -20) + 2.0 ** -23 * np.abs(b)), k
    tr.close()
