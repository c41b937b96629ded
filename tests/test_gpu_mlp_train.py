"""The passes of a training step (k_mlp_encode / _smem, k_mlp_train,
k_mlp_scatter) at the edges of their tiles: 16 rows a warp, 256 a CTA, 2^15
rows for the encoder that gathers from shared memory."""
import numpy as np
import pytest

from tests.test_gpu_mlp import LOG2, N_MAX, _cfg, _rows, net  # noqa: F401  (net: a fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 15, 17, 255, 256, 257, 300])
def test_tile_edges_match_oracle(net, oracle, n):  # noqa: F811
    """Every row counts once, none beyond the batch: against the FP64 oracle
    within the BF16 tolerance of summed gradients (12% in the table, as for
    96 rows in test_gpu_mlp)."""
    r, t, w = net
    rows = _rows(np.random.default_rng(n), n)
    loss, dw, dt = r.mlp_gradients(rows, log2_table=LOG2)
    rloss, rdw, rdt = oracle.mlp_grad(_cfg(oracle), t, w, rows[:, 0:3], rows[:, 3:6], rows[:, 6:9], rows[:, 9:12])
    assert loss == pytest.approx(rloss, rel=0.02)
    for l, used in enumerate([64, 64, 64, 64, 3]):
        assert np.linalg.norm(dw[l, :used] - rdw[l, :used]) < 0.12 * np.linalg.norm(rdw[l, :used])
    assert np.linalg.norm(dt - rdt) < 0.12 * np.linalg.norm(rdt)


@pytest.mark.parametrize("half", [1 << 14, (1 << 14) + 129])
def test_large_batch_is_the_mean_of_its_halves(net, half):  # noqa: F811
    """2 x half rows (levels gathered from shared memory) against the two
    halves (from L2).  The loss's 1/n differs by a power of two, so every BF16
    rounding is the same and only the FP32 sums' order differs: <= 2^15 terms
    of random sign, rounding 6e-8 each, over a sum not below a hundredth of
    their norm: 1e-4 relative."""
    r, _, _ = net
    rows = _rows(np.random.default_rng(8), 2 * half)
    loss, dw, dt = r.mlp_gradients(rows, log2_table=LOG2)
    a, b = (r.mlp_gradients(x, log2_table=LOG2) for x in (rows[:half], rows[half:]))
    assert loss == pytest.approx(0.5 * (a[0] + b[0]), rel=1e-4)
    for got, x, y in ((dw, a[1], b[1]), (dt, a[2], b[2])):
        ref = 0.5 * (x.astype(np.float64) + y)
        assert np.linalg.norm(got - ref) <= 1e-4 * np.linalg.norm(ref)


def test_training_wraps_around_the_rows(vct, net):  # noqa: F811
    """Batches that do not divide the rows, and a batch larger than them,
    train without leaving the sample buffer."""
    r, _, _ = net
    rows = _rows(np.random.default_rng(9), 1000, smooth=True)
    for batch in (333, 4096):
        rep = r.mlp_train_samples(rows, vct.mlp_desc(log2_table=LOG2, n_max=N_MAX, steps=30, batch=batch, lr=1e-3))
        assert np.isfinite(rep["loss_last"]) and rep["loss_last"] <= rep["loss_first"]
