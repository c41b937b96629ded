"""Training by value: batches that wrap around the rows train on the rows they
name, and the gradients of a large batch are as near their FP64 values as BF16
operands with rounded FP32 sums of 16 rows leave them."""
import math

import numpy as np
import pytest

from tests.test_gpu_mlp import LOG2, N_MAX, _rows

pytestmark = pytest.mark.gpu

LR = 1e-3


def _fresh(vct, r, log2=LOG2, n_max=N_MAX):
    """Random parameters and Adam at its start."""
    rng = np.random.default_rng(7)
    table = rng.uniform(-0.5, 0.5, (16, 1 << log2, 2)).astype(np.float32)
    w = (rng.uniform(-1, 1, (5, 64, 64)) * np.sqrt(6 / 64)).astype(np.float32)
    w[4, 3:] = 0
    r.mlp_init(vct.mlp_desc(log2_table=log2, n_max=n_max, seed=3))
    r.mlp_set_params(table, w)
    return table, w


@pytest.mark.parametrize("n", [1, 5, 15])
def test_a_batch_larger_than_the_rows(vct, n):
    """Fewer rows than the smallest batch, 16: each counts as often as the
    batch meets it.  Loss within FP32 summation of 48 terms (1e-5); Adam's
    first step moves a parameter by lr against the sign of its gradient (to
    the rounding of a parameter below 1, 6e-8 of lr 1e-3, and of the step,
    1e-6: 1e-3 of lr asked) where the gradient is clear of rounding and of the
    weights' decay, a hundredth of the largest, and not at all where it is 0."""
    rows = _rows(np.random.default_rng(n), n)
    r = vct.Renderer(16, 16, grid_res=16)
    table, w = _fresh(vct, r)
    loss, dw, dt = r.mlp_gradients(rows[np.arange(16) % n], log2_table=LOG2)
    rep = r.mlp_train_samples(rows, vct.mlp_desc(log2_table=LOG2, n_max=N_MAX, steps=1, batch=16, lr=LR))
    t1, w1 = r.mlp_get_params(log2_table=LOG2)
    r.close()
    assert rep["loss_first"] == pytest.approx(loss, rel=1e-5)
    for before, after, g in ((table, t1, dt), (w[:4], w1[:4], dw[:4]), (w[4, :3], w1[4, :3], dw[4, :3])):
        clear = np.abs(g) > 0.01 * np.abs(g).max()
        assert clear.any()
        step = after.astype(np.float64) - before
        assert np.abs(step[clear] + LR * np.sign(g[clear])).max() <= 1e-3 * LR
    assert (t1 == table)[dt == 0].all()


def test_a_batch_that_wraps(vct):
    """The fourth batch of 333 of 1000 rows is row 999, then rows 0 to 331; row
    0's target is far off, so its loss is most of the batch's.  With lr 1e-7
    the parameters are the first ones but for 4e-7 (of their BF16 copies at
    most one in a thousand takes the next value): the loss within 1e-3."""
    rows = _rows(np.random.default_rng(9), 1000)
    rows[0, 9:] = 60.0
    r = vct.Renderer(16, 16, grid_res=16)
    _fresh(vct, r)
    want, _, _ = r.mlp_gradients(rows[(999 + np.arange(333)) % 1000], log2_table=LOG2)
    other, _, _ = r.mlp_gradients(rows[666:999], log2_table=LOG2)
    rep = r.mlp_train_samples(rows, vct.mlp_desc(log2_table=LOG2, n_max=N_MAX, steps=4, batch=333, lr=1e-7))
    r.close()
    assert want > 5 * other
    assert rep["loss_last"] == pytest.approx(want, rel=1e-3)


def _fp64_gradients(torch, table, w, rows, log2, n_min=16, n_max=512):
    """Loss, dW and dTable in FP64 from BF16-rounded parameters and the
    kernels' FP32 grid positions."""
    bf = lambda x: torch.tensor(x).to(torch.bfloat16).double().cuda()  # noqa: E731
    n, r = rows.shape[0], torch.tensor(rows, device="cuda")
    tab, W = bf(table).requires_grad_(), bf(w).requires_grad_()
    b = math.exp((math.log(n_max) - math.log(n_min)) / 15)
    feats = []
    for l in range(16):
        res = int(math.floor(n_min * b ** l + 1e-6))
        x = r[:, 0:3] * np.float32(res)
        fl = torch.floor(x)
        fr, i0, f = (x - fl).double(), fl.long(), 0
        for k in range(8):
            c = [i0[:, d] + ((k >> d) & 1) for d in range(3)]
            wt = 1
            for d in range(3):
                wt = wt * (fr[:, d] if (k >> d) & 1 else 1 - fr[:, d])
            if (res + 1) ** 3 <= 1 << log2:
                c = [t.clamp(0, res) for t in c]
                idx = c[0] + (res + 1) * (c[1] + (res + 1) * c[2])
            else:
                idx = (c[0] ^ ((c[1] * 2654435761) & 0xffffffff) ^ ((c[2] * 805459861) & 0xffffffff)) & ((1 << log2) - 1)
            f = f + wt[:, None] * tab[l][idx]
        feats.append(f)
    nn = r[:, 3:6].double()
    nn = nn / nn.norm(dim=1, keepdim=True)
    one = torch.ones(n, 1, device="cuda", dtype=torch.float64)
    x = torch.cat(feats + [nn, r[:, 6:9].double(), one, one.new_zeros(n, 25)], 1)
    for l in range(4):
        x = torch.relu(x @ W[l].T)
    loss = ((x @ W[4][:3].T - r[:, 9:12].double()) ** 2).sum() / n
    loss.backward()
    return loss.item(), W.grad.cpu().numpy(), tab.grad.cpu().numpy()


def test_gradients_of_a_large_batch_against_fp64(vct):
    """65,536 rows, 2^15 entries a level.  The bounds are the errors, relative
    in L2, that a step had whose tensor products were added up in FP32 16 rows
    at a time, measured on these inputs: 1.128e-3, 7.164e-4, 4.373e-4,
    2.137e-4 and 2.400e-5 for the layers, 4.9485e-2 for the table (BF16
    gradients of the features), plus 1% for the order of the sums.  Chains of
    64 rows in the tensor core keep them; chains of 256 did not."""
    import torch

    log2, n = 15, 1 << 16
    rng = np.random.default_rng(3)
    table = rng.uniform(-0.3, 0.3, (16, 1 << log2, 2)).astype(np.float32)
    w = (rng.uniform(-1, 1, (5, 64, 64)) * math.sqrt(6 / 64)).astype(np.float32)
    w[4] *= .2
    w[4, 3:] = 0
    rows = np.concatenate([rng.random((n, 3), np.float32) * .96 + .02, rng.standard_normal((n, 3)), rng.random((n, 3)),
                           rng.random((n, 3))], 1).astype(np.float32)
    r = vct.Renderer(16, 16, grid_res=16)
    r.mlp_init(vct.mlp_desc(log2_table=log2))
    r.mlp_set_params(table, w)
    loss, dw, dt = r.mlp_gradients(rows, log2_table=log2)
    r.close()
    want, DW, DT = _fp64_gradients(torch, table, w, rows, log2)
    assert loss == pytest.approx(want, rel=1e-4)
    err = lambda a, b: np.linalg.norm(a.astype(np.float64) - b) / np.linalg.norm(b)  # noqa: E731
    for l, bound in enumerate([1.128e-3, 7.164e-4, 4.373e-4, 2.137e-4, 2.400e-5]):
        assert err(dw[l], DW[l]) <= 1.01 * bound, l
    assert err(dt, DT) <= 1.01 * 4.9485e-2
