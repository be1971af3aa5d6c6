"""The FP32 products of the warm-start network (tile_sum in mlp.cu) at the sizes
where they can go wrong: every tile size, remainders of tiles and of the
stages of 32 and 64 terms, aligned and odd row lengths, one row, and the rows
of a mini-batch picked in place; against the FP64 oracle."""
import numpy as np
import pytest

from oracle import mlp_oracle as MO

# (inputs, hidden, outputs, rows): tiles of 16 unless said
SIZES = [
    (1, 1, 1, 1),
    (64, 16, 16, 16),          # whole tiles, aligned rows
    (65, 17, 15, 17),          # one more / one less, odd rows: 4-byte copies
    (63, 36, 130, 31),
    (260, 256, 1681, 128),     # output layer in tiles of 32, its rows odd
    (128, 256, 1680, 129),     # the same, aligned
    (200, 64, 2501, 300),      # output layer in tiles of 64
]


def _net(inp, h, out, rows):
    rng = np.random.default_rng(inp + 7 * out + rows)
    scale = np.concatenate([np.full(inp * h + h, inp), np.full(h * h + h, h), np.full(h * out + out, h)])
    p = (rng.standard_normal(scale.size) / np.sqrt(scale)).astype(np.float32)
    return p, rng.standard_normal((rows, inp)).astype(np.float32), rng.standard_normal((rows, out)).astype(np.float32)


def _bound(terms):
    """A chain of `terms` FP32 fused multiply-adds moves the result by at most terms * eps of the sum of
    absolute products; products of O(1 / sqrt(terms)) weights and O(1) rows sum to O(sqrt(terms)) in absolute value."""
    return 4 * terms**1.5 * 2.0**-24


@pytest.mark.gpu
@pytest.mark.parametrize("inp,h,out,rows", SIZES)
def test_products_match_the_oracle(inp, h, out, rows):
    from pdal_gb300.learn import MLP

    p, X, Y = _net(inp, h, out, rows)
    net = MLP(inp, h, out, seed=1)
    net.set_params(p)
    tol = _bound(inp) + 2 * _bound(h)
    P, _ = MO.forward(p, X, inp, h, out)
    assert np.abs(net.predict(X, bf16=False) - P).max() <= tol * (1 + np.abs(P).max())
    loss, g = net.loss_grad(X, Y)
    lo, go = MO.loss_grad(p, X, Y, inp, h, out)
    assert abs(loss - lo) <= 2 * tol * (1 + lo)
    # a hidden unit whose input rounds to the other side of zero changes its whole column: compared in the 2-norm
    tol += _bound(rows) + _bound(out)
    assert np.linalg.norm(g - go) <= tol * np.linalg.norm(go)
    assert net.loss_grad(X, Y, grad=False)[0] == loss


@pytest.mark.gpu
@pytest.mark.parametrize("rows,batch", [(48, 16), (37, 8), (20, 64)])
def test_one_epoch_is_the_steps_of_its_gradients(rows, batch):
    """A mini-batch run: Adam steps on gradients of the batches (the fused update against the same update in
    FP64, with the gradients the library gives for the rows): a full batch, whose order does not matter, exactly; several
    batches through the loss, which falls."""
    from pdal_gb300.learn import MLP

    inp, h, out = 33, 20, 27
    p, X, Y = _net(inp, h, out, rows)
    net = MLP(inp, h, out, seed=1)
    net.set_params(p)
    net.set_data(X, Y)
    lr, b1, b2, eps = 1e-3, 0.9, 0.999, 1e-8
    if batch >= rows:
        first = net.loss_grad(X, Y)
        loss = net.train(1, batch, lr, seed=3)
        assert loss == pytest.approx(first[0], rel=1e-5)
        g = first[1].astype(np.float64)
        m, v = (1 - b1) * g / (1 - b1), (1 - b2) * g * g / (1 - b2)
        # FP32 of 1 - 0.999: relative 2^-24 / 1e-3 in v, half of that in its root
        want = p - lr * m / (np.sqrt(v) + eps)
        big = np.abs(g) > 1e-4
        assert np.abs(net.get_params() - want)[big].max() <= lr * 2e-4 + 2.0**-23 * np.abs(p).max()
    else:
        before = net.loss_grad(X, Y, grad=False)[0]
        assert net.train(30, batch, lr, seed=3) < before
        a = net.get_params()
        net.set_params(p)
        net.train(30, batch, lr, seed=3)
        assert np.array_equal(a, net.get_params())
