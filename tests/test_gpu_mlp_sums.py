"""The order in which a training pass's gradients are summed, and the row shares
of the weight gradients.

A bias gradient adds 32 rows at a time, rows r, r + 8, r + 16, r + 24 one after
another for r = 0 .. 7 and then those eight in order; the groups arrive in any
order. So the output layer's over 128 rows is, bit for bit, one of the 24 orders
of four such sums, worked out here in f32 from the network's own predictions.

A weight gradient adds shares of 512 rows (up to 4096 rows, then eight shares),
each one chain of products. With 64 outputs the loss's 1 / (rows x outputs) is a
power of two, so every value scales exactly: the gradient of 1024 rows is half
the sum of those of its two halves, bit for bit, and repeats.

Shares that end inside a 128-row tile and batches of one to eight shares against
the oracle that rounds the same quantities to BF16: 5e-3 per layer, as for the
training widths (a share of 1/8 of the rows left out moves it by 0.3)."""
import itertools

import numpy as np
import pytest

from omg_audio_gb300.surrogate import Mlp

pytestmark = pytest.mark.gpu


def _xy(rows, n_in, n_out, seed):
    rng = np.random.default_rng(seed)
    return (rng.standard_normal((rows, n_in)).astype(np.float32),
            rng.standard_normal((rows, n_out)).astype(np.float32))


@pytest.mark.parametrize("n_out", [64, 256])
def test_bias_gradient_order(ctx, n_out):
    rows = 128
    net = Mlp(ctx, 6, 64, 2, n_out, 1, seed=5)
    x, y = _xy(rows, 6, n_out, n_out)
    e = net.predict(x)[0] - y
    d = (np.float32(2) * e) * (np.float32(1) / (np.float32(rows) * np.float32(n_out)))
    groups = []
    for g in range(4):
        q = d[32 * g:32 * g + 32].reshape(4, 8, n_out)
        r = ((q[0] + q[1]) + q[2]) + q[3]
        t = r[0]
        for k in range(1, 8):
            t = t + r[k]
        groups.append(t)
    orders = np.stack([((p[0] + p[1]) + p[2]) + p[3] for p in itertools.permutations(groups)])
    assert orders.dtype == np.float32
    for _ in range(4):
        gb = net.grad(x, y)[1][-1][1]
        assert (orders == gb[None]).any(0).all()
    net.close()


@pytest.mark.parametrize("n_in,hidden", [(38, 256), (6, 64), (300, 128)])
def test_weight_gradients_are_sums_of_512_rows(ctx, n_in, hidden):
    net = Mlp(ctx, n_in, hidden, 3, 64, 2, seed=6)
    x, y = _xy(1024, n_in, 64, hidden)

    def weights(a, b):
        return [w for w, _ in net.grad(x[a:b], y[a:b], 1)[1]]

    lo, hi, both = weights(0, 512), weights(512, 1024), weights(0, 1024)
    for _ in range(3):
        for k in range(4):
            assert np.array_equal(both[k], np.float32(0.5) * (lo[k] + hi[k])), k
        lo, both = weights(0, 512), weights(0, 1024)
    net.close()


@pytest.mark.parametrize("n_in,hidden,n_out", [(38, 256, 192), (6, 16, 3), (300, 64, 17)])
@pytest.mark.parametrize("rows", [640, 1152, 4224, 5120])
def test_shares_hold_every_row(ctx, n_in, hidden, n_out, rows):
    from oracle import mlp_oracle as MO
    net = Mlp(ctx, n_in, hidden, 2, n_out, 1, seed=7)
    x, y = _xy(rows, n_in, n_out, rows)
    loss, grads = net.grad(x, y)
    ol, og = MO.loss_and_grads(net.layers(0), x, y, bf=True)
    assert abs(loss - ol) <= 1e-3 * ol
    for k, ((gw, gb), (ow, ob)) in enumerate(zip(grads, og)):
        assert np.linalg.norm(gw - ow) <= 5e-3 * np.linalg.norm(ow), k
        assert np.linalg.norm(gb - ob) <= 5e-3 * np.linalg.norm(ob), k
    net.close()
