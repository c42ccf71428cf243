"""The surrogate network's whole-pass kernels at the sizes where their tiles
end: widths of 16, 192, 240 and 256, inputs beyond one 256-wide step, row counts
around a 128-row tile and a chunk, one to many row tiles a share.

Inference against the FP64 network on the BF16-rounded weights and inputs: the
activations are rounded to BF16 (2^-9 relative) per layer, as in the oracle, so
the relative error stays below 1e-2; rows beyond the last tile do not matter.
Gradients against the oracle that rounds the same quantities to BF16: 5e-3 per
layer, as for the training widths. Training with a batch of the whole set
equals AdamW run on those gradients: the first step's update has the learning
rate's size for every weight, so the loss falls and matches epoch by epoch
within 2 %."""
import numpy as np
import pytest

from omg_audio_gb300.surrogate import Mlp

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float(np.linalg.norm(np.asarray(a) - np.asarray(b)) / max(np.linalg.norm(np.asarray(b)), 1e-30))


NETS = [(38, 256, 4, 192), (6, 16, 1, 3), (1, 240, 2, 256), (300, 64, 2, 17), (1024, 128, 1, 48)]


@pytest.mark.parametrize("n_in,hidden,n_hidden,n_out", NETS)
@pytest.mark.parametrize("rows", [1, 127, 129, 6000])
def test_inference_equals_the_network(ctx, n_in, hidden, n_hidden, n_out, rows):
    from oracle import mlp_oracle as MO
    members = 3
    net = Mlp(ctx, n_in, hidden, n_hidden, n_out, members, seed=3)
    x = np.random.default_rng(rows + n_in).standard_normal((rows, n_in)).astype(np.float32)
    mean, std = net.predict(x)
    ys = []
    for e in range(members):
        a = x.astype(np.float64)
        layers = net.layers(e)
        for k, (w, b) in enumerate(layers):
            z = MO.bf16(a.astype(np.float32)).astype(np.float64) @ MO.bf16(w.astype(np.float32)).astype(np.float64).T + b
            a = z if k + 1 == len(layers) else 0.5 * z * (1 + np.tanh(0.7978845608028654 * (z + 0.044715 * z ** 3)))
        ys.append(a)
    assert _rel(mean, np.mean(ys, 0)) <= 1e-2
    assert _rel(std, np.std(ys, 0)) <= 2e-2
    m2, spread = net.query(x, 0.0)
    assert np.array_equal(m2, mean)
    want = np.where(mean >= 0.0, std, 0.0).max(1)
    assert np.array_equal(spread, want)
    net.close()


@pytest.mark.parametrize("n_in,hidden,n_hidden,n_out", NETS)
@pytest.mark.parametrize("rows", [128, 384, 2560])
def test_gradients_match_the_oracle(ctx, n_in, hidden, n_hidden, n_out, rows):
    from oracle import mlp_oracle as MO
    net = Mlp(ctx, n_in, hidden, n_hidden, n_out, 2, seed=4)
    rng = np.random.default_rng(rows * 3 + n_in)
    x = rng.standard_normal((rows, n_in)).astype(np.float32)
    y = rng.standard_normal((rows, n_out)).astype(np.float32)
    for member in (1, 0):
        loss, grads = net.grad(x, y, member)
        ol, og = MO.loss_and_grads(net.layers(member), x, y, bf=True)
        assert abs(loss - ol) <= 1e-3 * ol
        for k, ((gw, gb), (ow, ob)) in enumerate(zip(grads, og)):
            assert _rel(gw, ow) <= 5e-3, k
            assert _rel(gb, ob) <= 5e-3, k
    net.close()


def test_whole_set_training_follows_adamw(ctx):
    """One batch an epoch (its order does not matter): the losses of 12 epochs
    against AdamW in FP64 on the oracle's gradients."""
    from oracle import mlp_oracle as MO
    n, lr = 256, 1e-2
    rng = np.random.default_rng(8)
    x = rng.standard_normal((n, 6)).astype(np.float32)
    y = np.stack([np.sin(x[:, 0]), x[:, 1] * x[:, 2], x[:, 3]], 1).astype(np.float32)
    net = Mlp(ctx, 6, 64, 2, 3, 2, seed=9)
    start = [net.layers(e) for e in range(2)]
    net.set_data(x, y)
    losses = net.train(12, n, lr=lr, lr_final=lr, weight_decay=1e-2)
    xs = (x - x.mean(0, dtype=np.float64)) / x.std(0, dtype=np.float64)
    ys = (y - y.mean(0, dtype=np.float64)) / y.std(0, dtype=np.float64)
    for e in range(2):
        layers = [[w.copy(), b.copy()] for w, b in start[e]]
        m = [[np.zeros_like(w), np.zeros_like(b)] for w, b in layers]
        v = [[np.zeros_like(w), np.zeros_like(b)] for w, b in layers]
        for t in range(12):
            loss, g = MO.loss_and_grads([tuple(l) for l in layers], xs.astype(np.float32), ys.astype(np.float32),
                                        bf=True)
            assert abs(losses[e, t] - loss) <= 2e-2 * loss, (e, t)
            for k in range(len(layers)):
                for j in range(2):
                    m[k][j] = 0.9 * m[k][j] + 0.1 * g[k][j]
                    v[k][j] = 0.999 * v[k][j] + 0.001 * g[k][j] ** 2
                    mh, vh = m[k][j] / (1 - 0.9 ** (t + 1)), v[k][j] / (1 - 0.999 ** (t + 1))
                    wd = 1e-2 if j == 0 else 0.0
                    layers[k][j] -= lr * (mh / (np.sqrt(vh) + 1e-8) + wd * layers[k][j])
    net.close()
