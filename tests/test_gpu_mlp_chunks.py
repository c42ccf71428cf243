"""The inference buffers when a network's calls alternate: a small predict, a larger
query (which has no use for the full spread) and a predict of that size again, in
one chunk of rows and in two. Every result equals, bit for bit, that of a network of
the same weights which has run nothing else."""
import numpy as np
import pytest

from omg_audio_gb300.surrogate import Mlp

pytestmark = pytest.mark.gpu


def _wave(members):
    """Rows of one chunk at most: the row tiles of all members fill the multiprocessors once."""
    import torch
    return 128 * max(1, torch.cuda.get_device_properties(0).multi_processor_count // members)


@pytest.mark.parametrize("members,n_out", [(4, 192), (3, 17), (1, 3)])
@pytest.mark.parametrize("chunks", [1, 2])
@pytest.mark.parametrize("small", [1, 64])
def test_predict_after_a_larger_query(ctx, members, n_out, chunks, small):
    big = 1000 if chunks == 1 else _wave(members) + 200
    x = np.random.default_rng(members * 10 + chunks).standard_normal((big, 24)).astype(np.float32)
    nets = []

    def fresh():
        nets.append(Mlp(ctx, 24, 64, 2, n_out, members, seed=11))
        return nets[-1]

    want_small, want_big = fresh().predict(x[:small]), fresh().predict(x)
    want_query = fresh().query(x, 0.0)
    net = fresh()
    for got, want in [(net.predict(x[:small]), want_small), (net.query(x, 0.0), want_query),
                      (net.predict(x), want_big), (net.predict(x[:small]), want_small),
                      (net.query(x[:small], 0.0), (want_query[0][:small], want_query[1][:small])),
                      (net.predict(x), want_big)]:
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    for n in nets:
        n.close()
