"""The band MLP's training step at the edges of its row blocks (128 rows) and
of its row-sum tiles (1,024 rows).  A batch of 2 m rows against its two halves:
1 / (2 m) is half of 1 / m exactly, so every rounding to BF16 is the same and
the mean of the halves' gradients differs from the batch's by the order of the
FP32 sums alone (at most 2,100 terms: 2,100 x 2^-24 of the terms' size)."""
import numpy as np
import pytest

from oracle import band_mlp as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 31, 64, 127, 128, 129, 512, 513, 1024, 1050])
def test_gradient_at_row_edges(m):
    from biovoltron_b200.pairhmm import PairHMMEngine
    rng = np.random.default_rng(m)
    w = M.init_weights(3, out_scale=1.0)
    x = rng.uniform(0, 1, (2 * m, M.FEAT)).astype(np.float32)
    t = rng.normal(0, 4, (2 * m, 2)).astype(np.float32)
    with PairHMMEngine() as e:
        out, loss, g = e.band_mlp_eval(w, x, t, alpha=8.0)
        again = e.band_mlp_eval(w, x, t, alpha=8.0)
        only, _, none = e.band_mlp_eval(w, x, t, alpha=8.0, grad=False)
        h0, h1 = (e.band_mlp_eval(w, x[s], t[s], alpha=8.0) for s in (slice(0, m), slice(m, 2 * m)))
    assert np.array_equal(out, again[0]) and np.array_equal(g, again[2]) and np.array_equal(out, only) and none is None
    assert np.array_equal(out, np.concatenate([h0[0], h1[0]]))
    assert abs(loss - (h0[1] + h1[1]) / 2) <= 1e-3 * loss
    assert np.linalg.norm(g - (h0[2] + h1[2]) / 2) <= 1e-3 * np.linalg.norm(g)


def test_ragged_last_minibatch():
    """Training whose last minibatch of an epoch is a single row, and one whose
    minibatch exceeds the row-sum tile, end with finite weights, the same twice."""
    from biovoltron_b200 import workloads as W
    from biovoltron_b200.pairhmm import PairHMMEngine
    b = W.config1(seed=51, n_regions=1)
    with PairHMMEngine() as e:
        n = e.band_train(b, epochs=1, batch_size=16)["labelled"]
        for batch in (16 if n % 16 == 1 else n - 1, 3000):
            got = []
            for _ in range(2):
                e.band_train(b, epochs=2, batch_size=batch)
                got.append(e.band_weights())
            assert np.all(np.isfinite(got[0])) and np.array_equal(got[0], got[1])
