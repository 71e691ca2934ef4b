"""Training over several epochs: the captured epoch's buffers, and the row orders and targets that the
device gets, against the same steps taken one at a time through gradient()."""
import numpy as np
import pytest

import biwfa_gpu_pii2025_gb300 as pkg

pytestmark = pytest.mark.gpu


@pytest.fixture()
def aligners():
    al = [pkg.BatchAligner(0), pkg.BatchAligner(0)]
    yield al
    for a in al:
        a.close()


def _orders(n, epochs, seed):
    """The epochs' row orders: a Fisher-Yates shuffle driven by splitmix64, carried from epoch to epoch."""
    mask, x, rows = (1 << 64) - 1, seed, list(range(n))
    for _ in range(epochs):
        for i in range(n - 1, 0, -1):
            x = (x + 0x9E3779B97F4A7C15) & mask
            z = ((x ^ (x >> 30)) * 0xBF58476D1CE4E5B9) & mask
            z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
            j = ((z ^ (z >> 31)) * (i + 1)) >> 64
            rows[i], rows[j] = rows[j], rows[i]
        yield np.array(rows)


@pytest.mark.parametrize("n,batch,epochs", [(700, 300, 1), (700, 300, 2), (700, 300, 5), (33, 16, 3)])
def test_epochs_take_their_own_row_orders_and_targets(aligners, n, batch, epochs):
    """Tolerance: both sides run the same train step; their sums of up to 300 fp32 terms in another order
    differ by about 1e-6 of the gradient, which Adam's division makes visible only where a gradient is
    itself rounding. 1 % of the way that the parameters went is far above that, and far below what
    another order of the rows or other targets do."""
    b = pkg.PairBatch.generate(2, n, seed=8)
    scores = -np.random.default_rng(3).integers(0, 3000, n).astype(np.int32)
    al, one = aligners
    al.upload(b)
    a, s = pkg.ScorePredictor(al, seed=5), pkg.ScorePredictor(one, seed=5)
    p = a.params().astype(np.float64)
    start, m, v, step, losses = p.copy(), np.zeros_like(p), np.zeros_like(p), 0, []
    got = a.train(scores, epochs=epochs, batch_rows=batch, lr=2e-3, seed=9)
    for rows in _orders(n, epochs, 9):
        total = 0.0
        for k in range(0, n, batch):
            at = rows[k:k + batch]
            one.upload(b.subset(at))
            s.set_params(p.astype(np.float32))
            loss, g = s.gradient(np.log1p(np.abs(scores[at].astype(np.float64))).astype(np.float32))
            total += loss * at.size
            step += 1
            g = g.astype(np.float64)
            m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
            p = p - 2e-3 * (m / (1 - 0.9 ** step)) / (np.sqrt(v / (1 - 0.999 ** step)) + 1e-8)
        losses.append(total / n)
    end = a.params().astype(np.float64)
    a.close()
    s.close()
    assert np.linalg.norm(end - p) <= 1e-2 * np.linalg.norm(p - start)
    np.testing.assert_allclose(got, losses, rtol=1e-2)


def test_training_after_a_larger_gradient_batch(aligners):
    """A larger batch's gradient() replaces the model's buffers; training at the earlier size then runs on
    the new ones and ends where a model that never saw the larger batch does."""
    al, _ = aligners
    small, large = pkg.PairBatch.generate(2, 100, seed=8), pkg.PairBatch.generate(2, 5000, seed=9)
    scores = -np.random.default_rng(3).integers(0, 3000, 100).astype(np.int32)
    al.upload(large)
    a, fresh = pkg.ScorePredictor(al, seed=5), pkg.ScorePredictor(al, seed=5)
    a.features()  # the context's feature buffer has its largest size from here on
    al.upload(small)
    start = a.params()
    a.train(scores, epochs=2, batch_rows=64)
    al.upload(large)
    a.gradient(np.zeros(5000, np.float32))
    al.upload(small)
    a.set_params(start)
    got, want = a.train(scores, epochs=2, batch_rows=64), fresh.train(scores, epochs=2, batch_rows=64)
    end, ref = a.params().astype(np.float64), fresh.params().astype(np.float64)
    a.close()
    fresh.close()
    np.testing.assert_allclose(got, want, rtol=1e-2)
    assert np.linalg.norm(end - ref) <= 1e-2 * np.linalg.norm(ref - start)  # see the test above
