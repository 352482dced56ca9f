"""GPU: training on one cluster (mlp_train_kernel) against a float64 restatement of the same steps
(oracle/es_mlp_ref.py's gradient, Adam, the trainer's seeded order): batches below a tile, between
tiles, of exactly eight tiles and above (several rounds per step), a last batch that is short, both
hidden widths and odd input widths.  FP32 sums of at most 64 terms carry a relative error of about
64 x 2^-24 = 4e-6 per step at worst and Adam's normalised steps are at most lr = 2e-3 of unit-size
weights, so parameters may differ by 2e-5 of their norm after these few steps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _order(n, epochs, seed):
    mask, s, perm = (1 << 64) - 1, seed, list(range(n))
    for _ in range(epochs):
        for i in range(n - 1, 0, -1):
            s = (s + 0x9e3779b97f4a7c15) & mask
            z = ((s ^ (s >> 30)) * 0xbf58476d1ce4e5b9) & mask
            z = ((z ^ (z >> 27)) * 0x94d049bb133111eb) & mask
            j = (z ^ (z >> 31)) % (i + 1)
            perm[i], perm[j] = perm[j], perm[i]
        yield np.array(perm)


@pytest.mark.parametrize("n,D,H,O,batch,epochs", [(1, 1, 32, 1, 1, 3), (70, 34, 64, 2, 32, 3), (500, 34, 64, 2, 256, 4),
                                                  (300, 7, 32, 3, 100, 3), (700, 64, 64, 8, 300, 3),
                                                  (1025, 33, 64, 2, 512, 3), (257, 5, 32, 2, 1000, 5)])
def test_training_steps_match_float64(native, n, D, H, O, batch, epochs):
    import es_learned
    import es_mlp_ref as R
    rng = np.random.default_rng(n + D)
    X = rng.normal(size=(n, D)).astype(np.float32)
    T = rng.normal(size=(n, O)).astype(np.float32)
    net = es_learned.MLP(D, O, H, seed=9)
    P = net.params().astype(np.float64)
    loss = net.train(X, T, epochs=epochs, batch=batch, lr=2e-3, seed=4)
    m, v, step = np.zeros_like(P), np.zeros_like(P), 0
    for perm in _order(n, epochs, 4):
        for at in range(0, n, batch):
            rows = perm[at:at + batch]
            _, g = R.loss_grad(P, X[rows], T[rows], D, H, O)
            step += 1
            m = 0.9 * m + 0.1 * g
            v = 0.999 * v + 0.001 * g * g
            P = P - 2e-3 * (m / (1 - 0.9 ** step)) / (np.sqrt(v / (1 - 0.999 ** step)) + 1e-8)
    got = net.params()
    assert np.linalg.norm(got - P) <= 2e-5 * np.linalg.norm(P)
    want = R.loss_grad(P, X, T, D, H, O)[0]
    assert abs(loss - want) <= 1e-4 * max(1.0, abs(want))
    # a second call goes on with the moments and the step count of the first
    net.train(X, T, epochs=1, batch=batch, lr=2e-3, seed=5)
    assert np.all(np.isfinite(net.params())) and not np.array_equal(net.params(), got)
