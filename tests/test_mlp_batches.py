"""The scheduler network's kernels at the edges of their tiles: batches that do
not fill a CTA's samples, positions with the most active inputs, the padded rows
of a prediction, and training through an order against one-step gradients."""
import numpy as np
import pytest

import perft_gpu_2026_b200 as pg
from perft_gpu_2026_b200 import mlp_ref

pytestmark = pytest.mark.gpu

FULL = "rnbqkbnr/pppppp1p/8/8/4PPp1/8/PPPP2PP/RNBQKBNR b KQkq f3 0 1"  # 32 pieces, 4 rights, en passant


@pytest.fixture(scope="module")
def eng():
    e = pg.Engine(device=0, use_tt=False, arena_bytes=1 << 30)
    yield e
    e.close()


def _batch(n, seed):
    pos = [pg.parse_fen(FULL), pg.parse_fen("4k3/8/8/8/8/8/8/4K3 w - - 0 1")]
    pos += list(pg.random_playouts(seed, n, 0, 60))
    t = np.random.default_rng(seed).uniform(0, 20, size=(n, 4)).astype(np.float32)
    return pos[:n], t


@pytest.mark.parametrize("n", [64, 192, 320, 4160])
def test_gradients_at_partial_tiles(eng, n):
    """64 is two parts of 32 samples, 4160 is 130 parts and 32.5 GEMM tiles."""
    eng.mlp_init(seed=5, out_bias=[4.0, 9.0, 14.0, 19.0])
    pos, t = _batch(n, n)
    g, loss = eng.mlp_gradients(pos, t)
    y, want_loss, want = mlp_ref.forward_backward(eng.mlp_params(), mlp_ref.features(pos), t)
    assert abs(loss - want_loss) <= 1e-3 * want_loss
    for a, b in [(mlp_ref.OFF_W1, mlp_ref.OFF_B1), (mlp_ref.OFF_B1, mlp_ref.OFF_W2), (mlp_ref.OFF_W2, mlp_ref.OFF_B2),
                 (mlp_ref.OFF_B2, mlp_ref.OFF_W3), (mlp_ref.OFF_W3, mlp_ref.OFF_B3), (mlp_ref.OFF_B3, mlp_ref.N_PARAMS)]:
        # BF16 rounding points differ in order only: the bound of the network's gradient test
        assert np.linalg.norm(g[a:b] - want[a:b]) <= 0.02 * np.linalg.norm(want[a:b]) + 1e-6
    again, _ = eng.mlp_gradients(pos, t)  # nothing is left over from the first call
    assert np.linalg.norm(again - g) <= 1e-5 * np.linalg.norm(g)


@pytest.mark.parametrize("n", [1, 63, 65, 8191, 8193])
def test_predictions_do_not_depend_on_the_batch(eng, n):
    eng.mlp_init(seed=5, out_bias=[4.0, 9.0, 14.0, 19.0])
    pos, _ = _batch(max(n, 2), 9)
    y = eng.mlp_predict(pos[:n])
    for k in {0, n // 2, n - 1}:
        assert np.array_equal(eng.mlp_predict([pos[k]])[0], y[k])


def test_training_steps_through_the_order(eng):
    """Two epochs of three steps equal Adam on mlp_gradients of the same
    batches in the same order (splitmix64 Fisher-Yates), step by step."""
    n, batch, lr = 200, 64, 1e-3
    pos, t = _batch(n, 77)
    eng.mlp_init(seed=3, out_bias=[4.0, 9.0, 14.0, 19.0])
    p0 = eng.mlp_params()
    loss = eng.mlp_train(pos, t, epochs=2, batch=batch, lr=lr, seed=11)
    got = eng.mlp_params()
    p, m, v = p0.astype(np.float64), 0.0, 0.0
    order, state, step, losses = list(range(n)), 11, 0, []
    for _ in range(2):
        losses = []
        for i in range(n - 1, 0, -1):
            r, state = pg.splitmix64(state)
            j = (r * (i + 1)) >> 64
            order[i], order[j] = order[j], order[i]
        for b in range(0, n - batch + 1, batch):
            at = order[b:b + batch]
            eng.mlp_set_params(p.astype(np.float32))
            g, one = eng.mlp_gradients([pos[k] for k in at], t[at])
            losses.append(one)
            step += 1
            m = 0.9 * m + 0.1 * g
            v = 0.999 * v + 0.001 * g.astype(np.float64) ** 2
            p = p - lr * (m / (1 - 0.9 ** step)) / (np.sqrt(v / (1 - 0.999 ** step)) + 1e-8)
    assert abs(loss - np.mean(losses)) <= 1e-4 * abs(np.mean(losses))
    # six steps of at most about lr each; orders of summation may flip the sign of a step of a near-zero gradient
    assert np.abs(got - p).max() <= 12 * lr
    assert np.linalg.norm(got - p) <= 0.02 * np.linalg.norm(got - p0)


def test_training_sets_of_several_pieces(eng):
    """Positions go to the device 1 M at a time.  1.5 M samples, the last third
    other positions than the first two, with the network's own predictions as
    targets: the loss of an epoch that changes no weight is zero (to the rounding
    of the predictions' last bits) only if every sample has its own features."""
    eng.mlp_init(seed=5, out_bias=[4.0, 9.0, 14.0, 19.0])
    a, b = pg.random_playouts(51, 64, 0, 60, packed=True), pg.random_playouts(52, 64, 0, 60, packed=True)
    n_a, n_b = (1 << 20) // 64, (1 << 19) // 64
    pos = (pg.Pos * (64 * (n_a + n_b))).from_buffer_copy(bytes(a) * n_a + bytes(b) * n_b)
    t = np.concatenate([np.tile(eng.mlp_predict(a), (n_a, 1)), np.tile(eng.mlp_predict(b), (n_b, 1))])
    apart = float(((eng.mlp_predict(a) - eng.mlp_predict(b)) ** 2).mean())
    assert apart > 1e-3  # the loss of a third of the samples, had they the others' features
    assert eng.mlp_train(pos, t, epochs=1, batch=65536, lr=0.0) < 1e-8
    # one position per sample wrong on purpose, in the last piece
    t[-1] += 64.0
    assert abs(eng.mlp_train(pos, t, epochs=1, batch=65536, lr=0.0) - 64.0 ** 2 / len(pos)) < 1e-6
