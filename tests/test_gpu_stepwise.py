"""Layouts run a few epochs at a time, whose lists are read ahead from call to call."""
import numpy as np
import pytest

import oracle
from test_gpu_sgd_memory import MB, in_use, layout

pytestmark = pytest.mark.gpu

EPOCHS = 60


@pytest.mark.parametrize("n,num_dim", [(300, 2), (60000, 2), (500, 3)])   # both list buffers, one, a copied layout
def test_same_epochs_however_called(umap, n, num_dim):
    """At a rate of 1e-9 every interaction moves points by its gradient at the start, whatever runs beside it, but for
    parts of 1e-9 x 60 epochs x some 30 steps of at most 4 (1e-5 of the sum): an epoch left out, repeated or taken from
    another's list changes the sum by a sixtieth."""
    X = oracle.gaussian_mixture(n, 10, 4, 4.0, seed=5, dtype=np.float64 if n < 1000 else np.float32).astype(np.float64)
    Y0 = np.random.default_rng(2).normal(scale=5.0, size=(n, num_dim))
    idx, dist = umap.knn(X.astype(np.float32), 10)
    moves = []
    for calls in ([60], [1] * 60, [1, 2, 3, 9, 1, 1, 1, 20, 8, 8, 1, 1, 4], [7, 50, 1, 1, 1], [1, 1, 1, 57], [8] * 7 + [4]):
        assert sum(calls) == EPOCHS
        Y = Y0.copy()
        status = umap.initialize_knn_matrix(idx, dist.astype(np.float64), num_dim, Y, umap.Options(
            num_epochs=EPOCHS, learning_rate=1e-9, initialize_method=umap.InitializeMethod.NONE))
        for c in calls:
            status.run(Y, status.epoch() + c)
        assert status.epoch() == EPOCHS
        moves.append(Y - Y0)
    largest = np.abs(moves[0]).max()
    assert largest > 1e-8
    for m in moves[1:]:
        assert np.max(np.abs(m - moves[0])) <= 1e-3 * largest


def test_what_is_read_ahead_is_bounded_and_given_back(umap, monkeypatch):
    monkeypatch.setenv("UMAPB_SGD_WINDOW_BYTES", str(32 * MB))
    status, Y = layout(umap, epochs=40)
    held = in_use(umap)
    for e in range(1, 30):
        status.run(Y, e)
        assert in_use(umap) <= held + 1.125 * 32 * MB / 2 + 2 * MB   # (buckets and the segments' offsets)
    status.run(Y)
    assert in_use(umap) <= held + MB
