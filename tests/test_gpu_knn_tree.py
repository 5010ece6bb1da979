"""The ordering of the points before the pruned search, at sizes around a tile
(128 points), a segment that one block splits (2048) and their multiples, on
data with and without clusters and with many equal points: whatever the order,
the search finds the FP64 oracle's neighbours."""
import numpy as np
import pytest

import oracle
from helpers import same_neighbors

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("clusters", [1, 40])
@pytest.mark.parametrize("n", [129, 256, 257, 2047, 2048, 2049, 4096, 4229])
def test_sizes(umap, n, clusters):
    X = oracle.gaussian_mixture(n, 7, clusters, 6.0 if clusters > 1 else 0.0, seed=n, dtype=np.float32)
    idx, dist = umap.knn(X, 9)
    ridx, rdist = oracle.knn(X, 9)
    assert same_neighbors(idx, ridx, rdist) == 0
    np.testing.assert_allclose(dist.astype(np.float64), rdist, rtol=1e-6, atol=1e-30)


@pytest.mark.parametrize("n,distinct", [(2048, 1), (2300, 3), (5000, 40)])
def test_equal_points(umap, n, distinct):
    rng = np.random.default_rng(n)
    X = rng.normal(size=(distinct, 5)).astype(np.float32)[rng.integers(0, distinct, n)]
    X[0] += 1.0   # one point apart
    idx, dist = umap.knn(X, 6)
    _, rdist = oracle.knn(X, 6)
    np.testing.assert_allclose(dist.astype(np.float64), rdist, rtol=1e-6, atol=1e-30)
    assert all(len(set(r.tolist())) == 6 and i not in r for i, r in enumerate(idx))


def test_batch_of_small_instances(umap):
    sizes = np.array([20, 128, 129, 2048, 2049, 700], np.int32)
    X = oracle.gaussian_mixture(int(sizes.sum()), 6, 5, 5.0, seed=4, dtype=np.float32)
    Y = np.zeros((len(X), 2), np.float32)
    umap.batch_run(X, sizes, 2, Y, umap.Options(num_neighbors=8, num_epochs=10, learning_rate=1e-30,
                                                 initialize_method=umap.InitializeMethod.RANDOM))
    assert np.all(np.isfinite(Y))
