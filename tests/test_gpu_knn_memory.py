"""Neighbour searches where device memory is short: what the CUDA-core search has room for is searched, and the
shards of a search are the same ones whatever memory each of them had."""
import numpy as np
import pytest

import oracle
from helpers import same_neighbors
from test_gpu_sgd_memory import in_use

pytestmark = pytest.mark.gpu

KB, MB = 1 << 10, 1 << 20


class limited:
    """At most this much device workspace beyond what is in use."""

    def __init__(self, umap, room):
        self.umap, self.room = umap, room

    def __enter__(self):
        self.before = self.umap.lib().umapb_set_workspace_limit(in_use(self.umap) + self.room)

    def __exit__(self, *args):
        self.umap.lib().umapb_set_workspace_limit(self.before)


@pytest.mark.parametrize("nref,nq,dim,k", [(3000, 3000, 2, 15), (2000, 1500, 3, 40)])
def test_query_with_the_memory_of_one_list(umap, monkeypatch, nref, nq, dim, k):
    """The memory that the search takes without tensor cores is enough with them (the workspace may give an array a
    block that is a quarter larger)."""
    X = oracle.gaussian_mixture(nref + nq, dim, 5, 4.0, seed=k, dtype=np.float32)

    def search(room):
        with limited(umap, room):
            return umap.knn_query(X[:nref], X[nref:], k)

    lo, hi = 0, 64 * MB
    with monkeypatch.context() as m:
        m.setenv("UMAPB_KNN_TENSOR_CORES", "0")
        while hi - lo > 4 * KB:
            mid = (lo + hi) // 2
            try:
                search(mid)
                hi = mid
            except umap.UmapbError:
                lo = mid
    idx, dist = search(hi + hi // 4)
    ridx, rdist = oracle.knn_query(X[:nref], X[nref:], k)
    assert same_neighbors(idx, ridx, rdist) == 0
    np.testing.assert_allclose(dist.astype(np.float64), rdist, rtol=1e-6, atol=1e-30)


@pytest.mark.parametrize("k", [10, 30])
def test_shards_agree_whatever_memory_they_have(umap, k):
    n = 6000
    X = oracle.gaussian_mixture(n, 20, 6, 4.0, seed=2, dtype=np.float32)
    idx, dist = umap.knn(X, k)
    rows0, idx0, _ = umap.knn_shard(X, k, 0, 2)
    found = 0
    for room in list(range(512, 12 * 1024, 256)) + [1 << 20]:
        try:
            with limited(umap, room * KB):
                rows1, idx1, dist1 = umap.knn_shard(X, k, 1, 2)
        except umap.UmapbError:
            continue
        found += 1
        assert np.array_equal(np.sort(np.concatenate([rows0, rows1])), np.arange(n)), room
        np.testing.assert_allclose(dist1, dist[rows1], rtol=1e-6)
        assert same_neighbors(idx1, idx[rows1], dist[rows1]) == 0
    assert found > 1
