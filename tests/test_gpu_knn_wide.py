"""Neighbour searches with more candidates than a thread's registers hold (the
tensor-core search in several passes) and of queries against a reference set
(its references split over several candidate lists), against the FP64 oracle:
the same neighbours, except for exchanges of distances equal to 1e-6 relative,
and distances rounded to float."""
import numpy as np
import pytest

import oracle
from helpers import same_neighbors

pytestmark = pytest.mark.gpu


def check(idx, dist, ridx, rdist):
    assert same_neighbors(idx, ridx, rdist) == 0
    np.testing.assert_allclose(dist.astype(np.float64), rdist, rtol=1e-6, atol=1e-30)


@pytest.mark.parametrize("n,dim,k", [(700, 10, 25), (2900, 20, 40), (1500, 63, 56), (1300, 64, 57), (900, 127, 120),
                                     (3000, 5, 88), (130, 3, 120), (400, 130, 40)])
def test_knn_many_neighbours(umap, n, dim, k):
    X = oracle.gaussian_mixture(n, dim, 4, 3.0, seed=n + k, dtype=np.float32)
    check(*umap.knn(X, k), *oracle.knn(X, k))


@pytest.mark.parametrize("k", [30, 70])
def test_knn_many_neighbours_with_ties(umap, k):
    # points of a small lattice: every distance many times, more equal ones than a pass lists
    X = np.random.default_rng(5).integers(0, 4, size=(2000, 3)).astype(np.float32)
    idx, dist = umap.knn(X, k)
    ridx, rdist = oracle.knn(X, k)
    np.testing.assert_allclose(dist.astype(np.float64), rdist, rtol=1e-6, atol=1e-30)
    for row in idx:
        assert len(set(row.tolist())) == k


def test_knn_many_neighbours_without_scale(umap):
    X = np.zeros((300, 6), np.float32)   # no finite non-zero maximum: the CUDA-core search
    idx, dist = umap.knn(X, 40)
    assert np.all(dist == 0) and np.all(idx >= 0)


@pytest.mark.parametrize("nref,nq,dim,k", [(1023, 20, 8, 15), (1024, 130, 8, 15), (4096, 1, 8, 15), (5000, 129, 63, 15), (6000, 700, 64, 8), (5001, 300, 127, 24),
                                           (4500, 260, 20, 30), (4200, 70, 30, 110), (4300, 40, 140, 15)])
def test_query_against_references(umap, nref, nq, dim, k):
    X = oracle.gaussian_mixture(nref + nq, dim, 5, 4.0, seed=nref + k, dtype=np.float32)
    ref, new = X[:nref], np.vstack([X[nref:], X[:2]])   # the last two coincide with references
    idx, dist = umap.knn_query(ref, new, k)
    check(idx, dist, *oracle.knn_query(ref, new, k))
    assert np.all(idx[-2:, 0] == np.arange(2)) and np.all(dist[-2:, 0] == 0)


def test_query_far_from_references(umap):
    # the queries set the scale of the search: the references' distances lose bits and are searched again in FP64
    X = oracle.gaussian_mixture(4400, 12, 4, 3.0, seed=9, dtype=np.float32)
    new = X[4100:] + np.float32(3000.0)
    check(*umap.knn_query(X[:4100], new, 10), *oracle.knn_query(X[:4100], new, 10))


def far(n, dim, seed):
    """Points a thousand units from the origin: the tensor cores' bound certifies no query."""
    return oracle.gaussian_mixture(n, dim, 4, 3.0, seed=seed, dtype=np.float32) + np.float32(1000.0)


# sizes around the blocks of 128 queries and 32 points, dimensions around 32 columns
@pytest.mark.parametrize("n,dim,k", [(33, 3, 15), (129, 32, 8), (1000, 33, 15), (2000, 10, 24), (3001, 20, 40), (1500, 40, 119), (2500, 4, 57)])
def test_knn_far_from_origin(umap, n, dim, k):
    X = far(n, dim, n + k)
    check(*umap.knn(X, k), *oracle.knn(X, k))


@pytest.mark.parametrize("nref,nq,dim,k", [(1024, 1, 5, 15), (4100, 300, 12, 15), (4100, 129, 40, 30), (2000, 40, 8, 110)])
def test_query_far_from_origin(umap, nref, nq, dim, k):
    X = far(nref + nq, dim, nref + k)
    check(*umap.knn_query(X[:nref], X[nref:], k), *oracle.knn_query(X[:nref], X[nref:], k))


@pytest.mark.parametrize("copies,k", [(1, 20), (100, 20), (140, 20), (100, 60), (240, 60), (270, 60)])   # within and beyond the 128 (256) points collected
def test_knn_far_copies(umap, copies, k):
    X = np.repeat(far(1400 // copies, 6, 3), copies, axis=0)
    idx, dist = umap.knn(X, k)
    ridx, rdist = oracle.knn(X, k)
    np.testing.assert_array_equal(idx, ridx)   # FP64 distances of equal points are equal: the lower index first
    np.testing.assert_allclose(dist.astype(np.float64), rdist, rtol=1e-6, atol=1e-30)


def test_far_from_origin_costs_little(umap):
    """20,000 x 20 points around the origin and a thousand units away, 60 neighbours."""
    import time

    X = oracle.gaussian_mixture(20000, 20, 10, 4.0, seed=1, dtype=np.float32)
    seconds = []
    for Z in (X, X + np.float32(1000.0)):
        umap.knn(Z, 60)
        best = 1e9
        for _ in range(3):
            t = time.perf_counter()
            umap.knn(Z, 60)
            best = min(best, time.perf_counter() - t)
        seconds.append(best)
    assert seconds[1] <= 3 * seconds[0], seconds


@pytest.mark.parametrize("n,dim,k,few", [(150, 2, 25, True), (1075, 2, 30, True), (1076, 2, 30, False), (499, 50, 56, True),
                                         (500, 50, 56, False), (150, 2, 57, False), (60, 100, 30, False)])
def test_few_points_take_the_short_search(umap, monkeypatch, n, dim, k, few):
    """Few points with 25 to 56 neighbours are searched as without tensor cores (the same launches)."""
    X = oracle.gaussian_mixture(n, dim, 4, 3.0, seed=n, dtype=np.float32)
    launches = []
    for cores in (None, "0"):
        if cores:
            monkeypatch.setenv("UMAPB_KNN_TENSOR_CORES", cores)
        umap.knn(X, k)
        before = umap.lib().umapb_launch_count()
        result = umap.knn(X, k)
        launches.append(umap.lib().umapb_launch_count() - before)
        check(*result, *oracle.knn(X, k))
    assert (launches[0] == launches[1]) == few, launches


@pytest.mark.parametrize("nref,dim,k,few", [(1505, 3, 8, True), (1506, 3, 8, False), (1023, 60, 5, True), (1024, 60, 5, False),
                                            (1023, 3, 9, True), (1024, 3, 9, False)])
def test_few_references_take_the_short_search(umap, monkeypatch, nref, dim, k, few):
    """Queries against few references are searched as without tensor cores (the same launches)."""
    X = oracle.gaussian_mixture(nref + 300, dim, 4, 3.0, seed=nref, dtype=np.float32)
    launches = []
    for cores in (None, "0"):
        if cores:
            monkeypatch.setenv("UMAPB_KNN_TENSOR_CORES", cores)
        umap.knn_query(X[:nref], X[nref:], k)
        before = umap.lib().umapb_launch_count()
        result = umap.knn_query(X[:nref], X[nref:], k)
        launches.append(umap.lib().umapb_launch_count() - before)
        check(*result, *oracle.knn_query(X[:nref], X[nref:], k))
    assert (launches[0] == launches[1]) == few, launches
