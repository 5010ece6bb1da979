"""The eigensolver's device steps on graphs whose spectrum is known: complete
graphs and stars, where the Krylov space closes after two or three steps and
the basis goes on from fresh directions, with rows from 1 edge to all.  With
residuals below 1e-10 of the largest eigenvalue the eigenvalues of a symmetric
matrix are within 1e-10 of it; the eigenvectors come back at the requested
scale and satisfy the eigen equation to the residual."""
import numpy as np
import pytest

import oracle
from helpers import csr_tuple

pytestmark = pytest.mark.gpu


def complete(n):
    j = np.arange(n)
    idx = np.concatenate([np.delete(j, i) for i in range(n)]).astype(np.int32)
    return oracle.CSR(np.arange(n + 1, dtype=np.int64) * (n - 1), idx, np.full(n * (n - 1), 0.7))


def star(n):
    ptr = np.concatenate([[0], n - 1 + np.arange(n, dtype=np.int64)])
    idx = np.concatenate([np.arange(1, n), np.zeros(n - 1)]).astype(np.int32)
    return oracle.CSR(ptr, idx, np.full(2 * (n - 1), 0.3))


@pytest.mark.parametrize("make,n", [(complete, 4), (complete, 17), (complete, 18), (complete, 65), (complete, 300),
                                    (star, 4), (star, 33), (star, 4736), (star, 4737), (star, 20000)])
def test_known_spectrum(umap, make, n):
    g = make(n)
    ok, Y, ev = umap.spectral_init(csr_tuple(g), 2, irlba=umap.IrlbaOptions(convergence_tolerance=1e-10),
                                   return_evals=True)
    assert ok
    second = 1 - 1 / (n - 1) if make is complete else 1.0
    assert np.max(np.abs(ev - np.array([2.0, second, second]))) <= 2e-9
    assert np.all(np.isfinite(Y)) and abs(np.abs(Y).max() - 10) < 1e-9
    # the eigen equation, W applied by rows
    deg = np.add.reduceat(g.val, g.ptr[:-1])
    rows = np.repeat(np.arange(n), np.diff(g.ptr))
    for d in range(2):
        v = Y[:, d] / np.linalg.norm(Y[:, d])
        av = v + np.bincount(rows, g.val * v[g.idx] / np.sqrt(deg[rows] * deg[g.idx]), minlength=n)
        assert np.linalg.norm(av - ev[d + 1] * v) <= 1e-8
