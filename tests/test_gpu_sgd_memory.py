"""Device memory of the layout epochs' interaction lists: what a layout holds between and after its runs."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

MB = 1 << 20


def in_use(umap):
    """Bytes of device workspace in use: the least limit under which an allocation of 512 bytes still passes."""
    lib = umap.lib()
    before = lib.umapb_set_workspace_limit(0)
    lo, hi = 1, 1 << 40
    try:
        while lo < hi:
            mid = (lo + hi) // 2
            lib.umapb_set_workspace_limit(mid)
            try:
                umap.random_init(1, 1, dtype=np.float32)
                hi = mid
            except umap.UmapbError:
                lo = mid + 1
    finally:
        lib.umapb_set_workspace_limit(before)
    return lo - 512


def layout(umap, n=20000, epochs=100, **options):
    X = oracle.gaussian_mixture(n, 10, 8, 4.0, seed=3, dtype=np.float32)
    Y = np.zeros((n, 2), dtype=np.float32)
    return umap.initialize_from_data(X, 2, Y, umap.Options(
        num_epochs=epochs, initialize_method=umap.InitializeMethod.RANDOM, **options)), Y


def test_layouts_keep_no_lists(umap):
    """A layout that has been run holds what it held before: its lists (some 200 MB
    here while it runs) are given back, when all epochs are done and when it was stopped between two long runs."""
    start = in_use(umap)
    status, Y = layout(umap)
    held = in_use(umap) - start
    assert 0 < held < 64 * MB
    status.run(Y, 50)
    assert in_use(umap) - start <= held + MB
    status.run(Y)
    assert in_use(umap) - start <= held + MB
    del status
    assert in_use(umap) == start
