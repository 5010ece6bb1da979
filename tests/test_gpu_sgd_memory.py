"""Device memory of the layout epochs' interaction lists: what a layout holds between and after its runs."""
import os
import subprocess
import sys

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


WINDOW_SCRIPT = """
import sys
sys.path[:0] = [%r, %r]
import torch
import umappp_b200
from test_gpu_sgd_memory import layout
status, Y = layout(umappp_b200, epochs=60, negative_sample_rate=100.0, learning_rate=0.01)
status.run(Y, 1)
torch.cuda.synchronize()
free = torch.cuda.mem_get_info()[0]
status.run(Y)
torch.cuda.synchronize()
print(free - torch.cuda.mem_get_info()[0])
"""


def test_window_bytes_bound_the_lists(umap):
    """100 samples per firing edge: an epoch's lists take some 55 MB, 8 epochs (which a window of 32 MB had with 5
    samples) 430 MB per buffer.  The workspace cache keeps what a run took, so the device's free memory tells."""
    tests = os.path.dirname(os.path.abspath(__file__))
    r = subprocess.run([sys.executable, "-c", WINDOW_SCRIPT % (os.path.dirname(tests), tests)], capture_output=True,
                       text=True, env=dict(os.environ, UMAPB_SGD_WINDOW_BYTES=str(256 * MB)))
    assert r.returncode == 0, r.stderr
    assert int(r.stdout) <= 1.25 * 256 * MB


@pytest.mark.parametrize("num_dim", [2, 3])
def test_runs_short_of_memory(umap, monkeypatch, num_dim):
    """With less and less device memory a run takes shorter windows, one after the other where two do not fit; where
    even one epoch (some 6 MB here) does not, it fails and leaves the layout and the epoch as they were, so that it can
    be run again."""
    torch = pytest.importorskip("torch")
    monkeypatch.setenv("UMAPB_SGD_WINDOW_BYTES", str(64 * MB))
    n = 20000
    X = torch.from_numpy(oracle.gaussian_mixture(n, 10, 8, 4.0, seed=3, dtype=np.float32)).cuda()
    Y = torch.from_numpy(np.random.default_rng(1).normal(scale=5.0, size=(n, num_dim)).astype(np.float32)).cuda()
    start = Y.clone()
    torch.cuda.synchronize()
    status = umap.initialize_from_data(X, num_dim, Y, umap.Options(
        num_epochs=30, initialize_method=umap.InitializeMethod.NONE))
    held, failed = in_use(umap), 0
    for room in list(np.arange(0.5, 12, 0.5)) + [12]:
        before = umap.lib().umapb_set_workspace_limit(held + int(room * MB))
        try:
            status.run(Y)
        except umap.UmapbError:
            failed += 1
            assert status.epoch() == 0 and torch.equal(Y, start), room
        finally:
            umap.lib().umapb_set_workspace_limit(before)
        if status.epoch():
            break
    assert failed > 0 and status.epoch() == 30 and not torch.equal(Y, start)
