"""The epochs' interaction lists (sgd_lists.cu) and the kernels that walk them,
at the sizes where they change form: layouts of every lane split, rows shorter
and longer than a segment of the list builder, edges with more negative samples
than are staged, one epoch per window, and layouts that are not aligned to
vectors.

Where rows share nothing that moves, a layout is determined by its inputs and
is compared with the oracle's serial FP64 run to 1e-9 of its extent (the
device's pow and the host's may differ in the last bit, and every step adds
less than 1e-15 of the extent):
- transform: only the new points move, with the device's negative samples;
- one row that holds all edges, with no repulsion (strength 0): its head meets
  every tail once an epoch, and no other row moves any.
"""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

TOL = 1e-9


@pytest.mark.parametrize("num_dim,rate,num_new", [(1, 5.0, 33), (2, 5.0, 600), (2, 60.0, 65), (2, 0.0, 40), (3, 5.0, 64),
                                                  (4, 9.0, 31), (5, 5.0, 40), (9, 5.0, 17), (17, 13.0, 16), (40, 5.0, 9)])
def test_lists_match_serial_transform(umap, num_dim, rate, num_new):
    X = oracle.gaussian_mixture(900 + num_new, 8, 4, 4.0, seed=num_dim, dtype=np.float64)
    ref, new = X[:900], X[900:]
    Yref = np.random.default_rng(num_dim).normal(scale=4.0, size=(900, num_dim))
    opt = umap.Options(negative_sample_rate=rate)
    Y = umap.transform(ref, Yref, new, opt, num_epochs=70)   # windows of 32, 32 and 6 epochs
    a, b = oracle.find_ab(1.0, 0.1)
    Yo, _, _, _ = oracle.transform(ref, Yref, new, 15, 70, a, b, negative_sample_rate=rate, seed=opt.optimize_seed)
    assert np.max(np.abs(Y - Yo)) <= TOL * np.abs(Yref).max()


def star(umap, edges, epochs, num_dim, dtype, seed=3):
    """Row 0 with 'edges' edges of random weight among edges + 70 points; the other rows empty."""
    rng = np.random.default_rng(seed)
    n = edges + 70
    w = rng.uniform(0.02, 1.0, size=edges).astype(dtype)
    g = oracle.CSR(np.concatenate([[0], np.full(n, edges, dtype=np.int64)]),
                   (1 + rng.permutation(n - 1)[:edges]).astype(np.int32), w)
    return oracle.similarities_to_epochs(g, epochs, 5.0), rng.normal(scale=3.0, size=(n, num_dim)).astype(dtype)


def device_epochs(umap, ep):
    return umap.EpochData(ep.ptr.copy(), ep.targets.copy(), ep.eps.copy(), ep.enext.copy(), ep.enneg.copy(),
                          total_epochs=ep.total_epochs, current_epoch=0)


@pytest.mark.parametrize("window_bytes", [None, 1])
@pytest.mark.parametrize("edges,num_dim", [(1, 2), (255, 2), (257, 3), (384, 2), (385, 2), (1300, 2), (1300, 6)])
def test_long_rows_match_serial(umap, monkeypatch, edges, num_dim, window_bytes):
    if window_bytes:
        monkeypatch.setenv("UMAPB_SGD_WINDOW_BYTES", str(window_bytes))   # one epoch per window
    monkeypatch.setenv("UMAPB_CHECK_SCHEDULE", "1")
    ep, Y = star(umap, edges, 40, num_dim, np.float64)
    dev = device_epochs(umap, ep)
    Yd = Y.copy()
    umap.optimize_layout(num_dim, Yd, dev, 1.577, 0.895, 0.0, 1.0, 99, 40, 5.0)
    oracle.optimize_layout(num_dim, Y, ep, 1.577, 0.895, 0.0, 1.0, 99, 40)
    assert np.max(np.abs(Yd - Y)) <= TOL * np.abs(Y).max()
    assert np.array_equal(dev.epoch_of_next_sample, ep.enext)
    assert np.array_equal(dev.epoch_of_next_negative_sample, ep.enneg)


def stars(n, heads, num_dim, dtype, seed=5):
    """n points of which the first 'heads' have edges, up to 90 each (every fifth none), to tails that no other has."""
    rng = np.random.default_rng(seed)
    count = np.zeros(n, dtype=np.int64)
    count[:heads] = np.where(np.arange(heads) % 5 == 4, 0, rng.integers(1, 91, size=heads))
    assert heads + count.sum() <= n
    w = rng.uniform(0.02, 1.0, size=count.sum()).astype(dtype)
    g = oracle.CSR(np.concatenate([[0], np.cumsum(count)]), (heads + np.arange(count.sum())).astype(np.int32), w)
    return oracle.similarities_to_epochs(g, 40, 5.0), rng.normal(scale=3.0, size=(n, num_dim)).astype(dtype)


# 49,152 points have 6,144 rows in flight, the most that relays take; 49,160 are taken by single warps
@pytest.mark.parametrize("n,heads", [(900, 9), (12000, 250), (49152, 700), (49160, 700)])
@pytest.mark.parametrize("num_dim,dtype", [(1, np.float32), (2, np.float32), (3, np.float32), (7, np.float32),
                                           (1, np.float64), (2, np.float64), (3, np.float64), (40, np.float64)])
def test_separate_rows_match_serial(umap, n, heads, num_dim, dtype):
    """Rows without common points and no repulsion: the serial run's layout, to TOL in FP64.  In FP32 a step's
    gradient is off by 2^-19 of at most 4 (the approximate logarithm, power and reciprocal and four products), a
    position by half a unit (at most 2^-20 below 32), and a row's head takes at most 90 steps an epoch at rates that
    add up to 2.05; four times their sum, as early errors may grow where a step overshoots."""
    ep, Y = stars(n, heads, num_dim, dtype)
    dev = device_epochs(umap, ep)
    Yd = Y.copy()
    umap.optimize_layout(num_dim, Yd, dev, 1.577, 0.895, 0.0, 0.1, 99, 40, 5.0)
    start = Y.copy()
    oracle.optimize_layout(num_dim, Y, ep, 1.577, 0.895, 0.0, 0.1, 99, 40)
    tol = TOL * np.abs(Y).max() if dtype == np.float64 else 4 * (90 * 2.05 * 4 * 2.0 ** -19 + 90 * 40 * 2.0 ** -20)
    assert np.max(np.abs(Y - start)) > 10 * tol
    assert np.max(np.abs(Yd - Y)) <= tol


# where relays end with more lanes per row: 1,536, 1,024 and 3,072 rows in flight
@pytest.mark.parametrize("n,num_dim,dtype", [(12288, 20, np.float32), (12289, 20, np.float32), (8192, 20, np.float64), (8193, 40, np.float64),
                                             (24576, 10, np.float64), (24577, 16, np.float64)])
def test_separate_rows_where_relays_end(umap, n, num_dim, dtype):
    test_separate_rows_match_serial(umap, n, 150, num_dim, dtype)


@pytest.mark.parametrize("num_dim", [2, 3, 4])
def test_unaligned_layout(umap, num_dim):
    torch = pytest.importorskip("torch")
    ep, Y = star(umap, 300, 20, num_dim, np.float32)
    out = []
    for offset in (0, 1):   # floats past a 256-byte boundary
        store = torch.zeros(Y.size + 8, device="cuda")
        view = store[offset:offset + Y.size]
        view.copy_(torch.from_numpy(Y).reshape(-1))
        torch.cuda.synchronize()
        dev = device_epochs(umap, ep)
        umap._lib.check(umap.lib().umapb_optimize_layout(
            0, num_dim, view.data_ptr(), len(Y), dev.cumulative_num_edges.ctypes.data, dev.edge_targets.ctypes.data,
            dev.epochs_per_sample.ctypes.data, dev.epoch_of_next_sample.ctypes.data,
            dev.epoch_of_next_negative_sample.ctypes.data, 5.0, 20, umap.ctypes.byref(umap.ctypes.c_int(0)), 1.577, 0.895,
            0.0, 1.0, 99, 20))
        out.append(store.cpu().numpy()[offset:offset + Y.size].copy())
        assert np.all(np.delete(store.cpu().numpy(), np.arange(offset, offset + Y.size)) == 0)
    assert np.array_equal(out[0], out[1])


def test_fewer_edges_take_no_longer(umap):
    """Three million points of which nearly all have no edge: a thousand edges in all, or four hundred thousand."""
    import time

    n, rng = 3000000, np.random.default_rng(4)
    seconds = []
    for edges in (1000, 400000):
        count = np.zeros(n, dtype=np.int64)
        count[np.sort(rng.choice(n, edges // 10, replace=False))] = 10
        g = oracle.CSR(np.concatenate([[0], np.cumsum(count)]), rng.integers(0, n, edges).astype(np.int32),
                       rng.uniform(0.1, 1.0, edges).astype(np.float32))
        ep = oracle.similarities_to_epochs(g, 200, 5.0)
        Y = np.zeros((n, 2), dtype=np.float32)
        best = 1e9
        for _ in range(3):
            dev = device_epochs(umap, ep)
            t = time.perf_counter()
            umap.optimize_layout(2, Y, dev, 1.577, 0.895, 1.0, 1.0, 99, 200, 5.0)
            best = min(best, time.perf_counter() - t)
        seconds.append(best)
    assert seconds[0] <= 1.2 * seconds[1], seconds
