"""Pageable host arrays to the device and back (host_copy.cu): a layout that is
loaded and stored by a run of no epochs comes back as it was, at sizes around
those where the copy takes another way (1 MiB) and where it starts another slot
(2 MiB), from one thread and from several at once."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def round_trip(umap, n, seed):
    Y = np.random.default_rng(seed).integers(0, 2**31, size=(n, 1)).astype(np.int32).view(np.float32)
    want = Y.copy()
    none = np.zeros(0, np.float32)
    ep = umap.EpochData(np.zeros(n + 1, np.int64), np.zeros(0, np.int32), none, none, none, total_epochs=10, current_epoch=3)
    umap.optimize_layout(1, Y, ep, 1.5, 0.9, 1.0, 1.0, 1, 3, 5.0)
    assert np.array_equal(Y.view(np.int32), want.view(np.int32))


@pytest.mark.parametrize("nbytes", [4, MIB - 4, MIB, MIB + 4, 2 * MIB, 2 * MIB + 4, 8 * MIB, 8 * MIB + 4, 19 * MIB + 12])
def test_round_trip(umap, nbytes):
    for seed in range(3):
        round_trip(umap, nbytes // 4, seed)


def test_round_trips_at_once(umap):
    failures = []

    def work(i):
        try:
            for k in range(6):
                round_trip(umap, (3 + i) * MIB // 4 + 7 * k, 10 * i + k)
        except BaseException as e:   # noqa: BLE001 - reported below
            failures.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures


# pieces of half a MiB below 5 MiB, of two from there on; four slots
@pytest.mark.parametrize("nbytes", [MIB + MIB // 2, MIB + MIB // 2 + 4, 2 * MIB + MIB // 2 + 8, 4 * MIB + 4, 5 * MIB - 4, 5 * MIB,
                                    5 * MIB + 4, 12 * MIB + 4])
def test_round_trip_in_pieces(umap, nbytes):
    for seed in range(3):
        round_trip(umap, nbytes // 4, seed)


@pytest.mark.parametrize("nbytes", [MIB, 5 * MIB, 8 * MIB - 4, 8 * MIB])
def test_into_untouched_pages(umap, nbytes):
    """Search results into arrays whose pages nobody has written yet, or the middle one only."""
    import mmap

    X = np.random.default_rng(1).normal(size=(nbytes // 40, 3)).astype(np.float32)
    want = umap.knn(X, 10)
    for touch in (False, True):
        out = []
        for t, a in ((np.int32, want[0]), (np.float32, want[1])):
            m = np.frombuffer(mmap.mmap(-1, a.nbytes + 4096), dtype=t)[:a.size]
            if touch:
                m[a.size // 2] = 7
            out.append(m)
        umap._lib.check(umap.lib().umapb_knn(0, 3, len(X), X.ctypes.data, 10, out[0].ctypes.data, out[1].ctypes.data))
        assert np.array_equal(out[0].reshape(want[0].shape), want[0])
        assert np.array_equal(out[1].reshape(want[1].shape), want[1])
