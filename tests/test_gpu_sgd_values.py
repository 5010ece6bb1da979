"""The layout epochs' steps by value, with repulsion and with rows that pull on one another (sgd.cu: relays up to
49,152 points, single warps above, with one lane per row and with lane groups), against the serial steps of
optimize_layout.hpp:136-180 with the device's negative samples."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

A, B, SEED = 1.577, 0.895, 99


def attract(diff):
    d2 = max((diff * diff).sum(), 2.0 ** -52)
    q = d2 ** B
    return np.clip(-2 * A * B * q / (d2 * (A * q + 1)) * diff, -4, 4)


def repulse(diff, gamma):
    d2 = max((diff * diff).sum(), 2.0 ** -52)
    return np.clip(2 * gamma * B / ((0.001 + d2) * (A * d2 ** B + 1)) * diff, -4, 4)


def interactions(ep, n, epochs, rate):
    """(epoch, head, target, samples) of every firing edge, heads in order, edges in stored order."""
    enext, enneg = ep.enext.copy(), ep.enneg.copy()
    dt = ep.eps.dtype.type
    heads = np.repeat(np.arange(n), np.diff(ep.ptr))
    for e in range(epochs):
        for j in np.nonzero(enext <= e)[0]:
            epns = ep.eps[j] / dt(rate)
            nn = int((dt(e) - enneg[j]) / epns)
            enext[j] += ep.eps[j]
            enneg[j] += dt(nn) * epns
            h, t = int(heads[j]), int(ep.targets[j])
            yield e, h, t, oracle.negstream_draws(h, t, e, SEED, n, max(nn, 0))


def run(umap, ep, Y, num_dim, gamma, lr, epochs):
    dev = umap.EpochData(ep.ptr.copy(), ep.targets.copy(), ep.eps.copy(), ep.enext.copy(), ep.enneg.copy(),
                         total_epochs=epochs, current_epoch=0)
    out = Y.copy()
    umap.optimize_layout(num_dim, out, dev, A, B, gamma, lr, SEED, epochs, 5.0)
    return out


@pytest.mark.parametrize("n", [49100, 49160])
@pytest.mark.parametrize("num_dim,dtype", [(1, np.float32), (2, np.float32), (3, np.float32), (4, np.float32),
                                           (1, np.float64), (2, np.float64), (3, np.float64), (4, np.float64), (7, np.float64), (40, np.float64)])
def test_row_with_repulsion_matches_serial(umap, n, num_dim, dtype):
    """One row whose samples are never its tails: the serial layout.  FP64 to 1e-9 of the extent, as steps differ by
    less than 1e-15 of it.  FP32: a step's gradient is off by 2^-19 of at most 4 and a position by half a unit (2^-19
    below 64); 12 edges take at most 84 steps an epoch, at rates that add up to 1.05 over 20 epochs; four times their
    sum, as early errors may grow where a step overshoots."""
    epochs, edges, gamma, lr = 20, 12, 50.0, 0.1
    for attempt in range(20):   # tails that no sample meets
        rng = np.random.default_rng(100 * num_dim + attempt)
        tails = np.sort(1 + rng.permutation(n - 1)[:edges])
        g = oracle.CSR(np.concatenate([[0], np.full(n, edges, dtype=np.int64)]), tails.astype(np.int32),
                       rng.uniform(0.1, 1.0, size=edges).astype(dtype))
        ep = oracle.similarities_to_epochs(g, epochs, 5.0)
        steps = list(interactions(ep, n, epochs, 5.0))
        if not np.isin(np.concatenate([s[3] for s in steps]), tails).any():
            break
    else:
        raise AssertionError("no such tails")
    Y = rng.normal(scale=10.0, size=(n, num_dim)).astype(dtype)
    want = []
    for strength in (0.0, gamma):
        Z = Y.astype(np.float64)
        for e, h, t, samples in steps:
            alpha = lr * (1 - e / epochs)
            move = alpha * attract(Z[h] - Z[t])
            Z[h] += move
            Z[t] -= move
            for k in samples:
                if k != h:
                    Z[h] += alpha * repulse(Z[h] - Z[k], strength)
        want.append(Z)
    tol = 1e-9 * np.abs(Y).max() if dtype == np.float64 else 4 * (84 * 1.05 * 4 * 2.0 ** -19 + 84 * 20 * 2.0 ** -19)
    got = run(umap, ep, Y, num_dim, gamma, lr, epochs)
    assert np.max(np.abs(want[1][0] - want[0][0])) > 10 * tol   # the samples count
    assert np.max(np.abs(got - want[1])) <= tol


@pytest.mark.parametrize("n", [600, 49100, 49160])
@pytest.mark.parametrize("num_dim", [1, 2, 3, 7])
def test_moves_of_a_hub_and_its_neighbours_add_up(umap, n, num_dim):
    """A hub with 120 edges that all fire (some 720 entries an epoch, so that its head takes over the other rows' pulls
    twice) and 120 rows whose edge is the hub.  At a rate of 1e-9 every step is the gradient at the start but for parts
    of 1e-9 x some 15,000 steps of at most 4 (6e-5): each point's move is the sum of its gradients, however the rows
    run beside one another."""
    epochs, edges, gamma, lr = 12, 120, 2.0, 1e-9
    rng = np.random.default_rng(num_dim)
    count = np.zeros(n, dtype=np.int64)
    count[0] = edges
    count[1:edges + 1] = 1
    targets = np.concatenate([np.arange(1, edges + 1), np.zeros(edges)]).astype(np.int32)
    g = oracle.CSR(np.concatenate([[0], np.cumsum(count)]), targets, np.ones(2 * edges))
    ep = oracle.similarities_to_epochs(g, epochs, 5.0)
    Y = rng.normal(scale=3.0, size=(n, num_dim))
    want = np.zeros_like(Y)
    for e, h, t, samples in interactions(ep, n, epochs, 5.0):
        alpha = lr * (1 - e / epochs)
        move = alpha * attract(Y[h] - Y[t])
        want[h] += move
        want[t] -= move
        for k in samples:
            if k != h:
                want[h] += alpha * repulse(Y[h] - Y[k], gamma)
    got = run(umap, ep, Y, num_dim, gamma, lr, epochs) - Y
    assert np.abs(want[0]).max() > 1e-8
    assert np.max(np.abs(got - want)) <= 1e-3 * np.abs(want[1:edges + 1]).max()
