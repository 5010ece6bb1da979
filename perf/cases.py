"""What the framework's users have it do, as timed cases: whole layouts, from small to a million points, in both
precisions and in two and three dimensions; batches of small data sets; the spectral initial layout; the neighbour
search by itself; new points placed into a finished layout; and the gradient of the layout's loss.

listed() gives the cases, draw(rng) more of the same ranges, prepare(case, seed) the arrays a program holds before the
call, run(state) one call through the public entry points, work(case) the bytes and operations such a call cannot do
without, and exact(case, seed) the result in 64 bits, computed with torch alone.

Data are Gaussian mixtures in 'd' dimensions: 'clusters' centres of standard deviation 'spread' and unit noise, so
that 'spread' 0 gives one connected cloud.  The layouts here ("fit" and "batch") start from a given layout and refine
it at a small learning rate, as a program does that has an older layout of the same data
(InitializeMethod.NONE): the rows of an epoch run concurrently, and from a random start at the full rate two runs on
the same inputs end in different, equally good layouts, which cannot be compared value by value.  The work of an epoch
does not depend on the rate.
"""
import math

import numpy as np
import torch

import umappp_b200 as U

A, B = 1.577, 0.895          # the curve of min_dist 0.1 and spread 1
LAYOUT_SCALE = 100.0         # half the extent of a given layout
RATE_EPOCHS = 20.0           # learning rate x epochs of a refinement


def listed():
    return [
        # the smallest everyday call: one sample of an interactive session; bound by latency and launches
        fit("fit_1k", 1000, 20, 5, epochs=500),
        # a typical single experiment, at the default 500 epochs
        fit("fit_10k", 10007, 50, 10, epochs=500),
        # a large experiment, with more neighbours than the default
        fit("fit_100k_k30", 100000, 50, 20, k=30, epochs=200),
        # the headline size: a million points, 200 epochs
        fit("fit_1m", 1000000, 50, 100, spread=5.0, epochs=200),
        # three dimensions, for rotating views
        fit("fit_20k_3d", 20011, 50, 10, dims=3, epochs=200),
        # double precision, the type of the R and Python callers
        fit("fit_2k_f64", 2003, 20, 5, dtype="f64", epochs=200),
        # many independent samples laid out in one call
        {"name": "batch_32", "kind": "batch", "instances": 32, "lo": 300, "hi": 10000, "d": 30, "clusters": 5,
         "spread": 5.0, "k": 15, "epochs": 200},
        # everything before the first epoch on connected data: neighbours, weights, graph and spectral layout
        {"name": "spectral_20k", "kind": "init", "n": 20000, "d": 30, "clusters": 1, "spread": 0.0, "k": 15,
         "dims": 2},
        # the neighbour search as a host program calls it, at the default number of neighbours
        {"name": "knn_100k", "kind": "knn", "n": 100003, "d": 50, "clusters": 20, "spread": 4.0, "k": 15,
         "dtype": "f32"},
        # and at the larger neighbourhoods that global structure asks for
        {"name": "knn_30k_k50", "kind": "knn", "n": 30011, "d": 30, "clusters": 10, "spread": 4.0, "k": 50,
         "dtype": "f32"},
        # new points placed into a finished layout (encoding of unseen data)
        {"name": "transform_100k_10k", "kind": "transform", "n": 100000, "new": 10000, "d": 50, "clusters": 20,
         "spread": 4.0, "k": 15},
        # the backward direction: loss and gradient of a layout, for programs that optimise it themselves
        {"name": "loss_grad_100k", "kind": "loss_grad", "n": 100000, "pairs": 10, "dims": 2},
    ]


def fit(name, n, d, clusters, spread=4.0, k=15, dims=2, dtype="f32", epochs=200):
    c = {"kind": "fit", "n": n, "d": d, "clusters": clusters, "spread": spread, "k": k, "dims": dims, "dtype": dtype,
         "epochs": epochs}
    return dict(c, name=name) if name else c


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["fit", "fit", "fit", "fit_3d", "fit_f64", "batch", "init", "knn", "knn", "transform", "loss_grad"])
    d, clusters = size(5, 100), rng.randint(3, 20)
    if kind == "fit":
        return fit(None, size(1000, 200000), d, clusters, k=size(5, 50), epochs=rng.choice([100, 200, 500]))
    if kind == "fit_3d":
        return fit(None, size(1000, 20000), d, clusters, k=size(5, 30), dims=rng.choice([3, 3, 5]), epochs=100)
    if kind == "fit_f64":
        return fit(None, size(500, 5000), d, clusters, k=size(5, 30), dims=rng.choice([2, 2, 3]), dtype="f64",
                   epochs=100)
    if kind == "batch":
        return {"kind": "batch", "instances": rng.randint(4, 48), "lo": size(200, 600), "hi": size(1000, 10000),
                "d": d, "clusters": 5, "spread": 5.0, "k": size(5, 20), "epochs": rng.choice([100, 200])}
    if kind == "init":
        return {"kind": "init", "n": size(1000, 50000), "d": size(5, 50), "clusters": 1, "spread": 0.0,
                "k": size(10, 30), "dims": rng.choice([2, 2, 3])}
    if kind == "knn":
        dtype = rng.choice(["f32", "f32", "f32", "f64"])
        return {"kind": "knn", "n": size(1000, 100000 if dtype == "f32" else 20000), "d": d, "clusters": clusters,
                "spread": 4.0, "k": size(5, 60), "dtype": dtype}
    if kind == "transform":
        return {"kind": "transform", "n": size(2000, 100000), "new": size(100, 10000), "d": d, "clusters": clusters,
                "spread": 4.0, "k": size(5, 30)}
    return {"kind": "loss_grad", "n": size(1000, 200000), "pairs": rng.randint(5, 12), "dims": rng.choice([2, 2, 3])}


# ------------------------------------------------------------------- inputs --

DTYPES = {"f32": torch.float32, "f64": torch.float64}


def _mixture(g, n, d, clusters, spread, dtype=torch.float32):
    """Points of a Gaussian mixture on the GPU, and the cluster of each."""
    centres = torch.randn(clusters, d, device="cuda", generator=g) * spread
    label = torch.randint(0, clusters, (n,), device="cuda", generator=g)
    return (torch.randn(n, d, device="cuda", generator=g) + centres[label]).to(dtype), label


def _layout(g, label, clusters, dims, dtype=torch.float32):
    """An older layout of these points: their clusters apart, each a unit cloud."""
    centres = (torch.rand(clusters, dims, device="cuda", generator=g) * 2 - 1) * LAYOUT_SCALE
    return (centres[label] + torch.randn(len(label), dims, device="cuda", generator=g)).to(dtype)


def _batch_sizes(case):
    m, lo, hi = case["instances"], case["lo"], case["hi"]
    return np.array([round(lo * (hi / lo) ** (i / max(m - 1, 1))) for i in range(m)], dtype=np.int32)


def _refine(case):
    return U.Options(num_neighbors=case["k"], num_epochs=case["epochs"], learning_rate=RATE_EPOCHS / case["epochs"],
                     initialize_method=U.InitializeMethod.NONE)


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    s = {"case": case}
    if kind == "fit":
        dtype = DTYPES[case["dtype"]]
        s["data"], label = _mixture(g, case["n"], case["d"], case["clusters"], case["spread"], dtype)
        s["layout"] = _layout(g, label, case["clusters"], case["dims"], dtype)
        s["options"] = _refine(case)
    elif kind == "batch":
        s["sizes"] = _batch_sizes(case)
        parts = []
        for m in s["sizes"]:
            x, label = _mixture(g, int(m), case["d"], case["clusters"], case["spread"])
            parts.append((x, _layout(g, label, case["clusters"], 2)))
        s["data"], s["layout"] = (torch.cat([p[i] for p in parts]) for i in (0, 1))
        s["options"] = _refine(case)
    elif kind == "init":
        s["data"], _ = _mixture(g, case["n"], case["d"], case["clusters"], case["spread"])
        s["options"] = U.Options(num_neighbors=case["k"])
    elif kind == "knn":
        x, _ = _mixture(g, case["n"], case["d"], case["clusters"], case["spread"], DTYPES[case["dtype"]])
        s["data"] = x.cpu().numpy()
    elif kind == "transform":
        x, label = _mixture(g, case["n"] + case["new"], case["d"], case["clusters"], case["spread"])
        y = _layout(g, label, case["clusters"], 2)
        x, y = x.cpu().numpy(), y.cpu().numpy()
        s["data"], s["new"], s["layout"] = x[:case["n"]], x[case["n"]:], np.ascontiguousarray(y[:case["n"]])
        s["options"] = U.Options(num_neighbors=case["k"], a=A, b=B)
    else:
        s["graph"], s["layout"] = _graph(g, case["n"], case["pairs"], case["dims"])
    torch.cuda.synchronize()   # the library works on its own streams
    return s


def _graph(g, n, pairs, dims):
    """A symmetric weighted graph of neighbours along a curve, the points in random order, and a layout near it."""
    order = torch.randperm(n, device="cuda", generator=g)
    offset = torch.rand(n, 60, device="cuda", generator=g).argsort(dim=1)[:, :pairs] + 1
    i = torch.arange(n, device="cuda")[:, None].expand(n, pairs)
    j = (i + offset).reshape(-1)
    i = i.reshape(-1)[j < n]
    j = j[j < n]
    w = torch.exp(-4 * torch.rand(len(i), device="cuda", generator=g))
    row, col = torch.cat([order[i], order[j]]), torch.cat([order[j], order[i]])
    at = torch.argsort(row * n + col)
    row, col, w = row[at], col[at], torch.cat([w, w])[at]
    ptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    ptr[1:] = torch.cumsum(torch.bincount(row, minlength=n), 0)
    t = torch.arange(n, device="cuda") * (20.0 / n)
    curve = torch.stack([20 * torch.cos(t * (c + 1) * 0.7 + c) for c in range(dims)], 1)
    y = torch.empty(n, dims, device="cuda")
    y[order] = curve + 0.3 * torch.randn(n, dims, device="cuda", generator=g)
    return (ptr.cpu().numpy(), col.to(torch.int32).cpu().numpy(), w.cpu().numpy()), y.cpu().numpy()


# --------------------------------------------------------------------- runs --

def run(s):
    kind = s["case"]["kind"]
    if kind == "fit":
        y = s["layout"].clone()
        torch.cuda.current_stream().synchronize()   # the library's streams do not wait for torch's
        status = U.initialize_from_data(s["data"], s["case"]["dims"], y, s["options"])
        status.run(y)
        return {"layout": y, "edges": status.num_edges()}
    if kind == "batch":
        y = s["layout"].clone()
        torch.cuda.current_stream().synchronize()
        U.batch_run(s["data"], s["sizes"], 2, y, s["options"])
        return {"layout": y}
    if kind == "init":
        y = torch.empty(s["case"]["n"], s["case"]["dims"], device="cuda")
        status = U.initialize_from_data(s["data"], s["case"]["dims"], y, s["options"])
        return {"layout": y, "edges": status.num_edges()}
    if kind == "knn":
        indices, distances = U.knn(s["data"], s["case"]["k"])
        return {"indices": indices, "distances": distances}
    if kind == "transform":
        return {"layout": U.transform(s["data"], s["layout"], s["new"], s["options"])}
    loss, grad, grad_ab = U.loss_grad(s["graph"], s["layout"], A, B)
    return {"loss": loss, "grad": grad, "grad_ab": np.array(grad_ab)}


def _epoch_work(edges, epochs, dims, size):
    """Bytes and operations of the epochs over 'edges' stored edges: about 0.28 of them fire in an epoch, each with
    five negative samples; a step is some 25 operations plus 5 a dimension."""
    fired = 0.28 * edges * epochs
    return (edges * size * epochs + fired * (12 + 4 * dims * size + 4 * size) + fired * 5 * dims * size,
            fired * 6 * (25 + 5 * dims))


def work(case):
    kind = case["kind"]
    size = 8 if case.get("dtype") == "f64" else 4
    if kind == "loss_grad":
        edges = 2 * case["n"] * case["pairs"]
        return {"bytes": edges * 8 + case["n"] * (8 + 8 * case["dims"]), "flops": edges * (30 + 6 * case["dims"])}
    n = int(_batch_sizes(case).sum()) if kind == "batch" else case["n"]
    new = case.get("new", 0)
    k, d = case["k"], case["d"]
    lists = (new or n) * k
    nbytes, flops = (n + new) * d * size, lists * 2 * d   # data in once, the listed distances
    if kind == "knn":
        return {"bytes": nbytes + lists * (4 + size), "flops": flops}
    if kind == "transform":
        epochs = 100 if new <= 10000 else 30
        fired = 0.4 * lists * epochs
        return {"bytes": nbytes + (n + 2 * new) * 8 + fired * 6 * 8, "flops": flops + fired * 6 * 35}
    edges = 1.7 * lists
    nbytes, flops = nbytes + lists * 16 + edges * (4 + 4 * size), flops + lists * 200
    if kind == "init":
        return {"bytes": nbytes + n * case["dims"] * size, "flops": flops}
    dims = case.get("dims", 2)
    eb, ef = _epoch_work(edges, case["epochs"], dims, size)
    return {"bytes": nbytes + eb + 2 * n * dims * size, "flops": flops + ef}


# ------------------------------------------------------------ 64-bit values --

def exact(case, seed):
    kind = case["kind"]
    if kind in ("fit", "batch"):
        return None   # the order in which concurrent rows meet is part of the result: no value is the exact one
    if kind == "init" and case["n"] > 30000:
        return None
    s = prepare(case, seed)
    if kind == "loss_grad":
        return _loss_grad(s["graph"], s["layout"])
    x = torch.as_tensor(s["data"], device="cuda").double()
    if kind == "knn":
        return {"indices": None, "distances": _neighbours(x, None, case["k"])[1]}
    if kind == "transform":
        return {"layout": _transform(x, torch.as_tensor(s["new"], device="cuda").double(),
                                     torch.as_tensor(s["layout"], device="cuda").double(), case)}
    return {"layout": _spectral(*_neighbours(x, None, case["k"]), case["dims"]), "edges": None}


def _neighbours(x, q, k):
    """The k nearest rows of x to every row of q (None: to its own rows, without themselves), by distance."""
    own = q is None
    q = x if own else q
    idx, dist = [], []
    norm = (x * x).sum(1)
    step = max(1, min(len(q), (1 << 28) // len(x)))
    for b in range(0, len(q), step):
        part = q[b:b + step]
        d2 = norm[None, :] - 2 * part @ x.T
        if own:
            d2[torch.arange(len(part), device="cuda"), torch.arange(b, b + len(part), device="cuda")] = math.inf
        near = d2.topk(min(k + 4, d2.shape[1]), largest=False).indices
        true = (part[:, None, :] - x[near]).square().sum(2).sqrt()
        true = torch.where(torch.isinf(d2.gather(1, near)), math.inf, true)
        true, at = true.sort(dim=1)
        idx.append(near.gather(1, at)[:, :k])
        dist.append(true[:, :k])
    return torch.cat(idx), torch.cat(dist)


def _weights(dist):
    """Membership weights of sorted positive distances: exp(-(d - rho) / sigma), the sigma at which they sum to
    log2(k + 1), found by bisection; sigma at least 1e-3 of the mean distance."""
    n, k = dist.shape
    far = (dist - dist[:, :1]).clamp_min(0)
    lo, hi = torch.zeros(n, 1, device="cuda", dtype=torch.float64), far[:, -1:] * 1e4
    for _ in range(200):
        mid = (lo + hi) / 2
        over = torch.exp(-far / mid).sum(1, keepdim=True) > math.log2(k + 1)
        lo, hi = torch.where(over, lo, mid), torch.where(over, mid, hi)
    sigma = torch.maximum((lo + hi) / 2, dist.mean(1, keepdim=True) * 1e-3)
    return torch.where(far > 0, torch.exp(-far / sigma), 1.0)


def _spectral(idx, dist, dims):
    """The eigenvectors 2 .. dims + 1 of I + D^-1/2 W D^-1/2, W the union of the weighted neighbours, by Lanczos with
    full orthogonalisation; signed by their largest entry and scaled to 10."""
    n, k = idx.shape
    w = _weights(dist)
    i = torch.arange(n, device="cuda").repeat_interleave(k)
    m = torch.sparse_coo_tensor(torch.stack([i, idx.reshape(-1)]), w.reshape(-1), (n, n)).coalesce()
    t = m.t().coalesce()
    both = (m + t).coalesce()
    c = torch.sparse_coo_tensor(torch.cat([m.indices(), t.indices()], 1),
                                torch.cat([torch.log1p(-m.values().clamp_max(1 - 1e-300)),
                                           torch.log1p(-t.values().clamp_max(1 - 1e-300))]), (n, n)).coalesce()
    a, ai = -torch.expm1(c.values()), both.indices()   # w + w' - w w'
    root = torch.zeros(n, device="cuda", dtype=torch.float64).index_add_(0, ai[0], a).sqrt()
    lap = torch.sparse_coo_tensor(ai, a / (root[ai[0]] * root[ai[1]]), (n, n)).coalesce().to_sparse_csr()
    steps = min(n, 400)
    v = torch.zeros(steps + 1, n, device="cuda", dtype=torch.float64)
    v[0] = torch.randn(n, device="cuda", dtype=torch.float64, generator=torch.Generator(device="cuda").manual_seed(1))
    v[0] /= v[0].norm()
    h = torch.zeros(steps, steps, dtype=torch.float64)
    for j in range(steps):
        u = v[j] + (lap @ v[j][:, None])[:, 0]
        h[j, j] = float(v[j] @ u)
        for _ in range(2):
            u = u - v[:j + 1].T @ (v[:j + 1] @ u)
        beta = float(u.norm())
        if beta < 1e-13:
            steps = j + 1
            break
        if j + 1 < steps:
            h[j, j + 1] = h[j + 1, j] = beta
        v[j + 1] = u / beta
    _, z = torch.linalg.eigh(h[:steps, :steps])
    y = v[:steps].T @ z[:, -dims - 1:-1].flip(1).cuda()
    y = y / y.norm(dim=0)
    big = y.abs().argmax(0)
    y = y * torch.sign(y[big, torch.arange(dims, device="cuda")])
    return y * (10 / y.abs().max())


def _philox(c0, c1, c2, c3, k0, k1):
    """Philox4x32-7 on int64 tensors that hold 32-bit words."""
    mask = 0xFFFFFFFF
    for _ in range(7):
        p0, p1 = c0 * 0xD2511F53, c2 * 0xCD9E8D57   # below 2^64: the wrapped product's halves are its bits
        c0, c1, c2, c3 = (((p1 >> 32) & mask) ^ c1 ^ k0, p1 & mask, ((p0 >> 32) & mask) ^ c3 ^ k1, p0 & mask)
        k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
    return torch.stack([c0, c1, c2, c3])


def _transform(x, q, layout, case):
    """The new points' positions: the weighted mean of their neighbours', then the epochs at a quarter of the rate
    with the neighbours and the sampled reference points fixed.  Which edges fire, and how many samples each draws,
    is decided in the data's 32 bits as the schedule is defined; positions are 64 bits."""
    n, new, k = case["n"], case["new"], case["k"]
    idx, dist = _neighbours(x, q, k)
    w = _weights(dist.float().double()).float()
    y = (w.double()[:, :, None] * layout[idx]).sum(1) / w.double().sum(1, keepdim=True)
    epochs = 100 if new <= 10000 else 30
    top = w.max()
    keep = w >= top / epochs
    eps = torch.where(keep, top / w, torch.inf).float()
    step = eps / 5.0
    due, neg_due = eps.clone(), step.clone()
    head = torch.arange(n, n + new, device="cuda")
    seed = 1234567890
    k0, k1 = (seed & 0xFFFFFFFF) ^ 0x4E454731, seed >> 32

    def move(y, at, other, attract, alpha, on):
        diff = y - other
        d2 = diff.square().sum(1).clamp_min(1.1920929e-07)
        p = d2 ** B
        c = -2 * A * B * p / (d2 * (A * p + 1)) if attract else 2 * B / ((0.001 + d2) * (A * p + 1))
        return torch.where(on[:, None], y + alpha * (c[:, None] * diff).clamp(-4, 4), y)

    for e in range(epochs):
        alpha = 0.25 * (1.0 - e / epochs)
        for j in range(k):
            fire = due[:, j] <= e
            if not bool(fire.any()):
                continue
            count = torch.where(fire, ((e - neg_due[:, j]) / step[:, j]).trunc(), 0.0)
            due[:, j] = torch.where(fire, due[:, j] + eps[:, j], due[:, j])
            neg_due[:, j] = torch.where(fire, neg_due[:, j] + count * step[:, j], neg_due[:, j])
            y = move(y, head, layout[idx[:, j]], True, alpha, fire)
            most = int(count.max())
            c3 = torch.zeros_like(head)
            words = torch.cat([_philox(head, idx[:, j], torch.full_like(head, e), c3 + b, k0, k1)
                               for b in range((most + 3) // 4 + 1)])
            at = torch.zeros_like(head)
            for r in range(most):
                m = words.gather(0, at[None])[0] * n
                while bool((bad := (m & 0xFFFFFFFF) < (2 ** 32 - n) % n).any()):
                    at = torch.where(bad, at + 1, at)
                    m = words.gather(0, at[None].clamp_max(len(words) - 1))[0] * n
                at = (at + 1).clamp_max(len(words) - 1)
                y = move(y, head, layout[m >> 32], False, alpha, count > r)
    return y


def _loss_grad(graph, layout):
    ptr, col, w = (torch.as_tensor(v, device="cuda") for v in graph)
    y = torch.as_tensor(layout, device="cuda").double()
    n = len(y)
    i, j, w = torch.repeat_interleave(torch.arange(n, device="cuda"), ptr.diff()), col.long(), w.double()
    diff = y[i] - y[j]
    d2 = diff.square().sum(1)
    p = A * d2 ** B
    loss = (w * torch.log1p(p) + (1 - w) * (torch.log1p(p) - torch.log(p))).sum()
    dd2 = w * B * p / (d2 * (1 + p)) - (1 - w) * B / (d2 * (1 + p))
    grad = torch.zeros_like(y)
    grad.index_add_(0, i, 2 * dd2[:, None] * diff)
    grad.index_add_(0, j, -2 * dd2[:, None] * diff)
    share = w * p / (1 + p) - (1 - w) / (1 + p)
    return {"loss": loss, "grad": grad, "grad_ab": torch.stack([(share / A).sum(), (share * torch.log(d2)).sum()])}
