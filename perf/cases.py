"""What a user of this library has it do, as measurable cases.

A case is a dict of plain values.  `op` says which public entry point it goes through:

  minibatch  de_minibatch_noalloc: one epoch of single-minibatch calls on the
             caller's own device memory
  train      Handle: embedding in, some epochs, embedding out (FP32 or BF16 storage)
  batch      Batch: many small graphs in one launch, host embeddings in and out
  serve      Server: a burst of jobs, all submitted and then waited for
  spmm       Handle.spmm into a device tensor
  sparse     Handle.sparse_embedding on pinned host rows, in place
  csr        coo_to_csr: host COO entries to a host CSR

Graphs are symmetrised kNN graphs of Gaussian mixtures and R-MAT graphs, the two kinds
this repository's configurations, tests and benchmark use, drawn from the seed.
"""
import math

import numpy as np
import torch

import distembed_gb300 as de
from distembed_gb300 import graphgen as gg

DEV = "cuda"
LR = 0.02  # the reference driver's rate


def listed():
    return [
        # the smallest call: a caller that owns the device heap steps a small graph
        # through its minibatches, one call each
        dict(name="minibatch-knn-2k", op="minibatch", kind="knn", n=2000, dim=64, batch=256, ns=5),
        # a small job at the driver's default minibatch: one minibatch per epoch, so
        # launches and per-epoch overheads are most of it
        dict(name="train-knn-1k5", op="train", kind="knn", n=1507, deg=10, dim=32, batch=16384, ns=5, epochs=20,
             precision="fp32", loss=True),
        # the CPU-runnable workload: 20,000 points in 64-D, k = 15, 30 epochs of 79 small
        # minibatches at a decaying rate, with the loss a user watches
        dict(name="train-knn-20k", op="train", kind="knn", n=20000, deg=15, points=64, dim=128, batch=256, ns=5,
             epochs=30, decay=True, precision="fp32", loss=True),
        # a job of the served stream's middle, vertex count odd and minibatches ragged
        dict(name="train-rmat-100k", op="train", kind="rmat", n=100003, deg=16, dim=64, batch=16384, ns=5, epochs=2,
             precision="fp32", loss=False),
        # the large FP32 workload: R-MAT of 2^20 vertices, dim 128, minibatch 4096
        dict(name="train-rmat-s20", op="train", kind="rmat", n=1 << 20, deg=16, dim=128, batch=4096, ns=5, epochs=1,
             precision="fp32", loss=False),
        # BF16 storage with 1024 shared negatives: the repulsion is two GEMMs
        dict(name="train-bf16-s20", op="train", kind="rmat", n=1 << 20, deg=16, dim=256, batch=8192, ns=1024,
             epochs=1, precision="bf16", loss=False),
        # many small graphs at once, BF16 rows, the team shape the autotuner keeps for
        # such a suite; the loss of the last epoch
        dict(name="batch-bf16-64", op="batch", graphs=64, n_lo=500, n_hi=50000, dim=64, batch=256, ns=5, epochs=2,
             precision="bf16", shape="staged"),
        # few small graphs, FP32, as a first call makes it: the default team shape
        dict(name="batch-fp32-24", op="batch", graphs=24, n_lo=500, n_hi=5000, dim=32, batch=256, ns=5, epochs=3,
             precision="fp32", shape="default"),
        # a burst of served jobs of mixed sizes, dims and kinds (the R-MAT jobs, on which
        # rounding grows quickly from epoch to epoch, take two epochs)
        dict(name="serve-8", op="serve", jobs=8, n_lo=1000, n_hi=60000, batch=16384, ns=5, epochs=10),
        # the SpMM step on the large graph
        dict(name="spmm-rmat-s20", op="spmm", kind="rmat", n=1 << 20, deg=16, dim=128, batch=4096),
        # the sparse embedding: five iterations with pruning to half of each row
        dict(name="sparse-rmat-s17", op="sparse", kind="rmat", n=1 << 17, deg=16, dim=128, batch=4096, iterations=5,
             density=0.5),
        # start-up: the COO entries of a file as a reader has them, to CSR
        dict(name="csr-rmat-s18", op="csr", n=1 << 18, deg=8, mirror=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["minibatch", "train", "train", "train", "bf16", "batch", "serve", "spmm", "sparse", "csr"])
    kind = rng.choice(["knn", "rmat"])
    hi = 40000 if kind == "knn" else 300000  # exact neighbours of more points are slow to prepare
    deg = rng.randint(4, 20)
    if op == "minibatch":
        dim = rng.choice([32, 64, 128, 256])
        return dict(op=op, kind=kind, n=_log(rng, 300, 20000), dim=dim, batch=_log(rng, 64, 1024),
                    ns=_log(rng, 1, 16))
    if op == "train":
        n = _log(rng, 500, hi)
        return dict(op="train", kind=kind, n=n, deg=deg, dim=rng.choice([32, 64, 128, 256]),
                    batch=max(_log(rng, 64, 16384), n // 500), ns=_log(rng, 1, 20),
                    epochs=rng.randint(1, 4) if kind == "knn" else 1, precision="fp32", loss=rng.random() < 0.5)
    if op == "bf16":
        n = _log(rng, 2000, hi)
        return dict(op="train", kind=kind, n=n, deg=deg, dim=rng.choice([64, 128, 256]), batch=_log(rng, 512, 16384),
                    ns=_log(rng, 3, 1024), epochs=1, precision="bf16", loss=rng.random() < 0.5)
    if op == "batch":
        lo = _log(rng, 200, 2000)
        return dict(op=op, graphs=rng.randint(2, 48), n_lo=lo, n_hi=lo * rng.randint(2, 20),
                    dim=rng.choice([32, 64, 128]), batch=_log(rng, 100, 1024), ns=rng.randint(1, 16),
                    epochs=rng.randint(1, 2), precision=rng.choice(["fp32", "bf16"]),
                    shape=rng.choice(["default", "staged"]))
    if op == "serve":
        lo = _log(rng, 500, 4000)
        return dict(op=op, jobs=rng.randint(1, 8), n_lo=lo, n_hi=lo * rng.randint(2, 10),
                    batch=_log(rng, 1024, 16384), ns=rng.randint(1, 10), epochs=rng.randint(1, 10))
    if op == "spmm":
        return dict(op=op, kind=kind, n=_log(rng, 1000, hi), deg=deg, dim=rng.choice([32, 64, 128, 256]),
                    batch=_log(rng, 256, 16384))
    if op == "sparse":
        return dict(op=op, kind=kind, n=_log(rng, 1000, min(hi, 100000)), deg=deg, dim=rng.choice([32, 64, 128, 256]),
                    batch=_log(rng, 256, 8192), iterations=rng.randint(2, 5), density=rng.choice([0.25, 0.5, 0.75]))
    return dict(op="csr", n=_log(rng, 1000, 262144), deg=rng.randint(2, 8), mirror=rng.random() < 0.5)


# ------------------------------------------------------------------ inputs

def _graph(kind, n, deg, seed, points=32):
    if kind == "knn":
        return gg.knn_csr(n, points, min(deg, n - 1), 10, seed, device=DEV)[1:]
    return gg.rmat_csr_torch(n, deg, seed, DEV)[1:]


def _uniform(shape, seed, dtype=torch.float32):
    """Rows as every form starts them: uniform in [-0.5, 0.5)."""
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return torch.rand(shape, generator=g, device=DEV, dtype=torch.float32).sub_(0.5).to(dtype)


def _pinned(x):
    out = torch.empty(x.shape, dtype=x.dtype, pin_memory=True)
    out.copy_(x)
    return out


def _rates(case):
    """One rate per epoch: constant, or falling linearly to zero."""
    e = np.arange(case["epochs"])
    return LR * (1.0 - e / case["epochs"]) if case.get("decay") else np.full(case["epochs"], LR)


def _suite(count, n_lo, n_hi, seed):
    """`count` graphs, sizes log-uniform, even ones kNN and odd ones R-MAT (graph_suite's mix);
    the sizes are the suite's, whatever the seed."""
    rng = np.random.Generator(np.random.PCG64(3))
    sizes = np.rint(np.exp(rng.uniform(np.log(n_lo), np.log(n_hi), size=count))).astype(int)
    return [_graph("knn", int(n), 10, seed * 1000 + i) if i % 2 == 0 else _graph("rmat", int(n), 8, seed * 1000 + i)
            for i, n in enumerate(sizes)]


def _draws(n, seed, ns):
    """The negatives of one minibatch: ns values uniform on 0..n inclusive from the
    48271 multiplicative generator, each a rejected-and-scaled state."""
    m = 2147483647
    s = seed % m or 1
    span = m - 2  # states are 1 .. m - 1, so state - 1 is 0 .. m - 2
    scale = span // (n + 1)
    out = []
    while len(out) < ns:
        s = s * 48271 % m
        if s - 1 < (n + 1) * scale:
            out.append((s - 1) // scale)
    return out


def _job_rates(case, job):
    return np.full(case["epochs"] if job % 2 == 0 else min(case["epochs"], 2), LR)


def _minibatches(n, batch):
    return -(-n // batch)


def _inputs(case, seed):
    """Graphs and start rows of a case, the same for prepare() and exact()."""
    op = case["op"]
    if op == "minibatch":
        rp, col = _graph(case["kind"], case["n"], 10, seed)
        return rp, col, _uniform((case["n"], case["dim"]), seed)
    if op in ("train", "spmm"):
        rp, col = _graph(case["kind"], case["n"], case["deg"], seed, case.get("points", 32))
        return rp, col, _uniform((case["n"], case["dim"]), seed)
    if op == "sparse":
        rp, col = _graph(case["kind"], case["n"], case["deg"], seed)
        return rp, col, _uniform((case["n"], case["dim"]), seed, torch.float64)
    if op == "batch":
        graphs = _suite(case["graphs"], case["n_lo"], case["n_hi"], seed)
        return graphs, _uniform((sum(len(rp) - 1 for rp, _ in graphs), case["dim"]), seed)
    if op == "serve":
        graphs = _suite(case["jobs"], case["n_lo"], case["n_hi"], seed)
        return graphs, [_uniform((len(rp) - 1, (32, 64, 128)[i % 3]), seed + i) for i, (rp, _) in enumerate(graphs)]
    # a file's entries: every vertex has `deg` edges to vertices at seeded distances, the
    # vertices are relabelled, an eighth of the entries comes twice, in no order
    n, deg = case["n"], case["deg"]
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    far = 1 + torch.randperm((n - 1) // 2, generator=g, device=DEV)[:deg]
    label = torch.randperm(n, generator=g, device=DEV)
    v = torch.arange(n, device=DEV).repeat_interleave(len(far))
    r, c = label[v], label[(v + far.repeat(n)) % n]
    r, c = torch.cat([r, r[: len(r) // 8]]), torch.cat([c, c[: len(c) // 8]])
    order = torch.randperm(len(r), generator=g, device=DEV)
    return r[order].cpu().numpy(), c[order].cpu().numpy()


# ------------------------------------------------------------------ the calls

def prepare(case, seed):
    op = case["op"]
    s = dict(case=case)
    if op == "minibatch":
        rp, col, x = _inputs(case, seed)
        b = _minibatches(case["n"], case["batch"])
        s.update(x=x, rp=torch.from_numpy(rp).to(DEV, torch.int32), col=torch.from_numpy(col).to(DEV, torch.int32),
                 negs=torch.tensor([_draws(case["n"], j, case["ns"]) for j in range(b)], dtype=torch.int32, device=DEV))
    elif op == "train":
        rp, col, x = _inputs(case, seed)
        s.update(x0=x, out=torch.empty_like(x), lr=_rates(case),
                 h=de.Handle(rp, col, case["dim"], precision=case["precision"], compute_loss=case["loss"]))
    elif op == "batch":
        graphs, x = _inputs(case, seed)
        b = de.Batch(graphs, case["dim"], precision=case["precision"])
        if case["shape"] == "staged":
            b.set_shape("staged", team_warps=16 if case["dim"] <= 64 else 8, edge_cap=16, pairs=2, stages=3, team_ctas=2)
        b.set_loss("last")
        x = _pinned(x)
        s.update(b=b, x0=x.numpy(), out=torch.empty(x.shape, pin_memory=True).numpy())
    elif op == "serve":
        graphs, xs = _inputs(case, seed)
        s.update(srv=de.Server(slots=16, hbm_bytes=2 << 30), graphs=graphs,
                 lr=[_job_rates(case, i) for i in range(case["jobs"])], x0=[_pinned(x).numpy() for x in xs],
                 out=[torch.empty(x.shape, pin_memory=True).numpy() for x in xs])
    elif op == "spmm":
        rp, col, x = _inputs(case, seed)
        h = de.Handle(rp, col, case["dim"])
        h.set_embeddings(x)
        s.update(h=h, out=torch.empty_like(x))
    elif op == "sparse":
        rp, col, x = _inputs(case, seed)
        s.update(h=de.Handle(rp, col, case["dim"]), x=_pinned(x).numpy(),
                 coll=torch.empty((case["batch"], case["dim"]), dtype=torch.float64, pin_memory=True).numpy())
    else:
        s["r"], s["c"] = _inputs(case, seed)
    return s


def _logged(loss):
    """The loss as a log keeps it: a sum of FP32 terms, read as FP32."""
    return np.asarray(loss).astype(np.float32)


def run(s):
    c = s["case"]
    op = c["op"]
    if op == "minibatch":
        call, n, stream = de.lib().de_minibatch_noalloc, c["n"], torch.cuda.current_stream().cuda_stream
        for j in range(_minibatches(n, c["batch"])):
            rc = call(n, s["rp"].data_ptr(), s["col"].data_ptr(), c["dim"], s["x"].data_ptr(), j, c["batch"],
                      s["negs"].data_ptr() + 4 * j * c["ns"], c["ns"], c["batch"], 1, LR, 5.0, None, stream)
            if rc:
                raise RuntimeError(f"de_minibatch_noalloc: {rc}")
        return s["x"]
    if op == "train":
        s["h"].set_embeddings(s["x0"])
        loss = s["h"].run(c["epochs"], c["batch"], c["ns"], s["lr"], want_loss=c["loss"])
        s["h"].get_embeddings(out=s["out"])
        return {"x": s["out"], "loss": _logged(loss)} if c["loss"] else s["out"]
    if op == "batch":
        s["b"].set_embeddings(-1, s["x0"])
        loss = s["b"].run(c["epochs"], c["batch"], c["ns"], LR)
        return {"x": s["b"].get_embeddings(-1, out=s["out"]), "loss": _logged(loss)}
    if op == "serve":
        ids = [s["srv"].submit(rp, col, x0, len(lr), c["batch"], c["ns"], lr, out=out)
               for (rp, col), x0, out, lr in zip(s["graphs"], s["x0"], s["out"], s["lr"])]
        done = [s["srv"].wait(i) for i in ids]
        return {"x": [d[0] for d in done], "loss": [_logged(d[1]) for d in done]}
    if op == "spmm":
        return s["h"].spmm(c["batch"], LR, out=s["out"])
    if op == "sparse":
        return s["h"].sparse_embedding(s["x"], c["iterations"], c["batch"], 5, LR, c["density"], inplace=True,
                                       coll=s["coll"])
    rows, cols, rp, col = de.coo_to_csr(c["n"], c["n"], s["r"], s["c"], mirror=c["mirror"])
    return {"rowptr": rp, "col": col}


# ------------------------------------------------------------------ work

def _entries(kind, n, deg):
    """CSR entries of a symmetrised graph, about: 1.4 k per vertex, or 1.9 ef per vertex."""
    return n * deg * (1.4 if kind == "knn" else 1.9)


def _train_work(kind, n, deg, dim, ns, epochs):
    """Each epoch reads the CSR and reads and writes every row; a pair costs about 7 dim operations."""
    nnz = _entries(kind, n, deg)
    return {"bytes": epochs * (4 * nnz + 4 * n + 8 * n * dim), "flops": epochs * 7.0 * dim * (nnz + n * ns)}


def work(case):
    op = case["op"]
    if op == "minibatch":
        return _train_work(case["kind"], case["n"], 10, case["dim"], case["ns"], 1)
    if op == "train":
        return _train_work(case["kind"], case["n"], case["deg"], case["dim"], case["ns"], case["epochs"])
    if op in ("batch", "serve"):
        count = case["graphs"] if op == "batch" else case["jobs"]
        lo, hi = case["n_lo"], case["n_hi"]
        n = count * (hi - lo) / math.log(hi / lo)  # the mean of a log-uniform size
        w = _train_work("knn", n, 11, case.get("dim", 75), case["ns"], case["epochs"])
        return {"bytes": w["bytes"] + 8 * n * case.get("dim", 75), "flops": w["flops"]}
    n = case["n"]
    if op == "spmm":
        nnz = _entries(case["kind"], n, case["deg"])
        return {"bytes": 4 * nnz + 4 * n + 8 * n * case["dim"], "flops": 2.0 * nnz * case["dim"]}
    if op == "sparse":
        nnz, it = _entries(case["kind"], n, case["deg"]), case["iterations"]
        return {"bytes": it * (4 * nnz + 4 * n * case["dim"]) + 16 * n * case["dim"],
                "flops": 7.0 * nnz * case["dim"] * it}
    m = n * case["deg"]
    return {"bytes": 18 * m + 8 * (m * (2 if case["mirror"] else 1) + n), "flops": 0}


# ------------------------------------------------------------------ 64-bit values

def _pair_rows(upd, loss, xi, xj, attract, lr):
    """Adds lr * clip(c (xi - xj)) over the last-but-one axis' pairs; returns update and loss."""
    d = xi - xj
    r = d.square().sum(-1)
    c = -2.0 / (1.0 + r) if attract else 2.0 / ((r + 1e-6) * (1.0 + r))
    d.mul_(c.unsqueeze(-1)).clamp_(-5.0, 5.0).mul_(lr)
    loss += float((torch.log1p(r) if attract else torch.log((1.0 + r) / (r + 1e-6))).sum())
    return d, loss


def _attract(x, rp, rows, col, lo, hi, skip, lr):
    """Attractive update and loss of rows [lo, hi)."""
    upd = torch.zeros((hi - lo, x.shape[1]), dtype=torch.float64, device=DEV)
    loss, step = 0.0, max(1, (1 << 27) // x.shape[1])
    for e in range(int(rp[lo]), int(rp[hi]), step):
        f = min(int(rp[hi]), e + step)
        src, dst = rows[e:f], col[e:f]
        if skip >= 0:
            src, dst = src[dst != skip], dst[dst != skip]
        d, loss = _pair_rows(upd, loss, x[src], x[dst], True, lr)
        upd.index_add_(0, src - lo, d)
    return upd, loss


def _repulse(x, lo, hi, draws, lr):
    keep = [k for k in draws if k < x.shape[0]]
    upd, loss = torch.zeros((hi - lo, x.shape[1]), dtype=torch.float64, device=DEV), 0.0
    if keep:
        neg = x[torch.tensor(keep, device=DEV)]
        step = max(1, (1 << 27) // (len(keep) * x.shape[1]))
        for a in range(lo, hi, step):
            b = min(hi, a + step)
            d, loss = _pair_rows(upd, loss, x[a:b].unsqueeze(1), neg.unsqueeze(0), False, lr)
            upd[a - lo:b - lo] = d.sum(1)
    return upd, loss


def _train64(rp, col, x, batch, ns, rates):
    """Minibatch SGD in 64 bits, with the one-rank behaviour the handles keep: edges into
    the last vertex are dropped, and from the second epoch on the repulsion covers as many
    rows as the last minibatch has."""
    n, x = x.shape[0], x.double()
    cols = torch.from_numpy(col).to(DEV)
    rows = torch.repeat_interleave(torch.arange(n, device=DEV), torch.from_numpy(np.diff(rp)).to(DEV))
    mb, losses = _minibatches(n, batch), []
    last = n - batch * (mb - 1)
    for e, lr in enumerate(float(np.float32(v)) for v in rates):
        losses.append(0.0)
        for j in range(mb):
            lo, hi = j * batch, min(n, (j + 1) * batch)
            upd, la = _attract(x, rp, rows, cols, lo, hi, n - 1, lr)
            top = lo + min(hi - lo, last if e else batch)
            rep, lb = _repulse(x, lo, top, _draws(n, e + j, ns), lr)
            upd[: top - lo] += rep
            x[lo:hi] += upd
            losses[-1] += la + lb
    return x, np.array(losses)


def exact(case, seed):
    op = case["op"]
    if op == "minibatch":
        rp, col, x = _inputs(case, seed)
        return _train64(rp, col, x, case["batch"], case["ns"], [LR])[0]
    if op == "train":
        rp, col, x = _inputs(case, seed)
        y, loss = _train64(rp, col, x, case["batch"], case["ns"], _rates(case))
        return {"x": y, "loss": loss} if case["loss"] else y
    if op == "batch":
        graphs, x = _inputs(case, seed)
        parts, losses, at = [], np.zeros((len(graphs), case["epochs"])), 0
        for g, (rp, col) in enumerate(graphs):
            y, loss = _train64(rp, col, x[at:at + len(rp) - 1], case["batch"], case["ns"], _rates(case))
            parts.append(y)
            losses[g, -1] = loss[-1]  # the others report 0
            at += len(rp) - 1
        return {"x": torch.cat(parts), "loss": losses}
    if op == "serve":
        graphs, xs = _inputs(case, seed)
        got = [_train64(rp, col, x, case["batch"], case["ns"], _job_rates(case, i))
               for i, ((rp, col), x) in enumerate(zip(graphs, xs))]
        return {"x": [y for y, _ in got], "loss": [loss for _, loss in got]}
    if op == "spmm":
        rp, col, x = _inputs(case, seed)
        n, x, cols = case["n"], x.double(), torch.from_numpy(col).to(DEV)
        rows = torch.repeat_interleave(torch.arange(n, device=DEV), torch.from_numpy(np.diff(rp)).to(DEV))
        y, step = torch.zeros_like(x), (1 << 27) // case["dim"]
        for e in range(0, len(col), step):
            src, dst = rows[e:e + step], cols[e:e + step]
            y.index_add_(0, src[dst != n - 1], x[dst[dst != n - 1]])
        return y.mul_(float(np.float32(LR)))
    if op == "sparse":
        rp, col, x = _inputs(case, seed)
        n, dim, batch, keep = case["n"], case["dim"], case["batch"], int(case["dim"] * case["density"])
        cols = torch.from_numpy(col).to(DEV)
        rows = torch.repeat_interleave(torch.arange(n, device=DEV), torch.from_numpy(np.diff(rp)).to(DEV))
        coll = torch.zeros((batch, dim), dtype=torch.float64, device=DEV)
        slot = torch.arange(n, device=DEV) % batch
        for i in range(case["iterations"]):
            coll.index_add_(0, slot, _attract(x, rp, rows, cols, 0, n, -1, float(np.float32(LR)))[0])
            if i == 0 and case["iterations"] > 1 and dim > keep:
                low = torch.argsort(x, dim=1, stable=True)[:, : dim - keep]
                x.scatter_(1, low, 0.0)
        return x, coll
    r, c = (torch.from_numpy(a).to(DEV) for a in _inputs(case, seed))
    n = case["n"]
    key = r * n + c
    if case["mirror"]:
        key = torch.cat([key, (c * n + r)[r != c]])
    key = torch.unique(key)
    rowptr = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    rowptr[1:] = torch.cumsum(torch.bincount(key // n, minlength=n), 0)
    return {"rowptr": rowptr, "col": key % n}
