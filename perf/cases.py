"""Performance cases of the engine: what a program that uses it has it do.

``listed()`` names the cases, ``draw(rng)`` gives further ones of the same
ranges, ``prepare(case, seed)`` makes the inputs and the handle a user's
program holds before the call, ``run(state)`` is one pass through the public
entry points, ``work(case)`` the bytes and operations that pass cannot do
without, and ``exact(case, seed)`` the value in 64 bits where the outputs have
one (the distances of an exact kNN).

The layout of a graph with more than 16,384 embedding floats is a Hogwild
optimisation whose positions differ from run to run, so the cases of large
inputs ask for the spectral embedding (``n_epochs=0``: kNN, fuzzy graph and
initialisation), which is reproducible; the layout itself is covered by the
fits of small inputs, which run it deterministically, and by the transforms.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from umapers_b200 import Umap, _lib
from umapers_b200._umapers import UmapCore

DEVICE = "cuda" if torch.cuda.is_available() else "cpu"


# ------------------------------------------------------------------ cases --
def listed() -> list[dict]:
    return [
        # The quick start of the documentation: a thousand rows of noise, the
        # latency of one small fit.
        dict(name="fit 1000x32", kind="fit", n=1000, d=32, k=15, epochs=200, comps=0,
             metric="euclidean", nc=2, labels=False),
        # A laboratory table with the estimator's default parameters (500
        # epochs, exact neighbours at this size); rows are no multiple of a tile.
        dict(name="fit 4200x96 defaults", kind="fit", n=4200, d=96, k=15, epochs=-1, comps=6,
             metric="euclidean", nc=2, labels=False),
        # The precision workload: wide rows on the tensor-core kNN, host buffers.
        dict(name="spectral 20000x192", kind="spectral", n=20000, d=192, k=15, comps=10,
             metric="euclidean", nc=2, approx=False, device=False),
        # The large fit, rows resident in device memory.
        dict(name="spectral 1000000x64", kind="spectral", n=1_000_000, d=64, k=15, comps=50,
             metric="euclidean", nc=2, approx=False, device=True),
        # A large table with the default neighbour search (NN-descent above
        # 16,384 rows), odd sizes, from host memory.
        dict(name="spectral 100003x100 nn-descent", kind="spectral", n=100_003, d=100, k=15,
             comps=20, metric="euclidean", nc=2, approx=True, device=False),
        # Bags of words: sparse rows under the cosine metric.
        dict(name="sparse 100000x2000 cosine", kind="sparse", n=100_000, d=2000, nnz=20, k=30,
             metric="cosine", nc=2),
        # Serving: one new row at a time.
        dict(name="transform 1 row", kind="transform", n=4000, d=32, k=15, comps=8, nq=1,
             device=False),
        # A batch of new rows, resident on the device.
        dict(name="transform 1000000x128", kind="transform", n=8000, d=128, k=15, comps=20,
             nq=1_000_000, device=True),
        # The same batch through the learned surrogate with its gate.
        dict(name="surrogate 1000000x128", kind="surrogate", n=8000, d=128, k=15, comps=20,
             nq=1_000_000, device=True),
        # Neighbours of new rows among stored rows, from host memory.
        dict(name="knn 50000 of 200000x128", kind="knn", n=200_000, d=128, k=15, comps=20,
             nq=50_000, metric="euclidean"),
        # Neighbours within embedding vectors under the cosine metric, a longer
        # list, ragged sizes.
        dict(name="knn 60013x100 cosine k30", kind="knn", n=60_013, d=100, k=30, comps=20, nq=0,
             metric="cosine"),
        # Embedded points mapped back to the data space.
        dict(name="inverse 2000", kind="inverse", n=4000, d=24, k=15, comps=8, nq=2000),
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng) -> dict:
    kind = rng.choice(["fit", "fit", "spectral", "spectral", "sparse", "transform", "transform",
                       "surrogate", "knn", "knn", "inverse"])
    if kind == "fit":
        epochs = rng.choice([200, -1])
        nc = rng.choice([2, 2, 2, 3])
        return dict(kind=kind, n=_log_int(rng, 200, 4200 if epochs < 0 else 5400),
                    d=_log_int(rng, 12, 200), k=rng.choice([10, 15, 15, 30]), epochs=epochs,
                    comps=rng.choice([0, 3, 8]), metric=rng.choice(["euclidean", "cosine"]), nc=nc,
                    labels=rng.random() < 0.25)
    if kind == "spectral":
        n = _log_int(rng, 5000, 1_000_000)
        return dict(kind=kind, n=n, d=_log_int(rng, 16, 64 if n > 200_000 else 256),
                    k=rng.choice([10, 15, 15, 30 if n < 300_000 else 15]),
                    comps=rng.choice([1, 10, 50]),
                    metric=rng.choice(["euclidean", "euclidean", "cosine"]),
                    nc=rng.choice([2, 2, 3]), approx=rng.random() < 0.4 and n < 400_000,
                    device=rng.random() < 0.5)
    if kind == "sparse":
        return dict(kind=kind, n=_log_int(rng, 3000, 100_000), d=_log_int(rng, 1000, 8000),
                    nnz=rng.randint(8, 24), k=rng.choice([10, 15, 30]),
                    metric=rng.choice(["cosine", "euclidean"]), nc=2)
    if kind in ("transform", "surrogate"):
        return dict(kind=kind, n=_log_int(rng, 1000 if kind == "transform" else 3000, 8000),
                    d=_log_int(rng, 16, 128), k=rng.choice([10, 15]), comps=rng.choice([8, 20]),
                    nq=_log_int(rng, 1, 1_000_000), device=rng.random() < 0.5)
    if kind == "knn":
        query = rng.random() < 0.5
        n = _log_int(rng, 500, 200_000)
        return dict(kind=kind, n=n, d=_log_int(rng, 8, 128 if n > 60_000 else 300),
                    k=rng.choice([5, 15, 30]), comps=rng.choice([1, 20]),
                    nq=_log_int(rng, 1, 50_000) if query else 0,
                    metric=rng.choice(["euclidean", "cosine"]))
    return dict(kind=kind, n=_log_int(rng, 500, 4000), d=_log_int(rng, 12, 96),
                k=rng.choice([10, 15]), comps=8, nq=_log_int(rng, 1, 2000))


# ----------------------------------------------------------------- inputs --
def _gen(seed: int) -> torch.Generator:
    return torch.Generator(device=DEVICE).manual_seed(seed)


def _rows(n: int, d: int, comps: int, seed: int, draw_seed: int | None = None) -> torch.Tensor:
    """n x d rows on the device: N(0, 1) for comps = 0, else an equal-weight
    mixture of axis-aligned Gaussians (means ~ N(0, 4^2), per-dimension standard
    deviations ~ U(0.5, 1.5)).  ``seed`` fixes the mixture, ``draw_seed`` the rows."""
    g = _gen(seed)
    if comps == 0:
        return torch.randn(n, d, generator=g, device=DEVICE)
    means = 4.0 * torch.randn(comps, d, generator=g, device=DEVICE)
    stds = 0.5 + torch.rand(comps, d, generator=g, device=DEVICE)
    if draw_seed is not None:
        g = _gen(draw_seed)
    lab = torch.randint(0, comps, (n,), generator=g, device=DEVICE)
    x = torch.randn(n, d, generator=g, device=DEVICE)
    return x.mul_(stds[lab]).add_(means[lab])


def _host(x: torch.Tensor) -> np.ndarray:
    return np.ascontiguousarray(x.cpu().numpy())


def _csr(n: int, d: int, nnz: int, seed: int):
    """CSR arrays: `nnz` uniform columns a row (repeats merged), LogNormal(0, 1) values."""
    g = _gen(seed)
    cols = torch.randint(0, d, (n, nnz), generator=g, device=DEVICE).sort(dim=1).values
    keep = torch.ones_like(cols, dtype=torch.bool)
    keep[:, 1:] = cols[:, 1:] != cols[:, :-1]
    vals = torch.randn(n, nnz, generator=g, device=DEVICE).exp_()
    indptr = torch.zeros(n + 1, dtype=torch.int64, device=DEVICE)
    indptr[1:] = keep.sum(dim=1).cumsum(0)
    return _host(indptr), _host(cols[keep]), _host(vals[keep])


def prepare(case: dict, seed: int) -> dict:
    kind, n, d, k = case["kind"], case["n"], case["d"], case["k"]
    st: dict = {"kind": kind, "case": case}
    if kind == "fit":
        x = _rows(n, d, case["comps"], seed)
        st["x"] = _host(x)
        st["y"] = (np.random.default_rng(seed).integers(-1, 4, n).astype(np.int64)
                   if case["labels"] else None)
        st["model"] = Umap(n_neighbors=k, n_components=case["nc"], metric=case["metric"],
                           n_epochs=None if case["epochs"] < 0 else case["epochs"],
                           target_metric="categorical" if case["labels"] else None)
    elif kind == "spectral":
        x = _rows(n, d, case["comps"], seed)
        kw = dict(n_neighbors=k, n_components=case["nc"], metric=case["metric"], n_epochs=0)
        if case["device"]:
            st["x"] = x.contiguous()
            st["core"] = UmapCore(use_approximate_knn=case["approx"], **kw)
            st["out"] = torch.empty(n, case["nc"], device=DEVICE)
        else:
            st["x"] = _host(x)
            st["model"] = Umap(use_approximate_knn=case["approx"], **kw)
    elif kind == "sparse":
        st["csr"] = _csr(n, d, case["nnz"], seed)
        st["core"] = UmapCore(n_neighbors=k, n_components=case["nc"], metric=case["metric"],
                              n_epochs=0)
    elif kind in ("transform", "surrogate"):
        core = UmapCore(n_neighbors=k)
        core.fit(_host(_rows(n, d, case["comps"], seed)))
        if kind == "surrogate":
            core.fit_surrogate(batch_size=1024, epochs=100)
        q = _rows(case["nq"], d, case["comps"], seed, seed + 1_000_003)
        st["core"] = core
        if case["device"]:
            st["q"] = q.contiguous()
            st["out"] = torch.empty(case["nq"], 2, device=DEVICE)
            st["flags"] = torch.empty(case["nq"], dtype=torch.uint8, device=DEVICE)
        else:
            st["q"] = _host(q)
    elif kind == "knn":
        nq = case["nq"]
        st["r"] = _host(_rows(n, d, case["comps"], seed))
        st["q"] = _host(_rows(nq, d, case["comps"], seed, seed + 1_000_003)) if nq else None
        rows = nq or n
        st["idx"] = np.empty((rows, k), np.int64)
        st["dist"] = np.empty((rows, k), np.float32)
    elif kind == "inverse":
        core = UmapCore(n_neighbors=k)
        core.fit(_host(_rows(n, d, case["comps"], seed)))
        rng = np.random.default_rng(seed)
        emb = core.embedding
        z = emb[rng.integers(0, n, case["nq"])]
        st["q"] = np.ascontiguousarray(z + rng.normal(0.0, 0.05, z.shape), np.float32)
        st["core"] = core
    return st


# ------------------------------------------------------------------- pass --
def run(st: dict):
    kind, case = st["kind"], st["case"]
    lib = _lib.load()
    if kind == "fit":
        return st["model"].fit_transform(st["x"], st["y"])
    if kind == "spectral":
        if "model" in st:
            return st["model"].fit_transform(st["x"])
        x, out = st["x"], st["out"]
        _lib.check(lib.umapb_fit_transform_device(st["core"]._handle, x.data_ptr(), x.shape[0],
                                                  x.shape[1], out.data_ptr(), None, None))
        return out
    if kind == "sparse":
        indptr, indices, values = st["csr"]
        return st["core"].fit_transform_sparse_csr(indptr, indices, values, case["d"])
    if kind == "transform":
        if not case["device"]:
            return st["core"].transform(st["q"])
        q, out = st["q"], st["out"]
        _lib.check(lib.umapb_transform_device(st["core"]._handle, q.data_ptr(), q.shape[0],
                                              q.shape[1], out.data_ptr()))
        return out
    if kind == "surrogate":
        if not case["device"]:
            return st["core"].transform_surrogate(st["q"])
        q, out, flags = st["q"], st["out"], st["flags"]
        _lib.check(lib.umapb_surrogate_transform_device(
            st["core"]._handle, q.data_ptr(), q.shape[0], q.shape[1], 1, out.data_ptr(),
            flags.data_ptr(), None))
        return out, flags
    if kind == "knn":
        r, q, idx, dist = st["r"], st["q"], st["idx"], st["dist"]
        metric = _lib.METRICS[case["metric"]]
        if q is None:
            _lib.check(lib.umapb_knn_exact(r.ctypes.data, r.shape[0], r.shape[1], case["k"],
                                           metric, 0, idx.ctypes.data, dist.ctypes.data, None))
        else:
            _lib.check(lib.umapb_knn_query(q.ctypes.data, q.shape[0], r.ctypes.data, r.shape[0],
                                           r.shape[1], case["k"], metric, 0, idx.ctypes.data,
                                           dist.ctypes.data))
        return idx, dist
    return st["core"].inverse_transform(st["q"])


# ------------------------------------------------------------------- work --
def work(case: dict) -> dict:
    kind, n, d, k = case["kind"], float(case["n"]), float(case["d"]), float(case["k"])
    nc = float(case.get("nc", 2))
    nq = float(case.get("nq", 0))
    edges = 1.6 * n * k  # the symmetric graph's directed edges
    sample = 6 * (20.0 + 6.0 * nc)  # one attractive and five negative updates
    if kind == "fit":
        epochs = case["epochs"] if case["epochs"] >= 0 else 500
        return {"bytes": 4 * n * (d + nc),
                "flops": 2 * n * n * d + 257 * 2 * edges * 6 * (nc + 1)
                + 0.35 * edges * epochs * sample}
    if kind == "spectral":
        knn = 14 * 50 * 3 * n * d if case["approx"] else 2 * n * n * d
        return {"bytes": 4 * n * (d + nc), "flops": knn + 257 * 2 * edges * 6 * (nc + 1)}
    if kind == "sparse":
        nnz = float(case["nnz"])
        return {"bytes": 12 * n * nnz + 4 * n * nc,
                "flops": 2 * n * n * nnz * nnz / d + 257 * 2 * edges * 6 * (nc + 1)}
    if kind == "transform":
        epochs = 100 if nq <= 10000 else 30
        return {"bytes": 4 * (nq * d + n * d + 2 * nq),
                "flops": 2 * nq * n * d + 0.5 * nq * k * epochs * sample}
    if kind == "surrogate":
        pad = 128 * math.ceil(d / 128)
        return {"bytes": 4 * nq * d + 9 * nq,
                "flops": 2 * nq * (pad * 512 + 512 * 512 + 2 * 512 + 256 * pad)}
    if kind == "knn":
        rows = nq or n
        return {"bytes": 4 * d * (n + nq) + 12 * rows * k, "flops": 2 * rows * n * d}
    return {"bytes": 4 * (2 * nq + nq * d + n * (d + 2)),
            "flops": 2 * nq * n * 2 + 0.5 * nq * k * 100 * 6 * (5 * d + 20)}


# ------------------------------------------------------------------ exact --
def exact(case: dict, seed: int):
    """The sorted distances of the k nearest rows in 64 bits, for the exact
    kNN; the other paths draw random numbers and have no such value."""
    if case["kind"] != "knn":
        return None
    n, d, k, nq = case["n"], case["d"], case["k"], case["nq"]
    cosine = case["metric"] == "cosine"
    r = _rows(n, d, case["comps"], seed).double()
    q = _rows(nq, d, case["comps"], seed, seed + 1_000_003).double() if nq else r
    if cosine:
        q = q / q.norm(dim=1, keepdim=True)
        r = r / r.norm(dim=1, keepdim=True)
    r2 = (r * r).sum(1)
    dist = torch.empty(q.shape[0], k, dtype=torch.float64, device=q.device)
    step = max(1, (1 << 27) // n)
    for s in range(0, q.shape[0], step):
        b = q[s:s + step]
        near = torch.addmm(r2, b, r.T, alpha=-2.0).topk(k, dim=1, largest=False).indices
        if cosine:
            val = 1.0 - (b[:, None, :] * r[near]).sum(2)
        else:
            val = (b[:, None, :] - r[near]).square().sum(2).sqrt()
        dist[s:s + step] = val.sort(dim=1).values
    return [None, dist]
