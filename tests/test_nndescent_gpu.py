"""NN-descent on the GPU: recall against exact kNN (the reference's
thresholds, rust_umap/src/lib.rs:6733-6764) and against the oracle's own
recall on the same data."""
import ctypes

import numpy as np
import pytest

from umapers_b200 import _lib, workloads
from tests import gpu_util as gu

pytestmark = pytest.mark.gpu


def recall(exact, approx):
    hits = sum(len(set(exact[i, 1:]) & set(approx[i, 1:])) for i in range(exact.shape[0]))
    return hits / (exact.shape[0] * (exact.shape[1] - 1))


def test_recall_reference_threshold_euclidean(orc):
    x = workloads.reference_synthetic(240, 8)
    ex, _ = orc.exact_knn(x, 12)
    ap, ad, ran = gu.nndescent(x, 12, 30, 8, 0x123456789ABCDEF0)
    assert recall(ex, ap) >= 0.70
    assert ran >= 1 and np.all(np.diff(ad, axis=1) >= 0)
    assert np.all(ap[:, 0] == np.arange(240))


def test_recall_reference_threshold_cosine(orc):
    x = workloads.reference_synthetic(220, 9)
    ex, _ = orc.exact_knn(x, 10, metric="cosine")
    ap, _, _ = gu.nndescent(x, 10, 28, 8, 0xCAFEBABEDEADC0DE, metric="cosine")
    assert recall(ex, ap) >= 0.65


def test_recall_tracks_oracle_on_mixture(orc):
    x = workloads.anisotropic_mixture(20_000, 64, 20, seed=11)
    rows = np.random.default_rng(0).choice(20_000, 500, replace=False)
    exr, _ = orc.exact_knn_rows(x, rows, 15)
    ap, ad, _ = gu.nndescent(x, 15, 30, 10, 99)
    oa, _, _ = orc.nndescent(x, 15, 30, 10, 99)
    r_gpu = recall(exr, ap[rows])
    r_orc = recall(exr, oa[rows])
    print("recall gpu", r_gpu, "oracle", r_orc)
    assert r_gpu >= r_orc - 0.02
    # distances are exact FP32 distances of the returned pairs
    d_chk = np.sqrt(((x[rows, None, :] - x[ap[rows]]) ** 2).sum(-1))
    np.testing.assert_allclose(ad[rows], d_chk, rtol=1e-5, atol=1e-5)


M64 = (1 << 64) - 1


def _mix64(z):
    z = (z + 0x9E3779B97F4A7C15) & M64
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & M64
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & M64
    return z ^ (z >> 31)


def _below(seed, a, b, n):
    return ((_mix64(_mix64(seed ^ _mix64(a)) ^ b) >> 32) * n) >> 32


def replay(full, k, candidates, iters, seed):
    """The candidate rule step by step on a matrix of exact distances."""
    n = full.shape[0]
    ck = max(candidates, k)
    pool, maxc = min(ck, n - 1), 4 * ck + 1
    expl = min(max(k // 2, 4), maxc)

    def best(i, cand):
        return sorted((full[i, j], j) for j in cand)[:k]

    lists = []
    for i in range(n):
        cand, ctr = [i], 0
        while len(cand) < pool + 1:
            j = _below(seed, i, ctr, n)
            ctr += 1
            if j not in cand:
                cand.append(j)
        lists.append(best(i, cand))
    for it in range(1, iters + 1):
        new = []
        for i in range(n):
            nb = [j for _, j in lists[i]]
            c = set(nb) | {j for q in nb for _, j in lists[q]} | {i}
            c |= {_below(seed, i, (it << 40) + e, n) for e in range(expl)}
            c = sorted(c)
            if len(c) > maxc:
                for s in range(maxc):
                    r = s + _below(seed, i, (it << 40) + (1 << 20) + s, len(c) - s)
                    c[s], c[r] = c[r], c[s]
                c = c[:maxc]
            new.append(best(i, c))
        done = new == lists
        lists = new
        if done:
            break
    return lists


@pytest.mark.parametrize("n,d,k,candidates,iters", [
    (40, 6, 2, 4, 3), (90, 8, 3, 3, 3), (150, 63, 5, 5, 2), (200, 64, 10, 12, 2),
    (300, 100, 15, 15, 2), (300, 101, 15, 50, 2), (260, 72, 22, 22, 2), (300, 20, 31, 31, 2),
    (300, 66, 31, 40, 2)])
def test_nndescent_follows_the_rule_step_by_step(orc, n, d, k, candidates, iters):
    # every register width of the sort, the random cut (pools below the lists'
    # reach), and row lengths with and without whole 16-byte quads
    x = np.random.default_rng(d).normal(size=(n, d)).astype(np.float32)
    idx, dist = orc.exact_knn(x, n)
    full = np.empty((n, n), np.float32)
    np.put_along_axis(full, idx.astype(np.int64), dist, axis=1)
    gi, gd, _ = gu.nndescent(x, k, candidates, iters, 99)
    ref = replay(full, k, candidates, iters, 99)
    assert np.array_equal(gi, [[j for _, j in r] for r in ref])
    assert np.array_equal(gd, np.array([[v for v, _ in r] for r in ref], np.float32))


# row lengths and list widths (256, 512 and 1,024 candidates) on both sides of
# where whole 16-byte quads stop being read two lanes a candidate
@pytest.mark.parametrize("d,k", [(800, 15), (804, 15), (480, 20), (484, 20), (804, 31)])
def test_long_rows_follow_the_rule_step_by_step(orc, d, k):
    test_nndescent_follows_the_rule_step_by_step(orc, 300, d, k, k, 2)


def _against_the_rule(got, full, k, candidates, iters, seed):
    gi, gd = got
    ref = replay(full, k, candidates, iters, seed)
    assert np.array_equal(gi, [[j for _, j in r] for r in ref])
    assert np.array_equal(gd, np.array([[v for v, _ in r] for r in ref], np.float32))


@pytest.mark.parametrize("n,d,k,candidates,iters", [
    (40, 6, 2, 4, 3), (150, 63, 5, 5, 2), (200, 64, 10, 12, 2), (300, 60, 15, 15, 2),
    (300, 101, 15, 50, 2), (260, 72, 22, 22, 2), (300, 66, 31, 40, 2), (300, 804, 15, 15, 2)])
def test_cosine_rows_follow_the_rule_step_by_step(orc, n, d, k, candidates, iters):
    # the forms of four rows and of sixteen, narrow and wide rows, with and
    # without a tail; a zero row and a repeated one
    x = np.random.default_rng(d).normal(size=(n, d)).astype(np.float32)
    x[5], x[7] = 0.0, 2.0 * x[6]
    idx, dist = orc.exact_knn(x, n, metric="cosine")
    full = np.empty((n, n), np.float32)
    np.put_along_axis(full, idx.astype(np.int64), dist, axis=1)
    got = gu.nndescent(x, k, candidates, iters, 99, metric="cosine")[:2]
    _against_the_rule(got, full, k, candidates, iters, 99)


@pytest.mark.parametrize("metric", ["euclidean", "cosine"])
@pytest.mark.parametrize("n,nnz,k,candidates", [(40, 3, 2, 4), (150, 4, 5, 5), (200, 13, 10, 12),
                                                (300, 21, 15, 50), (260, 30, 22, 22),
                                                (300, 7, 31, 31), (300, 33, 31, 40)])
def test_csr_rows_follow_the_rule_step_by_step(n, nnz, k, candidates, metric):
    # every register width on CSR rows; the longest row is and is not a
    # multiple of four, some rows are empty
    rng, d, iters, seed = np.random.default_rng(n + nnz), 3 * nnz, 2, 99
    counts = rng.integers(0, nnz + 1, n)
    counts[3], counts[11] = nnz, 0
    ip = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    ix = np.concatenate([np.sort(rng.choice(d, c, replace=False)) for c in counts]).astype(np.int64)
    dv = rng.lognormal(0.0, 1.0, len(ix)).astype(np.float32)
    lib, m = _lib.load(), gu.METRIC[metric]
    # all distances from the exact sparse kNN, 20 reference rows at a time
    full = np.empty((n, n), np.float32)
    for r0 in range(0, n, 20):
        c = min(20, n - r0)
        rp = ip[r0:r0 + c + 1] - ip[r0]
        rx, rv = ix[ip[r0]:ip[r0 + c]], dv[ip[r0]:ip[r0 + c]]
        i, v = np.empty((n, c), np.int64), np.empty((n, c), np.float32)
        _lib.check(lib.umapb_knn_csr_query(gu._p(ip), gu._p(ix), gu._p(dv), n, gu._p(rp),
                                           gu._p(rx), gu._p(rv), c, d, c, m, gu._p(i), gu._p(v)))
        np.put_along_axis(full, r0 + i, v, axis=1)
    np.fill_diagonal(full, 0.0)
    gi, gd = np.empty((n, k), np.int64), np.empty((n, k), np.float32)
    ran, ev, sec = ctypes.c_int64(), ctypes.c_int64(), ctypes.c_double()
    _lib.check(lib.umapb_nndescent_csr(gu._p(ip), gu._p(ix), gu._p(dv), n, d, k, m, candidates,
                                       iters, seed, gu._p(gi), gu._p(gd), ctypes.byref(ran),
                                       ctypes.byref(ev), ctypes.byref(sec)))
    _against_the_rule((gi, gd), full, k, candidates, iters, seed)
