"""NN-descent on the GPU: recall against exact kNN (the reference's
thresholds, rust_umap/src/lib.rs:6733-6764) and against the oracle's own
recall on the same data."""
import numpy as np
import pytest

from umapers_b200 import workloads
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
