"""transform on the GPU: kNN to the training rows, bipartite membership,
weighted-mean init and per-query SGD (rust_umap/src/lib.rs:1604-1780),
compared with the oracle's transform from the same fitted embedding."""
import numpy as np
import pytest

from umapers import Umap
from umapers_b200 import diagnostics, workloads

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fitted():
    fit, q = workloads.transform_mixture(n_fit=4000, n_query=1500, d=32, n_comp=8)
    m = Umap(n_neighbors=15, random_seed=3)
    emb = m.fit_transform(fit)
    return m, fit, q, emb


def test_transform_matches_oracle(orc, fitted):
    m, fit, q, emb = fitted
    a, b = m._core.ab_params
    g = m.transform(q)
    o = orc.transform(fit, emb, q, a, b, n_neighbors=15, random_seed=3)
    assert g.shape == (1500, 2) and np.all(np.isfinite(g))
    scale = np.linalg.norm(emb.std(0))
    disp = np.linalg.norm(g - o, axis=1)
    print("median displacement / scale", np.median(disp) / scale)
    assert np.median(disp) < 0.1 * scale
    both_g = np.vstack([fit, q]), np.vstack([emb, g])
    both_o = np.vstack([emb, o])
    tg = diagnostics.quality(both_g[0], both_g[1])["trustworthiness"]
    to = diagnostics.quality(both_g[0], both_o)["trustworthiness"]
    assert abs(tg - to) <= 0.01


def test_transform_of_training_rows_lands_near_fit(fitted):
    m, fit, _, emb = fitted
    g = m.transform(fit[:300])
    scale = np.linalg.norm(emb.std(0))
    assert np.median(np.linalg.norm(g - emb[:300], axis=1)) < 0.2 * scale


def test_transform_out_buffer_empty_and_errors(fitted):
    m, _, q, _ = fitted
    out = np.empty((10, 2), np.float32)
    assert m.transform(q[:10], out=out) is out
    assert m.transform(np.zeros((0, 32), np.float32)).shape == (0, 2)
    with pytest.raises(ValueError, match="feature mismatch"):
        m.transform(np.zeros((3, 31), np.float32))
    bad = q[:5].copy()
    bad[2, 1] = np.inf
    with pytest.raises(ValueError, match="non-finite value at row 2"):
        m.transform(bad)


@pytest.mark.parametrize("k,rate", [(15, 5), (16, 12), (20, 5)])
def test_transform_does_not_depend_on_the_lanes_per_query(k, rate):
    # Small requests give a query 16, 8 or 4 lanes, larger ones one thread.
    # Repeating a request's rows changes neither its largest weight nor its mean
    # distance, and a row's random stream is keyed by its position, so the
    # first copy's positions must come out the same bit for bit (rows of more
    # than 16 edges and more than 8 negatives an edge take paths of their own).
    fit, q = workloads.transform_mixture(n_fit=1500, n_query=9000, d=24, n_comp=6)
    m = Umap(n_neighbors=k, n_epochs=20, negative_sample_rate=rate, random_seed=5)
    m.fit(fit)
    q[3] = fit[10]  # a fitted point
    for n in (1, 31, 700, 4096, 4097, 8193):
        whole = np.tile(q[:n], (16385 // n + 1, 1))
        assert np.array_equal(m.transform(q[:n]), m.transform(whole)[:n])


@pytest.mark.parametrize("n", [1, 4097, 8193, 16385])
def test_transform_device_writes_to_any_float_address(n):
    # 16, 8 and 4 lanes a query and one thread a query: the same positions in
    # an array that starts one float off a vector boundary, nothing around it
    import torch

    from umapers_b200 import _lib

    fit, q = workloads.transform_mixture(n_fit=1000, n_query=n, d=16, n_comp=4)
    m = Umap(n_neighbors=10, n_epochs=10, random_seed=5)
    m.fit(fit)
    qd = torch.from_numpy(q).cuda()
    flat = torch.full((2 * n + 3,), -7.0, device="cuda")
    assert flat.data_ptr() % 8 == 0
    want = torch.empty((n, 2), device="cuda")
    torch.cuda.synchronize()
    for out in (want.data_ptr(), flat.data_ptr() + 4):
        _lib.check(_lib.load().umapb_transform_device(m._core._handle, qd.data_ptr(), n, 16, out))
    assert torch.equal(flat[1:-2].reshape(n, 2), want)
    assert flat[0] == -7.0 and (flat[-2:] == -7.0).all()


def test_transform_at_the_largest_request_of_several_lanes():
    # 14,208 queries fit the GPU at four lanes each, one more takes a thread
    # each; whole copies of a request leave its largest weight and mean distance
    fit, q = workloads.transform_mixture(n_fit=1500, n_query=7104, d=24, n_comp=6)
    m = Umap(n_neighbors=15, n_epochs=20, random_seed=5)
    m.fit(fit)
    for n, few, many in ((7104, 2, 3), (1093, 12, 13)):  # 14,208; 14,209 = 13 x 1,093
        a, b = (m.transform(np.tile(q[:n], (c, 1)))[:n] for c in (few, many))
        assert np.array_equal(a, b)
