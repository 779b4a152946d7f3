"""Host arrays in and out: large uploads through pinned buffers on several
threads, row indices widened and narrowed on the device, and CSR checks on
several threads."""
import threading

import numpy as np
import pytest
import torch

from umapers_b200 import _lib
from umapers_b200._umapers import UmapCore
from tests import gpu_util as gu

pytestmark = pytest.mark.gpu

STAGED = 64 << 20  # bytes from which an upload is staged
BUF = 1 << 20      # bytes of a staging buffer


def _self_neighbours(r, rows):
    """Every probed row of r is its own neighbour at distance zero only if its
    bytes have arrived: all values of r are distinct draws."""
    idx, dist = gu.knn_query(r[rows], r, 1)
    assert np.array_equal(idx[:, 0], rows) and not dist.any()


# just below and at the bound, one float past a buffer, and a ragged end
@pytest.mark.parametrize("n,d", [(STAGED // 64 - 1, 16), (STAGED // 64, 16),
                                 (STAGED // 4 + BUF // 4 + 1, 1), (1_000_003, 19)])
@pytest.mark.parametrize("pinned", [False, True])
def test_every_buffer_of_a_large_upload_arrives(n, d, pinned):
    g = torch.Generator().manual_seed(n)
    r = torch.randn(n, d, generator=g)
    if d == 1:
        # distinct values, increasing: rows probed by their nearest neighbour
        r = (torch.arange(n) - n // 2).float()[:, None]
    if pinned:
        r = r.pin_memory()
    r = r.numpy()
    edges = np.arange(0, n * d * 4, BUF) // (4 * d)
    rows = np.unique(np.clip(np.concatenate([edges - 1, edges, edges + 1, [n - 1]]), 0, n - 1))
    _self_neighbours(r, rows.astype(np.int64))


def test_uploads_of_several_threads_do_not_mix():
    n, d = 300_007, 64  # 76.8 MB each: more threads than pinned sets
    data = [np.random.default_rng(t).standard_normal((n, d), np.float32) for t in range(4)]
    rows = np.arange(0, n, 4099)
    failed = []

    def one(t):
        try:
            for _ in range(2):
                _self_neighbours(data[t], rows)
        except BaseException as e:  # noqa: BLE001 - reported below
            failed.append((t, e))

    team = [threading.Thread(target=one, args=(t,)) for t in range(4)]
    for th in team:
        th.start()
    for th in team:
        th.join()
    assert not failed


# indices below, at and above the 2M that are widened at a time
@pytest.mark.parametrize("nq", [5, 65_535, 65_536, 65_537, 131_073])
def test_indices_are_widened_chunk_by_chunk(nq):
    k = 32
    rng = np.random.default_rng(nq)
    r, q = rng.standard_normal((500, 8), np.float32), rng.standard_normal((nq, 8), np.float32)
    idx, dist = gu.knn_query(q, r, k)
    half = nq // 2
    for part in (slice(0, half), slice(half, nq)):
        i, d = gu.knn_query(q[part], r, k)
        assert np.array_equal(idx[part], i) and np.array_equal(dist[part], d)
    assert idx.min() >= 0 and idx.max() < 500


def _csr(n_rows, per_row, n_cols, seed):
    rng = np.random.default_rng(seed)
    start = rng.integers(0, n_cols - 2 * per_row, n_rows)
    step = np.cumsum(rng.integers(1, 3, (n_rows, per_row)), axis=1)
    indices = (start[:, None] + step).astype(np.int64)
    data = rng.uniform(0.5, 1.5, (n_rows, per_row)).astype(np.float32)
    return np.arange(n_rows + 1, dtype=np.int64) * per_row, indices.ravel(), data.ravel()


# nonzeros at and past the 2M that are narrowed at a time
@pytest.mark.parametrize("n_rows", [4096, 4097])
def test_column_indices_are_narrowed_chunk_by_chunk(n_rows):
    per_row, n_cols, k = 512, 1100, 4
    ip, ix, dv = _csr(n_rows, per_row, n_cols, n_rows)
    dense = np.zeros((n_rows, n_cols), np.float32)
    dense[np.repeat(np.arange(n_rows), per_row), ix] = dv
    idx = np.empty((n_rows, k), np.int64)
    dist = np.empty((n_rows, k), np.float32)
    _lib.check(_lib.load().umapb_knn_csr(gu._p(ip), gu._p(ix), gu._p(dv), n_rows, n_cols, k, 0,
                                         gu._p(idx), gu._p(dist)))
    want = gu.knn_exact(dense, k)[1]
    # distances near 20 from sums of 1,024 squares below 4 in FP32: the sums'
    # orders differ by at most 1,024 * 6e-8 of them
    assert np.abs(dist - want)[:, 1:].max() <= 20 * 1024 * 6e-8


# faults in the first and the last thread's rows, and two at once: the first
# in row order is named, columns before values
@pytest.mark.parametrize("faults,message", [
    ({"late": 0}, "csr row 2999 indices must be strictly increasing"),
    ({"early": 0, "late": 0}, "csr row 7 indices must be strictly increasing"),
    ({"range": 1500}, "csr row 1500 has column index 1100 out of bounds for n_cols=1100"),
    ({"nan": 2998}, "csr data must be finite"),
    ({"nan": 3, "late": 0}, "csr row 2999 indices must be strictly increasing"),
    ({}, "not fitted"),
])
def test_large_csr_faults_are_named_in_row_order(faults, message):
    per_row, n_cols = 512, 1100  # 1.5M nonzeros: four threads
    ip, ix, dv = _csr(3000, per_row, n_cols, 1)
    if "early" in faults:
        ix[7 * per_row + 3] = ix[7 * per_row + 2]
    if "late" in faults:
        ix[2999 * per_row + 511] = ix[2999 * per_row + 510]
    if "range" in faults:
        ix[faults["range"] * per_row + 511] = n_cols
    if "nan" in faults:
        dv[faults["nan"] * per_row] = np.nan
    core = UmapCore(n_neighbors=5, n_components=2)
    with pytest.raises(Exception, match=message):
        core.transform_sparse_csr(ip, ix, dv, n_cols)


# below and at the bound: an error of the call, after which the next one works
@pytest.mark.parametrize("n", [1000, STAGED // 64 - 1, STAGED // 64, STAGED // 32])
def test_a_null_array_is_an_error(n):
    lib, k = _lib.load(), 3
    r = np.random.default_rng(0).standard_normal((50, 16), np.float32)
    idx, dist = np.empty((n, k), np.int64), np.empty((n, k), np.float32)
    assert lib.umapb_knn_exact(None, n, 16, k, 0, 0, gu._p(idx), gu._p(dist), None) != 0
    assert lib.umapb_knn_query(None, n, gu._p(r), 50, 16, k, 0, 0, gu._p(idx), gu._p(dist)) != 0
    assert lib.umapb_knn_query(gu._p(r), 50, None, n, 16, k, 0, 0, gu._p(idx), gu._p(dist)) != 0
    _self_neighbours(r, np.arange(50))


# indices up to the 16,384 that the host widens, and one query more
@pytest.mark.parametrize("nq", [1, 512, 513])
def test_few_indices_are_widened_on_the_host(nq):
    test_indices_are_widened_chunk_by_chunk(nq + 1)
    rng = np.random.default_rng(nq)
    r = rng.standard_normal((500, 8), np.float32)
    q = rng.standard_normal((nq, 8), np.float32)
    idx, dist = gu.knn_query(q, r, 32)
    full = np.sqrt(((q[:, None, :].astype(np.float64) - r[None]) ** 2).sum(-1))
    # each row's distances, looked up by the indices, are the ones returned
    assert np.abs(np.take_along_axis(full, idx, 1) - dist).max() <= 1e-5
    assert np.abs(np.sort(full, 1)[:, :32] - dist).max() <= 1e-5


# as many nonzeros as the host narrows, and one row more
@pytest.mark.parametrize("n_rows", [32, 33])
def test_few_column_indices_are_narrowed_on_the_host(n_rows):
    test_column_indices_are_narrowed_chunk_by_chunk(n_rows)


# an odd number of indices goes through the distances' memory in three pieces,
# and distances come out before their memory is used
@pytest.mark.parametrize("nq,k", [(16_385, 1), (5_463, 3), (99_999, 5)])
@pytest.mark.parametrize("pinned", [False, True])
def test_indices_are_widened_through_the_memory_of_the_distances(nq, k, pinned):
    rng = np.random.default_rng(nq)
    r, q = rng.standard_normal((300, 5), np.float32), rng.standard_normal((nq, 5), np.float32)
    idx = torch.full((nq, k), -1, dtype=torch.int64)
    dist = torch.full((nq, k), -1.0)
    if pinned:
        idx, dist = idx.pin_memory(), dist.pin_memory()
    idx, dist = idx.numpy(), dist.numpy()
    _lib.check(_lib.load().umapb_knn_query(gu._p(q), nq, gu._p(r), 300, 5, k, 0, 0, gu._p(idx),
                                           gu._p(dist)))
    full = np.sqrt(((q[:, None, :].astype(np.float64) - r[None]) ** 2).sum(-1))
    assert np.abs(np.take_along_axis(full, idx, 1) - dist).max() <= 1e-5
    assert np.abs(np.sort(full, 1)[:, :k] - dist).max() <= 1e-5


def test_an_odd_number_of_column_indices_is_narrowed():
    per_row, n_rows, n_cols, k = 5, 3277, 40, 3  # 16,385 nonzeros
    ip, ix, dv = _csr(n_rows, per_row, n_cols, 3)
    dense = np.zeros((n_rows, n_cols), np.float32)
    dense[np.repeat(np.arange(n_rows), per_row), ix] = dv
    idx, dist = np.empty((n_rows, k), np.int64), np.empty((n_rows, k), np.float32)
    _lib.check(_lib.load().umapb_knn_csr(gu._p(ip), gu._p(ix), gu._p(dv), n_rows, n_cols, k, 0,
                                         gu._p(idx), gu._p(dist)))
    want = gu.knn_exact(dense, k)[1]
    # squared distances up to 40 as sums in two orders, 10 products each: 40 * 20 * 6e-8
    # apart, and the root of a difference as small as that
    assert np.abs(dist - want).max() <= np.sqrt(40 * 20 * 6e-8)
