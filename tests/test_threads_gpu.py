"""Calls of several threads at once that run the same kernels with different
amounts of shared memory: each gives what it gives alone."""
import threading

import numpy as np
import pytest

from umapers import Umap
from tests import gpu_util as gu

pytestmark = pytest.mark.gpu


def _rows(n, d):
    return np.random.default_rng(n + d).normal(size=(n, d)).astype(np.float32)


def _fit(n):
    return lambda: (Umap(n_neighbors=15, n_epochs=100, random_seed=7).fit_transform(_rows(n, 16)),)


def _knn(d, k, backend):
    return lambda: gu.knn_exact(_rows(700, d), k, backend=backend)[:2]


def _nd(d, k):
    return lambda: gu.nndescent(_rows(600, d), k, 20, 4, 5)[:2]


@pytest.mark.parametrize("calls", [
    [_fit(n) for n in (300, 900, 1500, 2400)],
    [_knn(d, k, "plain") for d, k in ((8, 5), (33, 40), (130, 15), (200, 3))],
    [_knn(d, k, "tensor") for d, k in ((8, 5), (33, 40), (130, 15), (500, 3))],
    [_nd(d, k) for d, k in ((4, 15), (70, 15), (300, 15), (900, 15))],
], ids=["fit", "plain", "tensor", "nndescent"])
def test_calls_of_several_threads_do_not_disturb_one_another(calls):
    want = [c() for c in calls]
    got = [[] for _ in calls]

    def work(i):
        for _ in range(6):
            got[i].append(calls[i]())

    team = [threading.Thread(target=work, args=(i,)) for i in range(len(calls))]
    for t in team:
        t.start()
    for t in team:
        t.join()
    for g, w in zip(got, want):
        assert len(g) == 6
        assert all(np.array_equal(a, b) for r in g for a, b in zip(r, w))
