"""The deterministic layout of small graphs against a sequential NumPy replay:
edges coloured greedily in graph order, each epoch's due edges one after
another by (colour, graph order), negatives from the epoch's starting
positions (rust_umap/src/lib.rs:5172-5318 per edge)."""
import ctypes
import gc
import threading

import numpy as np
import pytest

from umapers import Umap
from umapers_b200 import _lib
from tests.gpu_util import optimize_layout

pytestmark = pytest.mark.gpu

M64 = (1 << 64) - 1
F = np.float32


def mix64(z):
    z = (z + 0x9E3779B97F4A7C15) & M64
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & M64
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & M64
    return z ^ (z >> 31)


def replay(emb, h, t, w, n_epochs, a, b, lr, rate, seed):
    cur = emb.astype(np.float64)
    n, m = len(emb), len(h)
    used, color = [0] * n, np.zeros(m, np.int64)
    for e in range(m):
        u = used[h[e]] | used[t[e]]
        c = (~u & (u + 1)).bit_length() - 1
        color[e] = c
        used[h[e]] |= 1 << c
        used[t[e]] |= 1 << c
    order = np.lexsort((np.arange(m), color))
    ns = F(n_epochs) * (w.astype(F) / F(max(w.max(), 1e-12)))
    eps = np.where(ns > 0, F(n_epochs) / np.where(ns > 0, ns, F(1)), F(np.inf)).astype(F)
    en = (eps / F(rate)).astype(F)
    nxt, nneg = eps.copy(), en.copy()
    streams = [mix64(seed ^ mix64(e)) for e in range(m)]
    for ep in range(n_epochs):
        snap = cur.copy()
        alpha = float(F(lr) * (F(1) - F(ep) / F(n_epochs)))
        for e in order:
            if nxt[e] > F(ep):
                continue
            i, j = h[e], t[e]
            x = cur[i].copy()
            if i != j:
                d2 = ((x - cur[j]) ** 2).sum()
                if d2 > 0:
                    pb = d2 ** b
                    mv = np.clip(-2 * a * b * pb / d2 / (a * pb + 1) * (x - cur[j]), -4, 4) * alpha
                    x = x + mv
                    cur[j] = cur[j] - mv
            nxt[e] = F(nxt[e] + eps[e])
            if np.isfinite(en[e]) and en[e] > 0:
                k = int(max(np.floor(F(F(ep) - nneg[e]) / en[e]), 0))
                for s in range(k):
                    o = ((mix64(streams[e] ^ ((ep << 32) | s)) >> 32) * n) >> 32
                    if o == i:
                        continue
                    d2 = ((x - snap[o]) ** 2).sum()
                    if d2 > 0:
                        gc = 2 * b / ((0.001 + d2) * (a * d2 ** b + 1))
                        x = x + np.clip(gc * (x - snap[o]), -4, 4) * alpha
                nneg[e] = F(nneg[e] + F(k) * en[e])
            cur[i] = x
    return cur


def random_graph(n, deg, rng):
    h = np.repeat(np.arange(n), deg)
    t = rng.integers(0, n, n * deg)
    hh, tt = np.concatenate([h, t]), np.concatenate([t, h])
    o = np.lexsort((tt, hh))  # self edges and duplicates stay in
    return hh[o].astype(np.int32), tt[o].astype(np.int32)


def star(n):
    h = np.concatenate([np.zeros(n - 1), np.arange(1, n)])
    t = np.concatenate([np.arange(1, n), np.zeros(n - 1)])
    return h.astype(np.int32), t.astype(np.int32)


# (vertices, dimensions, degree or 0 for a star, epochs, negative rate): one
# edge, every position width (packed up to 3, plain above, run-time above 4), the
# largest vertex counts of each, negatives beyond the stored 14, a star whose
# centre's chain runs past the start-time buckets.
CASES = [(2, 2, 1, 4, 5), (33, 1, 3, 6, 5), (700, 2, 4, 4, 5), (300, 3, 4, 4, 1),
         (300, 4, 4, 4, 5), (200, 7, 3, 4, 5), (150, 2, 4, 3, 40), (8192, 2, 1, 3, 2),
         (16384, 1, 1, 2, 1), (5461, 3, 1, 2, 2), (2500, 2, 0, 3, 5)]


@pytest.mark.parametrize("n,dim,deg,n_epochs,rate", CASES)
def test_small_layout_matches_sequential_replay(n, dim, deg, n_epochs, rate):
    rng = np.random.default_rng(n + dim)
    h, t = random_graph(n, deg, rng) if deg else star(n)
    w = rng.uniform(0.3, 1.0, len(h)).astype(np.float32)
    emb = rng.normal(0, 3, (n, dim)).astype(np.float32)
    # A step of at most 4 lr moves a point; its coefficient is within 5e-5
    # relative of the replay's.  At lr = 0.01 a vertex with k updates is off by
    # at most k * 0.04 * 5e-5, grown by its neighbours' at most as much again;
    # a missing, repeated or misordered update moves it by 1e-3 and more.
    lr, a, b, seed = 0.01, 1.577, 0.895, 77
    got = optimize_layout(emb, h, t, w, n_epochs, a, b, lr=lr, neg_rate=rate, seed=seed)
    again = optimize_layout(emb, h, t, w, n_epochs, a, b, lr=lr, neg_rate=rate, seed=seed)
    assert np.array_equal(got, again)
    ref = replay(emb, h, t, w, n_epochs, a, b, lr, rate, seed)
    k = (np.bincount(h, minlength=n) * (1 + rate) + np.bincount(t, minlength=n)) * (n_epochs - 1)
    bound = 2 * k * 4 * lr * 5e-5 + 1e-6 * np.abs(emb).max()
    assert (np.abs(got - ref).max(1) <= bound).all()


def test_an_event_may_wait_longer_than_the_limit_on_idle_polls():
    # Two edges with one head: the second waits for the first one's 8,000,000
    # negatives, 1.5 s, longer than the limit on polls without any update.
    # Vertex 3 has no edge, and every point must stay finite and have moved.
    h, t = np.array([0, 0], np.int32), np.array([1, 2], np.int32)
    emb = np.random.default_rng(0).normal(0, 3, (4, 2)).astype(np.float32)
    got = optimize_layout(emb, h, t, np.ones(2, np.float32), 2, 1.577, 0.895, neg_rate=8_000_000,
                          seed=3)
    assert np.isfinite(got).all() and np.array_equal(got[3], emb[3])
    assert (got[:3] != emb[:3]).any(1).all()


# positions wider than a word, polled by their counter alone: the first and the
# last such width, and the most vertices of the last
@pytest.mark.parametrize("n,dim,deg", [(200, 5, 3), (200, 9, 3), (200, 16, 3), (1024, 16, 1)])
def test_wide_positions_match_sequential_replay(n, dim, deg):
    test_small_layout_matches_sequential_replay(n, dim, deg, 3, 5)


def _fit(x, seed):
    m = Umap(n_neighbors=15, n_epochs=200, random_seed=seed)
    return m, m.fit_transform(x)


def test_models_alive_share_the_work_space():
    # 1,000 rows of 32 columns ask for 224 MB of it, and for about 1 MB else
    lib = _lib.load()
    reserved, used = ctypes.c_int64(0), ctypes.c_int64(0)

    def pool():
        _lib.check(lib.umapb_pool_bytes(ctypes.byref(reserved), ctypes.byref(used)))
        return used.value

    x = np.random.default_rng(0).normal(size=(1000, 32)).astype(np.float32)
    before = pool()
    models = [_fit(x, 1)]
    one = pool()
    models += [_fit(x, 1) for _ in range(4)]
    assert one - before <= 272 << 20 and pool() - one <= 4 * (16 << 20)
    assert all(np.array_equal(e, models[0][1]) for _, e in models)
    models.clear()
    gc.collect()
    assert pool() <= before + (256 << 20)  # models of other tests may be alive


def test_fits_of_several_threads_keep_their_work_spaces_apart():
    rng = np.random.default_rng(1)
    data = [rng.normal(size=(n, 16)).astype(np.float32) for n in (300, 900, 1500, 2400)]
    want = [_fit(x, 7)[1] for x in data]
    got = [[] for _ in data]

    def work(i):
        for _ in range(3):
            got[i].append(_fit(data[i], 7)[1])

    team = [threading.Thread(target=work, args=(i,)) for i in range(len(data))]
    for t in team:
        t.start()
    for t in team:
        t.join()
    for g, w in zip(got, want):
        assert len(g) == 3 and all(np.array_equal(e, w) for e in g)
