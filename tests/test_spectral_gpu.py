"""Spectral initialisation on the GPU against the oracle: the same
embedding subspace for connected graphs, and component separation for
disconnected ones (rust_umap/src/lib.rs:7541-7694)."""
import numpy as np
import pytest

from umapers_b200 import workloads
from tests import gpu_util as gu

pytestmark = pytest.mark.gpu


def _ratio(e, labels, n):
    cents = np.stack([e[labels == c].mean(0) for c in range(n)])
    sep = min(np.linalg.norm(cents[i] - cents[j]) for i in range(n) for j in range(i + 1, n))
    std = max(np.sqrt(((e[labels == c] - cents[c]) ** 2).mean(0).sum()) for c in range(n))
    return sep / (std + 1e-6)


def test_connected_spectral_matches_oracle_subspace(orc):
    x = workloads.gaussian(2000, 32, seed=4)
    idx, dist = orc.exact_knn(x, 15)
    h, t, w, _, _ = orc.fuzzy_graph(idx, dist, n_epochs=500)
    g, used = gu.spectral_init(x, h, t, w, 2, 42)
    o, oused, ncomp = orc.spectral_init(x, h, t, w, 2, 42)
    assert used and oused and ncomp == 1
    assert np.abs(g).max() == pytest.approx(10.0, abs=1e-2)
    assert gu.linear_fit_r2(o, g) > 0.98 and gu.linear_fit_r2(g, o) > 0.98


def test_disconnected_spectral_beats_random(orc):
    x, labels = workloads.disconnected_components(4, 60)
    idx, dist = orc.exact_knn(x, 10)
    h, t, w, _, _ = orc.fuzzy_graph(idx, dist)
    g, used = gu.spectral_init(x, h, t, w, 2, 42)
    assert used
    rnd = orc.random_init(x.shape[0], 2, 42)
    assert _ratio(g, labels, 4) > _ratio(rnd, labels, 4) * 1.2


def test_large_disconnected_components_stay_structured(orc):
    # components above 128 nodes take the batched iterative path
    x, labels = workloads.disconnected_components(3, 152)
    idx, dist = orc.exact_knn(x, 12)
    h, t, w, _, _ = orc.fuzzy_graph(idx, dist)
    g, used = gu.spectral_init(x, h, t, w, 2, 42)
    assert used and np.all(np.isfinite(g))
    rnd = orc.random_init(x.shape[0], 2, 42)
    assert _ratio(g, labels, 3) > _ratio(rnd, labels, 3) * 1.2


def test_mixture_components_follow_oracle_layout(orc):
    x = workloads.isotropic_mixture(3000, 64, 6, 6.0, seed=8)
    idx, dist = orc.exact_knn(x, 15)
    h, t, w, _, _ = orc.fuzzy_graph(idx, dist, n_epochs=500)
    g, used = gu.spectral_init(x, h, t, w, 2, 7)
    o, oused, ncomp = orc.spectral_init(x, h, t, w, 2, 7)
    assert used and oused and ncomp >= 2
    # component anchors are deterministic (meta layout); within-component
    # coordinates agree up to the eigenvector sign per component
    np.testing.assert_allclose(g.mean(0), o.mean(0), atol=0.5)


def hub_graph(n_blocks=5, seed=3):
    """Blocks of random edges, loosely joined, with rows whose lengths lie at
    the edges of the product's quads, chunks and row kinds."""
    rng = np.random.default_rng(seed)
    sizes = [230 + 30 * b for b in range(n_blocks)]
    start = np.concatenate([[0], np.cumsum(sizes)])
    n = int(start[-1])
    w = np.zeros((n, n), np.float32)
    for b, sz in enumerate(sizes):
        i = start[b] + np.repeat(np.arange(sz), 12)
        j = start[b] + rng.integers(0, sz, i.shape[0])
        w[i, j] = rng.uniform(0.3, 1.0, i.shape[0])
    for b, c in enumerate(range(1, n_blocks)):
        i = start[b] + rng.integers(0, sizes[b], 80 + 60 * b)
        j = start[c] + rng.integers(0, sizes[c], 80 + 60 * b)
        w[i, j] = 0.5
    w = np.maximum(w, w.T)
    np.fill_diagonal(w, 0.0)
    want = [95, 96, 97, 127, 128, 129, 255, 256, 257]
    hubs = start[-2] + 3 + 7 * np.arange(len(want))
    for row, length in zip(hubs, want):  # grown by edges to rows that are no hubs
        free = [j for j in range(start[-2], n) if j not in hubs and j != row and w[row, j] == 0]
        add = rng.choice(free, length - int((w[row] > 0).sum()), replace=False)
        w[row, add] = w[add, row] = rng.uniform(0.3, 1.0, add.shape[0])
    assert [int((w[r] > 0).sum()) for r in hubs] == want
    return w


@pytest.mark.parametrize("dim", [1, 2, 3, 4])
def test_long_rows_give_the_dense_eigenvectors(dim):
    w = hub_graph()
    h, t = np.nonzero(w)
    deg = w.astype(np.float64).sum(1)
    a = w / np.sqrt(deg[:, None] * deg[None, :])
    val, vec = np.linalg.eigh(a)
    assert np.min(-np.diff(val[::-1][:dim + 2])) > 1e-3  # separated eigenvalues
    x = np.zeros((w.shape[0], 16), np.float32)
    g, used = gu.spectral_init(x, h.astype(np.int32), t.astype(np.int32), w[h, t], dim, 42)
    assert used
    ref = vec[:, ::-1][:, 1:dim + 1]
    ref = ref * 10.0 / np.abs(ref).max()
    ref = ref * np.sign((ref * g).sum(0))
    # N(0, 1e-4) noise on every coordinate (6 sigma), FP32 products (6e-8)
    # over eigenvalue gaps of 1e-3 at a scale of 10
    assert np.abs(g - ref).max() < 6e-4 + 10 * 6e-8 / 1e-3 * 2


def equitable_graph(blocks, m, seed=11):
    """A path of blocks of m nodes: six random m-cycles inside each block, node
    i of a block tied to node i of the next.  Every node of a block has the same
    weight to each block, so the leading eigenvectors of the normalised matrix
    are constant on the blocks and come from the blocks x blocks quotient."""
    rng = np.random.default_rng(seed)
    h, t, w = [], [], []
    tie = 0.3 + 0.17 * np.arange(blocks - 1)
    for b in range(blocks):
        for _ in range(6):
            cyc = rng.permutation(m) + b * m
            h.append(cyc), t.append(np.roll(cyc, 1)), w.append(np.full(m, 0.5))
        if b + 1 < blocks:
            i = np.arange(m) + b * m
            h.append(i), t.append(i + m), w.append(np.full(m, tie[b]))
    h, t, w = np.concatenate(h), np.concatenate(t), np.concatenate(w)
    n = blocks * m
    key, inv = np.unique(np.concatenate([h * n + t, t * n + h]), return_inverse=True)
    weight = np.bincount(inv, np.concatenate([w, w])).astype(np.float32)
    deg = 6.0 + np.append(tie, 0.0) + np.append(0.0, tie)
    q = np.diag(6.0 / deg)
    for b in range(blocks - 1):
        q[b, b + 1] = q[b + 1, b] = tie[b] / np.sqrt(deg[b] * deg[b + 1])
    return (key // n).astype(np.int32), (key % n).astype(np.int32), weight, q


# one chunk of rows and one row more than it, a whole bundle of 16 chunks and
# one more, more chunks than are split over CTAs, chunks of more than 1024 rows
@pytest.mark.parametrize("dim,m", [(1, 342), (2, 256), (2, 257), (2, 4096), (2, 4097),
                                   (3, 6001), (4, 341), (4, 25_271), (2, 38_001), (2, 77_003)])
def test_orthonormalisation_at_its_chunk_edges(dim, m):
    blocks = dim + 2
    h, t, w, q = equitable_graph(blocks, m)
    val, vec = np.linalg.eigh(q)
    val = val[::-1]
    assert np.min(-np.diff(val)) > 4e-3 and val[dim] > 0.7  # the cycles' bulk ends near 0.55
    x = np.zeros((blocks * m, 16), np.float32)
    g, used = gu.spectral_init(x, h, t, w, dim, 42)
    assert used
    ref = np.repeat(vec[:, ::-1][:, 1:dim + 1], m, axis=0)
    ref = ref * 10.0 / np.abs(ref).max()
    ref = ref * np.sign((ref * g).sum(0))
    # N(0, 1e-4) noise on every coordinate (6 sigma), FP32 products (6e-8)
    # over eigenvalue gaps of 4e-3 at a scale of 10
    assert np.abs(g - ref).max() < 6e-4 + 10 * 6e-8 / 4e-3 * 2


# rows and features below, at and above the groups and tiles of the centroid sum
@pytest.mark.parametrize("n_rows,d", [(5, 3), (15, 63), (16, 64), (17, 65), (100, 200)])
def test_component_layout_follows_its_centroids(n_rows, d):
    """Five rings of n_rows or n_rows + 1 rows.  A ring's own layout has mean
    zero, so its mean is its place in the layout of the centroids: the second
    and third eigenvectors of the normalised Laplacian of exp(-distance^2)."""
    rng = np.random.default_rng(n_rows)
    h, t, x = [], [], []
    base = 0
    size = [n_rows + c % 2 for c in range(5)]
    centre = rng.standard_normal((5, d))
    centre *= 0.9 / np.linalg.norm(centre, axis=1, keepdims=True)
    for c, m in enumerate(size):
        i = np.arange(m)
        h += [base + i, base + (i + 1) % m]
        t += [base + (i + 1) % m, base + i]
        x.append((rng.standard_normal((m, d)) * 0.3 + centre[c]).astype(np.float32))
        base += m
    h, t = np.concatenate(h), np.concatenate(t)
    order = np.lexsort((t, h))
    g, used = gu.spectral_init(np.concatenate(x), h[order].astype(np.int32),
                               t[order].astype(np.int32), np.ones(h.size, np.float32), 2, 42)
    assert used
    mid = np.array([p.mean(0) for p in np.split(g.astype(np.float64), np.cumsum(size)[:-1])])
    cent = np.array([p.astype(np.float64).mean(0) for p in x])
    aff = np.exp(-((cent[:, None] - cent[None]) ** 2).sum(-1))
    deg = aff.sum(1)
    val, vec = np.linalg.eigh(np.eye(5) - aff / np.sqrt(deg[:, None] * deg[None]))
    assert np.diff(val)[:3].min() > 1e-3
    ref = vec[:, 1:3] * (10.0 / np.abs(vec[:, 1:3]).max())
    ref *= np.sign((ref * mid).sum(0))
    # N(0, 1e-4) noise on the places and on the rows (6 sigma each), FP32
    # coordinates near 10 and their mean (6e-8 each)
    assert np.abs(mid - ref).max() < 1.2e-3 + 4 * 10 * 6e-8
