"""The structural step launchers (csrc/launchers.cu) where their kernels change:
one block and several (2,048 items each), ranges of edges and of root words that
end within a block, rows of 64 and 65 entries, empty rows in a warp's range of rows.
Against a restatement, bit for bit."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from labelpropcuda_gb300 import DeviceArray
from labelpropcuda_gb300 import _native as N

ACTIVE, DELETED, GT = 0, 1, 2
F = np.float32


def graph(n, edges, seed):
    """Random rows; vertices 5 and 6 have 64 and 65 entries, every 50th vertex none."""
    rng = np.random.default_rng(seed)
    owner = rng.integers(0, n, edges)
    owner = owner[(owner % 50 != 0) & (owner != 5) & (owner != 6)]
    owner = np.sort(np.concatenate([owner, np.full(64, 5), np.full(65, 6)]))
    row = np.zeros(n + 1, np.int32)
    row[1:] = np.cumsum(np.bincount(owner, minlength=n))
    col = rng.integers(0, n, owner.size).astype(np.int32)
    col[rng.random(col.size) < 0.05] = -1
    return row, col, rng.random(col.size, dtype=F), rng


SIZES = [(100, 300), (2047, 2048), (2049, 2049), (5000, 30011), (70000, 400003)]


@pytest.mark.gpu
@pytest.mark.parametrize("n,edges", SIZES)
def test_mark_deletions(gpu, n, edges):
    row, col, _, rng = graph(n, edges, n)
    status = rng.choice([ACTIVE, DELETED, GT], size=n, p=[0.8, 0.1, 0.1]).astype(np.int32)
    deleted = rng.permutation(n)[:max(1, n // 20)].astype(np.int32)
    deleted[0] = 6
    affected = (rng.random(n) < 0.1).astype(np.int32)
    d = [DeviceArray(x) for x in (row, col, status, affected, deleted)]
    N.check(N.lib().dlp_mark_deletions(*[x.ptr for x in d], deleted.size, n, None))
    owner = np.repeat(np.arange(n), np.diff(row))
    now = status.copy()
    now[deleted] = DELETED
    of_deleted = np.isin(owner, deleted)
    affected[col[of_deleted & (col >= 0)]] = 1
    col = col.copy()
    col[of_deleted] = -1
    col[(now[owner] != DELETED) & (col >= 0) & (now[col] == DELETED)] = -1
    np.testing.assert_array_equal(d[1].get(), col)
    np.testing.assert_array_equal(d[2].get(), now)
    np.testing.assert_array_equal(d[3].get(), affected)


def batch(n, edges, rng):
    inserted = rng.permutation(n)[:max(2, n // 3)].astype(np.int32)
    is_new = np.zeros(n, np.int32)
    is_new[inserted] = 1
    # most edges between new vertices, in runs of neighbours along a random order
    src = inserted[rng.integers(0, inserted.size - 1, edges)]
    dst = np.where(rng.random(edges) < 0.97, inserted[rng.integers(0, inserted.size, edges)], rng.integers(0, n, edges))
    return inserted, is_new, src.astype(np.int32), dst.astype(np.int32), rng.random(edges, dtype=F)


@pytest.mark.gpu
@pytest.mark.parametrize("n,edges", SIZES)
def test_sparsification(gpu, n, edges):
    rng = np.random.default_rng(n)
    inserted, is_new, src, dst, weight = batch(n, edges, rng)
    tau = F(0.4)
    weight[:3] = tau  # not above it
    affected = np.zeros(n, np.int32)
    d = [DeviceArray(x) for x in (affected, src, dst, weight, inserted, is_new)]
    sub_col, sub_val = DeviceArray(np.full(2 * edges, -7, np.int32)), DeviceArray(np.full(2 * edges, -7, F))
    nodes, kept = ctypes.c_int(-1), ctypes.c_int(-1)
    N.check(N.lib().dlp_build_sparsified_subgraph(
        None, None, None, d[0].ptr, None, d[1].ptr, d[2].ptr, d[3].ptr, edges, d[4].ptr, inserted.size, d[5].ptr, tau,
        None, sub_col.ptr, sub_val.ptr, ctypes.byref(nodes), ctypes.byref(kept), None))
    keep = (weight > tau) & (is_new[src] == 1) & (is_new[dst] == 1)
    assert (nodes.value, kept.value) == (inserted.size, 2 * keep.sum())
    want_col, want_val = np.full(2 * edges, -7, np.int32), np.full(2 * edges, -7, F)
    want_col[:kept.value] = np.stack([dst[keep], src[keep]], 1).ravel()
    want_val[:kept.value] = np.repeat(weight[keep], 2)
    np.testing.assert_array_equal(sub_col.get(), want_col)
    assert sub_val.get().tobytes() == want_val.tobytes()
    heavy = np.concatenate([src[weight > tau], dst[weight > tau]])
    affected[heavy[heavy < inserted.size]] = 1
    np.testing.assert_array_equal(d[0].get(), affected)


def components(n, inserted, src, dst):
    """Smallest member of each component of the inserted vertices; -1 (a vertex that
    is not inserted) takes over what it touches."""
    root = np.full(n, -1, np.int64)
    root[inserted] = inserted
    while True:
        before = root.copy()
        low = np.minimum(root[src], root[dst])
        for x in (src, dst):
            own = before[x]
            np.minimum.at(root, own[own >= 0], low[own >= 0])
        while True:
            up = np.where(root >= 0, root[root], -1)
            if np.array_equal(up, root):
                break
            root = up
        if np.array_equal(root, before):
            return root


@pytest.mark.gpu
@pytest.mark.parametrize("n,edges", SIZES)
@pytest.mark.parametrize("share", [1.0, 0.2])  # of the edges: few and many components
def test_components(gpu, n, edges, share):
    rng = np.random.default_rng(n + 1)
    inserted, is_new, src, dst, _ = batch(n, edges, rng)
    m = max(1, int(share * min(edges, inserted.size)))
    src, dst = src[:m], dst[:m]
    if share == 1.0:
        dst = np.where(is_new[dst] == 1, dst, src)
    d = [DeviceArray(x) for x in (src, dst, inserted, np.full(n, -7, np.int32))]
    count = ctypes.c_int(-1)
    N.check(N.lib().dlp_connected_components(d[0].ptr, d[1].ptr, m, d[2].ptr, inserted.size, d[3].ptr,
                                             ctypes.byref(count), n, None))
    root = components(n, inserted, src, dst)
    roots = np.unique(root[root >= 0])
    want = np.where(root >= 0, np.searchsorted(roots, root), -1)
    assert count.value == roots.size
    np.testing.assert_array_equal(d[3].get(), want)


@pytest.mark.gpu
@pytest.mark.parametrize("n,edges", SIZES)
@pytest.mark.parametrize("count", [1, 37, None])  # components; None: one per inserted vertex
def test_label_initialisation(gpu, n, edges, count):
    row, col, val, rng = graph(n, edges, n + 2)
    inserted = rng.permutation(n)[:max(8, n // 3)].astype(np.int32)
    inserted[:2] = 5, 6
    inserted = np.unique(inserted).astype(np.int32)
    count = inserted.size if count is None else count
    comp = np.full(n, -1, np.int32)
    comp[inserted] = rng.integers(-1, count + 1, inserted.size)  # none, and ids out of range
    gt = rng.choice([-1, 0, 1], size=n, p=[0.9, 0.05, 0.05]).astype(np.int32)
    labels = rng.random(n, dtype=F)
    d = [DeviceArray(x) for x in (row, col, val, labels, comp, inserted, gt)]
    N.check(N.lib().dlp_label_initialization(d[0].ptr, d[1].ptr, d[2].ptr, d[3].ptr, None, d[4].ptr, count, d[5].ptr,
                                             inserted.size, d[6].ptr, n, None))
    owner = np.repeat(np.arange(n), np.diff(row))
    new = np.zeros(n, bool)
    new[inserted] = True
    use = new[owner] & (comp[owner] >= 0) & (comp[owner] < count) & (col >= 0)
    fixed = np.rint(val.astype(np.float64) * 2.0**32).astype(np.int64)
    share = np.zeros((2, count), np.int64)
    for c in (0, 1):
        pick = use & (gt[col] == c)
        np.add.at(share[c], comp[owner[pick]], fixed[pick])
    w = (share.astype(np.float64) / 2.0**32).astype(F)
    den = w[0] + w[1]
    by_comp = np.where(den > F(1e-10), w[1] / np.where(den > F(1e-10), den, F(1)), F(0.5))
    want = labels.copy()
    inside = (comp[inserted] >= 0) & (comp[inserted] < count)
    want[inserted] = np.where(inside, by_comp[np.where(inside, comp[inserted], 0)], F(0.5))
    for c in (0, 1):
        want[inserted[gt[inserted] == c]] = c
    assert d[3].get().tobytes() == want.tobytes()
