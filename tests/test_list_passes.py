"""Passes over frontier lists: what a launch takes that does not run on owned rows,
because its frontier marks have no memory (here: no room in the budget) or because
it has too many vertices. The engine against the oracle, the launchers against
a restatement in fp32 and the oracle's recompute, all bit for bit."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

import labelpropcuda_gb300 as dlp
from labelpropcuda_gb300 import DeviceArray
from labelpropcuda_gb300 import _native as N
from parity_checks import EXACT_STATS

ACTIVE, DELETED, GT = 0, 1, 2
F = np.float32


def without_marks(probs, **kw):
    """An engine whose budget holds the graphs and nothing more."""
    budget = sum(dlp.Engine.graph_bytes(p.num_nodes, p.num_edges) for p in probs)
    eng = dlp.Engine(len(probs), memory_budget_bytes=budget, **kw)
    return eng, [eng.add_problem(p) for p in probs]


@pytest.mark.gpu
@pytest.mark.parametrize("lanes,solo", [(1, 0), (4, 0), (8, 0), (8, 7), (16, 0), (32, 0), (32, 7)])
def test_continued_batches_of_several_graphs(gpu, oracle, lanes, solo):
    """Every lane width, batches that go on in later launches beside ones that
    start, rows of 9 to 32 and of more than 32 entries, with frontiers that take one
    lane per short row and ones that do not."""
    probs = [dlp.Problem(n, d, 3, s, cache_dir="") for n, d, s in ((1500, 5, 1), (64, 3, 2), (3000, 34, 3), (90000, 9, 4))]
    cap = 50
    orcs = [oracle.OracleRun.from_problem(p, threads=4, max_iterations=cap) for p in probs]
    eng, ids = without_marks(probs, max_iterations=cap, small_frontier_solo=solo, narrow_lanes=lanes)
    dev = [[dlp.DeviceBatch(b) for b in p.batches] for p in probs]
    nxt, step = [0] * len(probs), 0
    while any(x < 3 for x in nxt) or any(eng.in_progress(g) for g in ids):
        start = [i for i, g in enumerate(ids) if nxt[i] < 3 and not eng.in_progress(g) and (step + i) % 2 == 0]
        done, _ = eng.step_sliced([(ids[i], nxt[i], dev[i][nxt[i]]) for i in start], pass_budget=17)
        for i in start:
            nxt[i] += 1
        for g in done:
            i = ids.index(g)
            want, got = orcs[i].apply(nxt[i] - 1, probs[i].batches[nxt[i] - 1]), eng.stats(g, nxt[i] - 1)
            for k in EXACT_STATS:
                assert got[k] == want[k], (i, nxt[i] - 1, k)
            assert eng.labels(g).tobytes() == orcs[i].labels().tobytes(), (i, nxt[i] - 1)
        step += 1


@pytest.mark.gpu
@pytest.mark.parametrize("n", [3068320, 3068321])  # the most that 151 blocks own in the engine, and one more
def test_around_the_most_vertices_on_owned_rows(gpu, oracle, n):
    p = dlp.Problem(n, 3, 200, 5, cache_dir="")
    orc = oracle.OracleRun.from_problem(p, threads=0, max_iterations=12)  # 8 passes over lists come first
    sess = dlp.Session.from_problem(p, max_iterations=12, small_frontier_solo=0)
    for b, batch in enumerate(p.batches[:3]):
        got, want = sess.apply(b, batch), orc.apply(b, batch)
        for k in EXACT_STATS:
            assert got[k] == want[k], (b, k)
        assert sess.labels().tobytes() == orc.labels().tobytes(), b


# ---------------------------------------------------------------- launchers --

@pytest.fixture(scope="module")
def large():
    """3,706,145 vertices (one more than the launchers' blocks own), rows of up to 32
    entries but the first, which has 40."""
    n = 3706145
    p = dlp.Problem(n, 3, 1, 9, cache_dir="")
    rng = np.random.default_rng(9)
    row, col, val = p.row_ptr.astype(np.int64), p.col_ind, p.values
    assert np.diff(row).max() <= 32
    extra = rng.integers(1, n, 40 - row[1]).astype(np.int32)
    col, val = np.concatenate([col[:row[1]], extra, col[row[1]:]]), np.concatenate(
        [val[:row[1]], rng.random(extra.size, dtype=F), val[row[1]:]])
    row[1:] += extra.size
    status = rng.choice([ACTIVE, DELETED, GT], size=n, p=[0.86, 0.06, 0.08]).astype(np.int32)
    status[0] = ACTIVE
    gt = np.where(status == GT, (p.true_labels >= 0.5).astype(np.int32), -1).astype(np.int32)
    labels = rng.random(n, dtype=F)
    affected = (rng.random(n) < 0.004).astype(np.int32)
    affected[0] = 1
    return row.astype(np.int32), col, val, labels, status, gt, affected


def cut(g, n):
    """The first n vertices."""
    row, col, val, labels, status, gt, affected = g
    col = np.where(col < n, col, -1).astype(np.int32)[:row[n]]
    return row[:n + 1], col, val[:row[n]], labels[:n], status[:n], gt[:n], affected[:n]


def new_labels(row, col, val, src, status, front):
    """src/iterativePropagation.cu:126-168 for many rows of at most 64 entries: slot
    t holds entry t, strides 32 to 1 (those above add zeros)."""
    at = row[front][:, None] + np.arange(64)
    use = at < row[front + 1][:, None]
    at = np.where(use, at, 0)
    c = np.where(use, col[at], -1)
    use = (c >= 0) & (status[c] != DELETED)
    w = np.where(use, val[at], F(0))
    x = np.where(use, val[at] * src[c], F(0))
    h = 32
    while h:
        w = w[:, :h] + w[:, h:2 * h]
        x = x[:, :h] + x[:, h:2 * h]
        h //= 2
    w, x = w[:, 0], x[:, 0]
    out = np.where(w > F(1e-10), x / np.where(w > F(1e-10), w, F(1)), src[front])
    return np.clip(out, F(0), F(1)).astype(F), np.where(use, c, -1)


def propagate(row, col, val, labels, status, gt, affected, delta, limit):
    buf, aff = [labels.copy(), labels.copy()], affected.copy()
    free = (status == ACTIVE) & (gt < 0)
    front, k = np.nonzero(free & (aff == 1))[0], 0
    while front.size and k < limit:
        src, dst = buf[k & 1], buf[1 - (k & 1)]
        nl, c = new_labels(row, col, val, src, status, front)
        dst[front] = nl
        moved = np.abs(nl - src[front]) > F(delta)
        hit = c[moved].ravel()
        hit = hit[hit >= 0]
        aff = np.zeros_like(aff)
        aff[front[moved]] = 1
        aff[hit[gt[hit] < 0]] = 1
        front = np.nonzero(free & (aff == 1))[0]
        k += 1
    out = buf[k & 1].copy()
    out[gt == 0], out[gt == 1] = 0, 1
    return out, aff, k


@pytest.mark.gpu
@pytest.mark.parametrize("n", [3706144, 3706145])  # owned rows, lists
@pytest.mark.parametrize("limit", [1, 7])
def test_propagation_launcher_around_its_limit(gpu, large, n, limit):
    g = cut(large, n)
    want = propagate(*g, 1e-3, limit)
    row, col, val, labels, status, gt, affected = g
    d = [DeviceArray(x) for x in (row, col, val, labels, labels, status, gt, affected)]
    used = ctypes.c_int(-1)
    N.check(N.lib().dlp_iterative_propagation(*[x.ptr for x in d], n, ctypes.c_float(1e-3), limit, ctypes.byref(used),
                                              None))
    assert used.value == want[2]
    assert d[3].get().tobytes() == want[0].tobytes()
    np.testing.assert_array_equal(d[7].get(), want[1])


@pytest.mark.gpu
@pytest.mark.parametrize("frontier", [20, 200])  # one block alone, the whole grid
def test_propagation_launcher_over_lists_small_frontiers(gpu, large, frontier):
    row, col, val, labels, status, gt, _ = large
    affected = np.zeros(labels.size, np.int32)
    affected[np.random.default_rng(frontier).integers(1, labels.size, frontier)] = 1
    want = propagate(row, col, val, labels, status, gt, affected, 0.2, 30)
    assert want[2] > 2
    d = [DeviceArray(x) for x in (row, col, val, labels, labels, status, gt, affected)]
    used = ctypes.c_int(-1)
    N.check(N.lib().dlp_iterative_propagation(*[x.ptr for x in d], labels.size, ctypes.c_float(0.2), 30,
                                              ctypes.byref(used), None))
    assert used.value == want[2]
    assert d[3].get().tobytes() == want[0].tobytes()
    np.testing.assert_array_equal(d[7].get(), want[1])


@pytest.mark.gpu
@pytest.mark.parametrize("n,limit", [(3400000, 3), (3706145, 1), (3706145, 6)])  # owned rows, lists, lists
def test_recompute_launcher_on_large_graphs(gpu, oracle, large, n, limit):
    row, col, val, labels, status, gt, _ = cut(large, n)
    labels = np.where(gt >= 0, gt, labels).astype(F)
    want, passes, _ = oracle.irlp(n, row, col, val, status, gt, labels, delta=1e-3, max_iterations=limit, threads=8)
    d = [DeviceArray(x) for x in (row, col, val, labels, status, gt)]
    used = ctypes.c_int(-1)
    N.check(N.lib().dlp_irlp(*[x.ptr for x in d], n, ctypes.c_float(1e-3), limit, ctypes.byref(used), None))
    assert used.value == passes
    assert d[3].get().tobytes() == want.tobytes()
