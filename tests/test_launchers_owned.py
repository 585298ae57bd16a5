"""The propagation and recompute launchers on owned rows (csrc/launchers.cu)
against a plain restatement of the passes in fp32 (row sums in the 256-slot tree
order, IEEE division), bit for bit, where their paths change: vertex counts
around a tile, rows of more than 32 entries, frontiers below and above what one
block takes, vertices without ground truth that are not active, soft-deleted
entries, ground-truth labels that are not 0 or 1, and pass limits of 0, 1 and 2."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from labelpropcuda_gb300 import DeviceArray, Problem
from labelpropcuda_gb300 import _native as N

ACTIVE, DELETED, GT = 0, 1, 2
F = np.float32


def inputs(n, degree, affected, seed):
    p = Problem(n, degree, 1, seed, cache_dir="")
    rng = np.random.default_rng(seed)
    status = rng.choice([ACTIVE, DELETED, GT], size=n, p=[0.86, 0.06, 0.08]).astype(np.int32)
    gt = np.where((status == GT) & (rng.random(n) < 0.7), (p.true_labels >= 0.5).astype(np.int32), -1).astype(np.int32)
    labels = rng.random(n, dtype=np.float32)
    col = p.col_ind.copy()
    col[(status[col] == DELETED) & (rng.random(col.size) < 0.5)] = -1
    return p.row_ptr, col, p.values, labels, status, gt, (rng.random(n) < affected).astype(np.int32)


def new_label(row, col, val, src, status, u):
    """src/iterativePropagation.cu:126-168."""
    w, l = np.zeros(256, F), np.zeros(256, F)
    for i, e in enumerate(range(row[u], row[u + 1])):
        v = col[e]
        if v >= 0 and status[v] != DELETED:
            assert i < 256
            w[i] = val[e]
            l[i] = F(val[e]) * F(src[v])
    h = 128
    while h:
        w[:h] += w[h:2 * h]
        l[:h] += l[h:2 * h]
        h //= 2
    x = l[0] / w[0] if w[0] > F(1e-10) else src[u]
    return F(min(max(x, F(0)), F(1)))


def propagate(row, col, val, labels, status, gt, affected, delta, limit):
    buf, aff = [labels.copy(), labels.copy()], affected.copy()
    front = [v for v in range(labels.size) if aff[v] == 1 and status[v] == ACTIVE and gt[v] < 0]
    k = 0
    while front and k < limit:
        src, dst = buf[k & 1], buf[1 - (k & 1)]
        marks = set()
        for u in front:
            nl = new_label(row, col, val, src, status, u)
            dst[u] = nl
            if abs(nl - src[u]) > F(delta):
                marks.add(u)
                marks.update(int(v) for v in col[row[u]:row[u + 1]]
                             if v >= 0 and status[v] != DELETED and gt[v] < 0)
        front = [v for v in sorted(marks) if status[v] == ACTIVE and gt[v] < 0]
        aff = np.zeros_like(aff)
        aff[list(marks)] = 1
        k += 1
    out = buf[k & 1].copy()
    out[gt == 0], out[gt == 1] = 0, 1
    return out, aff, k


def recompute(row, col, val, labels, status, gt, delta, limit):
    """src/validation.cu:47-139, :169-197."""
    buf, k = [labels.copy(), labels.copy()], 0
    while k < limit:
        src, dst = buf[k & 1], buf[1 - (k & 1)]
        moved = False
        for u in range(labels.size):
            if gt[u] < 0 and status[u] == ACTIVE:
                dst[u] = new_label(row, col, val, src, status, u)
                moved |= bool(abs(dst[u] - src[u]) > F(delta))
            else:
                dst[u] = 0 if gt[u] == 0 else 1 if gt[u] == 1 else src[u]
        k += 1
        if not moved:
            break
    return buf[k & 1], k


CASES = [(31, 4, 0.5, 60), (33, 4, 0.5, 2), (64, 3, 1.0, 1), (700, 34, 0.02, 8), (1500, 5, 0.7, 12), (300, 9, 0.3, 0),
         (2000, 3, 0.05, 40)]


@pytest.mark.gpu
@pytest.mark.parametrize("entry", ["dlp_iterative_propagation", "dlp_iterative_propagation_noalloc"])
@pytest.mark.parametrize("n,degree,affected,limit", CASES)
def test_propagation_matches_restatement(gpu, entry, n, degree, affected, limit):
    row, col, val, labels, status, gt, aff = inputs(n, degree, affected, n + degree)
    want = propagate(row, col, val, labels, status, gt, aff, 1e-3, limit)
    d = [DeviceArray(x) for x in (row, col, val, labels, labels, status, gt, aff)]
    used = ctypes.c_int(-1)
    N.check(getattr(N.lib(), entry)(*[x.ptr for x in d], n, ctypes.c_float(1e-3), limit, ctypes.byref(used), None))
    assert used.value == want[2]
    assert d[3].get().tobytes() == want[0].tobytes()
    np.testing.assert_array_equal(d[7].get(), want[1])


@pytest.mark.gpu
@pytest.mark.parametrize("n,degree,limit", [(31, 4, 60), (33, 4, 1), (64, 3, 2), (400, 34, 5), (1500, 5, 6), (300, 9, 0)])
def test_recompute_matches_restatement(gpu, n, degree, limit):
    row, col, val, labels, status, gt, _ = inputs(n, degree, 0.0, n + degree)
    want = recompute(row, col, val, labels, status, gt, 1e-3, limit)
    d = [DeviceArray(x) for x in (row, col, val, labels, status, gt)]
    used = ctypes.c_int(-1)
    N.check(N.lib().dlp_irlp(*[x.ptr for x in d], n, ctypes.c_float(1e-3), limit, ctypes.byref(used), None))
    assert used.value == want[1]
    assert d[3].get().tobytes() == want[0].tobytes()


@pytest.mark.gpu
@pytest.mark.parametrize("n,degree,limit", [(70, 60, 3), (600, 100, 6), (5000, 34, 2)])
def test_long_rows_are_dealt_out(gpu, n, degree, limit):
    """Most rows of more than 32 entries, in blocks of one tile and of two."""
    row, col, val, labels, status, gt, aff = inputs(n, degree, 0.6, n + degree)
    for entry in ("dlp_iterative_propagation", "dlp_irlp"):
        d = [DeviceArray(x) for x in (row, col, val, labels, labels, status, gt, aff)]
        used = ctypes.c_int(-1)
        if entry == "dlp_irlp":
            want = recompute(row, col, val, labels, status, gt, 1e-3, limit)
            N.check(N.lib().dlp_irlp(*[d[i].ptr for i in (0, 1, 2, 3, 5, 6)], n, ctypes.c_float(1e-3), limit,
                                     ctypes.byref(used), None))
        else:
            want = propagate(row, col, val, labels, status, gt, aff, 1e-3, limit)
            N.check(N.lib().dlp_iterative_propagation(*[x.ptr for x in d], n, ctypes.c_float(1e-3), limit,
                                                      ctypes.byref(used), None))
            np.testing.assert_array_equal(d[7].get(), want[1])
        assert used.value == want[-1]
        assert d[3].get().tobytes() == want[0].tobytes()
