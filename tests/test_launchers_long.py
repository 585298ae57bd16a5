"""The propagation launcher (csrc/launchers.cu) over more passes than a row's
visit counter and a stint's pass limit hold, with rows of more than 32 entries
in the same block."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from labelpropcuda_gb300 import DeviceArray
from labelpropcuda_gb300 import _native as N

F = np.float32


@pytest.mark.gpu
def test_rows_updated_more_often_than_a_counter_holds(gpu):
    """More than 1,024 vertices per block. In the first 151 tiles (a block each):
    a row of 33 entries that a wave along a path reaches after some 34,000
    passes; two vertices that swap their labels and settle only shortly before,
    after more than 32,768 updates; and two that swap theirs for ever. Nothing
    may touch the settled ones again, which shows in the buffer that the last
    pass leaves, if the numbers of passes have the right parity."""
    n, tiles, delta, eps = 160000, 151, F(0.5), F(2.06e-5)
    u, v, settled = F(1), F(0), 0  # u, v after `settled` passes
    while True:
        one = F(1) + eps
        nu, nv = F(F(v + eps * F(0.5)) / one), F(F(u + eps * F(0.5)) / one)
        old, settled = (u, v), settled + 1
        moved = abs(nu - u) > delta
        assert moved == (abs(nv - v) > delta)
        u, v = nu, nv
        if not moved:
            break
    assert settled > 32769
    length, limit = settled + 300, settled + 305
    rows: list[list[tuple[int, float]]] = [[] for _ in range(n)]
    labels, affected = np.full(n, 0.25, F), np.zeros(n, np.int32)
    gt, status = np.full(n, -1, np.int32), np.zeros(n, np.int32)
    half = n - 1  # a ground-truth vertex whose label reads as 0.5
    gt[half], status[half], labels[half] = 0, 2, 0.5
    path = np.arange(32 * tiles, 32 * tiles + length + 1)
    for a, b in zip(path[:-1].tolist(), path[1:].tolist()):
        rows[b].append((a, 1.0))
        rows[a].append((b, 0.0))
    labels[path], labels[path[0]], affected[path[1]] = 0, 1, 1
    wide = [32 * t for t in range(tiles)]
    for t, w in enumerate(wide):
        rows[w] = [(n - 2 - i, 1.0) for i in range(33)]
        rows[int(path[-1])].append((w, 0.0))
        a, b, c, d, e, f = range(w + 1, w + 7)
        rows[a], rows[b] = [(b, 1.0), (half, float(eps))], [(a, 1.0), (half, float(eps))]
        for x, y in ((c, d), (e, f)):
            rows[x], rows[y] = [(y, 1.0)], [(x, 1.0)]
        labels[[a, c, e]], labels[[b, d, f]] = 1, 0
        affected[a:f + 1] = 1
    row = np.zeros(n + 1, np.int32)
    row[1:] = np.cumsum([len(r) for r in rows])
    col = np.array([x for r in rows for x, _ in r], np.int32)
    val = np.array([x for r in rows for _, x in r], F)
    want = labels.copy()
    want[half] = 0
    want[path] = 1
    buffers = {settled & 1: (u, v), (settled & 1) ^ 1: old}
    # an update in the wave's pass would land in the older buffer, which the last pass leaves
    assert (length - settled) % 2 == 0 and (limit - length) % 2 == 1
    swapped = limit & 1
    for w in wide:
        want[w + 1], want[w + 2] = buffers[limit & 1]
        for x in (w + 3, w + 5):
            want[x], want[x + 1] = (0, 1) if swapped else (1, 0)
    d = [DeviceArray(x) for x in (row, col, val, labels, labels, status, gt, affected)]
    used = ctypes.c_int(-1)
    N.check(N.lib().dlp_iterative_propagation(*[x.ptr for x in d], n, ctypes.c_float(delta), limit, ctypes.byref(used),
                                              None))
    assert used.value == limit
    got = d[3].get()
    assert got.tobytes() == want.tobytes(), np.nonzero(got != want)[0][:20]
