"""Launchers, a session and an allocation-free call again after cudaDeviceReset (which
ends only this process's context), in a process of its own."""
from __future__ import annotations

import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

CHILD = r"""
import ctypes
import numpy as np
import labelpropcuda_gb300 as dlp
from labelpropcuda_gb300 import _native as N

n = 3001
p = dlp.Problem(n, 5, 2, 1, cache_dir="")
rng = np.random.default_rng(1)
status = rng.choice([0, 1, 2], size=n, p=[.88, .06, .06]).astype(np.int32)
gt = np.where(status == 2, (p.true_labels >= .5).astype(np.int32), -1).astype(np.int32)
labels, affected = rng.random(n, dtype=np.float32), np.ones(n, np.int32)


def run():
    out = []
    d = [dlp.DeviceArray(x) for x in (p.row_ptr, p.col_ind, p.values, labels, labels, status, gt, affected)]
    used = ctypes.c_int(0)
    for entry in ("dlp_iterative_propagation", "dlp_iterative_propagation_noalloc"):
        d[3].set(labels)
        d[7].set(affected)
        N.check(getattr(N.lib(), entry)(*[x.ptr for x in d], n, ctypes.c_float(1e-4), 30, ctypes.byref(used), None))
        out.append(d[3].get())
    d[3].set(labels)
    N.check(N.lib().dlp_irlp(*[d[i].ptr for i in (0, 1, 2, 3, 5, 6)], n, ctypes.c_float(1e-4), 30, ctypes.byref(used),
                             None))
    out.append(d[3].get())
    for x in d:
        x.free()
    s = dlp.Session.from_problem(p, max_iterations=50)
    for b, batch in enumerate(p.batches):
        s.apply(b, batch)
    out.append(s.labels())
    s.close()
    return out


runtime = ctypes.CDLL("libcudart.so.13")
first = run()
for _ in range(2):
    assert runtime.cudaDeviceReset() == 0
    assert all(a.tobytes() == b.tobytes() for a, b in zip(first, run()))
print("same")
"""


@pytest.mark.gpu
def test_calls_after_a_device_reset(gpu):
    out = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.strip() == "same", out.stderr[-2000:]
