"""The step launchers that return nothing to the host (deletion marks, label
initialisation) as part of a CUDA graph, captured as the first calls of a process."""
from __future__ import annotations

import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

CHILD = r"""
import ctypes, sys
import torch
import labelpropcuda_gb300 as dlp
from labelpropcuda_gb300 import _native as N

inserted = int(sys.argv[1])
n = 3 * inserted
gen = torch.Generator(device="cuda").manual_seed(inserted)
rint = lambda lo, hi, k: torch.randint(lo, hi, (k,), generator=gen, device="cuda", dtype=torch.int32)
length = rint(0, 9, n)
row = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
row[1:] = torch.cumsum(length, 0)
m = int(row[-1])
given = {"col": rint(-1, n, m), "status": rint(0, 3, n), "affected": rint(0, 2, n),
         "labels": torch.rand(n, generator=gen, device="cuda")}
val = torch.rand(m, generator=gen, device="cuda")
deleted = torch.randperm(n, generator=gen, device="cuda")[:n // 50].int()
new = torch.randperm(n, generator=gen, device="cuda")[:inserted].int()
gt, comp, comps = rint(-9, 2, n), rint(-1, 7, n), 7
now = {k: v.clone() for k, v in given.items()}
p = lambda t: ctypes.c_void_p(t.data_ptr())


def both():
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    for k, v in given.items():
        now[k].copy_(v)
    N.check(N.lib().dlp_mark_deletions(p(row), p(now["col"]), p(now["status"]), p(now["affected"]), p(deleted),
                                       deleted.numel(), n, s))
    N.check(N.lib().dlp_label_initialization(p(row), p(now["col"]), p(val), p(now["labels"]), None, p(comp), comps,
                                             p(new), inserted, p(gt), n, s))


torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    both()
out = []
for run in (graph.replay, graph.replay, both):
    for v in now.values():
        v.zero_()
    run()
    torch.cuda.synchronize()
    out.append({k: v.clone() for k, v in now.items()})
for other in out[1:]:
    assert all(torch.equal(out[0][k], other[k]) for k in now)
assert not torch.equal(out[0]["labels"], given["labels"])
print("same")
"""


@pytest.mark.gpu
@pytest.mark.parametrize("inserted", [300, 40000])  # one block, several
def test_steps_without_results_can_be_captured(gpu, inserted):
    pytest.importorskip("torch")
    out = subprocess.run([sys.executable, "-c", CHILD, str(inserted)], cwd=ROOT, capture_output=True, text=True,
                         timeout=300)
    assert out.returncode == 0 and out.stdout.strip() == "same", out.stderr[-2000:]
