"""The work that users of this library have it do, as measurable cases.

Three kinds of programs use the library, and each case is one of them:

  replay     a Session (one resident graph) that takes a stream of update
             batches one at a time: the plain per-batch path of runDynLP;
  mix        an Engine that advances many resident graphs by one batch each per
             step;
  serve      a Server that takes the requests of many resident graphs from a
             queue;
  update     the reference-layout step launchers on the caller's own device
             arrays, one batch: deletion marks, sparsification, components and
             label initialisation;
  propagate  the reference-layout propagation launcher;
  irlp       the full recompute of all labels on a snapshot.

Inputs come from a seed. The replay, mix, serve and irlp inputs are the
library's own synthetic problems (a spanning path plus uniform edges, 90% new
vertices, 1% ground truth and 9% deletions per batch); the launcher inputs are
the same kind of graph, built here on the GPU because they are large.
"""
from __future__ import annotations

import concurrent.futures
import ctypes

import numpy as np
import torch

import labelpropcuda_gb300 as dlp
from labelpropcuda_gb300 import _native as N

ACTIVE, DELETED, GROUND_TRUTH = 0, 1, 2

# What a batch's statistics hold besides times and counts that depend on how
# threads race (hook_rounds).
STATS = ("iterations", "num_components", "num_sub_edges", "hook_edges", "seed_frontier", "seed_marks",
         "affected_edges", "frontier_visits", "correct", "total", "init_branch", "hook_truncated", "dirty_rows",
         "dirty_entries")


def listed():
    return [
        # The smallest real stream: 200-vertex updates, where launches, barriers and the host path count.
        {"name": "replay_1k", "kind": "replay", "n": 1000, "degree": 3, "batches": 5, "max_iterations": 2000,
         "semantics": "ref", "arithmetic": "ieee", "device_batches": False},
        # The plain path at the small configuration: 5,000 vertices, 10 batches, default pass limit.
        {"name": "replay_5k", "kind": "replay", "n": 5000, "degree": 5, "batches": 10, "max_iterations": 100000,
         "semantics": "ref", "arithmetic": "ieee", "device_batches": False},
        # The default configuration: 50,000 vertices, 10 batches, long propagation on small frontiers.
        {"name": "replay_50k", "kind": "replay", "n": 50000, "degree": 5, "batches": 10, "max_iterations": 100000,
         "semantics": "ref", "arithmetic": "ieee", "device_batches": False},
        # A large graph whose frontiers fill the GPU.
        {"name": "replay_500k", "kind": "replay", "n": 500000, "degree": 7, "batches": 10, "max_iterations": 1000,
         "semantics": "ref", "arithmetic": "ieee", "device_batches": False},
        # The documented semantics (full affected set) with the reference's division, batches already on the device.
        {"name": "replay_spec_20k", "kind": "replay", "n": 20000, "degree": 7, "batches": 8, "max_iterations": 5000,
         "semantics": "spec", "arithmetic": "fast", "device_batches": True},
        # Many graphs of uneven size advanced together, one launch per step.
        {"name": "mix_32", "kind": "mix", "graphs": 32, "smallest": 1000, "largest": 100000, "batches": 10,
         "max_iterations": 1000},
        # The request queue of a server: every batch of 16 graphs, sliced steps.
        {"name": "serve_16", "kind": "serve", "graphs": 16, "smallest": 10000, "largest": 100000, "batches": 6,
         "max_iterations": 2000},
        # One small batch through the step launchers: call overhead.
        {"name": "update_1k", "kind": "update", "n": 1000, "degree": 5, "batches": 10},
        # One large batch through the step launchers: memory traffic.
        {"name": "update_2m", "kind": "update", "n": 2000003, "degree": 7, "batches": 10},
        # Propagation from a caller's own arrays at the default size, and on a large graph.
        {"name": "propagate_50k", "kind": "propagate", "n": 50000, "degree": 5, "affected": 0.02, "deleted": 0.06,
         "max_iterations": 2000, "no_alloc": False},
        {"name": "propagate_1m", "kind": "propagate", "n": 1000000, "degree": 7, "affected": 0.05, "deleted": 0.06,
         "max_iterations": 300, "no_alloc": True},
        # Full recompute of the labels after the last batch.
        {"name": "irlp_100k", "kind": "irlp", "n": 100000, "degree": 5, "batches": 10, "max_iterations": 1000},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["replay", "replay", "replay", "mix", "serve", "update", "propagate", "propagate", "irlp"])
    if kind == "replay":
        n = _log_uniform(rng, 1000, 500000)
        return {"kind": kind, "n": n, "degree": rng.choice([3, 4, 5, 6, 7]), "batches": rng.randint(3, 10),
                "max_iterations": _log_uniform(rng, 500, 5000 if n <= 50000 else 1000),
                "semantics": rng.choice(["ref", "ref", "spec"]), "arithmetic": rng.choice(["ieee", "ieee", "fast"]),
                "device_batches": rng.random() < 0.5}
    if kind in ("mix", "serve"):
        smallest = _log_uniform(rng, 1000, 10000)
        return {"kind": kind, "graphs": rng.randint(2, 32 if kind == "mix" else 16), "smallest": smallest,
                "largest": _log_uniform(rng, smallest, 100000), "batches": rng.randint(3, 10 if kind == "mix" else 6),
                "max_iterations": _log_uniform(rng, 200, 1000)}
    if kind == "update":
        return {"kind": kind, "n": _log_uniform(rng, 500, 2000003), "degree": rng.choice([3, 5, 7, 12]),
                "batches": rng.randint(2, 20)}
    if kind == "propagate":
        n = _log_uniform(rng, 1000, 1000000)
        return {"kind": kind, "n": n, "degree": rng.choice([3, 5, 7, 12]), "affected": round(rng.uniform(0.002, 0.1), 4),
                "deleted": round(rng.uniform(0.0, 0.1), 4), "max_iterations": _log_uniform(rng, 50, 300 if n > 200000 else 2000),
                "no_alloc": rng.random() < 0.3}
    return {"kind": kind, "n": _log_uniform(rng, 1000, 100000), "degree": rng.choice([3, 5, 7]),
            "batches": rng.randint(2, 10), "max_iterations": _log_uniform(rng, 100, 1000)}


def work(case):
    """Each input read once and each output written once; two operations (a
    multiply-add) per directed edge of the graph and per label of the result.
    The number of passes a propagation takes follows from the data and is not
    counted."""
    if case["kind"] in ("mix", "serve"):
        k, lo, hi = case["graphs"], case["smallest"], case["largest"]
        sizes = _sizes(k, lo, hi)
        n, m = sum(s for s, _ in sizes), sum(s * d for s, d in sizes)
    else:
        n, m = case["n"], case["n"] * case["degree"]
    if case["kind"] in ("replay", "mix", "serve"):
        # adjacency (8 B an entry), batch edges (12 B, half the entries), vertex ids, labels out
        return {"bytes": 8 * m + 6 * m + 8 * n + 4 * n, "flops": 2 * m}
    if case["kind"] == "update":
        new = m // (2 * case["batches"])
        # the caller's arrays come in and go out once (columns, status, marks, labels), the batch's edges once
        return {"bytes": 8 * m + 4 * n * 8 + 12 * new + 16 * new, "flops": 2 * new}
    return {"bytes": 8 * m + 4 * n * 7, "flops": 2 * m}


# ------------------------------------------------------------------ inputs --

def _sizes(count, smallest, largest):
    """Sizes spread evenly over the logarithm of the range, degrees 3, 5 and 7 in turn."""
    out = []
    for i in range(count):
        f = i / (count - 1) if count > 1 else 1.0
        out.append((int(round(smallest * (largest / smallest) ** f)), (3, 5, 7)[i % 3]))
    return out


def _problems(sizes, batches, seed):
    make = lambda x: dlp.Problem(x[1][0], x[1][1], batches, (seed * 1009 + x[0]) & 0x7fffffff, cache_dir="")
    with concurrent.futures.ThreadPoolExecutor(8) as pool:
        return list(pool.map(make, enumerate(sizes)))


def _graph(n, degree, seed):
    """A spanning path over a random order plus uniform edges, symmetric, rows
    sorted by column, weights by class; on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    rand = lambda k: torch.rand(k, generator=g, device="cuda")
    truth = (torch.randperm(n, generator=g, device="cuda") >= n // 2).int()
    path = torch.randperm(n, generator=g, device="cuda")
    extra = max(0, n * degree // 2 - (n - 1))
    a = torch.cat([path[:-1], torch.randint(0, n, (extra,), generator=g, device="cuda")])
    b = torch.cat([path[1:], torch.randint(0, n, (extra,), generator=g, device="cuda")])
    a, b = torch.minimum(a, b), torch.maximum(a, b)
    key = torch.unique(a * n + b)
    a, b = key // n, key % n
    a, b = a[a != b], b[a != b]
    w = torch.where(truth[a] == truth[b], 0.5 + 0.5 * rand(a.numel()), 0.01 + 0.49 * rand(a.numel()))
    return truth, a, b, w, g


def _csr(n, a, b, w):
    """Both directions of the edges (a, b, w) as CSR with sorted rows."""
    key = torch.cat([a * n + b, b * n + a])
    key, order = torch.sort(key)
    val = torch.cat([w, w])[order]
    row = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    row[1:] = torch.cumsum(torch.bincount(key // n, minlength=n), 0)
    return row.int(), (key % n).int(), val.contiguous()


def _prepare_update(case, seed):
    n = case["n"]
    truth, a, b, w, g = _graph(n, case["degree"], seed)
    rand = lambda k: torch.rand(k, generator=g, device="cuda")
    order = torch.randperm(n, generator=g, device="cuda")
    arrival = torch.empty(n, dtype=torch.int64, device="cuda")
    arrival[order] = torch.arange(n, device="cuda") * case["batches"] // n
    now = case["batches"] // 2                       # the batch that is applied
    keep = torch.maximum(arrival[a], arrival[b]) <= now
    row, col, val = _csr(n, a[keep], b[keep], w[keep])
    new_edge = torch.maximum(arrival[a], arrival[b]) == now
    is_new = (arrival == now).int()
    inserted = order[arrival[order] == now].int()
    present = arrival <= now
    gt = torch.where(present & (rand(n) < 0.01), truth, torch.full_like(truth, -1))
    status = torch.where(present, ACTIVE, DELETED).int()
    status[gt >= 0] = GROUND_TRUTH
    deleted = torch.nonzero((arrival < now) & (gt < 0) & (rand(n) < 0.02)).flatten().int()
    labels = torch.where(gt >= 0, gt.float(), (0.2 + 0.6 * truth.float() + 0.4 * (rand(n) - 0.5)).float())
    s = {"n": n, "row": row, "col": col, "val": val, "status": status, "deleted": deleted, "inserted": inserted,
         "is_new": is_new, "gt": gt, "labels": labels, "src": a[new_edge].int(), "dst": b[new_edge].int(),
         "weight": w[new_edge].float().contiguous(), "tau": float(w.double().mean())}
    s["status_now"], s["labels_now"] = (torch.empty_like(s[k]) for k in ("status", "labels"))
    s["marks"], s["component"] = (torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(2))
    # buffers for the largest graph of this size and degree, as a program keeps them over its batches
    room = 2 * max(n - 1, n * case["degree"] // 2)
    s["col_now"] = torch.full((room,), -1, dtype=torch.int32, device="cuda")
    s["sub_row"] = torch.empty(n + 1, dtype=torch.int32, device="cuda")
    s["sub_col"] = torch.zeros(room, dtype=torch.int32, device="cuda")
    s["sub_val"] = torch.zeros(room, dtype=torch.float32, device="cuda")
    return s


def _prepare_propagate(case, seed):
    n = case["n"]
    truth, a, b, w, g = _graph(n, case["degree"], seed)
    rand = lambda k: torch.rand(k, generator=g, device="cuda")
    row, col, val = _csr(n, a, b, w)
    x = rand(n)
    status = torch.full((n,), ACTIVE, dtype=torch.int32, device="cuda")
    status[x < case["deleted"]] = DELETED
    status[x > 0.94] = GROUND_TRUTH
    gt = torch.where(status == GROUND_TRUTH, truth, torch.full_like(truth, -1))
    # settled labels lean to their class; a tenth of the vertices is new and starts undecided
    labels = (0.2 + 0.6 * truth.float() + 0.4 * (rand(n) - 0.5)).float()
    labels[rand(n) < 0.1] = 0.5
    labels = torch.where(gt >= 0, gt.float(), labels).contiguous()
    col = torch.where(status[col.long()] == DELETED, torch.full_like(col, -1), col).contiguous()
    affected = (rand(n) < case["affected"]).int()
    return {"n": n, "row": row, "col": col, "val": val, "labels": labels, "status": status, "gt": gt,
            "affected": affected, "labels_now": torch.empty_like(labels), "buffer": torch.empty_like(labels),
            "affected_now": torch.empty_like(affected), "max_iterations": case["max_iterations"],
            "call": "dlp_iterative_propagation_noalloc" if case["no_alloc"] else "dlp_iterative_propagation"}


def _prepare_irlp(case, seed):
    p = dlp.Problem(case["n"], case["degree"], case["batches"], seed & 0x7fffffff, cache_dir="")
    snap = dlp.irlp_snapshot(p)
    s = {k: torch.from_numpy(v).cuda() for k, v in (("row", snap.row_ptr), ("col", snap.col_ind), ("val", snap.values),
                                                    ("labels", snap.labels), ("status", snap.status),
                                                    ("gt", snap.gt_class))}
    s.update(n=case["n"], labels_now=torch.empty_like(s["labels"]), max_iterations=case["max_iterations"])
    return s


def _options(case):
    return {"max_iterations": case["max_iterations"],
            "semantics": dlp.SEMANTICS_SPEC if case.get("semantics") == "spec" else dlp.SEMANTICS_REF,
            "arithmetic": dlp.ARITH_REFERENCE_FAST_MATH if case.get("arithmetic") == "fast" else dlp.ARITH_IEEE}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "replay":
        p = _problems([(case["n"], case["degree"])], case["batches"], seed)[0]
        batches = [dlp.DeviceBatch(b) for b in p.batches] if case["device_batches"] else p.batches
        s = {"session": dlp.Session.from_problem(p, **_options(case)), "batches": batches}
    elif kind in ("mix", "serve"):
        probs = _problems(_sizes(case["graphs"], case["smallest"], case["largest"]), case["batches"], seed)
        engine = dlp.Engine(len(probs), **_options(case))
        ids = [engine.add_problem(p) for p in probs]
        s = {"engine": engine, "ids": ids, "problems": probs}
        if kind == "serve":
            s["server"] = dlp.Server(engine)
            for gid, p in zip(ids, probs):
                s["server"].reserve(gid, p.batches)
    else:
        s = {"update": _prepare_update, "propagate": _prepare_propagate, "irlp": _prepare_irlp}[kind](case, seed)
    s["kind"] = kind
    return s


# ------------------------------------------------------------------- passes --

def _numbers(stats):
    return np.array([[int(x[k]) for k in STATS] for x in stats], dtype=np.int64)


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def _run_replay(s):
    """The stream from its first batch, host batches with their statistics
    awaited, device batches queued and their statistics read at the end."""
    sess = s["session"]
    sess.reset()
    if isinstance(s["batches"][0], dlp.DeviceBatch):
        for i, b in enumerate(s["batches"]):
            sess.apply_device(i, b)
        sess.synchronize()
        stats = [sess.stats(i) for i in range(len(s["batches"]))]
    else:
        stats = [sess.apply(i, b) for i, b in enumerate(s["batches"])]
    return {"labels": sess.labels(), "stats": _numbers(stats)}


def _labels(s):
    return np.concatenate([s["engine"].labels(g) for g in s["ids"]])


def _run_mix(s):
    for g in s["ids"]:
        s["engine"].reset_graph(g)
    stats = []
    for b in range(len(s["problems"][0].batches)):
        stats += s["engine"].step([(g, b, p.batches[b]) for g, p in zip(s["ids"], s["problems"])])
    return {"labels": _labels(s), "stats": _numbers(stats)}


def _run_serve(s):
    """Every request queued at once; the server works the queue off."""
    for g in s["ids"]:
        s["engine"].reset_graph(g)
    trace = [(0.0, g, b, p.batches[b]) for b in range(len(s["problems"][0].batches))
             for g, p in zip(s["ids"], s["problems"])]
    results, _ = s["server"].replay(trace)
    return {"labels": _labels(s), "stats": _numbers([r["stats"] for r in results])}


def _run_update(s):
    """A batch as the reference's driver applies it: the caller's arrays come
    in (device copies here), then the four structural steps."""
    L, stream, n = N.lib(), _stream(), s["n"]
    col, status, labels, marks = s["col_now"], s["status_now"], s["labels_now"], s["marks"]
    col[:s["col"].numel()].copy_(s["col"])
    status.copy_(s["status"])
    labels.copy_(s["labels"])
    marks.zero_()
    edges, inserted = s["src"].numel(), s["inserted"].numel()
    N.check(L.dlp_mark_deletions(_ptr(s["row"]), _ptr(col), _ptr(status), _ptr(marks), _ptr(s["deleted"]),
                                 s["deleted"].numel(), n, stream))
    nodes, kept, comps = ctypes.c_int(0), ctypes.c_int(0), ctypes.c_int(0)
    N.check(L.dlp_build_sparsified_subgraph(_ptr(s["row"]), _ptr(col), _ptr(s["val"]), _ptr(marks), _ptr(status),
                                            _ptr(s["src"]), _ptr(s["dst"]), _ptr(s["weight"]), edges,
                                            _ptr(s["inserted"]), inserted, _ptr(s["is_new"]), s["tau"],
                                            _ptr(s["sub_row"]), _ptr(s["sub_col"]), _ptr(s["sub_val"]),
                                            ctypes.byref(nodes), ctypes.byref(kept), stream))
    N.check(L.dlp_connected_components(_ptr(s["src"]), _ptr(s["dst"]), min(kept.value, edges), _ptr(s["inserted"]),
                                       inserted, _ptr(s["component"]), ctypes.byref(comps), n, stream))
    N.check(L.dlp_label_initialization(_ptr(s["row"]), _ptr(col), _ptr(s["val"]), _ptr(labels), _ptr(status),
                                       _ptr(s["component"]), comps.value, _ptr(s["inserted"]), inserted, _ptr(s["gt"]),
                                       n, stream))
    return {"col": col, "status": status, "marks": marks, "sub_col": s["sub_col"], "sub_val": s["sub_val"],
            "component": s["component"], "labels": labels, "kept": kept.value, "components": comps.value}


def _run_propagate(s):
    used = ctypes.c_int(0)
    labels, affected = s["labels_now"], s["affected_now"]
    labels.copy_(s["labels"])
    affected.copy_(s["affected"])
    N.check(getattr(N.lib(), s["call"])(_ptr(s["row"]), _ptr(s["col"]), _ptr(s["val"]), _ptr(labels), _ptr(s["buffer"]),
                                        _ptr(s["status"]), _ptr(s["gt"]), _ptr(affected), s["n"],
                                        ctypes.c_float(1e-4), s["max_iterations"], ctypes.byref(used), _stream()))
    return {"labels": labels, "affected": affected, "iterations": used.value}


def _run_irlp(s):
    used = ctypes.c_int(0)
    labels = s["labels_now"]
    labels.copy_(s["labels"])
    N.check(N.lib().dlp_irlp(_ptr(s["row"]), _ptr(s["col"]), _ptr(s["val"]), _ptr(labels), _ptr(s["status"]),
                             _ptr(s["gt"]), s["n"], ctypes.c_float(1e-4), s["max_iterations"], ctypes.byref(used),
                             _stream()))
    return {"labels": labels, "iterations": used.value}


def run(state):
    return {"replay": _run_replay, "mix": _run_mix, "serve": _run_serve, "update": _run_update,
            "propagate": _run_propagate, "irlp": _run_irlp}[state["kind"]](state)


# ------------------------------------------------------------------ 64 bits --

def _exact_update(s):
    """Initial labels of the inserted vertices: the weighted share of class 1
    among the ground-truth neighbours of each vertex's component."""
    h = {k: s[k].cpu().numpy() for k in ("row", "col", "val", "status", "deleted", "inserted", "gt", "labels", "src",
                                        "dst", "weight", "is_new")}
    n = s["n"]
    status = h["status"].copy()
    status[h["deleted"]] = DELETED
    rows = np.repeat(np.arange(n), np.diff(h["row"]))
    col = h["col"].astype(np.int64)
    gone = (status[rows] == DELETED) | (status[col] == DELETED)
    kept = int((h["is_new"][h["src"]].astype(bool) & h["is_new"][h["dst"]].astype(bool) &
                (h["weight"] > np.float32(s["tau"]))).sum())
    hooked = min(2 * kept, h["src"].size)
    a, b = h["src"][:hooked].astype(np.int64), h["dst"][:hooked].astype(np.int64)
    root = np.full(n, -1, np.int64)
    root[h["inserted"]] = h["inserted"]
    while True:  # smallest member of each component; -1 (not inserted) takes over what it touches
        low = np.minimum(root[a], root[b])
        was = root.copy()
        np.minimum.at(root, a, low)
        np.minimum.at(root, b, low)
        for x, y in ((a, low), (b, low)):
            own = was[x]
            np.minimum.at(root, own[own >= 0], y[own >= 0])
        while True:
            up = np.where(root >= 0, root[root], -1)
            if np.array_equal(up, root):
                break
            root = up
        if np.array_equal(root, was):
            break
    share = np.zeros((2, n))
    use = ~gone & (h["is_new"][rows] == 1) & (root[rows] >= 0) & (h["gt"][col] >= 0)
    np.add.at(share, (h["gt"][col[use]], root[rows[use]]), h["val"][use].astype(np.float64))
    labels = h["labels"].astype(np.float64)
    ins = h["inserted"]
    r = root[ins]
    den = share[0][r] + share[1][r]
    new = np.where((r >= 0) & (den > 1e-10), share[1][r] / np.where(den > 0, den, 1), 0.5)
    labels[ins] = np.where(h["gt"][ins] >= 0, h["gt"][ins], new)
    return {"labels": labels}


def _exact_passes(s, full, limit):
    """The label passes in 64 bits: every active vertex (`full`), or the
    frontier of the vertices whose neighbourhood moved, from two buffers that
    keep what a pass does not write. None once over `limit` entries are read."""
    h = {k: s[k].cpu().numpy() for k in ("row", "col", "val", "status", "gt", "labels")}
    n, row, col, val = s["n"], h["row"].astype(np.int64), h["col"].astype(np.int64), h["val"].astype(np.float64)
    val = np.where((col >= 0) & (h["status"][col] != DELETED), val, 0.0)
    free = (h["status"] == ACTIVE) & (h["gt"] < 0)
    buf = [h["labels"].astype(np.float64), h["labels"].astype(np.float64)]
    front = np.nonzero(free & (np.ones(n, bool) if full else s["affected"].cpu().numpy() == 1))[0]
    read = 0
    for k in range(s["max_iterations"]):
        if not front.size:
            break
        src, dst = buf[k & 1], buf[1 - (k & 1)]
        length = row[front + 1] - row[front]
        read += int(length.sum())
        if read > limit:
            return None
        starts = np.cumsum(length) - length
        at = np.repeat(row[front] - starts, length) + np.arange(int(length.sum()))
        owner = np.repeat(np.arange(front.size), length)
        total = np.bincount(owner, val[at], front.size)
        pull = np.bincount(owner, val[at] * src[col[at]], front.size)
        new = np.clip(np.where(total > 1e-10, pull / np.where(total > 0, total, 1), src[front]), 0, 1)
        moved = np.abs(new - src[front]) > np.float32(1e-4)
        if full:
            dst[:] = np.where(h["gt"] >= 0, h["gt"], src)
        dst[front] = new
        if full:
            if not moved.any():
                k += 1
                return {"labels": dst}
            continue
        hit = col[at][moved[owner] & (val[at] > 0)]
        front = np.unique(np.concatenate([hit, front[moved]]))
        front = front[free[front]]
        if not front.size:
            return {"labels": np.where(h["gt"] >= 0, h["gt"], dst)}
    last = buf[s["max_iterations"] & 1]
    return {"labels": last if full else np.where(h["gt"] >= 0, h["gt"], last)}


def exact(case, seed):
    """Labels in 64 bits for one batch's structural steps, a propagation and a
    recompute. A stream of batches has no such value: how many passes a batch
    takes follows from the last bits of the labels (propagation stops at, or
    cycles around, the threshold), and the next batch starts from there."""
    if case["kind"] not in ("update", "propagate", "irlp"):
        return None
    s = prepare(case, seed)
    if case["kind"] == "update":
        got = _exact_update(s)
        return dict.fromkeys(("col", "status", "marks", "sub_col", "sub_val", "component", "kept", "components")) | got
    got = _exact_passes(s, case["kind"] == "irlp", 600_000_000)
    return None if got is None else dict.fromkeys(("affected", "iterations") if case["kind"] == "propagate" else ("iterations",)) | got
