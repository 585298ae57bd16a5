"""Full-grid passes on owned rows (csrc/owner_pass.cuh), bit-exact against the
oracle with the one-block mode off: graphs of two tiles, of two tiles and a vertex,
rows of 8, 9, 32 and 33 entries, several graphs in one launch (with pass limits
that end at different launch passes), and blocks whose rows do not fit their
shared memory."""
from __future__ import annotations

import pytest

import labelpropcuda_gb300 as dlp
from parity_checks import EXACT_STATS, check_batch


@pytest.mark.gpu
@pytest.mark.parametrize("n,degree,sem", [(63, 4, dlp.SEMANTICS_REF), (64, 4, dlp.SEMANTICS_SPEC),
                                          (65, 9, dlp.SEMANTICS_REF), (400, 33, dlp.SEMANTICS_SPEC),
                                          (9700, 8, dlp.SEMANTICS_REF)])
def test_owned_passes_match_oracle(gpu, oracle, n, degree, sem):
    p = dlp.Problem(n, degree, 5, 3, cache_dir="")
    cap = 120
    orc = oracle.OracleRun.from_problem(p, semantics=sem, record=True, threads=4, max_iterations=cap)
    sess = dlp.Session.from_problem(p, semantics=sem, record=True, max_iterations=cap, small_frontier_solo=0)
    for b, batch in enumerate(p.batches):
        check_batch(b, sess.apply(b, batch), orc.apply(b, batch), sess, orc, oracle)


@pytest.mark.gpu
def test_owned_passes_rows_beyond_shared_memory(gpu, oracle):
    p = dlp.Problem(160000, 30, 3, 5, cache_dir="")  # 1,060 vertices, 32,000 entries per block
    cap = 25
    orc = oracle.OracleRun.from_problem(p, threads=0, max_iterations=cap)
    sess = dlp.Session.from_problem(p, max_iterations=cap, small_frontier_solo=0)
    for b, batch in enumerate(p.batches):
        got, want = sess.apply(b, batch), orc.apply(b, batch)
        for k in EXACT_STATS:
            assert got[k] == want[k], (b, k)
        assert sess.labels().tobytes() == orc.labels().tobytes(), b


@pytest.mark.gpu
def test_owned_passes_of_continued_batches(gpu, oracle):
    """Graphs that continue a batch beside graphs that start one: their pass
    numbers, buffers and pass limits differ within a launch."""
    probs = [dlp.Problem(n, d, 4, s, cache_dir="") for n, d, s in ((1500, 5, 1), (64, 3, 2), (3000, 7, 3))]
    cap = 90
    orcs = [oracle.OracleRun.from_problem(p, threads=4, max_iterations=cap) for p in probs]
    eng = dlp.Engine(len(probs), max_iterations=cap, small_frontier_solo=0)
    ids = [eng.add_problem(p) for p in probs]
    dev = [[dlp.DeviceBatch(b) for b in p.batches] for p in probs]
    nxt, step = [0] * len(probs), 0
    while any(x < 4 for x in nxt) or any(eng.in_progress(g) for g in ids):
        start = [i for i, g in enumerate(ids) if nxt[i] < 4 and not eng.in_progress(g) and (step + i) % 2 == 0]
        done, _ = eng.step_sliced([(ids[i], nxt[i], dev[i][nxt[i]]) for i in start], pass_budget=37)
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
@pytest.mark.parametrize("n", [3706144, 3706145])  # the most that 151 blocks own, and one more
def test_owned_passes_up_to_the_limit(gpu, oracle, n):
    p = dlp.Problem(n, 3, 200, 5, cache_dir="")
    orc = oracle.OracleRun.from_problem(p, threads=0, max_iterations=6)
    sess = dlp.Session.from_problem(p, max_iterations=6, small_frontier_solo=0)
    for b, batch in enumerate(p.batches[:3]):
        got, want = sess.apply(b, batch), orc.apply(b, batch)
        for k in EXACT_STATS:
            assert got[k] == want[k], (b, k)
        assert sess.labels().tobytes() == orc.labels().tobytes(), b


@pytest.mark.gpu
def test_more_graphs_than_a_block_has_room_for(gpu, oracle):
    """As many vertices as the blocks own for one graph, but the 600 graphs' own
    records do not fit beside them."""
    p = dlp.Problem(6000, 3, 4, 9, cache_dir="")
    orc = oracle.OracleRun.from_problem(p, threads=4, max_iterations=8)
    eng = dlp.Engine(600, max_iterations=8, small_frontier_solo=0)
    ids = [eng.add_problem(p) for _ in range(600)]
    for b, batch in enumerate(p.batches):
        want, got = orc.apply(b, batch), eng.step([(g, b, batch) for g in ids])
        for g, st in zip(ids, got):
            for k in EXACT_STATS:
                assert st[k] == want[k], (g, b, k)
        for g in (ids[0], ids[299], ids[599]):
            assert eng.labels(g).tobytes() == orc.labels().tobytes(), (g, b)


@pytest.mark.gpu
def test_owned_passes_partial_tile_beyond_shared_memory(gpu, oracle):
    """At most 1,024 vertices per block (a tile per warp), a last tile of 17
    vertices, and about 30 entries per row, more than the blocks have room for."""
    p = dlp.Problem(150001, 30, 3, 6, cache_dir="")
    cap = 25
    orc = oracle.OracleRun.from_problem(p, threads=0, max_iterations=cap)
    sess = dlp.Session.from_problem(p, max_iterations=cap, small_frontier_solo=0)
    for b, batch in enumerate(p.batches):
        got, want = sess.apply(b, batch), orc.apply(b, batch)
        for k in EXACT_STATS:
            assert got[k] == want[k], (b, k)
        assert sess.labels().tobytes() == orc.labels().tobytes(), b


@pytest.mark.gpu
@pytest.mark.parametrize("solo", [0, 7])
def test_lists_before_owned_rows(gpu, oracle, solo):
    """From 1.75 million vertices on, a launch runs 8 full-grid passes over lists
    before it loads rows."""
    p = dlp.Problem(1800001, 4, 150, 5, cache_dir="")
    orc = oracle.OracleRun.from_problem(p, threads=0, max_iterations=20)
    sess = dlp.Session.from_problem(p, max_iterations=20, small_frontier_solo=solo)
    for b, batch in enumerate(p.batches[:4]):
        got, want = sess.apply(b, batch), orc.apply(b, batch)
        for k in EXACT_STATS:
            assert got[k] == want[k], (b, k)
        assert sess.labels().tobytes() == orc.labels().tobytes(), b


@pytest.mark.gpu
@pytest.mark.parametrize("solo", [0, 7])
def test_launches_of_few_passes_among_longer_ones(gpu, oracle, solo):
    """At most 3 passes run over lists, more on owned rows: batches that go through
    both, with pass limits that end in either."""
    probs = [dlp.Problem(n, d, 4, s, cache_dir="") for n, d, s in ((1500, 5, 1), (64, 3, 2), (3000, 34, 3))]
    cap, budgets = 61, (2, 5, 3, 1, 4)
    orcs = [oracle.OracleRun.from_problem(p, threads=4, max_iterations=cap) for p in probs]
    eng = dlp.Engine(len(probs), max_iterations=cap, small_frontier_solo=solo)
    ids = [eng.add_problem(p) for p in probs]
    dev = [[dlp.DeviceBatch(b) for b in p.batches] for p in probs]
    nxt, step = [0] * len(probs), 0
    while any(x < 4 for x in nxt) or any(eng.in_progress(g) for g in ids):
        start = [i for i, g in enumerate(ids) if nxt[i] < 4 and not eng.in_progress(g) and (step + i) % 2 == 0]
        done, _ = eng.step_sliced([(ids[i], nxt[i], dev[i][nxt[i]]) for i in start],
                                  pass_budget=budgets[step % len(budgets)])
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
@pytest.mark.parametrize("n,degree,solo", [(2000, 100, 0), (2000, 100, 7), (9700, 17, 0), (12000, 40, 7), (200000, 40, 0)])
def test_rows_that_take_a_tile_many_steps(gpu, oracle, n, degree, solo):
    """Rows of more than 8 and of more than 32 entries in most places: dealt out to
    all warps of a block, whether or not it owns more than 32 vertices per warp."""
    p = dlp.Problem(n, degree, 4, 7, cache_dir="")
    cap = 40
    orc = oracle.OracleRun.from_problem(p, record=n < 10000, threads=8, max_iterations=cap)
    sess = dlp.Session.from_problem(p, record=n < 10000, max_iterations=cap, small_frontier_solo=solo)
    for b, batch in enumerate(p.batches):
        if n < 10000:
            check_batch(b, sess.apply(b, batch), orc.apply(b, batch), sess, orc, oracle)
            continue
        got, want = sess.apply(b, batch), orc.apply(b, batch)
        for k in EXACT_STATS:
            assert got[k] == want[k], (b, k)
        assert sess.labels().tobytes() == orc.labels().tobytes(), b


@pytest.mark.gpu
def test_short_time_slices_among_longer_ones(gpu, oracle):
    """Slices of 10 us run over lists, of 40 us on owned rows; the results are those of
    batches run to their end."""
    probs = [dlp.Problem(n, d, 3, s, cache_dir="") for n, d, s in ((1500, 5, 1), (20000, 9, 2), (3000, 34, 3))]
    cap = 150
    orcs = [oracle.OracleRun.from_problem(p, threads=4, max_iterations=cap) for p in probs]
    eng = dlp.Engine(len(probs), max_iterations=cap)
    ids = [eng.add_problem(p) for p in probs]
    dev = [[dlp.DeviceBatch(b) for b in p.batches] for p in probs]
    nxt, step = [0] * len(probs), 0
    while any(x < 3 for x in nxt) or any(eng.in_progress(g) for g in ids):
        start = [i for i, g in enumerate(ids) if nxt[i] < 3 and not eng.in_progress(g)]
        done, _ = eng.step_sliced([(ids[i], nxt[i], dev[i][nxt[i]]) for i in start], slice_us=(10.0, 40.0)[step % 2])
        for i in start:
            nxt[i] += 1
        for g in done:
            i = ids.index(g)
            want, got = orcs[i].apply(nxt[i] - 1, probs[i].batches[nxt[i] - 1]), eng.stats(g, nxt[i] - 1)
            for k in EXACT_STATS:
                assert got[k] == want[k], (i, nxt[i] - 1, k)
            assert eng.labels(g).tobytes() == orcs[i].labels().tobytes(), (i, nxt[i] - 1)
        step += 1
