"""One-block passes (csrc/row_stint.cuh) where their layout changes: rows of 8
and 9 entries (one lane, four lanes), of 32 and 33 (four lanes, no stint), and
frontiers that fill the block's lanes or its vertex table. Bit-exact against
the oracle, with the frontier sizes recorded (the recording loop) and without
(the loops that gather before or after the marks are known)."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

import labelpropcuda_gb300 as dlp
from parity_checks import EXACT_STATS, check_batch


@pytest.mark.gpu
@pytest.mark.parametrize("n,degree", [(40, 3), (300, 8), (700, 16), (1100, 5), (1500, 33), (4200, 9)])
def test_one_block_passes_match_oracle(gpu, oracle, n, degree):
    p = dlp.Problem(n, degree, 5, 11, cache_dir="")
    cap = 700  # beyond the first look at the rows in use
    orc = oracle.OracleRun.from_problem(p, record=True, threads=4, max_iterations=cap)
    rec = dlp.Session.from_problem(p, record=True, max_iterations=cap, solo_entry=1024)
    plain = [dlp.Session.from_problem(p, max_iterations=cap, **kw)
             for kw in (dict(), dict(solo_entry=1024), dict(small_frontier_solo=3))]
    for b, batch in enumerate(p.batches):
        want = orc.apply(b, batch)
        check_batch(b, rec.apply(b, batch), want, rec, orc, oracle)
        for s in plain:
            got = s.apply(b, batch)
            for k in EXACT_STATS:
                assert got[k] == want[k], (b, k)
            assert s.labels().tobytes() == orc.labels().tobytes(), b


@pytest.mark.parametrize("scale_a,scale_b", [(-40, -33), (-40, 39), (39, -33), (39, 39), (0, 0), (-20, 3)])
def test_quotient_from_the_reciprocal_is_the_ieee_quotient(scale_a, scale_b):
    """divide() of csrc/common.cuh, restated with the C library's fmaf, over the
    range it serves: numerators of 2^-40 to 2^40 and 0, weight sums above 1e-10."""
    fma = ctypes.CDLL("libm.so.6").fmaf
    fma.restype, fma.argtypes = ctypes.c_float, [ctypes.c_float] * 3
    f32 = np.float32
    rng = np.random.default_rng([scale_a + 40, scale_b + 40])
    mant = np.concatenate([1 + rng.random(4000), [1, 1 + 2**-23, 2 - 2**-23, 1.5, 4 / 3, 5 / 3]]).astype(f32)
    a, b = np.ldexp(mant, scale_a), np.ldexp(rng.permutation(mant), scale_b)
    a[:8] = 0
    with np.errstate(all="raise"):
        for x, d in zip(a, b):
            y = f32(1) / d
            q0 = x * y
            q1 = fma(fma(-d, q0, x), y, q0)
            q = fma(fma(-d, q1, x), y, q1)
            assert f32(q) == x / d, (x, d)
