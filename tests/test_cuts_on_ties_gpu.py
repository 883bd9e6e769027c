"""Cuts and draws that fall on a boundary of the cumulative distribution, and beside one: rows of equal logits (every
exponential is 1, every partial sum exact), so that the device has to give the oracle's tokens whatever it decides from
partial sums and whatever it adds up again; and the same rows with the kept set recorded, which always adds up."""
import numpy as np
import pytest

import ferro_b200 as fb

pytestmark = pytest.mark.gpu

ROWS = 64


def rows_of(n, seed):
    rng = np.random.default_rng(seed)
    lg = np.full((ROWS, 1500), -80.0, dtype=np.float32)
    for r in range(ROWS):
        lg[r, rng.permutation(1500)[:n]] = 2.5
    lg[ROWS // 2:] += (0.3 * rng.standard_normal((ROWS // 2, 1500))).astype(np.float32)     # these have no ties
    p = fb.make_params(ROWS, top_k=n, repetition_penalty=1.0, temperature=0.7)
    p["seed"] = 1 + rng.integers(0, 1 << 40, ROWS)
    m = rng.integers(1, n + 1, ROWS)
    share = (m / n).astype(np.float32)
    p["top_p"] = np.where(np.arange(ROWS) % 4 == 3, 1.0, np.where(np.arange(ROWS) % 4 == 2, np.nextafter(share, np.float32(0)), share))
    p["min_p"] = np.array([0.0, 0.0, 1.0, 0.5, np.nextafter(np.float32(1), np.float32(0))])[np.arange(ROWS) % 5]
    return lg, p


@pytest.mark.parametrize("n", [1, 2, 3, 4, 8, 16, 17, 31, 32, 33, 48, 64, 65, 128, 255, 256])
def test_cuts_on_ties(engine, oracle, n):
    lg, p = rows_of(n, n)
    ref = oracle.sample_rows(p, oracle.new_rngs(p["seed"]), lg.copy(), [[]] * ROWS)
    for flags in (0, fb.KEEP_KEPT_SET):
        sids = engine.open_streams(p)
        tok = engine.sample_batch(sids, lg, [[]] * ROWS, flags=flags)
        for s in sids:
            engine.close_stream(int(s))
        assert (tok == ref["tokens"]).all(), (flags, np.nonzero(tok != ref["tokens"]))
