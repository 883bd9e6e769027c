"""Full-vocabulary rows with masked (minus infinity) logits: they are candidates of weight zero, in order behind the finite
ones, and their probability is exactly 0 - in the record, and where min-p looks at it."""
import numpy as np
import pytest

import ferro_b200 as fb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vocab,finite", [(300, 1), (300, 10), (300, 255), (300, 256), (300, 300), (2000, 40), (70001, 500)])
def test_masked_logits_have_probability_zero(oracle, vocab, finite):
    rows = 6
    rng = np.random.default_rng(vocab + finite)
    lg = np.full((rows, vocab), -np.inf, dtype=np.float32)
    for r in range(rows):
        lg[r, rng.permutation(vocab)[:finite]] = (rng.standard_normal(finite) * 2).astype(np.float32)
    p = fb.make_params(rows, temperature=0.9, top_k=0, repetition_penalty=1.0)
    p["top_p"] = [1.0, 1.0, 0.9, 0.999, 1.0, 0.5]
    p["min_p"] = [0.0, 1e-30, 0.0, 0.0, 0.05, 1e-30]
    p["seed"] = 3 + np.arange(rows)
    ref = oracle.sample_rows(p, oracle.new_rngs(p["seed"]), lg.copy(), [[]] * rows, cap=vocab)
    e = fb.Engine(device=0, max_rows=rows, max_vocab=vocab, max_hist_ids=64)
    tok = e.sample_batch(e.open_streams(p), lg, [[]] * rows, flags=fb.KEEP_KEPT_SET)
    for r in range(rows):
        ids, pr, n = e.last_kept(r)
        m, want = len(ids), ref["kept_pr"][r, :len(ids)]
        assert n == ref["n_keep"][r] and m == min(n, fb.MAX_CANDIDATE_K), r
        assert np.array_equal(ids, ref["kept_ids"][r, :m]), r
        assert np.abs(pr - want).max() <= 1e-12 and np.array_equal(pr[want == 0.0], want[want == 0.0]), r   # (a NaN fails both)
    e.close()
    assert np.array_equal(tok, ref["tokens"])
