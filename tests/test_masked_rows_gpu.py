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


@pytest.mark.parametrize("rows,vocab,top_k", [(6, 3, 2), (9, 300, 256), (65, 1000, 40), (8, 65537, 1), (8, 65537, 64), (64, 20000, 50), (40, 40000, 64),
                                              (150, 49155, 40), (150, 49155, 200), (4, 300, 0)])
def test_softcap_makes_masked_logits_finite(oracle, rows, vocab, top_k):
    """cap * tanh(-inf / cap) = -cap: a masked logit is a candidate like any other, and above one that the penalty has pushed
    below -cap.  Rows of few finite logits, some of them far below, all of them in the window; segments without any; rows
    whose best logits are all capped to -cap."""
    rng = np.random.default_rng(vocab + rows + top_k)
    lg = np.full((rows, vocab), -np.inf, dtype=np.float32)
    hists = []
    for r in range(rows):
        n = int(rng.integers(0, 1 + min(vocab, 2 * max(top_k, 3))))
        cols = rng.permutation(vocab)[:n] if r % 3 else np.arange(n)
        lg[r, cols] = rng.choice([-4e4, -2000.0, -95.0, -3.0, 2.0, 50.0], n) if r % 2 else -100.0 * rng.random(n)
        hists.append(np.concatenate([cols[: n if r % 4 else n // 2], rng.integers(0, vocab, 20)]).astype(np.int32))
    p = fb.make_params(rows, temperature=0.8 if top_k != 1 else 0.0, top_k=top_k, top_p=1.0)
    p["repetition_penalty"] = np.array([1.4, 3.0, 0.5, 1.0, 1e10], dtype=np.float32)[np.arange(rows) % 5]
    p["temperature"][::7] = 0.0
    p["temperature"][1::7] = 1e20       # all candidates alike: the draw goes by their order
    p["seed"] = 3 + np.arange(rows)
    seen = lg.copy()
    oracle.softcap(seen, 30.0)
    ref = oracle.sample_rows(p, oracle.new_rngs(p["seed"]), seen, hists, cap=256)
    e = fb.Engine(device=0, max_rows=rows, max_vocab=vocab, max_hist_ids=sum(map(len, hists)) + 64)
    e.set_softcap(30.0)
    tok = e.sample_batch(e.open_streams(p), lg, hists, flags=fb.KEEP_KEPT_SET)
    bad = []
    for r in range(rows):
        if p["temperature"][r] <= 0 or top_k == 1:
            continue
        ids, pr, n = e.last_kept(r)
        if n != ref["n_keep"][r] or not np.array_equal(ids, ref["kept_ids"][r, :len(ids)]) or not np.abs(pr - ref["kept_pr"][r, :len(ids)]).max() <= 1e-6:
            bad.append(r)
    e.close()
    assert not bad and np.array_equal(tok, ref["tokens"]), (bad, np.flatnonzero(tok != ref["tokens"]))
