"""Rows of several CTAs and segments at the size of the shared-memory ring, against the CPU oracle: the bound that the CTAs of a
row find together, the candidates they send to the first one, and what they do when too many logits reach it, or too few exist."""
import numpy as np
import pytest

import ferro_b200 as fb
from helpers import compare_with_oracle

pytestmark = pytest.mark.gpu

SHAPES = [  # rows, logits, top_k, window
    (1, 65535, 40, 3), (2, 65536, 64, 0), (2, 65537 + 3, 41, 70), (5, 65541, 17, 0),      # eight small CTAs, their ring full or just over it
    (12, 32768, 64, 30), (12, 32769, 63, 30), (20, 16391, 33, 12),                         # four, two
    (30, 131072, 40, 50), (30, 131077, 64, 50), (70, 65536, 50, 9), (70, 65543, 2, 9),     # four large CTAs, two
    (100, 32768, 64, 5), (100, 32773, 40, 5), (100, 1500, 64, 2), (60, 900, 64, 40), (90, 130, 64, 8), (60, 61, 64, 2), (60, 3, 2, 1),
    (14, 100000, 40, 20), (14, 131077, 64, 30), (15, 100001, 40, 9), (1, 262144, 64, 9),   # eight large CTAs
    (44, 40003, 64, 9), (64, 65535, 40, 5), (8, 16384, 64, 9), (9, 16384, 40, 9), (37, 16391, 5, 3), (2, 2050, 40, 3),   # four or eight small ones, short
    (200, 8192, 64, 5), (200, 8193, 40, 5), (200, 8188, 5, 0), (160, 70, 30, 3),           # one small CTA per row
]


@pytest.mark.parametrize("rows,vocab,top_k,window", SHAPES)
def test_row_bound(oracle, rows, vocab, top_k, window):
    rng = np.random.default_rng(rows + vocab)
    lg = (rng.standard_normal((rows, vocab)) * 3).astype(np.float32)
    part = max(1, vocab // 8)
    for r in range(rows):
        kind = r % 7
        if kind == 1:
            lg[r] = np.round(lg[r])                              # equal logits across all segments
        elif kind == 2:
            lg[r, part:2 * part] = lg[r].max() + 1               # all of one segment's reach the bound
        elif kind == 3:
            lg[r, part:] = -np.inf                               # one segment has any
        elif kind == 4:
            lg[r, rng.integers(0, vocab, max(1, vocab - top_k // 2))] = -np.inf     # hardly any
        elif kind == 5:
            lg[r, : max(1, vocab // 3)] = np.nan
            lg[r, -1] = 2.0
        elif kind == 6:
            lg[r, vocab - part:] += 9                            # all candidates in one segment
    p = fb.make_params(rows, temperature=0.8, top_k=top_k, top_p=0.95, repetition_penalty=1.3 if rows % 2 else 0.8)
    p["seed"] = 1 + np.arange(rows)
    p["temperature"][::5] = 0.0
    top = np.argsort(-np.nan_to_num(lg, nan=-1e30), axis=1)[:, :window // 2]
    hists = [np.concatenate([top[r], rng.integers(0, vocab, window - len(top[r]))]).astype(np.int32) for r in range(rows)]
    clean = np.nan_to_num(lg, nan=-np.inf, neginf=-np.inf)       # (a NaN is no candidate; the oracle's order knows none)
    keep = np.array([np.isfinite(clean[r]).sum() >= top_k or r % 7 != 5 for r in range(rows)])
    ref = oracle.sample_rows(p, oracle.new_rngs(p["seed"]), clean.copy(), hists, cap=fb.MAX_CANDIDATE_K)
    e = fb.Engine(device=0, max_rows=rows, max_vocab=vocab, max_hist_ids=rows * (window + 2) + 64)
    sids = e.open_streams(p)
    tok = e.sample_batch(sids, lg, hists, n_vocab=vocab, flags=fb.KEEP_KEPT_SET)
    hard, near, kept_bad = compare_with_oracle(e, tok, ref, p, vocab)
    e.close()
    bad = [h for h in hard if keep[h if np.isscalar(h) else h[0]]]
    bad_kept = [h for h in kept_bad if keep[h if np.isscalar(h) else h[0]]]
    assert not bad and not bad_kept and near <= 1, (bad[:3], bad_kept[:3], near)
