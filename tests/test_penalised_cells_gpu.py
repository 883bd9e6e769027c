"""Penalty windows kept by 16-byte cells (many whole rows on small CTAs), against the CPU oracle: at the shortest rows and the
longest windows of that layout and one beyond, with penalties that raise logits, tables half full, several ids per cell."""
import numpy as np
import pytest

import ferro_b200 as fb
from helpers import compare_with_oracle

pytestmark = pytest.mark.gpu

CASES = [  # rows, logits, top_k, window, repetition penalty, softcap
    (150, 8199, 40, 300, 1.3, 0.0), (150, 8200, 40, 300, 1.3, 0.0), (151, 8207, 64, 1024, 0.7, 0.0), (150, 16385, 64, 1025, 1.2, 0.0),
    (150, 16384, 50, 2046, 1.3, 0.0), (149, 16384, 50, 2047, 0.8, 0.0), (160, 12003, 33, 2045, 0.6, 30.0), (160, 12003, 33, 700, 1.4, 30.0),
    (149, 32771, 7, 64, 0.5, 0.0), (149, 65539, 64, 2046, 1.1, 0.0),
]


@pytest.mark.parametrize("rows,vocab,top_k,window,penalty,softcap", CASES)
def test_penalised_cells(oracle, rows, vocab, top_k, window, penalty, softcap):
    rng = np.random.default_rng(rows + vocab + window)
    base = (rng.standard_normal((12, vocab)) * 3).astype(np.float32)
    base[1] = np.round(base[1])             # equal logits
    base[2, 40:] = -np.inf                  # nearly all masked
    base[3] -= 9                            # few above 0: a penalty makes most smaller still
    lg = base[np.arange(rows) % 12]
    p = fb.make_params(rows, temperature=0.9, top_k=top_k, top_p=0.97, repetition_penalty=penalty, repeat_last_n=-1)
    p["seed"] = 1 + np.arange(rows)
    p["repetition_penalty"][::9] = 1.0
    top = np.argsort(-base, axis=1)
    spread = [window // 2, 8, window]
    hists = []
    for r in range(rows):
        n = min(spread[r % 3], vocab)       # windows of top logits: half, a few, all of it
        hists.append(np.concatenate([top[r % 12][:n], rng.integers(-3, vocab + 3, window - n), [0, vocab - 1]]).astype(np.int32))
    seen = lg.copy()
    if softcap:
        oracle.softcap(seen, softcap)
    ref = oracle.sample_rows(p, oracle.new_rngs(p["seed"]), seen.copy(), hists, cap=fb.MAX_CANDIDATE_K)
    e = fb.Engine(device=0, max_rows=rows, max_vocab=vocab, max_hist_ids=rows * (window + 2) + 64)
    if softcap:
        e.set_softcap(softcap)
    tok = e.sample_batch(e.open_streams(p), lg, hists, n_vocab=vocab, flags=fb.KEEP_KEPT_SET)
    hard, near, kept_bad = compare_with_oracle(e, tok, ref, p, vocab, check_kept=not softcap)    # (the device's tanhf may differ in the last place)
    e.close()
    assert not hard and not kept_bad and near <= 1, (hard[:3], kept_bad[:3], near)
