"""Every layout of a launch against the CPU oracle, at the sizes where one gives way to the next: CTA sizes, segments per
row, list lengths around 64, windows longer than the list of looked-up logits, descriptors and windows that go with the
launch, clusters of the full-vocabulary kernel."""
import numpy as np
import pytest

import ferro_b200 as fb
from helpers import compare_with_oracle

pytestmark = pytest.mark.gpu

PLANS = [
    # rows, logits, top_k, window, repetition penalty, softcap
    (8, 16385, 64, 32, 1.2, 0.0), (9, 16383, 65, 28, 0.8, 0.0),      # 8 rows and 256 ids go with the launch, more do not
    (8, 65537, 40, 33, 1.1, 0.0), (64, 4099, 50, 8, 1.1, 0.0), (65, 4099, 256, 0, 1.0, 0.0),
    (3, 65535, 50, 1500, 1.3, 0.0), (33, 65539, 64, 100, 1.1, 0.0), (34, 65536, 64, 100, 1.1, 0.0),   # clusters of four large CTAs, of two
    (5, 40001, 33, 1030, 0.7, 30.0), (38, 32769, 64, 64, 1.1, 0.0), (75, 32769, 128, 64, 1.1, 0.0), (148, 16384, 7, 50, 1.1, 0.0),
    (149, 8191, 64, 200, 1.2, 0.0), (149, 32768, 256, 20, 1.2, 0.0), (150, 16000, 200, 2000, 1.2, 0.0),
    (149, 65536, 1, 40, 1.5, 0.0), (223, 65536, 1, 40, 1.5, 0.0), (8, 65536, 1, 1100, 1.5, 0.0), (445, 65540, 1, 20, 1.5, 0.0),
    (300, 131076, 20, 40, 1.1, 0.0), (149, 65545, 64, 1022, 1.3, 0.0), (150, 65547, 9, 1023, 0.6, 0.0), (151, 65551, 50, 300, 1.2, 30.0),   # penalised cells
    (80, 400000, 40, 300, 1.1, 0.0), (2, 400003, 256, 300, 1.1, 0.0),  # bitmaps too long for large CTAs
]


@pytest.mark.parametrize("rows,vocab,top_k,window,penalty,softcap", PLANS)
def test_layouts_of_the_streaming_kernel(oracle, rows, vocab, top_k, window, penalty, softcap):
    rng = np.random.default_rng(rows * 7 + vocab)
    base = (rng.standard_normal((min(rows, 24), vocab)) * 3).astype(np.float32)
    lg = base[np.arange(rows) % len(base)]
    lg[0] = np.round(lg[0])                 # equal logits by the thousand
    lg[-1, 5:] = -np.inf                    # fewer finite logits than top_k
    p = fb.make_params(rows, temperature=0.9 if top_k > 1 else 0.0, top_k=top_k, top_p=0.97, repetition_penalty=penalty, repeat_last_n=-1)
    p["seed"] = 1 + np.arange(rows)
    top = np.argsort(-base, axis=1)[:, :window // 2]
    hists = [np.concatenate([top[r % len(base)], rng.integers(0, vocab, window - window // 2), [0, vocab - 1]]).astype(np.int32) for r in range(rows)]
    seen = lg.copy()
    if softcap:
        oracle.softcap(seen, softcap)
    ref = oracle.sample_rows(p, oracle.new_rngs(p["seed"]), seen.copy(), hists, cap=fb.MAX_CANDIDATE_K)
    e = fb.Engine(device=0, max_rows=rows, max_vocab=vocab, max_hist_ids=rows * (window + 2) + 64)
    if softcap:
        e.set_softcap(softcap)
    sids = e.open_streams(p)
    tok = e.sample_batch(sids, lg, hists, n_vocab=vocab, flags=fb.KEEP_KEPT_SET)
    hard, near, kept_bad = compare_with_oracle(e, tok, ref, p, vocab, check_kept=not softcap)    # (the device's tanhf may differ in the last place)
    e.close()
    assert not hard and not kept_bad and near <= 1, (hard[:3], kept_bad[:3], near)


@pytest.mark.parametrize("rows", [15, 16, 22, 23, 33, 34])
def test_clusters_of_the_full_vocabulary_kernel(oracle, rows):
    vocab = 20011
    rng = np.random.default_rng(rows)
    lg = (rng.standard_normal((rows, vocab)) * 3).astype(np.float32)
    p = fb.make_params(rows, temperature=1.0, top_k=0, top_p=0.9, repetition_penalty=1.1)
    p["seed"] = 5 + np.arange(rows)
    p["top_p"] = np.array([0.5, 0.7, 0.9, 1.0])[np.arange(rows) % 4]        # kept sets of some tens to all logits
    p["min_p"] = np.array([0.0, 0.05, 0.001])[np.arange(rows) % 3]
    p["top_k"] = np.array([0, 257, 768, 1025, 5000])[np.arange(rows) % 5]
    hists = [rng.integers(0, vocab, 100).astype(np.int32) for _ in range(rows)]
    ref = oracle.sample_rows(p, oracle.new_rngs(p["seed"]), lg.copy(), hists, cap=vocab)
    e = fb.Engine(device=0, max_rows=rows, max_vocab=vocab, max_hist_ids=rows * 100 + 64)
    sids = e.open_streams(p)
    tok = e.sample_batch(sids, lg, hists, n_vocab=vocab, flags=fb.KEEP_KEPT_SET)
    hard, near, kept_bad = compare_with_oracle(e, tok, ref, p, vocab)
    e.close()
    assert not hard and not kept_bad and near <= 1, (hard[:3], kept_bad[:3], near)
