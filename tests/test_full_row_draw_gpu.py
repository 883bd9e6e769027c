"""Rows over the whole vocabulary whose kept set is not recorded: the cut and the draw come from the candidates of a few bins, against
the CPU oracle - cuts by top-p, min-p, both or none, flat and peaked rows, equal logits, rows off 16-byte boundaries, draws that
fall into the last bin or on a boundary - and against the same call with the record, which looks at the row another way."""
import numpy as np
import pytest

import ferro_b200 as fb
from helpers import compare_with_oracle

pytestmark = pytest.mark.gpu

CASES = [  # rows, logits, row stride beyond them, softcap
    (12, 1000, 0, 0.0), (12, 4099, 1, 0.0), (16, 20011, 0, 0.0), (15, 32768, 4, 0.0), (16, 65536, 0, 0.0), (23, 65541, 3, 0.0),
    (14, 131072, 0, 0.0), (9, 262144, 0, 0.0), (6, 270001, 0, 0.0), (12, 30000, 0, 30.0), (12, 30001, 2, 30.0), (8, 266003, 2, 30.0),
]


@pytest.mark.parametrize("rows,vocab,pad,softcap", CASES)
def test_full_rows_without_a_record(oracle, rows, vocab, pad, softcap):
    rng = np.random.default_rng(rows + vocab)
    lg = (rng.standard_normal((rows, vocab + pad)) * 3).astype(np.float32)
    for r in range(rows):
        kind = r % 8
        if kind == 1:
            lg[r, rng.integers(0, vocab, 16)] += 12                     # peaked
        elif kind == 2:
            lg[r] = np.round(lg[r] * 2) / 2                             # equal logits by the hundred
        elif kind == 3:
            lg[r] *= 0.01                                               # flat: everything in a few temperatures
        elif kind == 4:
            lg[r, vocab // 3:] = -np.inf
        elif kind == 5:
            lg[r] = 1.25                                                # one value
        elif kind == 6:
            lg[r] = -30
            lg[r, rng.integers(0, vocab)] = 5                           # all but one far down: draws of the last bin
    p = fb.make_params(rows, temperature=1.0, top_k=0, repetition_penalty=1.2)
    p["temperature"] = rng.choice([0.3, 0.8, 1.0, 1.3, 3.0], rows)
    p["top_p"] = np.array([0.95, 1.0, 0.5, 0.999, 1.0])[np.arange(rows) % 5]
    p["min_p"] = np.array([0.0, 0.05, 0.0, 0.001, 0.0, 0.3])[(np.arange(rows) // 2) % 6]
    p["top_k"] = np.array([0, 0, 300, 0, 5000])[(np.arange(rows) // 3) % 5]
    hists = [np.concatenate([np.argsort(-lg[r, :vocab])[:20], rng.integers(-2, vocab + 2, 300), rng.integers(0, vocab, 300)[:r]]).astype(np.int32) for r in range(rows)]
    seen = lg[:, :vocab].copy()
    if softcap:
        oracle.softcap(seen, softcap)
    e = fb.Engine(device=0, max_rows=rows, max_vocab=vocab + pad, max_hist_ids=rows * 700 + 64)
    if softcap:
        e.set_softcap(softcap)
    for draw in range(3):
        p["seed"] = 1 + 1000 * draw + np.arange(rows)
        if draw == 0:
            ref = oracle.sample_rows(p, oracle.new_rngs(p["seed"]), seen.copy(), hists, cap=vocab)
        got = []
        for flags in (0, fb.KEEP_KEPT_SET):
            sids = e.open_streams(p)
            got.append(e.sample_batch(sids, lg, hists, n_vocab=vocab, flags=flags).copy())
            for s in sids:
                e.close_stream(int(s))
        assert (got[0] == got[1]).all(), (draw, np.nonzero(got[0] != got[1]))
        if draw == 0:
            hard, near, _ = compare_with_oracle(e, got[0], ref, p, vocab, check_kept=False)
            assert len(hard) <= (1 if softcap else 0) and near <= 1, (hard[:3], near)    # (softcap: the device's tanhf may differ in the last place)
    e.close()
