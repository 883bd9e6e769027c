"""All-greedy launches run a kernel of their own where no row has a penalty window, and one that knows windows where some row has: the
tokens of both against the oracle, for every layout, on rows of ties, masked logits and a maximum at either end."""
import numpy as np
import pytest

import ferro_b200 as fb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("windows", ["none", "off", "some", "all"])
@pytest.mark.parametrize("rows,vocab,pad", [(1, 3, 0), (1, 70001, 0), (8, 65536, 0), (9, 16384, 1), (64, 30001, 3), (70, 50000, 0), (136, 65536, 0), (148, 20003, 2), (200, 70000, 0), (450, 4099, 1)])
def test_greedy_rows_with_and_without_windows(oracle, rows, vocab, pad, windows):
    import torch
    rng = np.random.default_rng(rows + vocab)
    base = (np.round(rng.standard_normal((min(rows, 16), vocab)) * 8) / 4).astype(np.float32)   # the maximum several times
    base[:, ::7] = -np.inf
    lg = base[np.arange(rows) % len(base)].copy()
    lg[rows // 2] = -np.inf
    lg[-1, -1] = 50.0
    lg[0, 0] = 50.0
    p = fb.make_params(rows, temperature=0.0, repetition_penalty=1.0 if windows == "off" else 1.5)
    hists = [rng.integers(0, vocab, 40).astype(np.int32) for _ in range(rows)]
    best = lg.argmax(axis=1).astype(np.int32)
    for r in range(rows):
        hists[r][:2] = best[r]
        if windows == "none" or (windows == "some" and r % 3 != 1 and rows > 1):
            hists[r] = hists[r][:0]
    ref = oracle.sample_rows(p, oracle.new_rngs(p["seed"]), lg.copy(), hists)
    dev = torch.full((rows, vocab + pad), 99.0, device="cuda")
    dev[:, :vocab].copy_(torch.from_numpy(lg))
    e = fb.Engine(device=0, max_rows=rows, max_vocab=vocab, max_hist_ids=rows * 64)
    tok = e.sample_batch(e.open_streams(p), dev[:, :vocab], hists, n_vocab=vocab)
    e.close()
    assert np.array_equal(tok, ref["tokens"])
