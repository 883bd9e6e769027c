"""The fused softcap over bounds near zero, within four caps and far beyond, where it is flat and many logits become equal: the
device's tokens against the oracle's on capped logits."""
import numpy as np
import pytest

import ferro_b200 as fb
from helpers import compare_with_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,vocab,top_k,scale,shift", [(12, 65536, 50, 3.0, 0.0), (12, 65536, 50, 40.0, 0.0), (12, 65536, 64, 12.0, 60.0), (12, 65536, 20, 300.0, 0.0), (12, 65536, 40, 9.0, -150.0),
                                                          (64, 70001, 64, 25.0, 0.0), (40, 262144, 64, 20.0, 10.0), (160, 20003, 40, 30.0, 0.0), (20, 200000, 200, 25.0, 0.0)])
def test_softcap_bounds(oracle, rows, vocab, top_k, scale, shift):
    rng = np.random.default_rng(rows + vocab)
    base = (rng.standard_normal((min(rows, 12), vocab)) * scale + shift).astype(np.float32)
    lg = base[np.arange(rows) % len(base)]
    p = fb.make_params(rows, temperature=0.9, top_k=top_k, top_p=0.97, repetition_penalty=1.2)
    p["seed"] = 1 + np.arange(rows)
    p["temperature"][::4] = 0.0
    hists = [rng.integers(0, vocab, 60).astype(np.int32) for _ in range(rows)]
    seen = lg.copy()
    oracle.softcap(seen, 30.0)
    ref = oracle.sample_rows(p, oracle.new_rngs(p["seed"]), seen.copy(), hists, cap=fb.MAX_CANDIDATE_K)
    e = fb.Engine(device=0, max_rows=rows, max_vocab=vocab, max_hist_ids=rows * 64)
    e.set_softcap(30.0)
    tok = e.sample_batch(e.open_streams(p), lg, hists, n_vocab=vocab)
    hard, near, _ = compare_with_oracle(e, tok, ref, p, vocab, check_kept=False)
    e.close()
    # (the device's tanhf may differ from the C library's in the last place, which swaps neighbours: one row in twenty is allowed to)
    assert len(hard) <= max(1, rows // 20) and near <= 1, (len(hard), hard[:3], near)


@pytest.mark.parametrize("rows,vocab,top_k,window", [(64, 65536, 100, 512), (64, 65536, 200, 2048), (24, 131072, 100, 1024), (24, 131072, 200, 512), (20, 262144, 200, 1024),
                                                     (24, 131072, 50, 1024), (160, 8000, 100, 1024), (300, 16003, 65, 200)])
def test_only_logits_that_reach_the_bound_are_candidates(rows, vocab, top_k, window):
    """However the bound was come by, under the softcap too: a window of the row's smallest logits brings a segment's list no entry."""
    import torch
    torch.manual_seed(vocab + top_k)
    lg = torch.randn(rows, vocab, device="cuda") * 9
    lowest = torch.topk(lg, window, dim=1, largest=False).indices.to(torch.int32).cpu().numpy()
    lengths = []
    for penalty in (1.0, 1.2):
        p = fb.make_params(rows, temperature=0.9, top_k=top_k, top_p=0.97, repetition_penalty=penalty)
        p["seed"] = 1 + np.arange(rows)
        trace = torch.zeros(4096 * 8 + 64, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        e = fb.Engine(device=0, max_rows=rows, max_vocab=vocab, max_hist_ids=rows * window)
        e.set_softcap(30.0)
        e.set_trace_buffer(trace.data_ptr())
        e.sample_batch(e.open_streams(p), lg, list(lowest), n_vocab=vocab)
        e.set_trace_buffer(0)
        e.close()
        words = trace.cpu().numpy()[:4096 * 8].reshape(4096, 8)
        lengths.append(words[words[:, 0] != 0][:, 3])
    assert len(lengths[0]) >= rows and lengths[0].max() <= 1024, lengths[0]
    assert (lengths[0] == lengths[1]).all(), (lengths[0], lengths[1])
