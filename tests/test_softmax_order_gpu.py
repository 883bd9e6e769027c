"""The softmax denominator of the candidate path is the sequential sum over the candidates in order (src/sampler.cpp:40),
bit for bit.  Rows hold one logit x0 and k - 1 equal ones below it, so the denominator is (((1 + c) + c) + c) + ... with
c = exp((x1 - x0) / T): the device's exp and the C library's are both within an ulp of the true value, so c is one of five
numbers, and one of them has to give every recorded probability exactly.  (A sum in another order differs in three rows of
four at k = 40, in nine of ten at k = 256.)"""
import numpy as np
import pytest

import ferro_b200 as fb

pytestmark = pytest.mark.gpu

ROWS, VOCAB = 48, 4096


def rows_of(k, seed):
    rng = np.random.default_rng(seed)
    lg = np.full((ROWS, VOCAB), -60.0, dtype=np.float32)
    x0 = rng.uniform(1.0, 12.0, ROWS).astype(np.float32)
    x1 = (x0 - rng.uniform(0.05, 3.0, ROWS).astype(np.float32)).astype(np.float32)
    for r in range(ROWS):
        cols = rng.permutation(VOCAB)[:k]
        lg[r, cols] = x1[r]
        lg[r, cols[0]] = x0[r]
    p = fb.make_params(ROWS, top_k=k, top_p=1.0, repetition_penalty=1.0)
    p["temperature"] = rng.uniform(0.3, 1.5, ROWS).astype(np.float32)
    p["seed"] = 1 + np.arange(ROWS)
    return lg, p, x0, x1


def in_sequence(pr, x0, x1, temperature):
    c = np.exp(np.float64(x1 - x0) / np.float64(temperature))
    for ulps in range(-2, 3):
        e = np.concatenate([[1.0], np.full(len(pr) - 1, c + ulps * np.spacing(c))])
        total = np.float64(0.0)
        for v in e:
            total += v
        if np.array_equal(pr, e / total):
            return True
    return False


@pytest.mark.parametrize("k", [2, 16, 17, 33, 40, 64, 65, 255, 256])
def test_denominator_is_summed_in_candidate_order(engine, k):
    lg, p, x0, x1 = rows_of(k, k)
    sids = engine.open_streams(p)
    engine.sample_batch(sids, lg, [[]] * ROWS, flags=fb.KEEP_KEPT_SET)
    bad = []
    for r in range(ROWS):
        ids, pr, n = engine.last_kept(r)
        assert n == k
        if not in_sequence(pr, x0[r], x1[r], p["temperature"][r]):
            bad.append(r)
    for s in sids:
        engine.close_stream(int(s))
    assert not bad


@pytest.mark.parametrize("k", [40, 256])
def test_denominator_of_merged_lists_is_summed_in_candidate_order(k):
    import torch
    lg, p, x0, x1 = rows_of(k, 1000 + k)
    dev = torch.from_numpy(lg).cuda()
    half = VOCAB // 2
    engines, lists = [], torch.zeros((2, ROWS, k + 1), dtype=torch.int64, device="cuda")
    for g in range(2):
        e = fb.Engine(device=0, max_rows=ROWS, max_vocab=half, max_hist_ids=64)
        e.set_vocab_shard(g * half, VOCAB)
        b = e.prepare_batch(e.open_streams(p), [[]] * ROWS, half, ld=VOCAB, flags=fb.KEEP_KEPT_SET)
        b.shard_launch_packed(dev.data_ptr() + 4 * g * half, lists[g].data_ptr(), k + 1)
        engines.append((e, b))
    torch.cuda.synchronize()
    e, b = engines[0]
    b.merge_launch_packed(lists.data_ptr(), k + 1, 2, 0, ROWS)
    b.check()
    bad = [r for r in range(ROWS) if not in_sequence(e.last_kept(r)[1], x0[r], x1[r], p["temperature"][r])]
    for e, b in engines:
        b.free()
        e.close()
    assert not bad
