"""A captured fsb_batch_launch, replayed after fsb_batch_redraw, draws the new engine outputs: row counts on both sides of
the 64 descriptors that go with a launch, and a batch with full-vocabulary rows (which run on a second stream)."""
import numpy as np
import pytest

import ferro_b200 as fb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,mixed", [(1, False), (8, True), (64, False), (65, False)])
def test_replayed_launch_draws_what_the_redraw_drew(oracle, rows, mixed):
    import torch
    vocab = 5003
    rng = np.random.default_rng(rows)
    lg = rng.standard_normal((rows, vocab)).astype(np.float32)
    p = fb.make_params(rows, temperature=1.2, top_k=200, top_p=1.0, repetition_penalty=1.2)
    if mixed:
        p["top_k"][::2] = 0
    p["seed"] = 70 + np.arange(rows)
    hists = [rng.integers(0, vocab, 30).astype(np.int32) for _ in range(rows)]
    rngs = oracle.new_rngs(p["seed"])
    dev = torch.from_numpy(lg).cuda()
    stream = torch.cuda.Stream()
    e = fb.Engine(device=0, max_rows=rows, max_vocab=vocab, max_hist_ids=rows * 30 + 64)
    e.set_cuda_stream(stream.cuda_stream)
    b = e.prepare_batch(e.open_streams(p), hists, vocab)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        graph.capture_begin()
        b.launch(dev.data_ptr())
        graph.capture_end()
        for step in range(4):
            if step:
                b.redraw()
            graph.replay()
            want = oracle.sample_rows(p, rngs, lg.copy(), hists, cap=vocab)["tokens"]
            assert np.array_equal(b.tokens(), want), step
    torch.cuda.synchronize()
    b.free()
    e.close()
    del graph
