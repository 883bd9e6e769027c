"""Launches of a prepared batch in plain stream order, queued without waiting: each reads logits that a kernel writes just before it,
into the same buffer, and writes the same tokens; whatever overlap the launch attribute allows, the tokens are those of launches that
are waited for one by one."""
import numpy as np
import pytest

import ferro_b200 as fb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,vocab,top_k", [(1, 65536, 40), (24, 20000, 16), (40, 70001, 50), (148, 30000, 64), (200, 9000, 40), (450, 12000, 20), (20, 40000, 200), (130, 30000, 1)])
def test_chained_launches(rows, vocab, top_k):
    import torch
    torch.manual_seed(rows)
    base = torch.randn(rows, vocab, device="cuda") * 3
    p = fb.make_params(rows, temperature=0.9 if top_k > 1 else 0.0, top_k=top_k, top_p=0.95, repetition_penalty=1.2)
    p["seed"] = 1 + np.arange(rows)
    hists = [np.random.default_rng(r).integers(0, vocab, 60).astype(np.int32) for r in range(rows)]
    stream = torch.cuda.Stream()
    e = fb.Engine(device=0, max_rows=rows, max_vocab=vocab, max_hist_ids=rows * 64)
    e.set_cuda_stream(stream.cuda_stream)
    b = e.prepare_batch(e.open_streams(p), hists, vocab)

    class Ints:
        __cuda_array_interface__ = {"shape": (rows,), "typestr": "<i4", "data": (int(b.tokens_device_ptr), False), "version": 2}

    tokens = torch.as_tensor(Ints(), device="cuda")
    results = []
    for wait in (True, False):
        lg, out = torch.empty_like(base), torch.empty(12, rows, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            for i in range(12):
                lg.copy_(torch.roll(base, 1000 * i + 1, dims=1))
                lg.mul_(1.0 + 0.01 * i)
                b.launch(lg.data_ptr())
                if i % 3 == 2:
                    b.launch(lg.data_ptr())      # a launch right behind a launch
                if wait:
                    stream.synchronize()
                out[i].copy_(tokens)
        torch.cuda.synchronize()
        results.append(out.cpu().numpy())
    b.check()
    b.free()
    e.close()
    assert (results[0] == results[1]).all()
