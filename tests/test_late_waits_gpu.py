"""Waits for another CTA of a row that run out.  The library is built once more with waits that now and then give up at once, and a process
of its own runs batches of every layout of both kernels through it: each call either returns the tokens of the usual library or fails with
the status that says so, and the calls after it are as good as any."""
import json
import os
import shutil
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# rows, vocab, kept sets wanted, calls, parameters.  Streaming kernel: clusters of two, four and eight CTAs, small and large; full-vocabulary
# kernel: clusters of four to eight, cuts by either and by both, lists that do not fit, a k below the vocabulary, infinite logits and rows
# too long for shared memory (no bins)
CASES = [
    (1, 65536, False, 60, dict(top_k=40, top_p=0.9)),
    (8, 16384, False, 60, dict(top_k=64, min_p=0.02)),
    (30, 16384, False, 60, dict(top_k=50)),
    (14, 131072, False, 60, dict(top_k=40)),
    (32, 131072, True, 60, dict(top_k=60, top_p=0.95)),
    (64, 70001, False, 60, dict(top_k=64)),
    (8, 65536, False, 40, dict(top_k=0, top_p=0.95)),
    (16, 131072, False, 40, dict(top_k=0, min_p=0.05)),
    (23, 100003, False, 40, dict(top_k=0, top_p=0.9, min_p=0.01)),
    (32, 30000, False, 40, dict(top_k=0)),
    (4, 65536, True, 40, dict(top_k=0, top_p=0.9)),
    (8, 50000, False, 40, dict(top_k=3000, top_p=0.9)),
    (3, 300001, False, 20, dict(top_k=0, top_p=0.9)),
]


def batch(case, infinite):
    import ferro_b200 as fb
    rows, vocab, _, _, kw = CASES[case]
    rng = np.random.default_rng(case)
    lg = (rng.standard_normal((rows, vocab)) * 2).astype(np.float32)
    if rows > 2:
        lg[1] = np.round(lg[1])     # lists that do not fit
        lg[2] *= 0.01
    if infinite:
        lg[rows // 2, 7] = np.inf
    p = fb.make_params(rows, temperature=0.9, repetition_penalty=1.2, **kw)
    p["seed"] = 1 + np.arange(rows)
    return lg, p, [rng.integers(0, vocab, 100).astype(np.int32) for _ in range(rows)]


def run(case, infinite, calls):
    """Tokens of each call, or the error's text."""
    import torch

    import ferro_b200 as fb
    lg, p, hists = batch(case, infinite)
    rows, vocab, kept = CASES[case][:3]
    dev = torch.from_numpy(lg).cuda()
    torch.cuda.synchronize()
    e = fb.Engine(device=0, max_rows=rows, max_vocab=vocab, max_hist_ids=rows * 128)
    out = []
    for _ in range(calls):
        sids = e.open_streams(p)
        try:
            out.append(e.sample_batch(sids, dev, hists, n_vocab=vocab, flags=fb.KEEP_KEPT_SET if kept else 0).tolist())
        except fb.SamplerError as err:
            out.append(str(err))
        for s in sids:
            e.close_stream(s)
    e.close()
    return out


def all_cases(calls=None):
    return [run(c, infinite, calls or CASES[c][3]) for c in range(len(CASES)) for infinite in (False, True)]


def test_waits_that_run_out(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc on this machine")
    from ferro_b200 import _build
    _build.build()
    for d in ("ferro_b200", "include"):
        shutil.copytree(os.path.join(ROOT, d), str(tmp_path / d))
    csrc, lib = tmp_path / "ferro_b200" / "csrc", tmp_path / "ferro_b200" / "lib" / os.path.basename(_build.LIB_PATH)
    r = subprocess.run([nvcc, *_build.NVCC_FLAGS, "-t", "4", "-include", os.path.join(ROOT, "tests", "late_waits.cuh"), "-x", "cu", *(str(csrc / f) for f in _build.SOURCES), "-o", str(lib)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([sys.executable, os.path.abspath(__file__), str(tmp_path)], capture_output=True, text=True, timeout=500)
    assert r.returncode == 0, (r.stdout[-1000:], r.stderr[-3000:])
    got, want = json.loads(r.stdout.splitlines()[-1]), all_cases(1)
    failed = {"streaming": 0, "full vocabulary": 0}
    for i, (calls, (usual,)) in enumerate(zip(got, want)):
        assert not isinstance(usual, str), usual
        for tokens in calls:
            if isinstance(tokens, str):
                status = int(tokens.split("kernel status 0x")[1].split()[0], 16)
                assert status & 16 and status & ~(16 | 8) == 0, tokens
                failed["full vocabulary" if CASES[i // 2][4].get("top_k") in (0, 3000) else "streaming"] += 1
            else:
                assert tokens == usual, (CASES[i // 2], i % 2)
    print(failed, [sum(isinstance(t, str) for t in calls) for calls in got])
    assert min(failed.values()) >= 10, failed   # (each call has some hundred to some ten thousand waits that may give up)


if __name__ == "__main__":
    sys.path.insert(0, sys.argv[1])
    import ferro_b200
    assert ferro_b200.__file__.startswith(sys.argv[1]), ferro_b200.__file__
    print(json.dumps(all_cases()))
