"""What users of the sampler have it do, as cases that can be timed: one entry per way of calling it.

A case is a dict of plain values.  ``call`` names the public entry points that one pass goes through:

* ``step``      ``Engine.sample_batch``: one decode step of all slots, every slot's history handed over with the call,
                logits on the device - the loop of a scheduler that keeps its histories itself;
* ``class``     ``Sampler.sample``: the drop-in class, one row in host memory, penalised in place;
* ``resident``  ``Engine.sample_batch_resident`` with APPEND_SAMPLED: continuous batching over histories that live in
                the engine; one request ends and another begins (close, open, history_set) per pass;
* ``launch``    ``Batch.launch``: a prepared batch on the next logits buffer, nothing waited for - tokens stay on the
                device for the kernel that embeds them;
* ``windows``   ``Engine.verify_windows``: speculative verification windows with histories handed over;
* ``draft``     ``Engine.lookup_drafts`` and ``Engine.verify_windows_resident``: a speculative step with
                prompt-lookup drafts over resident histories;
* ``shard``     ``Batch.redraw``, ``shard_launch_packed``, ``merge_launch_packed``, ``check``: one rank's work in a
                vocabulary-sharded step (the other ranks' candidate lists are already here).

``sampler`` names the parameter mix: ``topk`` (top-k, then top-p), ``mixed`` (greedy, full-vocabulary and top-k rows
in turn), ``nucleus`` (no top-k: top-p and min-p over the whole vocabulary), ``greedy``.
"""
import numpy as np
import torch

import ferro_b200 as fb

EOS = 1            # end-of-sequence id of the drafting calls
DRAFTS = 8         # most drafts per stream of a drafting call


def _case(name=None, **kw):
    c = dict(call="step", sampler="topk", rows=1, vocab=65536, pad=0, dist="normal", temperature=0.8, top_k=40, top_p=0.9, min_p=0.0,
             penalty=1.1, hist=256, softcap=0.0, steps=1, window=1, shards=1)
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: one stream's decode step on a small vocabulary - launches and latency
        _case("one_row", rows=1, vocab=65536, temperature=0.7, top_k=40, top_p=0.95, hist=64),
        # the reference's own call site: one Sampler object, its default parameters, logits read back to the host
        _case("class_host_row", call="class", rows=1, vocab=65536, temperature=0.05, top_k=50, top_p=1.0, penalty=1.05, hist=256),
        # a small server's decode step: eight slots whose requests brought different parameters
        _case("slots_mixed", sampler="mixed", rows=8, vocab=65536, penalty=1.15, hist=256),
        # a vocabulary that is not a multiple of anything: rows start off 16-byte boundaries, the last tile is ragged
        _case("ragged_vocab", rows=24, vocab=100003, top_k=50, penalty=1.15, hist=300),
        # requests without top-k: the whole vocabulary is the candidate set
        _case("nucleus", sampler="nucleus", rows=16, vocab=131072, temperature=1.0, penalty=1.1, hist=256),
        # the benchmark's headline shape, launched back to back on prepared parameters
        _case("large_vocab_launch", call="launch", rows=64, vocab=262144, dist="student", temperature=1.0, top_k=64, top_p=0.95, hist=512),
        # the same shape as one synchronous step on raw logits, final-logit softcap fused in front
        _case("large_vocab_softcap", rows=64, vocab=262144, dist="raw", temperature=1.0, top_k=64, top_p=0.95, hist=512, softcap=30.0),
        # speculative verification, temperature 0: eight streams, windows of seventeen rows
        _case("windows_greedy", call="windows", sampler="greedy", rows=8, window=17, vocab=65536, temperature=0.0, penalty=1.0, hist=128),
        # a speculative step at temperature 0.8 with prompt-lookup drafts and the penalty over growing windows
        _case("draft_and_verify", call="draft", rows=8, window=1 + DRAFTS, vocab=131072, top_k=50, top_p=0.95, hist=1024),
        # continuous batching, a mid-sized server
        _case("resident_decode", call="resident", rows=32, vocab=131072, top_k=40, steps=4, hist=256),
        # continuous batching, a whole box's batch on one GPU: the largest
        _case("serving_resident", call="resident", rows=512, vocab=262144, dist="student", top_k=40, steps=2, hist=1024),
        # one rank of eight of a vocabulary-sharded step of the same batch: many rows, short shards
        _case("vocab_shard", call="shard", rows=512, vocab=32768, dist="student", top_k=40, shards=8, hist=1024),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    call = rng.choice(["step", "step", "step", "class", "resident", "resident", "launch", "windows", "draft", "shard"])
    c = _case(call=call, dist=rng.choice(["normal", "student"]), temperature=rng.choice([0.05, 0.3, 0.7, 0.8, 1.0, 1.2]),
              top_k=_log_int(rng, 2, 256), top_p=rng.choice([1.0, 0.95, 0.9, 0.8]), min_p=rng.choice([0.0, 0.0, 0.02, 0.05]),
              penalty=rng.choice([1.0, 1.05, 1.1, 1.2]), hist=_log_int(rng, 16, 2048))
    c["vocab"] = _log_int(rng, 16384, 262144)
    if rng.random() < 0.6:   # most vocabularies are padded to a round number, the rest are what the tokenizer gave
        c["vocab"] = c["vocab"] // 128 * 128
    most = lambda rows: max(1, min(rows, (512 * 262144) // c["vocab"]))  # noqa: E731
    if call == "step":
        c["sampler"] = rng.choice(["topk", "topk", "mixed", "nucleus", "greedy"])
        c["rows"] = most(_log_int(rng, 1, 32 if c["sampler"] in ("mixed", "nucleus") else 128))
        c["pad"] = rng.choice([0, 0, 0, 1, 4, 64])
        if c["sampler"] == "topk" and rng.random() < 0.25:
            c["softcap"], c["dist"] = 30.0, "raw"
    elif call == "class":
        c["sampler"] = rng.choice(["topk", "topk", "greedy", "nucleus"])
    elif call == "resident":
        c["steps"] = rng.randint(1, 4)
        c["rows"] = max(1, min(_log_int(rng, 4, 512), 2 * 512 * 262144 // (c["vocab"] * c["steps"])))
    elif call == "launch":
        c["rows"] = most(_log_int(rng, 4, 256))
    elif call == "windows":
        c["sampler"] = rng.choice(["greedy", "greedy", "topk"])
        c["rows"], c["window"] = _log_int(rng, 1, 16), rng.randint(2, 17)
    elif call == "draft":
        c["rows"], c["window"] = _log_int(rng, 1, 16), 1 + DRAFTS
        c["hist"] = max(c["hist"], 64)
    else:
        c["shards"] = rng.choice([2, 4, 8])
        c["rows"] = _log_int(rng, 16, 512)
        c["vocab"] = c["vocab"] // c["shards"] // 4 * 4
        c["top_k"] = min(c["top_k"], 200)
    if c["sampler"] == "greedy":
        c["temperature"] = 0.0
    return c


# ------------------------------------------------------------------------------------------------ inputs
def _params(c, n, seed):
    p = fb.make_params(n, temperature=c["temperature"], top_k=c["top_k"], top_p=c["top_p"], min_p=c["min_p"], repetition_penalty=c["penalty"])
    p["seed"] = 1 + (int(seed) * 1000003) % (1 << 40) + np.arange(n)
    if c["sampler"] == "mixed":      # two rows each: greedy, temperature only, top-k, top-p with min-p
        g = (np.arange(n) // 2) % 4
        p["temperature"] = np.array([0.0, 1.0, 0.8, 1.0])[g]
        p["top_k"] = np.array([50, 0, 50, 0])[g]
        p["top_p"] = np.array([1.0, 1.0, 1.0, 0.9])[g]
        p["min_p"] = np.array([0.0, 0.0, 0.0, 0.05])[g]
    elif c["sampler"] == "nucleus":  # top-p, min-p, both
        g = np.arange(n) % 3
        p["top_k"] = 0
        p["top_p"] = np.array([0.95, 1.0, 0.9])[g]
        p["min_p"] = np.array([0.0, 0.05, 0.02])[g]
    if c["call"] == "launch":        # the headline batch: every second request has the penalty off
        p["repetition_penalty"][::2] = 1.0
    if c["call"] == "resident":      # the server's --repeat-last-n: the window does not grow with the request
        p["repeat_last_n"] = c["hist"]
    return p


def _logits(c, gen, rows):
    """[rows][vocab + pad] fp32: normal rows with sixteen tokens well above the rest (a confident model), or the
    heavy-tailed rows of a soft-capped large-vocabulary model ("raw": before its softcap)."""
    V = c["vocab"]
    z = torch.randn(rows, V + c["pad"], device="cuda", generator=gen)
    if c["dist"] == "normal":
        z.mul_(2.0 if c["call"] == "windows" else 3.0)
        ids = torch.randint(V, (rows, 16), device="cuda", generator=gen)
        z.scatter_add_(1, ids, 8.0 + 6.0 * torch.rand(rows, 16, device="cuda", generator=gen))
    else:
        den = torch.zeros_like(z)
        for _ in range(3):
            den += torch.randn(rows, V + c["pad"], device="cuda", generator=gen).square_()
        z.mul_(4.0).div_(den.div_(3.0).sqrt_())
        if c["dist"] == "student":
            z.div_(30.0).tanh_().mul_(30.0)
    return z[:, :V]


def _histories(c, rng, logits, rows, n, offset=0):
    """Token ids with Zipf frequencies (low ids are common); one in eight is a token the model rates highly now, as
    recently used words are."""
    V = c["vocab"] * c["shards"]
    cdf = np.cumsum(1.0 / np.arange(1, V + 1) ** 1.1)
    ids = np.searchsorted(cdf / cdf[-1], rng.random((rows, n))).astype(np.int32).clip(0, V - 1)
    top = torch.topk(logits[:rows], 16, dim=1).indices.cpu().numpy().astype(np.int32) + offset
    hot = rng.random((rows, n)) < 0.125
    pick = np.take_along_axis(top, rng.integers(0, 16, (rows, n)), axis=1)
    return [np.ascontiguousarray(h) for h in np.where(hot, pick, ids)]


class _DeviceInts:
    """A device array of int32 as torch's tensor constructor can take it."""

    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<i4", "data": (int(ptr), False), "version": 2}


def prepare(case, seed):
    c = dict(case)
    rng = np.random.default_rng([seed, 17])
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    call, R, V = c["call"], c["rows"], c["vocab"]
    n_logits = R * c["window"]
    hist_ids = R * (c["hist"] + c["window"]) + 1024
    if call in ("resident", "draft"):   # regions of power-of-two size, with room for what is generated
        hist_ids = R * 4 * (c["hist"] + c["window"] + c["steps"] * R + 256)
    eng = fb.Engine(device=0, max_rows=n_logits, max_vocab=V, max_hist_ids=hist_ids)
    eng.set_cuda_stream(torch.cuda.current_stream().cuda_stream)
    if c["softcap"]:
        eng.set_softcap(c["softcap"])
    s = {"case": c, "engine": eng}
    p = _params(c, R, seed)

    if call == "class":
        lg = _logits(c, gen, 1)
        s["history"] = _histories(c, rng, lg, 1, c["hist"])[0]
        s["fresh"] = lg[0].cpu().numpy()
        s["row"] = s["fresh"].copy()
        s["sampler"] = fb.Sampler(p, eng)
        return s

    if call == "resident":
        s["logits"] = [_logits(c, gen, R) for _ in range(min(2, c["steps"]))]
        s["prompts"] = _histories(c, rng, s["logits"][0], R, c["hist"])
        s["params"], s["pass"] = p, 0
        s["sids"] = eng.open_streams(p)
        for sid, h in zip(s["sids"], s["prompts"]):
            eng.history_set(int(sid), h)
        return s

    if call == "shard":
        lg = _logits(c, gen, R)
        hists = _histories(c, rng, lg, R, c["hist"])
        eng.set_vocab_shard(0, V * c["shards"])
        s["logits"], s["sids"] = lg, eng.open_streams(p)
        s["batch"] = b = eng.prepare_batch(s["sids"], hists, V)
        s["stride"] = b.max_k + 1
        s["packed"] = torch.zeros(R, s["stride"], dtype=torch.int64, device="cuda")
        s["block"] = block = -(-R // c["shards"])   # the rows this rank finishes, as an all-to-all leaves them
        s["lists"] = torch.zeros(c["shards"], block, s["stride"], dtype=torch.int64, device="cuda")
        for g in range(1, c["shards"]):             # the other ranks' lists of those rows
            eng.set_vocab_shard(g * V, V * c["shards"])
            other = _logits(c, gen, R)
            b.shard_launch_packed(other.data_ptr(), s["packed"].data_ptr(), s["stride"])
            s["lists"][g].copy_(s["packed"][:block])
            b.check()
        eng.set_vocab_shard(0, V * c["shards"])
        s["packed"].zero_()
        s["tokens"] = torch.as_tensor(_DeviceInts(b.tokens_device_ptr, R), device="cuda")[:block]
        return s

    s["logits"] = lg = _logits(c, gen, n_logits)
    s["sids"] = eng.open_streams(p)
    if call in ("windows", "draft"):
        W = c["window"]
        first = lg.view(R, W, -1)[:, 0]
        hists = _histories(c, rng, first, R, c["hist"])
        best = torch.argmax(lg, dim=1).cpu().numpy().astype(np.int32).reshape(R, W)
        right = np.minimum(rng.geometric(0.3, R) - 1, W - 1)   # drafts that agree with the model, then some that do not
        drafts = np.where(np.arange(W - 1)[None, :] < right[:, None], best[:, :W - 1], rng.integers(2, V, (R, W - 1))).astype(np.int32)
        if call == "windows":
            s["rows"] = [np.concatenate([h[-1:], d]).astype(np.int32) for h, d in zip(hists, drafts)]
        else:   # somewhere in the prompt stands what the drafts repeat, behind the four ids the prompt ends with
            for h, d in zip(hists, drafts):
                at = int(rng.integers(0, len(h) - 4 - (W - 1) - 4 + 1))
                h[at:at + 4] = h[-4:]
                h[at + 4:at + 4 + len(d)] = d
            for sid, h in zip(s["sids"], hists):
                eng.history_set(int(sid), h)
            s["last"] = np.array([h[-1] for h in hists], dtype=np.int32)
    else:
        hists = _histories(c, rng, lg, R, c["hist"])
    s["hists"] = hists
    if call == "launch":
        s["batch"] = eng.prepare_batch(s["sids"], hists, V, ld=lg.stride(0))
        s["tokens"] = torch.as_tensor(_DeviceInts(s["batch"].tokens_device_ptr, R), device="cuda")
    return s


# ------------------------------------------------------------------------------------------------ one pass
def run(s):
    c, eng = s["case"], s["engine"]
    call = c["call"]
    if call == "step":
        return eng.sample_batch(s["sids"], s["logits"], s["hists"], n_vocab=c["vocab"])
    if call == "launch":
        s["batch"].launch(s["logits"].data_ptr())
        return s["tokens"]
    if call == "class":
        np.copyto(s["row"], s["fresh"])   # the model's logits, read back
        token = s["sampler"].sample(s["row"], c["vocab"], s["history"])
        return {"token": token, "row": s["row"]}
    if call == "resident":
        i = s["pass"] % c["rows"]
        s["pass"] += 1
        eng.close_stream(int(s["sids"][i]))
        s["sids"][i] = eng.open_stream(s["params"][i:i + 1])
        eng.history_set(int(s["sids"][i]), s["prompts"][i])
        return [eng.sample_batch_resident(s["sids"], s["logits"][t % len(s["logits"])].data_ptr(), n_vocab=c["vocab"], flags=fb.APPEND_SAMPLED)
                for t in range(c["steps"])]
    if call == "windows":
        tokens, accepted, confirmed = eng.verify_windows(s["sids"], s["rows"], s["logits"], s["hists"], n_vocab=c["vocab"])
        return {"tokens": np.concatenate(tokens), "accepted": accepted, "confirmed": confirmed}
    if call == "draft":
        drafts = eng.lookup_drafts(s["sids"], DRAFTS, 2, EOS)
        rows = [np.concatenate([s["last"][i:i + 1], d]) for i, d in enumerate(drafts)]
        tokens, accepted, confirmed = eng.verify_windows_resident(s["sids"], rows, s["logits"], n_vocab=c["vocab"])
        return {"drafts": np.concatenate(rows), "tokens": np.concatenate(tokens), "accepted": accepted, "confirmed": confirmed}
    b = s["batch"]
    b.redraw()
    b.shard_launch_packed(s["logits"].data_ptr(), s["packed"].data_ptr(), s["stride"])
    s["lists"][0].copy_(s["packed"][:s["block"]])   # this rank's own lists, where the exchange would leave them
    b.merge_launch_packed(s["lists"].data_ptr(), s["stride"], c["shards"], 0, s["block"])
    b.check()
    return {"tokens": s["tokens"], "lists": s["packed"]}


def work(case):
    """Each logit and each window id read once, one engine output read and one token written per row; one comparison
    per logit, an exponential (counted as 20) where the whole vocabulary is weighed, a tanh (20) under the softcap."""
    c = case
    rows = c["rows"] * c["window"] * c["steps"]
    bytes_ = rows * (4 * c["vocab"] + (4 * c["hist"] if c["penalty"] != 1.0 else 0) + 12)
    per_logit = 1 + (20 if c["sampler"] == "nucleus" else 10 if c["sampler"] == "mixed" else 0) + (20 if c["softcap"] else 0)
    if c["call"] == "shard":
        bytes_ += c["rows"] * (c["top_k"] + 1) * 8 * 2
    if c["call"] == "class":
        bytes_ += 4 * c["hist"]
    return {"bytes": bytes_, "flops": rows * c["vocab"] * per_logit}


def tolerance(case):
    """Token ids, candidate lists and penalised logits follow from the inputs bit for bit."""
    return "exact"
