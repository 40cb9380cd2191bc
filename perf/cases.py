"""Timed cases of the framework's public entry points, and what each has to move and compute.

A case is one call (or the few calls of one job) as a user's program makes it: one token with its logits, a self-loop on the GPU,
a prompt prefill, the logits of a whole text, a batch of jobs, a served set of sessions.  Models are the repository's own tiny and
3B shapes with random weights in the three formats it loads: fp16, int8 with one (scale, zero) per output row, and int8 with one per
row and group of 128 (the reference quantiser's files, "int8g").  A program keeps its model, so a model is loaded once for all
cases that follow each other on it; the checkpoints are written once per machine.
"""
import json
import math
import os
import tempfile

import numpy as np
import torch

import rwkv_rsv_b200 as rsv

# ---- the cases -----------------------------------------------------------------------------------------------------------------
# sampler: "argmax"; "chat" = temperature 0.8, top-k 50, top-p 0.9; "nucleus" = temperature 1, top-p 0.9 over the whole vocabulary.


def listed():
    return [
        # The smallest call: one token in, logits out, a model that fits the L2 (latency and launches count).
        {"name": "tiny token", "kind": "token", "shape": "tiny", "weights": "fp16", "tokens": 1},
        # Interactive decode with the sampler on the host: one token in, 65536 logits out.
        {"name": "3b int8 token", "kind": "token", "shape": "3b", "weights": "int8", "tokens": 1},
        # One user's greedy answer, generated on the GPU.
        {"name": "3b int8 greedy x1", "kind": "loop", "shape": "3b", "weights": "int8", "sessions": 1, "steps": 64, "sampler": "argmax"},
        # A few users at once.
        {"name": "3b int8 greedy x3", "kind": "loop", "shape": "3b", "weights": "int8", "sessions": 3, "steps": 16, "sampler": "argmax"},
        # The ordinary serving batch.
        {"name": "3b int8 chat x64", "kind": "loop", "shape": "3b", "weights": "int8", "sessions": 64, "steps": 16, "sampler": "chat"},
        # The largest batch of the decode sweep: the sessions' states are most of the traffic.
        {"name": "3b int8 nucleus x1024", "kind": "loop", "shape": "3b", "weights": "int8", "sessions": 1024, "steps": 4, "sampler": "nucleus"},
        # A long prompt in chunks.
        {"name": "3b int8 prefill 2048", "kind": "prefill", "shape": "3b", "weights": "int8", "tokens": 2048, "chunk": 512},
        # Continuous batching: prompts and generations of very different lengths packed into every step.
        {"name": "3b int8 serve x32", "kind": "serve", "shape": "3b", "weights": "int8", "sessions": 32, "longest": 512, "mean_new": 32, "sampler": "chat"},
        # A small batch on the reference's own int8 files.
        {"name": "3b int8g chat x16", "kind": "loop", "shape": "3b", "weights": "int8g", "sessions": 16, "steps": 8, "sampler": "chat"},
        # Scoring a text: logits at every position, ragged length.
        {"name": "3b int8g score 201", "kind": "score", "shape": "3b", "weights": "int8g", "tokens": 201},
        # One user's sampled answer.
        {"name": "3b fp16 chat x1", "kind": "loop", "shape": "3b", "weights": "fp16", "sessions": 1, "steps": 32, "sampler": "chat"},
        # A static batch of jobs: ragged prompts, then a fixed number of sampled tokens each.
        {"name": "3b fp16 jobs x20", "kind": "jobs", "shape": "3b", "weights": "fp16", "sessions": 20, "longest": 512, "steps": 12, "sampler": "chat"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["token", "loop", "loop", "loop", "prefill", "score", "jobs", "serve"])
    c = {"kind": kind, "shape": "tiny" if rng.random() < 0.2 else "3b", "weights": rng.choice(["fp16", "int8", "int8", "int8g"])}
    if kind == "token":
        c["tokens"] = _log_int(rng, 2, 32)
    elif kind == "loop":
        c["sessions"] = _log_int(rng, 1, 768)
        c["steps"] = max(2, min(rng.randint(8, 64), 2048 // c["sessions"]))
        c["sampler"] = rng.choice(["argmax", "chat", "nucleus"] if c["sessions"] >= 256 else ["argmax", "chat"])
    elif kind == "prefill":
        c["tokens"] = _log_int(rng, 16, 2048)
        c["chunk"] = rng.choice([128, 256, 512])
    elif kind == "score":
        c["tokens"] = _log_int(rng, 8, 256)
    elif kind == "jobs":
        c.update(sessions=_log_int(rng, 2, 16), longest=_log_int(rng, 48, 512), steps=rng.randint(4, 16), sampler=rng.choice(["argmax", "chat"]))
    else:
        c["weights"] = "fp16" if c["weights"] == "int8g" else c["weights"]
        c.update(sessions=_log_int(rng, 6, 40), longest=_log_int(rng, 48, 512), mean_new=_log_int(rng, 8, 32), sampler=rng.choice(["argmax", "chat"]))
    return c


def _prompt_lengths(c):
    """Log-uniform lengths from 16 to `longest`, one quantile per session, in an order that mixes short and long."""
    n = c["sessions"]
    return [int(16 * (c["longest"] / 16) ** ((i * 7 % n + 0.5) / n if n % 7 else (i + 0.5) / n)) for i in range(n)]


def _new_lengths(c):
    """Geometric generation lengths, one quantile per session, in another order than the prompts."""
    n, m = c["sessions"], c["mean_new"]
    return [max(1, min(4 * m, math.ceil(-m * math.log(1 - ((i * 11 % n if n % 11 else i) + 0.5) / n)))) for i in range(n)]


# ---- random-init checkpoints ---------------------------------------------------------------------------------------------------
_DIR = os.path.join(tempfile.gettempdir(), "rwkv7_cases_%d" % os.getuid())
_MODELS = {}


def _tensors(sh):
    """(name, shape, distribution) of every tensor: matrices N(0, 0.02), norms around 1, mixes uniform."""
    C, F, V, H, N = sh["n_embd"], sh["ffn_hidden"], sh["vocab"], sh["n_head"], sh["head_size"]
    small, one, unit = ("n", 0.0, 0.02), ("n", 1.0, 0.02), ("u", 0.0, 1.0)
    yield "emb.weight", (V, C), small
    for s, d in (("weight", one), ("bias", small)):
        yield "blocks.0.ln0." + s, (C,), d
        yield "ln_out." + s, (C,), d
    yield "head.weight", (V, C), small
    for i in range(sh["n_layer"]):
        p = "blocks.%d." % i
        for s, d in (("weight", one), ("bias", small)):
            for ln in ("ln1.", "ln2.", "att.ln_x."):
                yield p + ln + s, (C,), d
        for x in ("att.x_r", "att.x_w", "att.x_k", "att.x_v", "att.x_a", "att.x_g", "att.k_a", "ffn.x_k"):
            yield p + x, (1, 1, C), unit
        yield p + "att.w0", (1, 1, C), ("u", -6.0, -1.0)
        yield p + "att.a0", (1, 1, C), small
        yield p + "att.v0", (1, 1, C), small
        yield p + "att.k_k", (1, 1, C), ("u", 0.5, 1.5)
        yield p + "att.r_k", (H, N), small
        for x in "wavg":
            yield p + "att.%s1" % x, (C, sh[x + "_mid"]), small
            yield p + "att.%s2" % x, (sh[x + "_mid"], C), small
        for x in ("receptance", "key", "value", "output"):
            yield p + "att.%s.weight" % x, (C, C), small
        yield p + "ffn.key.weight", (F, C), small
        yield p + "ffn.value.weight", (C, F), small


def _quantised(name, weights):
    return weights != "fp16" and name.startswith("blocks.") and name.split(".")[-1] == "weight" and name.split(".")[-2] in ("receptance", "key", "value", "output")


def _quantise(w, weights):
    """[M, K] -> u8 codes and the u32 words (scale fp16 | zero fp16 << 16) of every row and group of 128."""
    M, K = w.shape
    if weights == "int8":  # symmetric per output row
        s = (w.abs().amax(1, keepdim=True) / 127).half()
        z = (-128 * s.float()).half()
        q = (w / s.float()).round().clamp(-127, 127) + 128
        s, z = s.expand(M, K // 128), z.expand(M, K // 128)
    else:  # the range of every group
        g = w.view(M, K // 128, 128)
        lo, hi = g.amin(2), g.amax(2)
        step = (hi - lo) / 255
        q = ((g - lo[:, :, None]) / step[:, :, None]).round().clamp(0, 255).view(M, K)
        s, z = step.half(), lo.half()
    words = torch.stack([s, z], 2).contiguous().view(torch.int32)
    return q.to(torch.uint8), words


def _checkpoint(shape, weights):
    path = os.path.join(_DIR, "%s_%s.safetensors" % (shape, weights))
    if os.path.exists(path):
        return path
    os.makedirs(_DIR, exist_ok=True)
    parts, header, at = [], {}, 0
    for name, dims, dist in _tensors(rsv.SHAPES[shape]):
        n = math.prod(dims)
        if _quantised(name, weights):
            pieces = [(name + ".int8_idx", "U8", dims, n), (name + ".int8_sz", "U32", (dims[0], dims[1] // 128), n // 128 * 4)]
        else:
            pieces = [(name, "F16", dims, 2 * n)]
        for key, dtype, d, size in pieces:
            header[key] = {"dtype": dtype, "shape": list(d), "data_offsets": [at, at + size]}
            at += size
        parts.append((name, dims, dist))
    text = json.dumps(header).encode()
    text += b" " * (-len(text) % 8)
    gen = torch.Generator("cuda").manual_seed(0)
    tmp = "%s.%d" % (path, os.getpid())
    with open(tmp, "wb") as f:
        f.write(len(text).to_bytes(8, "little") + text)
        for name, dims, (d, a, b) in parts:
            x = torch.randn(dims, generator=gen, device="cuda") * b + a if d == "n" else torch.rand(dims, generator=gen, device="cuda") * (b - a) + a
            x = x.half()
            for y in _quantise(x.float(), weights) if _quantised(name, weights) else (x,):
                y.cpu().numpy().tofile(f)
    os.replace(tmp, path)
    torch.cuda.empty_cache()
    return path


def _model(case):
    key = (case["shape"], case["weights"])
    if key not in _MODELS:
        _MODELS.clear()  # a program serves one model; what is still in use keeps its own reference
        _MODELS[key] = rsv.Model(_checkpoint(*key))
    return _MODELS[key]


# ---- preparation and one pass --------------------------------------------------------------------------------------------------
def _sampler(name, seed):
    return {"argmax": None, "chat": rsv.SamplerParams(temperature=0.8, top_k=50, top_p=0.9, seed=seed),
            "nucleus": rsv.SamplerParams(temperature=1.0, top_p=0.9, seed=seed)}[name]


def prepare(case, seed):
    m = _model(case)
    rng = np.random.default_rng(seed)
    tokens = lambda n: rng.integers(0, m.info().num_vocab, size=n).astype(np.uint32)  # noqa: E731
    s = {"case": case, "model": m}
    kind = case["kind"]
    if kind in ("token", "prefill", "score") or (kind == "loop" and case["sessions"] == 1):
        s["bundle"] = rsv.Bundle(m)
    if kind == "token":
        s["bundle"].infer_seq(tokens(32))
        s["tokens"] = tokens(case["tokens"])
    elif kind in ("prefill", "score"):
        s["tokens"] = tokens(case["tokens"])
    elif kind == "loop":
        # sessions in the middle of their answers, each with a context of its own
        if case["sessions"] == 1:
            s["bundle"].infer_seq(tokens(32))
            s["seeds"] = tokens(1)
        else:
            s["state"] = m.create_batch_state(case["sessions"])
            s["seeds"] = m.forward_seq_batch(s["state"], [tokens(8) for _ in range(case["sessions"])])
        s["sampler"] = _sampler(case["sampler"], seed % 1000003)
    elif kind == "jobs":
        s["state"] = m.create_batch_state(case["sessions"])
        s["prompts"] = [tokens(n) for n in _prompt_lengths(case)]
        s["sampler"] = _sampler(case["sampler"], seed % 1000003)
    else:
        s["scheduler"] = rsv.Scheduler(m, max_slots=case["sessions"], chunk=512, max_new_cap=4 * case["mean_new"])
        s["prompts"] = [tokens(n) for n in _prompt_lengths(case)]
        s["new"] = _new_lengths(case)
        s["samplers"] = [_sampler(case["sampler"], seed % 1000003 + 7919 * i) for i in range(case["sessions"])]
    return s


def run(s):
    case, m = s["case"], s["model"]
    kind = case["kind"]
    if kind == "token":
        return s["bundle"].infer_tokens(s["tokens"])
    if kind == "prefill":
        s["bundle"].reset()
        return s["bundle"].infer_chunked(s["tokens"], case["chunk"])
    if kind == "score":
        s["bundle"].reset()
        return s["bundle"].infer(rsv.RnnInput(s["tokens"], option=rsv.RnnOption.Full))
    if kind == "loop" and case["sessions"] == 1:
        b, first = s["bundle"], int(s["seeds"][0])
        out = b.infer_argmax_selfloop(first, case["steps"]) if s["sampler"] is None else b.infer_sample_selfloop(first, case["steps"], s["sampler"])
        s["seeds"] = out[-1:]
        return out
    if kind == "loop":
        out = m.collect_sample_selfloop_batch(m.submit_sample_selfloop_batch(s["state"], s["seeds"], case["steps"], s["sampler"]))
        s["seeds"] = out[:, -1]
        return out
    if kind == "jobs":
        s["state"].reset()
        seeds = m.forward_seq_batch(s["state"], s["prompts"])
        return m.collect_sample_selfloop_batch(m.submit_sample_selfloop_batch(s["state"], seeds, case["steps"], s["sampler"]))
    ids = [s["scheduler"].submit(p, n, sp) for p, n, sp in zip(s["prompts"], s["new"], s["samplers"])]
    done = s["scheduler"].run_until_done()
    return np.concatenate([done[i] for i in ids])


# ---- what a pass cannot do without ---------------------------------------------------------------------------------------------
def work(case):
    """Bytes: the layers' weights and the head once per step that depends on the step before it (a prefill is one step), the sessions'
    states read and written once per step, the embedding rows, the logits that are returned.  Operations: two per weight and row."""
    sh = rsv.SHAPES[case["shape"]]
    L, C, F, V, H, N = (sh[k] for k in ("n_layer", "n_embd", "ffn_hidden", "vocab", "n_head", "head_size"))
    big, rank = L * (4 * C * C + 2 * C * F), L * 2 * C * (sh["w_mid"] + sh["a_mid"] + sh["v_mid"] + sh["g_mid"])
    stored = {"fp16": 2 * big, "int8": big + L * (5 * C + F) * 4, "int8g": big + big // 32}[case["weights"]]
    layers = stored + 2 * rank + L * 19 * C * 4
    head, state = 2 * V * C, 4 * (L * (2 * C + H * N * N) + C)
    row_flops, head_flops = 2 * (big + rank) + 8 * L * H * N * N, 2 * V * C
    steps = lambda n, rows: {"bytes": n * (layers + head + rows * (2 * state + 2 * C)), "flops": n * rows * (row_flops + head_flops)}  # noqa: E731
    fill = lambda rows, sessions, logits: {"bytes": layers + (head if logits else 0) + sessions * 2 * state + rows * 2 * C,  # noqa: E731
                                           "flops": rows * row_flops + logits * head_flops}
    kind = case["kind"]
    if kind == "token":
        w = steps(case["tokens"], 1)
        w["bytes"] -= (case["tokens"] - 1) * head
        w["flops"] -= (case["tokens"] - 1) * head_flops
        w["bytes"] += 4 * V
    elif kind == "loop":
        w = steps(case["steps"], case["sessions"])
    elif kind in ("prefill", "score"):
        logits = case["tokens"] if kind == "score" else 1
        w = fill(case["tokens"], 1, logits)
        w["bytes"] += 4 * V * logits
    elif kind == "jobs":
        a, b = fill(sum(_prompt_lengths(case)), case["sessions"], 0), steps(case["steps"], case["sessions"])
        w = {k: a[k] + b[k] for k in a}
    else:
        new = _new_lengths(case)
        a, b, c = fill(sum(_prompt_lengths(case)), case["sessions"], case["sessions"]), steps(max(new) - 1, 0), steps(1, sum(new) - len(new))
        w = {"bytes": a["bytes"] + b["bytes"] + c["bytes"] - layers - head, "flops": a["flops"] + c["flops"]}
    return w


def tolerance(case):
    """Logits: fp32 activations and sums through all layers.  Tokens: a draw within rounding of a step of the distribution (or two
    logits within rounding of each other) takes the neighbour, and that session goes on from there."""
    return {"rel": 1e-5} if case["kind"] in ("token", "prefill", "score") else {"rel": 0.0, "differ": 0.01}
