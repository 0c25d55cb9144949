"""The work that users have this backend do, as cases that can be timed and compared.

Three things go through the public entry points:

  sampled    one conversation turn with the sampler on the host: Prefill of a prompt, then DecodeLogits for every
             token the host picked (the reference's call sequence with its CPU sampler, constrained decoding, scoring)
  greedy     one turn decoded on the device: Prefill, DecodeTokens, and the logits of the step after it
  group      several sessions over one weight copy: PrefillSession for each, DecodeTokensBatch in lockstep, then the
             logits of the next step of one session that leaves the group
  attention  split-KV decode attention over caller-owned device buffers (the allocation-free operator)

Every pass starts its sessions over (Reset), so it can be repeated on the same executor.
"""
import dataclasses
import math

import numpy as np
import torch

import __graft_entry__ as graft

pkg = graft.load_package()
mio = pkg.model_io

MIB = 1 << 20

#: KV cache type of each model, as the repository's configurations and bench use them.
KV = {"gemma3-1b": "fp32", "gemma3-4b-slice": "fp32", "gemma3-27b-slice": "bf16", "small-gqa": "bf16", "small": "fp32"}


# ------------------------------------------------------------------------------------------------- cases

def listed():
    return [
        # A short question to the 1B model, time to the first logits: launches, small token tiles, a ragged length.
        {"name": "first-logits-37", "kind": "sampled", "model": "gemma3-1b", "prompt": 37, "steps": 1},
        # The benchmark's prompt, time to the first logits.
        {"name": "first-logits-1024", "kind": "sampled", "model": "gemma3-1b", "prompt": 1024, "steps": 1},
        # A long document near the context limit: three work groups, the last one ragged.
        {"name": "first-logits-3001", "kind": "sampled", "model": "gemma3-1b", "prompt": 3001, "steps": 1},
        # The benchmark: 1024-token prompt, 256 greedy tokens.
        {"name": "greedy-1024-256", "kind": "greedy", "model": "gemma3-1b", "prompt": 1024, "steps": 256},
        # A chat turn whose tokens are picked on the host: every step's logits cross to host memory.
        {"name": "sampled-203-48", "kind": "sampled", "model": "gemma3-1b", "prompt": 203, "steps": 48},
        # A few conversations at once on the 1B model, prompts of different lengths.
        {"name": "group-4x300-64", "kind": "group", "model": "gemma3-1b", "sessions": 4, "prompt": 300, "steps": 64},
        # A small server on the 4B layer geometry: an odd number of sessions and ragged prompts.
        {"name": "group-9x511-48", "kind": "group", "model": "gemma3-4b-slice", "sessions": 9, "prompt": 511, "steps": 48},
        # The multi-session benchmark's load on one GPU, on the 4B layer geometry: 64 sessions of 1024 + 128.
        {"name": "group-64x1024-128", "kind": "group", "model": "gemma3-4b-slice", "sessions": 64, "prompt": 1024, "steps": 128},
        # The largest layers (27B geometry, bf16 cache): prompt and decode for one user.
        {"name": "greedy-27b-700-32", "kind": "greedy", "model": "gemma3-27b-slice", "prompt": 700, "steps": 32},
        # A tiny assistant model with grouped heads and a bf16 cache: overhead of every call.
        {"name": "greedy-small-50-12", "kind": "greedy", "model": "small-gqa", "prompt": 50, "steps": 12},
        # The attention operator: one query on a short fp32 cache ...
        {"name": "attention-1x1000", "kind": "attention", "batch": 1, "keys": 1000, "hq": 4, "hkv": 1, "hd": 256, "kv": "fp32",
         "window": 0, "splits": 3},
        # ... and 64 samples over one long shared prompt in bf16.
        {"name": "attention-64x32768", "kind": "attention", "batch": 64, "keys": 32768, "hq": 4, "hkv": 1, "hd": 256, "kv": "bf16",
         "window": 0, "splits": 31},
    ]


def _log(rng, lo, hi):
    """A whole number from lo to hi, spread over the logarithm."""
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def _splits(batch, keys, hq, hd):
    """What the attention benchmark asks for: one split per page, as far as the operator's scratch holds them."""
    room = (8 * MIB - 65536) // (batch * hq * (hd + 2) * 4)
    return max(1, min(64, keys // 256, room))


def draw(rng):
    kind = rng.choice(["sampled", "sampled", "greedy", "greedy", "group", "group", "attention", "attention"])
    if kind == "attention":
        hq, hkv, hd = rng.choice([(4, 1, 256), (4, 1, 256), (8, 4, 256), (32, 16, 128), (8, 4, 128)])
        batch, keys = _log(rng, 1, 64), _log(rng, 300, 32768)
        return {"kind": kind, "batch": batch, "keys": keys, "hq": hq, "hkv": hkv, "hd": hd, "kv": rng.choice(["bf16", "fp32"]),
                "window": rng.choice([0, 0, 512]), "splits": _splits(batch, keys, hq, hd)}
    if kind == "group":
        if rng.random() < 0.5:
            return {"kind": kind, "model": "gemma3-1b", "sessions": _log(rng, 2, 24), "prompt": _log(rng, 16, 700), "steps": _log(rng, 8, 64)}
        return {"kind": kind, "model": "gemma3-4b-slice", "sessions": _log(rng, 5, 64), "prompt": _log(rng, 16, 1024), "steps": _log(rng, 8, 64)}
    model = rng.choice(["gemma3-1b", "gemma3-1b", "gemma3-1b", "gemma3-4b-slice", "gemma3-27b-slice", "small", "small-gqa"])
    top = {"gemma3-1b": 3072, "gemma3-4b-slice": 1800, "gemma3-27b-slice": 1800, "small": 800, "small-gqa": 400}[model]
    return {"kind": kind, "model": model, "prompt": _log(rng, 8, top), "steps": _log(rng, 1, 64) if kind == "sampled" else _log(rng, 4, 96)}


# ------------------------------------------------------------------------------------------------- models

_owners = {}


def _int4(w):
    """Symmetric int4 rows as model_io.quantize_int4 packs them, on the GPU."""
    scale = w.abs().amax(dim=1).clamp_min(1e-12) / 7.0
    q = torch.round(w / scale[:, None]).clamp_(-7, 7).to(torch.int32) & 0xF
    return (q[:, 0::2] | (q[:, 1::2] << 4)).to(torch.uint8).cpu().numpy(), scale.cpu().numpy()


def _config(model):
    return dataclasses.replace(mio.CONFIGS[model](), kv_dtype=1 if KV[model] == "bf16" else 0)


def _owner(model):
    """One weight copy per model and process, as a server keeps it: random-init weights of the repository's
    distribution, N(0, 0.02) before quantisation, gains 1 + N(0, 0.02).  The two post-norm gains are a quarter of
    that, so that the residual stream keeps the token and the model is as sure of its next token as a trained one:
    greedy ids can then be compared one by one."""
    if model not in _owners:
        cfg = _config(model)
        gen = torch.Generator(device="cuda").manual_seed(cfg.seed + 1)
        tensors = {}

        def mat(name, rows, cols):
            parts = [_int4(torch.randn(min(32768, rows - r), cols, device="cuda", generator=gen) * 0.02) for r in range(0, rows, 32768)]
            tensors[name + ".q"] = np.concatenate([p[0] for p in parts])
            tensors[name + ".scale"] = np.concatenate([p[1] for p in parts])

        def gain(name, n, base):
            tensors[name] = ((1.0 + 0.02 * torch.randn(n, device="cuda", generator=gen)) * base).cpu().numpy()

        d, hd = cfg.d_model, cfg.head_dim
        mat("embed", cfg.vocab, d)
        for i in range(cfg.n_layers):
            p = "L%d." % i
            mat(p + "wqkv", cfg.n_qkv_rows, d)
            mat(p + "wo", d, cfg.n_q_heads * hd)
            mat(p + "wgate", cfg.ffn, d)
            mat(p + "wup", cfg.ffn, d)
            mat(p + "wdown", d, cfg.ffn)
            for name, n, base in (("pre_attn", d, 1.0), ("post_attn", d, 0.25), ("pre_ffn", d, 1.0), ("post_ffn", d, 0.25),
                                  ("q_norm", hd, 1.0), ("k_norm", hd, 1.0)):
                gain(p + name, n, base)
        gain("final_norm", d, 1.0)
        torch.cuda.empty_cache()
        image = mio.export_model_litertlm(cfg, mio.pack_weights_record(cfg, tensors))
        _owners[model] = pkg.B200LlmExecutor(image, max_num_tokens=256)
    return _owners[model]


def _lengths(case):
    """Prompt length of every session: the first has the full one, the others end up to a third earlier."""
    if case["kind"] != "group":
        return [case["prompt"]]
    n = case["prompt"]
    return [n - (37 * i) % (n // 3 + 1) for i in range(case["sessions"])]


# ------------------------------------------------------------------------------------------------- the interface

class State:
    pass


def prepare(case, seed):
    s = State()
    s.case = case
    if case["kind"] == "attention":
        gen = torch.Generator(device="cuda").manual_seed(seed)
        b, keys, hq, hkv, hd = case["batch"], case["keys"], case["hq"], case["hkv"], case["hd"]
        pages = -(-keys // 256)
        kv = torch.bfloat16 if case["kv"] == "bf16" else torch.float32
        s.q = torch.randn(b, (hq + 2 * hkv) * hd, device="cuda", generator=gen)
        s.k = torch.randn(pages, hkv, 256, hd, device="cuda", generator=gen).to(kv)
        s.v = torch.randn(pages, hkv, 256, hd, device="cuda", generator=gen).to(kv)
        s.table = torch.randperm(pages, device="cuda", generator=gen).to(torch.int32)
        s.out = torch.empty(b, hq, hd, device="cuda")
        s.call = dict(batch=b, s=keys, hq=hq, hkv=hkv, hd=hd, window=case["window"], kv_bf16=case["kv"] == "bf16", nsplit=case["splits"],
                      stream=torch.cuda.current_stream().cuda_stream)
        return s
    cfg = _config(case["model"])
    rng = np.random.Generator(np.random.PCG64(seed))
    sessions, steps = case.get("sessions", 1), case["steps"]
    s.ids = [rng.integers(0, cfg.vocab, n).astype(np.int32) for n in _lengths(case)]
    s.picked = [int(t) for t in rng.integers(0, cfg.vocab, steps)]     # what the host's sampler answers
    room = case["prompt"] + steps + 1
    s.ex = _owner(case["model"]).CreateShared(n_sessions=sessions, max_num_tokens=-(-room // 256) * 256)
    # logits land in page-locked memory, as a host sampler keeps them
    rows = steps if case["kind"] == "sampled" else 1
    s.pinned = torch.empty(rows, cfg.vocab, dtype=torch.float32, pin_memory=True)
    s.logits = s.pinned.numpy()
    return s


def run(s):
    case = s.case
    if case["kind"] == "attention":
        pkg.ops.attention_decode_static(s.q.data_ptr(), s.k.data_ptr(), s.v.data_ptr(), s.table.data_ptr(), s.out.data_ptr(), **s.call)
        return s.out
    ex = s.ex
    if case["kind"] == "group":
        for i, ids in enumerate(s.ids):
            ex.SelectSession(i)
            ex.Reset()
            ex.PrefillSession(i, ids, wait_for_completion=False)
        out = ex.DecodeTokensBatch(case["steps"])
        ex.SelectSession(case["sessions"] - 1)
        ex.DecodeLogits(out=s.logits)
        return {"ids": out, "logits": s.logits}
    ex.Reset()
    ex.Prefill(s.ids[0])
    if case["kind"] == "greedy":
        out = ex.DecodeTokens(case["steps"])
        ex.DecodeLogits(out=s.logits)
        return {"ids": out, "logits": s.logits}
    ex.DecodeLogits(out=s.logits[0])
    for k in range(1, case["steps"]):
        ex.DecodeLogits(s.picked[k], out=s.logits[k])
    return s.logits


def work(case):
    if case["kind"] == "attention":
        keys = min(case["keys"], case["window"]) if case["window"] else case["keys"]
        size = 2 if case["kv"] == "bf16" else 4
        rows = case["batch"] * case["hq"] * case["hd"]
        return {"bytes": 2.0 * keys * case["hkv"] * case["hd"] * size + 8.0 * rows, "flops": 4.0 * rows * keys}
    cfg = _config(case["model"])
    steps, sessions = case["steps"], case.get("sessions", 1)
    size = 2 if cfg.kv_dtype else 4
    d, hd, f = cfg.d_model, cfg.head_dim, cfg.ffn
    layer_bytes = cfg.layer_params() / 2 + 4.0 * (cfg.n_qkv_rows + 2 * d + 2 * f + 4 * d + 2 * hd)
    weights, head = cfg.n_layers * layer_bytes, cfg.vocab * (d / 2 + 4.0)
    n_glob = sum(1 for i in range(cfg.n_layers) if cfg.is_global(i))
    row = 2.0 * cfg.n_kv_heads * hd * size                                   # K and V of one position of one layer
    nbytes = flops = 0.0

    def step(positions, logits):
        """One decode step of the sessions at these positions: weights once, every visible K / V row once."""
        nonlocal nbytes, flops
        seen = sum(n_glob * (p + 1) + (cfg.n_layers - n_glob) * min(p + 1, cfg.window) for p in positions)
        nbytes += weights + head + row * (seen + cfg.n_layers * len(positions)) + (4.0 * cfg.vocab if logits else 0.0)
        flops += len(positions) * 2.0 * (cfg.n_layers * cfg.layer_params() + cfg.vocab * d) + 4.0 * hd * cfg.n_q_heads * seen

    lengths = _lengths(case)
    for n in lengths:                                                        # the last id is held back for the first step
        if n > 1:
            nbytes += weights + (n - 1) * (cfg.n_layers * row + d / 2)
            flops += cfg.prefill_flops(n - 1)
    for k in range(steps):
        step([n - 1 + k for n in lengths], case["kind"] == "sampled")
    if case["kind"] != "sampled":
        step([lengths[sessions - 1] - 1 + steps], True)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    if case["kind"] == "attention":
        return {"rel": 1e-5, "max": 1e-4}        # fp32 queries, sums and results; the cache enters exactly
    return {"rel": 1e-2, "max": 0.1}             # bf16 activations in prefill (and in groups of more than four); ids exactly
