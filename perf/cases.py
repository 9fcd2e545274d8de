"""The work that programs have this engine do, as a list of timed cases with their exact answers.

Every case goes through the model classes of `crane_b200` as a server or a script does.  Weights are random at the widths of the
configurations in `crane_b200.synth`; where one block is the subject, the model has one to four layers and a small vocabulary so that
the block is what takes the time.  `exact()` restates each model in 64-bit torch.
"""
import math
import zlib

import numpy as np
import torch

import crane_b200
from crane_b200 import synth

PAGE_V = 8192                    # vocabulary of the block-sized models

# widths of synth.QWEN3_0_6B, the text half of synth.QWEN3_VL_2B, and synth.QWEN3_8B
WIDTHS = {1024: (3072, 16, 8), 2048: (6144, 16, 8), 4096: (12288, 32, 8)}
# the recipes of `bench.py --config qwen3_8b_q4km` and of an all-Q8_0 file
RECIPES = {
    "q4_k_m": {"q_proj": "Q4_K", "k_proj": "Q4_K", "v_proj": "Q6_K", "o_proj": "Q4_K", "gate_proj": "Q4_K", "up_proj": "Q4_K", "down_proj": "Q6_K",
               "lm_head": "Q6_K", "embed_tokens": "Q4_K"},
    "q8_0": {n: "Q8_0" for n in ("q_proj", "k_proj", "v_proj", "o_proj", "gate_proj", "up_proj", "down_proj", "lm_head", "embed_tokens")},
}
BLOCK_BYTES = {"Q4_K": 144 / 256, "Q6_K": 210 / 256, "Q8_0": 34 / 32}
GGML = {"Q8_0": 8, "Q4_K": 12, "Q6_K": 14}


# ------------------------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # one user, one stream, the whole smallest model: forced tokens one by one at a chat prompt's length (the smallest call there is)
        {"name": "dense_token", "kind": "token", "width": 1024, "layers": 28, "vocab": 151936, "past": 128, "steps": 4},
        # a long prompt through one layer at the widest configuration
        {"name": "dense_prefill", "kind": "prefill", "width": 4096, "layers": 1, "rows": 4096, "past": 0},
        # the next turn of a conversation: a short odd-sized message behind a long cached prefix
        {"name": "dense_turn", "kind": "prefill", "width": 2048, "layers": 4, "rows": 77, "past": 1500},
        # plain bf16 operands and pages, as a server chooses that prefers speed to the last digits
        {"name": "dense_prefill_bf16", "kind": "prefill", "width": 2048, "layers": 4, "rows": 1111, "past": 0, "precision": "bf16"},
        # a server's decode rounds over 32 conversations of unequal lengths
        {"name": "dense_batch", "kind": "batch", "width": 4096, "layers": 2, "seqs": 32, "past": 900, "steps": 2},
        # the same from a quantised file, and its prompts
        {"name": "quant_batch", "kind": "batch", "width": 4096, "layers": 1, "seqs": 32, "past": 300, "steps": 2, "quant": "q4_k_m"},
        {"name": "quant_prefill", "kind": "prefill", "width": 4096, "layers": 1, "rows": 512, "past": 0, "quant": "q4_k_m"},
        # one user on a quantised file
        {"name": "quant_token", "kind": "token", "width": 2048, "layers": 2, "vocab": 32768, "past": 200, "steps": 4, "quant": "q8_0"},
        # the hybrid of recurrent and softmax layers: a long prompt, and tokens sampled from a shared prefix (fork, decode, free)
        {"name": "hybrid_prefill", "kind": "hybrid_prefill", "layers": 4, "rows": 4096},
        {"name": "hybrid_token", "kind": "hybrid_token", "layers": 8, "past": 1000, "steps": 8},
        # one 448 x 448 image through the whole vision tower
        {"name": "vision", "kind": "vision", "grid_h": 28, "grid_w": 28},
        # continuous batching on a layer-list model: portions of prompts beside decoded tokens, requests joining and leaving
        {"name": "ragged_serving", "kind": "ragged", "experts": 0, "requests": 5, "prompt": 420, "portion": 256, "tokens": 6},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["token", "prefill", "prefill", "batch", "batch", "quant_batch", "quant_prefill", "quant_token", "hybrid_prefill", "hybrid_token",
                       "vision", "ragged"])
    if kind == "token":
        w = rng.choice([1024, 2048, 4096])
        return {"kind": "token", "width": w, "layers": rng.randint(1, 4 if w > 1024 else 16), "vocab": rng.choice([PAGE_V, 32768, 50001]),
                "past": _log(rng, 2, 4000), "steps": rng.randint(1, 6)}
    if kind == "prefill":
        return {"kind": "prefill", "width": rng.choice([1024, 2048, 4096]), "layers": rng.randint(1, 2), "rows": _log(rng, 2, 3000),
                "past": rng.choice([0, 0, _log(rng, 1, 1000)]), "precision": rng.choice(["split", "split", "bf16"])}
    if kind == "batch":
        return {"kind": "batch", "width": rng.choice([1024, 2048, 4096]), "layers": rng.randint(1, 2), "seqs": _log(rng, 2, 48), "past": _log(rng, 20, 900),
                "steps": rng.randint(1, 3)}
    if kind == "quant_batch":
        return {"kind": "batch", "width": rng.choice([1024, 2048, 4096]), "layers": 1, "seqs": _log(rng, 2, 40), "past": _log(rng, 10, 60),
                "steps": rng.randint(1, 3), "quant": rng.choice(sorted(RECIPES))}
    if kind == "quant_prefill":
        return {"kind": "prefill", "width": rng.choice([1024, 2048, 4096]), "layers": 1, "rows": _log(rng, 2, 512), "past": 0,
                "quant": rng.choice(sorted(RECIPES))}
    if kind == "quant_token":
        return {"kind": "token", "width": rng.choice([1024, 2048, 4096]), "layers": rng.randint(1, 2), "vocab": PAGE_V, "past": _log(rng, 8, 100),
                "steps": rng.randint(2, 8), "quant": rng.choice(sorted(RECIPES))}
    if kind == "hybrid_prefill":
        return {"kind": "hybrid_prefill", "layers": rng.choice([4, 5]), "rows": _log(rng, 3, 3000)}
    if kind == "hybrid_token":
        return {"kind": "hybrid_token", "layers": rng.choice([4, 5, 8]), "past": _log(rng, 4, 1500), "steps": rng.randint(1, 8)}
    if kind == "vision":
        return {"kind": "vision", "grid_h": 2 * rng.randint(4, 16), "grid_w": 2 * rng.randint(4, 16)}
    return {"kind": "ragged", "experts": rng.choice([0, 8]), "requests": rng.randint(2, 6), "prompt": _log(rng, 5, 600), "portion": _log(rng, 32, 400),
            "tokens": rng.randint(2, 6)}


# ------------------------------------------------------------------------------------------------------------------ configurations
def _dense_config(case):
    ff, nh, nkv = WIDTHS[case["width"]]
    return dict(synth.QWEN3_8B, hidden_size=case["width"], intermediate_size=ff, num_attention_heads=nh, num_key_value_heads=nkv,
                num_hidden_layers=case["layers"], vocab_size=case.get("vocab", PAGE_V), tie_word_embeddings="quant" not in case)


def _hybrid_config(case):
    return dict(synth.QWEN3_5_0_8B, num_hidden_layers=case["layers"], vocab_size=PAGE_V)


def _vision_config():
    # the tower at full size; the text half is not run and is as small as its three DeepStack levels let it be
    text = dict(synth.QWEN3_VL_2B["text_config"], num_hidden_layers=3, vocab_size=1024, intermediate_size=512, num_attention_heads=2, num_key_value_heads=1)
    return dict(synth.QWEN3_VL_2B, text_config=text, image_token_id=1001, vision_start_token_id=1002, vision_end_token_id=1003)


def _ragged_config(case):
    return synth.fosovik_config(vocab=32768, blocks=1, moe=(case["experts"], 4, 896) if case["experts"] else None)


# ------------------------------------------------------------------------------------------------------------------ random tensors
def _gen(seed, name):
    return torch.Generator(device="cuda").manual_seed((int(seed) << 32) + zlib.crc32(name.encode()))


def _tensor(seed, name, shape, kind):
    """One bf16 tensor on the GPU with the distribution synth.make_tensor gives its kind."""
    fan = math.prod(shape[1:]) if len(shape) > 1 else 1
    mean, std = {"linear": (0.0, fan ** -0.5), "embed": (0.0, shape[1] ** -0.5 if len(shape) > 1 else 1.0), "norm": (1.0, 0.02), "norm0": (0.24, 0.05),
                 "a_log": (-2.0, 0.1), "dt_bias": (0.0, 1.0), "bias": (0.0, 0.02), "alpha": (0.5, 0.02)}[kind]
    g = _gen(seed, name)
    return torch.empty(shape or (1,), dtype=torch.bfloat16, device="cuda").normal_(mean, std, generator=g)


def _ids(seed, name, n, vocab):
    return torch.randint(0, vocab, (n,), generator=_gen(seed, name), device="cuda").cpu().numpy().astype(np.uint32)


_STAGE = {}


def _to_host(t):
    """A device tensor's bytes in host memory (one pinned buffer, used anew by the next call)."""
    n = t.numel() * t.element_size()
    if _STAGE.get("n", 0) < n:
        _STAGE.update(n=n, buf=torch.empty(n, dtype=torch.uint8, pin_memory=True))
    b = _STAGE["buf"][:n]
    b.copy_(t.contiguous().view(-1).view(torch.uint8))
    return b.numpy()


def _load_bf16(m, seed, name, shape, kind):
    m.load_tensor(name, _to_host(_tensor(seed, name, shape, kind)).view(np.uint16).reshape(shape or (1,)))


def _blocks(seed, name, rows, k, qt):
    """(ggml blocks [rows, bytes], their values in 64 bits on demand) of a random matrix with variance 1 / k; an embedding's is 1, so that the
    residual stream carries more than one layer adds to it, as it does in a trained model."""
    g = _gen(seed, name)
    ints = lambda lo, hi, *s: torch.randint(lo, hi, s, generator=g, device="cuda", dtype=torch.uint8)  # noqa: E731
    unit = torch.rand((rows, k // (32 if qt == "Q8_0" else 256)), generator=g, device="cuda") + 0.5
    unit = unit * (math.sqrt(k) if "embed" in name else 1.0)
    half = lambda x: x.to(torch.float16).contiguous().view(torch.uint8).reshape(*x.shape, 2)  # noqa: E731
    if qt == "Q8_0":
        d = unit / (73.0 * 1.04 * math.sqrt(k))
        q = ints(1, 255, rows, k // 32, 32)                       # two's complement bytes but -1 and 0: values spread over [-128, 127]
        raw = torch.cat([half(d), q], -1).reshape(rows, -1)
        return raw, lambda: (q.view(torch.int8).double() * d.to(torch.float16).double()[..., None]).reshape(rows, k)
    nb = k // 256
    if qt == "Q4_K":
        d = unit / (199.0 * math.sqrt(k))
        dm = 7.5 * d
        sc, qs = ints(16, 64, rows, nb, 8), ints(0, 256, rows, nb, 4, 32)
        mn = sc                                                    # a block's offset goes with its scale: values centred on zero
        head = torch.empty((rows, nb, 12), dtype=torch.uint8, device="cuda")
        head[..., 0:4] = sc[..., :4] | ((sc[..., 4:] >> 4) << 6)
        head[..., 4:8] = mn[..., :4] | ((mn[..., 4:] >> 4) << 6)
        head[..., 8:12] = (sc[..., 4:] & 15) | ((mn[..., 4:] & 15) << 4)
        raw = torch.cat([half(d), half(dm), head, qs.reshape(rows, nb, 128)], -1).reshape(rows, -1)

        def values():
            q = torch.stack([qs & 15, qs >> 4], 3).reshape(rows, nb, 8, 32).double()
            w = (d.to(torch.float16).double()[..., None] * sc)[..., None] * q - (dm.to(torch.float16).double()[..., None] * mn)[..., None]
            return w.reshape(rows, k)
        return raw, values
    d = unit / (18.5 * 85.0 * 1.04 * math.sqrt(k))
    ql, qh = ints(0, 256, rows, nb, 2, 64), ints(0, 256, rows, nb, 2, 32)
    sc = ints(32, 128, rows, nb, 16).to(torch.int8) * (1 - 2 * ints(0, 2, rows, nb, 16).to(torch.int8))
    raw = torch.cat([ql.reshape(rows, nb, 128), qh.reshape(rows, nb, 64), sc.view(torch.uint8), half(d)], -1).reshape(rows, -1)

    def values6():
        parts = [(ql[..., :32] & 15) | ((qh & 3) << 4), (ql[..., 32:] & 15) | (((qh >> 2) & 3) << 4), (ql[..., :32] >> 4) | (((qh >> 4) & 3) << 4),
                 (ql[..., 32:] >> 4) | ((qh >> 6) << 4)]
        q = torch.stack(parts, 3).reshape(rows, nb, 16, 16).double() - 32.0
        return (q * (d.to(torch.float16).double()[..., None] * sc.double())[..., None]).reshape(rows, k)
    return raw, values6


def _quant_of(case, name):
    r = RECIPES[case["quant"]] if "quant" in case else {}
    return r.get(name.split(".")[-2]) if name.endswith(".weight") else None


def _load(m, case, seed, specs):
    for name, shape, kind in specs:
        qt = _quant_of(case, name)
        if qt and len(shape) == 2:
            raw, _ = _blocks(seed, name, shape[0], shape[1], qt)
            m.load_tensor_ggml(name, GGML[qt], shape, _to_host(raw))
        else:
            _load_bf16(m, seed, name, shape, kind)
    m.finalize()


def _weights64(case, seed, specs):
    """name -> function that gives the tensor in 64 bits."""
    out = {}
    for name, shape, kind in specs:
        qt = _quant_of(case, name)
        if qt and len(shape) == 2:
            out[name] = lambda name=name, shape=shape, qt=qt: _blocks(seed, name, shape[0], shape[1], qt)[1]()
        else:
            out[name] = lambda name=name, shape=shape, kind=kind: _tensor(seed, name, shape, kind).double()
    return out


# ------------------------------------------------------------------------------------------------------------------ prepare and run
def _lengths(case, seed):
    """Cached lengths of a batch's conversations: unequal, up to the case's own."""
    r = np.random.default_rng(int(seed) * 7919 + 1)
    n = case["seqs"]
    return [max(2, int(case["past"] * f)) for f in r.permutation(np.linspace(0.15, 1.0, n))]


def _requests(case, seed):
    """[(arrival step, prompt ids, forced tokens)] of the serving case."""
    r = np.random.default_rng(int(seed) * 7919 + 2)
    out = []
    for i in range(case["requests"]):
        n = max(2, int(case["prompt"] * r.uniform(0.3, 1.0)))
        out.append((i, _ids(seed, f"prompt{i}", n, 32768), _ids(seed, f"forced{i}", case["tokens"], 32768)))
    return out


def _schedule(case, reqs):
    """Engine iterations: each live request gives its next prompt portion or its next token; a request leaves after its last token.
    -> [[(request, tokens, want, first, last)]]"""
    at = [0] * len(reqs)
    steps, t = [], 0
    while any(a < len(p) + len(f) for a, (_, p, f) in zip(at, reqs)):
        entries = []
        for i, (start, prompt, forced) in enumerate(reqs):
            if t < start or at[i] >= len(prompt) + len(forced):
                continue
            if at[i] < len(prompt):
                part = prompt[at[i]: at[i] + case["portion"]]
                done = at[i] + len(part) == len(prompt)
            else:
                part, done = forced[at[i] - len(prompt): at[i] - len(prompt) + 1], True
            first = at[i] == 0
            at[i] += len(part)
            entries.append((i, part, [len(part) - 1] if done else [], first, at[i] == len(prompt) + len(forced)))
        if entries:
            steps.append(entries)
        t += 1
    return steps


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind in ("token", "prefill"):
        cfg = _dense_config(case)
        n = case["steps"] if kind == "token" else case["rows"]
        m = crane_b200.Qwen3Model(cfg, max_seq_len=case["past"] + n + 64, **({"precision": case["precision"]} if "precision" in case else {}))
        _load(m, case, seed, synth.text_tensor_specs(cfg))
        st["ids"] = _ids(seed, "ids", n, cfg["vocab_size"])
        if case["past"]:
            m.forward_step_argmax(_ids(seed, "past", case["past"], cfg["vocab_size"]), 0)
    elif kind == "batch":
        cfg = _dense_config(case)
        m = crane_b200.Qwen3Model(cfg, max_seq_len=case["past"] + case["steps"] + 64, max_batch=case["seqs"])
        _load(m, case, seed, synth.text_tensor_specs(cfg))
        st["lens"] = _lengths(case, seed)
        st["slots"] = [0] + [m.seq_create() for _ in range(case["seqs"] - 1)]
        st["tokens"] = [_ids(seed, f"round{r}", case["seqs"], cfg["vocab_size"]) for r in range(case["steps"])]
        for s, n in zip(st["slots"], st["lens"]):
            m.seq_select(s)
            m.forward_step_argmax(_ids(seed, f"past{s}", n, cfg["vocab_size"]), 0)
    elif kind in ("hybrid_prefill", "hybrid_token"):
        cfg = _hybrid_config(case)
        n = case["rows"] if kind == "hybrid_prefill" else case["past"] + case["steps"]
        m = crane_b200.Qwen3_5Model(cfg, max_seq_len=n + 64, max_batch=2)
        _load(m, case, seed, synth.qwen3_5_tensor_specs(cfg))
        if kind == "hybrid_prefill":
            st["ids"] = _ids(seed, "ids", n, cfg["vocab_size"])
        else:
            m.forward_step_argmax(_ids(seed, "past", case["past"], cfg["vocab_size"]), 0)
            st["ids"] = _ids(seed, "ids", case["steps"], cfg["vocab_size"])
    elif kind == "vision":
        cfg = _vision_config()
        m = crane_b200.Qwen3VLModel(cfg, max_seq_len=128)
        _load(m, case, seed, list(synth.text_tensor_specs(cfg["text_config"], "model.language_model.")) + list(synth.vision_tensor_specs(cfg["vision_config"])))
        n = case["grid_h"] * case["grid_w"]
        st["pixels"] = np.random.default_rng(int(seed)).uniform(-1.0, 1.0, (n, 1536)).astype(np.float32)
        st["grid"] = np.array([[1, case["grid_h"], case["grid_w"]]], np.uint32)
    else:
        cfg = _ragged_config(case)
        m = crane_b200.FosovikModel(cfg, max_tokens=64 * 16 * case["requests"], max_batch=case["requests"] + 1)
        _load(m, case, seed, synth.fosovik_tensor_specs(cfg))
        st["steps"] = _schedule(case, _requests(case, seed))
    st["model"] = m
    return st


def run(st):
    case, m = st["case"], st["model"]
    kind = case["kind"]
    if kind == "token":                   # back to the cached prefix, then the program's own tokens, each step's logits in the program's hands
        m.set_kv_caches([], case["past"])
        return [m.forward_step(st["ids"][i: i + 1], case["past"] + i) for i in range(case["steps"])]
    if kind == "prefill":
        m.set_kv_caches([], case["past"])
        return m.forward_step(st["ids"], case["past"])
    if kind == "batch":                   # every conversation back to its prefix, then lock-step rounds
        for s, n in zip(st["slots"], st["lens"]):
            m.seq_select(s)
            m.set_kv_caches([], n)
        return [m.decode_batch(st["slots"], t, 1, want_logits=True)[1] for t in st["tokens"]]
    if kind == "hybrid_prefill":
        m.clear_kv_cache()
        return m.forward_step(st["ids"], 0)
    if kind == "hybrid_token":
        s = m.seq_fork(0)
        m.seq_select(s)
        out = [m.forward_step(st["ids"][i: i + 1], case["past"] + i) for i in range(case["steps"])]
        m.seq_free(s)
        return out
    if kind == "vision":
        return m.encode_images(st["pixels"], st["grid"], want_deepstack=3)
    out, slot = [], {}
    for entries in st["steps"]:
        for i, _, _, first, _ in entries:
            if first:
                slot[i] = m.seq_create()
        got = m.step_batch([(slot[i], part, want) for i, part, want, _, _ in entries])
        if got is not None:
            out.append(got)
        for i, _, _, _, last in entries:
            if last:
                m.seq_free(slot.pop(i))
    return np.concatenate(out)


# ------------------------------------------------------------------------------------------------------------------ work and tolerance
def _linear_work(case, specs, rows, head_rows):
    """Bytes of the matrices read once and the operations of `rows` rows through them (the head: `head_rows`)."""
    by = fl = 0.0
    for name, shape, _ in specs:
        if len(shape) < 2 or "embed" in name or name == "head":
            continue
        n = math.prod(shape)
        qt = _quant_of(case, name)
        by += n * (BLOCK_BYTES[qt] if qt else 2)
        fl += 2.0 * n * (head_rows if "lm_head" in name else rows)
    return by, fl


def work(case):
    kind = case["kind"]
    if kind in ("token", "prefill", "batch"):
        cfg = _dense_config(case)
        V, L, nh, nkv = cfg["vocab_size"], case["layers"], cfg["num_attention_heads"], cfg["num_key_value_heads"]
        specs = list(synth.text_tensor_specs(cfg))
        kvb = 2 * nkv * 128 * (2 if case.get("precision") == "bf16" else 4)
        if kind == "prefill":
            passes, rows, heads = 1, case["rows"], 1
            pairs = case["rows"] * (case["past"] + (case["rows"] + 1) / 2)
            cached = case["past"] + 2 * case["rows"]
        elif kind == "token":
            passes, rows, heads = case["steps"], 1, 1
            pairs = cached = case["past"] + 1
        else:
            passes, rows, heads = case["steps"], case["seqs"], case["seqs"]
            pairs = cached = 0.575 * case["past"] * case["seqs"]
        by, fl = _linear_work(case, specs, rows, heads)
        if "quant" not in case:            # the tied head
            by, fl = by + 2.0 * V * case["width"], fl + 2.0 * V * case["width"] * heads
        return {"bytes": passes * (by + L * kvb * cached + 4.0 * V * heads), "flops": passes * (fl + L * 4.0 * nh * 128 * pairs)}
    if kind in ("hybrid_prefill", "hybrid_token"):
        cfg = _hybrid_config(case)
        pre = kind == "hybrid_prefill"
        rows, passes = (case["rows"], 1) if pre else (1, case["steps"])
        full = sum(synth.is_full_attention_layer(cfg, i) for i in range(case["layers"]))
        by, fl = _linear_work(case, synth.qwen3_5_tensor_specs(cfg), rows, 1)
        head = 2.0 * PAGE_V * 1024
        cached = 2 * rows if pre else case["past"]
        pairs = rows * (rows + 1) / 2 if pre else case["past"]
        state = (case["layers"] - full) * 16 * 128 * 128
        return {"bytes": passes * (by + head + full * cached * 2 * 2 * 256 * 4 + state * 8),
                "flops": passes * (fl + head + full * 4.0 * 8 * 256 * pairs + rows * state * 7.0)}
    if kind == "vision":
        vc = _vision_config()["vision_config"]
        n = case["grid_h"] * case["grid_w"]
        by = fl = 0.0
        for name, shape, _ in synth.vision_tensor_specs(vc):
            if len(shape) >= 2 and "pos_embed" not in name:
                by += 2.0 * math.prod(shape)
                fl += 2.0 * math.prod(shape) * (n // 4 if "merger" in name else n)
        return {"bytes": by + n * 1536 * 4.0 + 4 * (n // 4) * 2048 * 4.0, "flops": fl + 24 * 4.0 * 1024 * n * n}
    cfg = _ragged_config(case)
    by = fl = 0.0
    for e in _schedule(case, [(i, np.zeros(int(case["prompt"] * 0.65) + 1, np.uint32), np.zeros(case["tokens"], np.uint32)) for i in range(case["requests"])]):
        rows, heads = sum(len(p) for _, p, _, _, _ in e), sum(len(w) for _, _, w, _, _ in e)
        share = min(1.0, rows * 4 / case["experts"]) if case["experts"] else 1.0
        for name, shape, _ in synth.fosovik_tensor_specs(cfg):
            if len(shape) < 2 or name in ("embed", "head"):
                continue
            expert = ".mlp.e" in name
            by += 2.0 * math.prod(shape) * (share if expert else 1.0)
            fl += 2.0 * math.prod(shape) * rows * (4 / case["experts"] if expert else 1.0)
        by += (2.0 * 32768 * 1024 + 4.0 * 32768 * heads) if heads else 0.0
        fl += 2.0 * 32768 * 1024 * heads
    return {"bytes": by, "flops": fl}


def tolerance(case):
    kind = case["kind"]
    if case.get("precision") == "bf16":
        return {"rel": 3e-2}
    if "quant" in case:                   # an activation on the border of two 8-bit codes takes either, a step of 1/128 of its block's largest value,
        return {"rel": 3e-2}              # and what one linear's codes move decides over many of the next one's: measured 1e-2
    if kind == "vision":
        return {"rel": 5e-5}
    return {"rel": 1e-4}


# ------------------------------------------------------------------------------------------------------------------ 64-bit answers
def _rms(x, w, eps):
    return x / torch.sqrt(x.square().mean(-1, keepdim=True) + eps) * w


def _silu(x):
    return x * torch.sigmoid(x)


def _codes(x, qt):
    """The activations a quantised linear multiplies by: their 8-bit block codes times the blocks' scales."""
    n, k = x.shape
    away = lambda v: torch.sign(v) * torch.floor(v.abs() + 0.5)  # noqa: E731
    if qt == "Q8_0":
        b = x.reshape(n, k // 32, 32)
        d = b.abs().amax(-1, keepdim=True) / 127.0
        return (away(torch.where(d > 0, b / d, torch.zeros_like(b))) * d.to(torch.float16).double()).reshape(n, k)
    b = x.reshape(n, k // 256, 256)
    big = b.gather(-1, b.abs().argmax(-1, keepdim=True))
    scale = torch.where(big != 0, -128.0 / big, torch.zeros_like(big))
    return (torch.clamp(away(scale * b), max=127.0) * torch.where(big != 0, 1.0 / scale, torch.zeros_like(big))).reshape(n, k)


def _linear(case, w, name, x):
    qt = _quant_of(case, name)
    return (_codes(x, qt) if qt else x) @ w[name]().T


def _attend(q, k, v, scale, causal=True, sink=None):
    """q [S, H, d] are the last S of T positions; k, v [T, G, d]."""
    S, H, _ = q.shape
    T, G, dv = v.shape
    out = torch.empty(S, H, dv, dtype=q.dtype, device=q.device)
    seen = torch.arange(T, device=q.device)[None, :] <= torch.arange(T - S, T, device=q.device)[:, None]
    for h in range(H):
        s = (q[:, h] @ k[:, h // (H // G)].T) * scale
        if causal:
            s = s.masked_fill(~seen, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(S, 1)], 1)
        out[:, h] = torch.softmax(s, -1)[:, :T] @ v[:, h // (H // G)]
    return out


def _angles(inv, n):
    """cos and sin of the 32-bit angles the rotary tables are made of."""
    a = torch.from_numpy(np.arange(n, dtype=np.float32)[:, None] * inv[None, :]).double().cuda()
    return a.cos(), a.sin()


def _rotate(x, cos, sin):
    h = cos.shape[-1]
    a, b = x[..., :h], x[..., h: 2 * h]
    c, s = cos[:, None], sin[:, None]
    return torch.cat([a * c - b * s, a * s + b * c, x[..., 2 * h:]], -1)


def _dense64(case, seed, seqs, want):
    """Logits of the last want[i] rows of every sequence."""
    cfg = _dense_config(case)
    w = _weights64(case, seed, synth.text_tensor_specs(cfg))
    nh, nkv, eps = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["rms_norm_eps"]
    inv = np.array([1.0 / cfg["rope_theta"] ** (i / 128) for i in range(0, 128, 2)]).astype(np.float32)
    cos, sin = _angles(inv, max(len(s) for s in seqs))
    table = w["model.embed_tokens.weight"]()
    x = torch.cat([table[torch.from_numpy(s.astype(np.int64)).cuda()] for s in seqs])
    at = np.cumsum([0] + [len(s) for s in seqs])
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        h = _rms(x, w[p + "input_layernorm.weight"](), eps)
        q, k, v = (_linear(case, w, p + f"self_attn.{n}_proj.weight", h).reshape(len(h), -1, 128) for n in "qkv")
        q, k = _rms(q, w[p + "self_attn.q_norm.weight"](), eps), _rms(k, w[p + "self_attn.k_norm.weight"](), eps)
        a = []
        for b, e in zip(at[:-1], at[1:]):
            a.append(_attend(_rotate(q[b:e], cos[: e - b], sin[: e - b]), _rotate(k[b:e], cos[: e - b], sin[: e - b]), v[b:e], 128 ** -0.5))
        x = x + _linear(case, w, p + "self_attn.o_proj.weight", torch.cat(a).reshape(len(x), nh * 128))
        h = _rms(x, w[p + "post_attention_layernorm.weight"](), eps)
        f = _silu(_linear(case, w, p + "mlp.gate_proj.weight", h)) * _linear(case, w, p + "mlp.up_proj.weight", h)
        x = x + _linear(case, w, p + "mlp.down_proj.weight", f)
    x = torch.cat([x[e - n: e] for e, n in zip(at[1:], want)])
    x = _rms(x, w["model.norm.weight"](), eps)
    return x @ table.T if cfg["tie_word_embeddings"] else _linear(case, w, "lm_head.weight", x)


def _hybrid64(case, seed, ids, want):
    cfg = _hybrid_config(case)
    w = _weights64(case, seed, synth.qwen3_5_tensor_specs(cfg))
    eps, S = cfg["rms_norm_eps"], len(ids)
    base = np.float32(cfg["rope_parameters"]["rope_theta"])
    inv = np.array([np.float32(1.0) / np.power(base, np.float32(i) * np.float32(2.0) / np.float32(64), dtype=np.float32) for i in range(32)], np.float32)
    cos, sin = _angles(inv, S)
    table = w["model.embed_tokens.weight"]()
    x = table[torch.from_numpy(ids.astype(np.int64)).cuda()]
    unit = lambda t: t / torch.sqrt(t.square().sum(-1, keepdim=True) + 1e-6)  # noqa: E731
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        h = _rms(x, 1.0 + w[p + "input_layernorm.weight"](), eps)
        if synth.is_full_attention_layer(cfg, i):
            qg = (h @ w[p + "self_attn.q_proj.weight"]().T).reshape(S, 8, 512)
            k, v = ((h @ w[p + f"self_attn.{n}_proj.weight"]().T).reshape(S, 2, 256) for n in "kv")
            q = _rotate(_rms(qg[..., :256], 1.0 + w[p + "self_attn.q_norm.weight"](), eps), cos, sin)
            k = _rotate(_rms(k, 1.0 + w[p + "self_attn.k_norm.weight"](), eps), cos, sin)
            o = (_attend(q, k, v, 1.0 / 16.0) * torch.sigmoid(qg[..., 256:])).reshape(S, 2048)
            x = x + o @ w[p + "self_attn.o_proj.weight"]().T
        else:
            p += "linear_attn."
            u = h @ w[p + "in_proj_qkv.weight"]().T
            cw = w[p + "conv1d.weight"]().reshape(-1, 4)
            pad = torch.cat([torch.zeros(3, u.shape[1], dtype=u.dtype, device=u.device), u])
            u = _silu(sum(pad[t: t + S] * cw[:, t] for t in range(4)))
            q, k, v = u[:, :2048].reshape(S, 16, 128), u[:, 2048:4096].reshape(S, 16, 128), u[:, 4096:].reshape(S, 16, 128)
            q, k = unit(q) / math.sqrt(128), unit(k)
            beta = torch.sigmoid(h @ w[p + "in_proj_b.weight"]().T)[..., None]
            decay = torch.exp(-torch.exp(w[p + "A_log"]()) * torch.log1p(torch.exp(h @ w[p + "in_proj_a.weight"]().T + w[p + "dt_bias"]())))
            s = torch.zeros(16, 128, 128, dtype=u.dtype, device=u.device)
            ys = []
            for t in range(S):
                s = s * decay[t][:, None, None]
                new = (v[t] - torch.einsum("hkv,hk->hv", s, k[t])) * beta[t]
                s = s + k[t][:, :, None] * new[:, None, :]
                ys.append(torch.einsum("hkv,hk->hv", s, q[t]))
            z = (h @ w[p + "in_proj_z.weight"]().T).reshape(S, 16, 128)
            y = _rms(torch.stack(ys), w[p + "norm.weight"](), eps) * _silu(z)
            x = x + y.reshape(S, 2048) @ w[p + "out_proj.weight"]().T
            p = f"model.layers.{i}."
        h = _rms(x, 1.0 + w[p + "post_attention_layernorm.weight"](), eps)
        x = x + (_silu(h @ w[p + "mlp.gate_proj.weight"]().T) * (h @ w[p + "mlp.up_proj.weight"]().T)) @ w[p + "mlp.down_proj.weight"]().T
    return _rms(x[S - want:], 1.0 + w["model.norm.weight"](), eps) @ table.T


def _vision64(case, seed):
    vc = _vision_config()["vision_config"]
    p0 = "model.visual."
    w = _weights64(case, seed, synth.vision_tensor_specs(vc))
    W = lambda n: w[p0 + n]()  # noqa: E731
    gh, gw, H, side = case["grid_h"], case["grid_w"], 1024, 48
    norm = lambda x, n: torch.nn.functional.layer_norm(x, (x.shape[-1],), W(n + ".weight"), W(n + ".bias"), 1e-6)  # noqa: E731
    blocks = lambda t: t.reshape(gh // 2, 2, gw // 2, 2, -1).permute(0, 2, 1, 3, 4).reshape(gh * gw, -1)  # noqa: E731  (2 x 2 patches side by side)

    def line(n):                           # the learned grid's coordinates of n evenly spread patches, in 32 bits as the tables are
        c = np.arange(n, dtype=np.float32) * (np.float32(side - 1) / np.float32(n - 1))
        f = np.floor(c).astype(np.int64)
        return f, np.minimum(np.ceil(c).astype(np.int64), side - 1), torch.from_numpy((c - f.astype(np.float32)).astype(np.float64)).cuda()
    pv = torch.from_numpy(np.random.default_rng(int(seed)).uniform(-1.0, 1.0, (gh * gw, 1536)).astype(np.float32)).cuda().double()
    x = pv @ W("patch_embed.proj.weight").reshape(H, -1).T + W("patch_embed.proj.bias")
    (hf, hc, dh), (wf, wc, dw), pos = line(gh), line(gw), W("pos_embed.weight").reshape(side, side, H)
    at = lambda r, c: pos[torch.from_numpy(r).cuda()[:, None], torch.from_numpy(c).cuda()[None, :]]  # noqa: E731
    dh, dw = dh[:, None, None], dw[None, :, None]
    x = x + blocks(at(hf, wf) * (1 - dh) * (1 - dw) + at(hf, wc) * (1 - dh) * dw + at(hc, wf) * dh * (1 - dw) + at(hc, wc) * dh * dw)
    inv = np.array([np.float32(1.0) / np.float32(10000.0) ** (np.float32(i) / np.float32(32)) for i in range(0, 32, 2)], np.float32)
    ang = torch.from_numpy(np.arange(max(gh, gw), dtype=np.float32)[:, None] * inv[None, :]).double().cuda()
    ang = torch.cat([ang[:gh, None].expand(gh, gw, 16), ang[None, :gw].expand(gh, gw, 16)], -1)
    ang = blocks(ang)
    cos, sin = ang.cos(), ang.sin()
    gelu = torch.nn.functional.gelu

    def merge(x, n, post):
        y = norm(x.reshape(-1, 4 * H), n + "norm") if post else norm(x, n + "norm").reshape(-1, 4 * H)
        y = gelu(y @ W(n + "linear_fc1.weight").T + W(n + "linear_fc1.bias"), approximate="tanh")
        return y @ W(n + "linear_fc2.weight").T + W(n + "linear_fc2.bias")
    deep = []
    for i in range(vc["depth"]):
        b = f"blocks.{i}."
        qkv = (norm(x, b + "norm1") @ W(b + "attn.qkv.weight").T + W(b + "attn.qkv.bias")).reshape(-1, 3, 16, 64)
        o = _attend(_rotate(qkv[:, 0], cos, sin), _rotate(qkv[:, 1], cos, sin), qkv[:, 2], 0.125, causal=False)
        x = x + o.reshape(-1, H) @ W(b + "attn.proj.weight").T + W(b + "attn.proj.bias")
        y = gelu(norm(x, b + "norm2") @ W(b + "mlp.linear_fc1.weight").T + W(b + "mlp.linear_fc1.bias"))
        x = x + y @ W(b + "mlp.linear_fc2.weight").T + W(b + "mlp.linear_fc2.bias")
        if i in vc["deepstack_visual_indexes"]:
            deep.append(merge(x, f"deepstack_merger_list.{len(deep)}.", True))
    return merge(x, "merger.", False), torch.stack(deep)


def _ragged64(case, seed):
    """The layer list over every request by itself, then the wanted rows in the order the schedule asks for them."""
    cfg = _ragged_config(case)
    w = _weights64(case, seed, synth.fosovik_tensor_specs(cfg))
    cache = {}
    W = lambda n: cache.setdefault(n, w[n]())  # noqa: E731
    eps = cfg["norm"]["eps"]
    norm = lambda x, n: torch.tanh(W(n + ".alpha") * x) * W(n) + W(n + ".b")  # noqa: E731
    one = lambda x: x / torch.sqrt(x.square().mean(-1, keepdim=True) + eps)  # noqa: E731

    def logits(ids):
        S = len(ids)
        x = W("embed")[torch.from_numpy(ids.astype(np.int64)).cuda()] * cfg["embedding"]["scale"]
        for i, L in enumerate(cfg["layers"]):
            m, p = L["mixer"], f"l{i}.mix."
            h = norm(x, f"l{i}.norm1")
            if L["type"] == "attention":
                q = one((h @ W(p + "q").T).reshape(S, m["heads"], m["dim"]))
                pos = torch.arange(S, device="cuda", dtype=torch.float64)
                q = q * (1.0 + m["q_temp"]["coef"] * torch.log(torch.floor((pos + 1.0) / m["q_temp"]["every"]) + 1.0))[:, None, None]
                k, v = one((h @ W(p + "k").T).reshape(S, m["kv_heads"], m["dim"])), (h @ W(p + "v").T).reshape(S, m["kv_heads"], m["vdim"])
                mix = _attend(q, k, v, m["scale"], sink=W(p + "sink")).reshape(S, -1) @ W(p + "o").T
            else:
                hm, pw, n, g = m["heads"], m["vdim"], m["state"], m["groups"]
                inner = hm * pw
                proj = h @ W(p + "in").T
                z, u, dt = proj[:, :inner], proj[:, inner: 2 * inner + 2 * g * n], proj[:, 2 * inner + 2 * g * n:]
                taps, cw = m["conv"], W(p + "conv")
                pad = torch.cat([torch.zeros(taps - 1, u.shape[1], dtype=u.dtype, device=u.device), u])
                u = _silu(sum(pad[t: t + S] * cw[:, t] for t in range(taps)) + W(p + "conv.b"))
                xs = u[:, :inner].reshape(S, hm, pw)
                b, c = (u[:, inner + j * g * n: inner + (j + 1) * g * n].reshape(S, g, n).repeat_interleave(hm // g, 1) for j in (0, 1))
                dt = torch.nn.functional.softplus(dt + W(p + "dt_bias"), threshold=100)
                decay = torch.exp(-torch.exp(W(p + "A_log")) * dt)
                s = torch.zeros(hm, n, pw, dtype=u.dtype, device=u.device)
                ys = []
                for t in range(S):
                    s = s * decay[t][:, None, None] + (dt[t][:, None] * b[t])[:, :, None] * xs[t][:, None, :]
                    ys.append(torch.einsum("hnp,hn->hp", s, c[t]))
                y = (torch.stack(ys) + W(p + "D")[:, None] * xs).reshape(S, inner) * _silu(z)
                mix = (one(y.reshape(S, m["norm_groups"], -1)).reshape(S, inner) * W(p + "norm")) @ W(p + "o").T
            f, p = L["mlp"], f"l{i}.mlp."
            if f["kind"] == "dense":
                gate = torch.clamp(h @ W(p + "gate").T, max=f["limit"])
                up = torch.clamp(h @ W(p + "up").T, min=-f["limit"], max=f["limit"])
                ff = (gate * torch.sigmoid(1.702 * gate) * (up + 1.0)) @ W(p + "down").T
            else:
                top, idx = torch.topk(torch.softmax(h @ W(p + "router").T, -1), f["router"]["top"])
                ff = torch.zeros_like(x)
                for e in range(f["router"]["experts"]):
                    r, k = (idx == e).nonzero(as_tuple=True)
                    ff.index_add_(0, r, top[r, k][:, None] * (torch.nn.functional.gelu(h[r] @ W(f"{p}e{e}.up").T) @ W(f"{p}e{e}.down").T))
            x = x + mix + ff
        return x
    reqs = _requests(case, seed)
    full = [logits(np.concatenate([p, f])) for _, p, f in reqs]
    at, rows = [0] * len(reqs), []
    for entries in _schedule(case, reqs):
        for i, part, want, _, _ in entries:
            rows += [full[i][at[i] + j] for j in want]
            at[i] += len(part)
    return norm(torch.stack(rows), "final.norm") @ W("head").T


def exact(case, seed):
    kind = case["kind"]
    V = case.get("vocab", PAGE_V)
    with torch.no_grad():
        if kind in ("token", "prefill"):
            n = case["steps"] if kind == "token" else case["rows"]
            ids = np.concatenate([_ids(seed, "past", case["past"], V), _ids(seed, "ids", n, V)]) if case["past"] else _ids(seed, "ids", n, V)
            got = _dense64(case, seed, [ids], [n if kind == "token" else 1])
            return list(got) if kind == "token" else got[0]
        if kind == "batch":
            r = case["steps"]
            forced = [_ids(seed, f"round{j}", case["seqs"], V) for j in range(r)]
            seqs = [np.concatenate([_ids(seed, f"past{s}", n, V), np.array([f[s] for f in forced])]) for s, n in enumerate(_lengths(case, seed))]
            got = _dense64(case, seed, seqs, [r] * len(seqs)).reshape(len(seqs), r, V)
            return [got[:, j] for j in range(r)]
        if kind == "hybrid_prefill":
            return _hybrid64(case, seed, _ids(seed, "ids", case["rows"], PAGE_V), 1)[0]
        if kind == "hybrid_token":
            ids = np.concatenate([_ids(seed, "past", case["past"], PAGE_V), _ids(seed, "ids", case["steps"], PAGE_V)])
            return list(_hybrid64(case, seed, ids, case["steps"]))
        if kind == "vision":
            return _vision64(case, seed)
        return _ragged64(case, seed)
