"""Passes of the serving engine as its users run them: the cases that its speed is judged by.

A case is one pass of ``ZStreamerEngine``'s runner over requests that are in its paged cache: a decode step (one token for
each of many sequences, through CUDA graphs), a packed prefill pass (whole prompts, or a chunk of a long one behind what is
cached already) or the verification of drafted tokens.  The models are Qwen2.5 and Gemma-2 shapes with random weights, in the
quantisations that ``.zse`` files come in.  One engine per model serves every batch, as in a server; a batch is its
sequences in the cache and the tokens that come next.  What is cached before the pass is drawn at random.

``exact`` evaluates the same models in 64 bits with plain torch.
"""
import gc
import itertools
import math
import os
import tempfile
import weakref
import zlib

import torch

GROUP = 128
# width, layers, query heads, kv heads, head size, feed-forward size, vocabulary, RoPE base, spread of the embedding
SHAPES = {
    "qwen2.5-7b": dict(H=3584, L=28, nh=28, nkv=4, hd=128, I=18944, V=152064, theta=1e6, embed=1.0, gemma=False),
    "qwen2.5-14b": dict(H=5120, L=48, nh=40, nkv=8, hd=128, I=13824, V=152064, theta=1e6, embed=1.0, gemma=False),
    "gemma2-9b": dict(H=3584, L=42, nh=16, nkv=8, hd=256, I=14336, V=256000, theta=1e4, embed=0.02, gemma=True),
}
WINDOW, SCORE_CAP, LOGIT_CAP = 4096, 50.0, 30.0       # Gemma-2
CACHE_TOKENS = {"qwen2.5-7b": 600_000, "qwen2.5-14b": 400_000, "gemma2-9b": 280_000}    # 34 to 96 GB beside the weights


def _case(name, model, quant, phase, seqs, past, new=(1, 1), sampled=False):
    c = {"model": model, "quant": quant, "phase": phase, "seqs": seqs, "past_lo": past[0], "past_hi": past[1],
         "new_lo": new[0], "new_hi": new[1], "sampled": sampled}
    return dict(c, name=name) if name else c


def listed():
    b7, b14, g9 = "qwen2.5-7b", "qwen2.5-14b", "gemma2-9b"
    return [
        # one user at a local chat: latency of a single token is all that counts
        _case("decode_1", b7, "int4", "decode", 1, (517, 517)),
        # time to first token of a short chat message
        _case("prompt_77", b7, "int4", "prefill", 1, (0, 0), (77, 77)),
        # a few agents with long documents in their context, sampling
        _case("decode_5_long", b7, "int4", "decode", 5, (6001, 20011), sampled=True),
        # a small server
        _case("decode_17", b7, "int4", "decode", 17, (100, 3000)),
        # a full server with short chats, sampling
        _case("decode_160", b7, "int4", "decode", 160, (64, 1100), sampled=True),
        # the next chunk of a long prompt
        _case("chunk_2048", b7, "int4", "prefill", 1, (14336, 14336), (2048, 2048)),
        # a document, 8-bit weights
        _case("prompt_int8_1500", b7, "int8", "prefill", 1, (0, 0), (1500, 1500)),
        # the family with soft caps and windows
        _case("decode_gemma_20", g9, "int4", "decode", 20, (64, 6000)),
        # short prompts of several requests packed into one pass, the windowed family
        _case("prompts_gemma_6", g9, "int4", "prefill", 6, (0, 0), (90, 800)),
        # the benchmark of the repository: 64 concurrent requests, prompts of 128 to 2048 tokens
        _case("decode_64", b14, "int4", "decode", 64, (128, 2300)),
        # drafts of four tokens for 32 requests, verified in one pass
        _case("verify_32", b14, "int4", "verify", 32, (500, 4000), (5, 5)),
        # a full pass of prompts of unequal length
        _case("prompts_5", b14, "int4", "prefill", 5, (0, 0), (600, 2660)),
    ]


def _spread(rng, lo, hi):
    """A whole number between lo and hi, even over the logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng):
    model, quant = rng.choice([("qwen2.5-7b", "int4"), ("qwen2.5-14b", "int4"), ("qwen2.5-7b", "int8"), ("gemma2-9b", "int4")])
    phase = "prefill" if quant == "int8" else rng.choice(["decode", "decode", "prefill", "prefill", "verify"])
    if phase == "decode":
        seqs = _spread(rng, 1, 200)
        hi = _spread(rng, 64, min(20000 if model == "qwen2.5-7b" else 6000, (66_000 if model == "gemma2-9b" else 95_000) // seqs))
        return _case("", model, quant, "decode", seqs, (rng.randint(hi // 8 + 1, hi), hi), sampled=rng.random() < 0.4)
    if phase == "verify":
        seqs, new = _spread(rng, 1, 32), rng.randint(3, 7)
        hi = _spread(rng, 64, 4000)
        return _case("", model, quant, "verify", seqs, (rng.randint(hi // 8 + 1, hi), hi), (new, new))
    if rng.random() < 0.3:                      # a chunk behind a cached past
        new = _spread(rng, 200, 2048)
        past = _spread(rng, 256, 14336 if model == "qwen2.5-7b" else 5000)
        return _case("", model, quant, "prefill", 1, (past, past), (new, new))
    total = _spread(rng, 100 if quant == "int8" else 9, 7800)
    seqs = min(_spread(rng, 1, 12), total // 9)
    hi = total // seqs
    return _case("", model, quant, "prefill", seqs, (0, 0), (rng.randint(hi * 4 // 5, hi), hi))


def _lengths(lo, hi, n):
    """n lengths from lo to hi, evenly apart."""
    return [lo + (hi - lo) * i // max(1, n - 1) for i in range(n)] if n > 1 else [hi]


def _spans(case):
    """(cached tokens, new tokens) of every sequence."""
    n = case["seqs"]
    return list(zip(_lengths(case["past_lo"], case["past_hi"], n), reversed(_lengths(case["new_lo"], case["new_hi"], n))))


# ---- weights: the same for every batch, made tensor by tensor ----------------------------------------------------------------

def _gen(*key):
    return torch.Generator(device="cuda").manual_seed(zlib.crc32(repr(key).encode()))


def _linears(s):
    q, kv = s["nh"] * s["hd"], s["nkv"] * s["hd"]
    return {"self_attn.q_proj": (q, s["H"]), "self_attn.k_proj": (kv, s["H"]), "self_attn.v_proj": (kv, s["H"]),
            "self_attn.o_proj": (s["H"], q), "mlp.gate_proj": (s["I"], s["H"]), "mlp.up_proj": (s["I"], s["H"]),
            "mlp.down_proj": (s["H"], s["I"])}


def _quantised(name, n, k, quant):
    """(codes, scales, zeros) on the GPU; int4 codes are packed two to a byte, the lower nibble first.  What joins the
    residual is smaller than the rest, as in deep models, so that rounding is not blown up from layer to layer."""
    g = _gen(name, n, k)
    groups = n * k // GROUP
    half = 0.03 + 0.03 * torch.rand(groups, device="cuda", generator=g)
    if "o_proj" in name or "down_proj" in name:
        half *= 0.05
    if quant == "int8":
        return torch.randint(-127, 128, (n, k), dtype=torch.int8, device="cuda", generator=g), (half / 127).half(), None
    q = torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device="cuda", generator=g)
    return q, (2 * half / 15).half(), (-half).half()


def _half(name, shape, std, mean=0.0):
    g = _gen(name, shape)
    return (torch.randn(shape, device="cuda", generator=g) * std + mean).half()


def _norm_weight(name, n, gemma):
    """(as stored, as applied): Gemma-2 files hold w - 1, and norms of what joins the residual are small there."""
    w = _half(name, (n,), 0.1, 1.0)
    if not gemma:
        return w, w
    stored = (w.float() * (0.1 if "post_" in name else 1.0) - 1).half()
    return stored, (stored.float() + 1).half()


def _norm_names(s):
    return ["input_layernorm", "post_attention_layernorm"] + (
        ["pre_feedforward_layernorm", "post_feedforward_layernorm"] if s["gemma"] else [])


def _model_file(model, quant):
    """The .zse file of a model, written once."""
    from zse_b200.format import synth
    from zse_b200.format.writer import ZSEWriter
    path = os.path.join(tempfile.gettempdir(), f"zse_cases_{os.getuid()}_{model}_{quant}.zse")
    if os.path.exists(path):
        return path
    s = SHAPES[model]
    w = ZSEWriter(f"{path}.{os.getpid()}")
    w.set_config(synth.shape_config(model, quant=quant))
    w.set_tokenizer(synth.byte_tokenizer(s["V"]).serialize())
    w.begin_weights()
    half = lambda name, shape, std, mean=0.0: w.add_weight_raw_fp16(name, shape, _half(name, shape, std, mean).cpu().numpy())

    def norm(name):
        w.add_weight_raw_fp16(name, (s["H"],), _norm_weight(name, s["H"], s["gemma"])[0].cpu().numpy())

    half("embed_tokens.weight", (s["V"], s["H"]), s["embed"])
    for i in range(s["L"]):
        for name, (n, k) in _linears(s).items():
            full = f"layers.{i}.{name}.weight"
            q, sc, z = _quantised(full, n, k, quant)
            if quant == "int8":
                w.add_weight_raw_int8(full, (n, k), q.cpu().numpy(), sc.cpu().numpy(), GROUP)
            else:
                w.add_weight_raw(full, (n, k), q.cpu().numpy(), sc.cpu().numpy(), z.cpu().numpy(), GROUP)
            if not s["gemma"] and name[-6:] in ("q_proj", "k_proj", "v_proj"):
                half(f"layers.{i}.{name}.bias", (n,), 0.02)
        for name in _norm_names(s):
            norm(f"layers.{i}.{name}.weight")
    norm("norm.weight")
    if not s["gemma"]:
        half("lm_head.weight", (s["V"], s["H"]), 0.02)
    w.finalize()
    os.replace(f"{path}.{os.getpid()}", path)
    return path


# ---- the engine, and batches in its cache ------------------------------------------------------------------------------------

_engine = {}                                    # the one engine that is alive, by model
_ids = itertools.count(1)


def _engine_for(model, quant):
    from zse_b200.config import EngineConfig
    from zse_b200.engine import ZStreamerEngine
    key = (model, quant)
    if key not in _engine:
        _engine.clear()
        gc.collect()
        torch.cuda.empty_cache()
        cfg = EngineConfig(max_batch_seqs=256, max_batch_tokens=8192, max_seq_len=32768, kv_tokens=CACHE_TOKENS[model])
        _engine[key] = ZStreamerEngine(_model_file(model, quant), config=cfg)
    return _engine[key]


class _Batch:
    """Sequences in the cache of an engine, their next tokens, and how they are sampled."""


def _order(case, seed):
    """The order of the lengths in the batch, and the tokens that come next."""
    g = torch.Generator().manual_seed(seed)
    spans = _spans(case)
    spans = [spans[i] for i in torch.randperm(len(spans), generator=g).tolist()]
    vocab = SHAPES[case["model"]]["V"]
    return spans, [torch.randint(0, vocab, (new,), generator=g).tolist() for _, new in spans]


def _past(s, seed, i, n):
    """Cached keys and values of sequence i: [layers, 2, kv heads, n, head size]."""
    g = torch.Generator(device="cuda").manual_seed(seed * 1009 + i)
    return torch.randn((s["L"], 2, s["nkv"], n, s["hd"]), dtype=torch.float16, device="cuda", generator=g)


def _release(cache, ids):
    for i in ids:
        cache.free_sequence(i)


def prepare(case, seed):
    from zse_b200.runtime.runner import SamplingRow
    engine, s = _engine_for(case["model"], case["quant"]), SHAPES[case["model"]]
    b, cache = _Batch(), engine.kv_cache
    spans, b.tokens = _order(case, seed)
    b.engine, b.runner, b.phase = engine, engine.runner, case["phase"]
    b.ids, b.past = [next(_ids) for _ in spans], [past for past, _ in spans]
    weakref.finalize(b, _release, cache, b.ids)
    for i, (sid, (past, new)) in enumerate(zip(b.ids, spans)):
        cache.allocate_sequence(sid, num_tokens=past + new)
        if past:
            blocks, bs = torch.tensor(cache.get_block_ids(sid), device="cuda"), cache.block_size
            kv = torch.nn.functional.pad(_past(s, seed, i, past), (0, 0, 0, len(blocks) * bs - past))
            cache.slab[:, blocks] = kv.view(s["L"], 2, s["nkv"], len(blocks), bs, s["hd"]).permute(0, 3, 1, 2, 4, 5)
    if b.phase == "decode":
        b.last = [t[0] for t in b.tokens]
    else:
        b.items = list(zip(b.ids, b.tokens, b.past))
    b.rows = sum(len(t) for t in b.tokens)
    b.sampling = [SamplingRow(0.8, 50, 0.95, seed + i) for i in range(len(spans))] if case["sampled"] else None
    return b


def run(b):
    """One pass.  Its results stay on the device: logits of the rows that choose a token, final hidden states of all rows."""
    if b.phase == "decode":
        b.runner.decode(b.ids, b.last, sampling=b.sampling)
        logits = b.runner.buf.logits[: len(b.ids)]
    elif b.phase == "verify":
        _, logits = b.runner.prefill(b.items, all_logits=True)
    else:
        b.runner.prefill(b.items)
        logits = b.runner.buf.logits[: len(b.ids)]
    return {"logits": logits, "hidden": b.runner.model.hidden_rows(b.runner.buf, b.rows)}


def _seen(past, new, window):
    """Keys seen by the new tokens, summed over them."""
    return sum(min(past + j + 1, window) if window else past + j + 1 for j in range(new))


def work(case):
    s = SHAPES[case["model"]]
    spans = _spans(case)
    rows = sum(n for _, n in spans)
    picks = rows if case["phase"] == "verify" else len(spans)
    params = sum(n * k for n, k in _linears(s).values())
    per = {"int4": 0.5 + 4 / GROUP, "int8": 1 + 2 / GROUP}[case["quant"]]
    nbytes = s["L"] * params * per + 2 * s["V"] * s["H"] + rows * s["H"] * 4 + picks * s["V"] * 2
    flops = 2 * rows * s["L"] * params + 2 * picks * s["V"] * s["H"]
    row = 4 * s["nkv"] * s["hd"]                # bytes of one token's keys and values in a layer
    for layer in range(s["L"]):
        window = WINDOW if s["gemma"] and layer % 2 == 0 else 0
        for past, new in spans:
            nbytes += row * (min(past, window + new) if window else past) + row * new
            flops += 4 * s["nh"] * s["hd"] * _seen(past, new, window)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # fp16 activations and probabilities through 28 to 48 layers: 1e-3 to 3e-3 from the 64-bit result, as measured; where the
    # reference maximum of a row moves (verification) two runs are 1.3e-3 apart
    return {"rel": 8e-3, "max": 0.15}


# ---- 64 bits -----------------------------------------------------------------------------------------------------------------

def _dense(name, n, k, quant):
    q, sc, z = _quantised(name, n, k, quant)
    if quant == "int8":
        return (q.double().view(-1, GROUP) * sc.double()[:, None]).view(n, k)
    q = torch.stack([q & 15, q >> 4], dim=-1).double().view(-1, GROUP)
    return (q * sc.double()[:, None] + z.double()[:, None]).view(n, k)


def _rms(x, name, gemma):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-6) * _norm_weight(name, x.shape[-1], gemma)[1].double()


def _turn(x, pos, theta):
    """Rotates the pairs (i, i + hd / 2) of x [tokens, heads, hd]."""
    half = x.shape[-1] // 2
    ang = pos.double()[:, None] * theta ** (-torch.arange(half, dtype=torch.float64, device=x.device) / half)
    c, s = torch.cos(ang)[:, None], torch.sin(ang)[:, None]
    a, b = x[..., :half], x[..., half:]
    return torch.cat([a * c - b * s, b * c + a * s], dim=-1)


def _attend(q, k, v, past, window, gemma):
    """q [new, heads, hd], k and v [kv heads, past + new, hd]; one kv head at a time."""
    new, nh, hd = q.shape
    rep = nh // k.shape[0]
    at = torch.arange(past, past + new, device=q.device)[:, None]
    col = torch.arange(past + new, device=q.device)[None]
    hidden = col > at
    if window:
        hidden = hidden | (col <= at - window)
    out = torch.empty_like(q)
    for h in range(k.shape[0]):
        scores = torch.matmul(q[:, h * rep:(h + 1) * rep].transpose(0, 1), k[h].T) * hd ** -0.5
        if gemma:
            scores = torch.tanh(scores / SCORE_CAP) * SCORE_CAP
        p = torch.softmax(scores.masked_fill(hidden, -math.inf), dim=-1)
        out[:, h * rep:(h + 1) * rep] = torch.matmul(p, v[h]).transpose(0, 1)
    return out


@torch.no_grad()
def exact(case, seed):
    s, quant = SHAPES[case["model"]], case["quant"]
    _engine.clear()
    gc.collect()
    torch.cuda.empty_cache()
    spans, tokens = _order(case, seed)
    pasts = [_past(s, seed, i, past) if past else None for i, (past, _) in enumerate(spans)]
    flat = torch.tensor(list(itertools.chain(*tokens)), device="cuda")
    pos = torch.cat([torch.arange(past, past + new) for past, new in spans]).cuda()
    embed = _half("embed_tokens.weight", (s["V"], s["H"]), s["embed"])
    h = embed[flat].double()
    if s["gemma"]:
        h = h * s["H"] ** 0.5
    for i in range(s["L"]):
        pre = f"layers.{i}."
        lin = lambda x, name: torch.matmul(x, _dense(f"{pre}{name}.weight", *_linears(s)[name], quant).T)
        x = _rms(h, pre + "input_layernorm.weight", s["gemma"])
        qkv = []
        for name, heads in (("q", s["nh"]), ("k", s["nkv"]), ("v", s["nkv"])):
            y = lin(x, f"self_attn.{name}_proj")
            if not s["gemma"]:
                y = y + _half(f"{pre}self_attn.{name}_proj.bias", (heads * s["hd"],), 0.02).double()
            y = y.view(-1, heads, s["hd"])
            qkv.append(y if name == "v" else _turn(y, pos, s["theta"]))
        q, k, v = qkv
        window = WINDOW if s["gemma"] and i % 2 == 0 else 0
        a, row = torch.empty_like(q), 0
        for (past, new), old in zip(spans, pasts):
            kn, vn = k[row:row + new].transpose(0, 1), v[row:row + new].transpose(0, 1)
            if old is not None:
                kn, vn = torch.cat([old[i, 0].double(), kn], 1), torch.cat([old[i, 1].double(), vn], 1)
            a[row:row + new] = _attend(q[row:row + new], kn, vn, past, window, s["gemma"])
            row += new
        y = lin(a.reshape(len(flat), -1), "self_attn.o_proj")
        if s["gemma"]:
            h = h + _rms(y, pre + "post_attention_layernorm.weight", s["gemma"])
            x = _rms(h, pre + "pre_feedforward_layernorm.weight", s["gemma"])
        else:
            h = h + y
            x = _rms(h, pre + "post_attention_layernorm.weight", s["gemma"])
        gate = lin(x, "mlp.gate_proj")
        gate = torch.nn.functional.gelu(gate, approximate="tanh") if s["gemma"] else torch.nn.functional.silu(gate)
        y = lin(gate * lin(x, "mlp.up_proj"), "mlp.down_proj")
        h = h + (_rms(y, pre + "post_feedforward_layernorm.weight", s["gemma"]) if s["gemma"] else y)
    h = _rms(h, "norm.weight", s["gemma"])
    picks = h if case["phase"] != "prefill" else h[torch.cumsum(torch.tensor([n for _, n in spans]), 0).cuda() - 1]
    head = embed if s["gemma"] else _half("lm_head.weight", (s["V"], s["H"]), 0.02)
    logits = torch.cat([torch.matmul(picks, part.double().T) for part in head.split(16384)], dim=1)
    if s["gemma"]:
        logits = torch.tanh(logits / LOGIT_CAP) * LOGIT_CAP
    return {"logits": logits, "hidden": h}
