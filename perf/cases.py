"""What a user has this framework do, as cases that can be timed and checked.

A case is one engine step, or a few in a row, through CudaModelRunner: a batch of prompts (prefill), decode
steps that continue cached sequences (decode), or both (generate).  Models are the repository's presets.  GPT-2
runs whole; of the others a case takes a block of a few full-width layers with a vocabulary of 4096, so that its
time is that of the layers and not of copying logits out.

  prepare  a loaded runner, the prompts, their block tables (pages in no order, as an engine's free list has them
           after a while) and, for decode, the cached prompts
  run      the steps; returns the logits after the last one (float32 [sequences, vocabulary]) and, for greedy
           decoding, the tokens [sequences, steps]
  exact    the same in float64 with plain torch, no caches, whole sequences at once

Lengths: a ragged batch spreads from half the longest prompt to the longest.  Greedy continuations are stable under
rounding, as a trained model's mostly are: the output head is the embedding table, whose entries are wide enough that a
random-weight model repeats its last token by a wide margin.
"""
import math
import random
from dataclasses import replace

import numpy as np
import torch

import nvllm_pkg

C = nvllm_pkg.sub("config")
W = nvllm_pkg.sub("weights")
R = nvllm_pkg.sub("runner")

BLOCK = C.KV_BLOCK_SIZE
VOCAB = 4096


def _hybrid():
    """A Mamba2 and an attention block at Llama-3.2-1B's width (64 heads of 64, state 128, 8 groups, 4 taps)."""
    return C.tiny_hybrid(vocab_size=VOCAB, hidden=2048, num_layers=2, num_heads=32, num_kv_heads=8, head_dim=64, ffn_dim=8192,
                         max_seq_len=8192, mamba_num_heads=64, mamba_head_dim=64, mamba_state_size=128, mamba_n_groups=8,
                         mamba_conv_kernel=4, hybrid_layers=(True, False))


def _zozonex():
    """A delta-rule and a window-attention layer at the same width, squared-ReLU feed-forward of 12288."""
    delta = C.LayerSpec(mixer=C.MIXER_DELTA, heads=16, kv_heads=8, dim=128, vdim=128, conv=4, mlp=C.MLP_DENSE, ff=12288,
                        act=C.FFN_RELU2)
    window = C.LayerSpec(mixer=C.MIXER_WINDOW_ATTENTION, heads=32, kv_heads=8, dim=64, vdim=64, window=1024, sink=1, qk_norm=1,
                         scale=0.125, mlp=C.MLP_DENSE, ff=12288, act=C.FFN_RELU2)
    return C.ListedModelConfig("zozonex", VOCAB, 2048, (delta, window), 1e-5, embedding_scale=2048.0 ** 0.5, arch=C.ARCH_ZOZONEX,
                               block_style=C.LBLOCK_SEQUENTIAL_POSTNORM, position=C.LPOS_SINUSOIDAL, tied_head=True,
                               norm_offset=1.0)


#: name -> (config, depth of the whole model, which sets the scale of the output projections)
MODELS = {
    "gpt2": (lambda: C.gpt2_small(), 12),
    "llama-1b": (lambda: replace(C.llama32_1b(), num_layers=4, vocab_size=VOCAB), 16),
    "llama-3b": (lambda: replace(C.llama32_3b(), num_layers=2, vocab_size=VOCAB), 28),
    "granite-moe": (lambda: replace(C.granite_moe_1b(), num_layers=4, vocab_size=VOCAB), 24),
    "falcon": (lambda: replace(C.falcon_7b(), num_layers=2, vocab_size=VOCAB), 32),
    "hybrid": (_hybrid, 16),
    "zozonex": (_zozonex, 16),
}


def _case(model, kind, seqs, tokens, ragged=True, steps=0, shared=0, f32=False, sampled=False):
    return {"model": model, "kind": kind, "seqs": seqs, "tokens": tokens, "ragged": ragged, "steps": steps, "shared": shared,
            "f32": f32, "sampled": sampled}


def listed():
    return [
        # one user, one short prompt, greedy decoding: a chain of the smallest launches
        dict(_case("gpt2", "decode", 1, 32, ragged=False, steps=16), name="gpt2-decode-1"),
        # the reference's own precision: four short prompts in float32
        dict(_case("gpt2", "prefill", 4, 100, f32=True), name="gpt2-prompts-f32"),
        # a full batch of prompts, as the scheduler packs them
        dict(_case("llama-1b", "prefill", 64, 512), name="llama-prompts-64"),
        # continuous batching: 64 conversations, all of them decoding
        dict(_case("llama-1b", "decode", 64, 640, steps=16), name="llama-decode-64"),
        # long prompts on a cached prefix: the first request fills the pages that the others find
        dict(_case("llama-3b", "prefill", 16, 4096, ragged=False, shared=3840), name="llama-prefix-16"),
        # prompts through routed experts
        dict(_case("granite-moe", "prefill", 64, 384), name="moe-prompts-64"),
        # a wide decode batch through routed experts
        dict(_case("granite-moe", "decode", 128, 256, steps=16), name="moe-decode-128"),
        # one long prompt, one K / V head for 71 query heads, odd widths
        dict(_case("falcon", "prefill", 1, 2048, ragged=False), name="falcon-prompt-1"),
        # a step with the reference's default sampling: temperature 1, repetition penalty over the history
        dict(_case("falcon", "decode", 8, 700, steps=1, sampled=True), name="falcon-sampled-8"),
        # prompts through a state-space block
        dict(_case("hybrid", "prefill", 16, 512), name="hybrid-prompts-16"),
        # longer prompts through a recurrence and windowed attention
        dict(_case("zozonex", "prefill", 16, 1500), name="zozonex-prompts-16"),
        # whole requests of a model with recurrent state: short prompts, then decoding
        dict(_case("zozonex", "generate", 32, 64, steps=16), name="zozonex-requests-32"),
    ]


#: (model, kind, most sequences, shortest and longest prompt, most tokens in the batch, further options)
RANGES = [
    ("gpt2", "decode", 8, 8, 900, 4000, {"steps": 16}),
    ("gpt2", "prefill", 4, 8, 256, 512, {"f32": True}),
    ("llama-1b", "prefill", 64, 16, 2048, 32768, {}),
    ("llama-1b", "decode", 128, 16, 2048, 40960, {"steps": 16}),
    ("llama-3b", "prefill", 16, 300, 4096, 65536, {"shared": True}),
    ("granite-moe", "prefill", 64, 16, 1024, 24576, {}),
    ("granite-moe", "decode", 128, 16, 1024, 32768, {"steps": 16}),
    ("falcon", "prefill", 4, 16, 2048, 2048, {}),
    ("falcon", "decode", 8, 16, 2000, 8000, {"steps": 1, "sampled": True}),
    ("hybrid", "prefill", 16, 16, 2048, 8192, {}),
    ("zozonex", "prefill", 16, 16, 3000, 24000, {}),
    ("zozonex", "generate", 32, 8, 128, 2048, {"steps": 16}),
]


def draw(rng):
    model, kind, most, low, high, total, more = rng.choice(RANGES)
    seqs = round(math.exp(rng.uniform(0.0, math.log(most))))
    high = max(low, min(high, total // seqs))
    tokens = round(math.exp(rng.uniform(math.log(low), math.log(high))))
    more = dict(more)
    if more.pop("shared", False):
        more["shared"] = BLOCK * rng.randint(0, (tokens - 1) // BLOCK)
    return _case(model, kind, seqs, tokens, ragged=rng.random() < 0.7 and not more.get("shared"), **more)


# ---- inputs

def _lengths(case):
    rng = random.Random(case["seqs"] * 100003 + case["tokens"])
    n, top = case["seqs"], case["tokens"]
    return [top] + [rng.randint(max(1, top // 2), top) if case["ragged"] else top for _ in range(n - 1)]


def _prompts(case, vocab, seed):
    rng = np.random.RandomState(seed % (1 << 31))
    common = rng.randint(0, vocab, case["shared"])
    return [np.concatenate([common, rng.randint(0, vocab, n - case["shared"])]).astype(np.int32) for n in _lengths(case)]


def _draws(case, seed):
    return np.random.RandomState((seed + 7) % (1 << 31)).random_sample(case["seqs"]).astype(np.float32) if case["sampled"] else None


def _tables(case, seed):
    """Block tables with room for the steps and one token more; prompts on a common prefix share its pages."""
    common = case["shared"] // BLOCK
    own = [-(-(n + case["steps"] + 1) // BLOCK) - common for n in _lengths(case)]
    total = common + sum(own)
    pages = np.random.RandomState((seed + 3) % (1 << 31)).permutation(total).astype(np.int32)
    tables, at = [], common
    for k in own:
        tables.append(np.concatenate([pages[:common], pages[at:at + k]]))
        at += k
    return tables, total


def _uniform_weights(cfg, depth, seed):
    """(weight id, layer, float32 tensor on the GPU holding bf16 values) in the layouts that the runner takes."""
    g = torch.Generator(device="cuda")
    for wid, layer, shape, std, mean in W.weight_specs(cfg):
        g.manual_seed((seed * 1000003 + wid * 7919 + (layer + 1) * 104729) & 0x7FFFFFFF)
        if wid in (C.W_O, C.W_FFN_W2, C.W_MOE_OUTPUT, C.W_MAMBA_OUT_PROJ):
            std = 0.02 / math.sqrt(2 * depth)
        elif wid == C.W_TOKEN_EMBEDDING and not cfg.embedding_multiplier:
            std = 0.1
        t = torch.empty(shape, dtype=torch.float32, device="cuda").normal_(mean, std, generator=g)
        yield wid, layer, t.to(torch.bfloat16)


def _named_weights(cfg, seed):
    g = torch.Generator(device="cuda")
    for i, (name, shape) in enumerate(cfg.tensor_shapes().items()):
        g.manual_seed((seed * 1000003 + i) & 0x7FFFFFFF)
        t = torch.empty(shape, dtype=torch.float32, device="cuda")
        if name.endswith("A_log"):
            t.uniform_(-3.0, 0.5, generator=g)
        elif name.endswith("dt_bias"):
            t.uniform_(-2.0, 1.0, generator=g)
        elif name.endswith("mix.norm"):
            t.normal_(1.0, 0.02, generator=g)
        elif len(shape) == 1:
            t.normal_(0.0, 0.02, generator=g)  # norm weights are stored around zero
        else:
            t.normal_(0.0, 0.02 if name == "embed" else shape[1] ** -0.5, generator=g)
        yield name, t.to(torch.bfloat16)


def _bits(t):
    return t.view(torch.int16).cpu().numpy().view(np.uint16)


def prepare(case, seed):
    make, depth = MODELS[case["model"]]
    cfg = make()
    tables, blocks = _tables(case, seed)
    prompts = _prompts(case, cfg.vocab_size, seed)
    if isinstance(cfg, C.ListedModelConfig):
        weights = ((name, _bits(t)) for name, t in _named_weights(cfg, seed))
    else:
        weights = ((wid, layer, _bits(t)) for wid, layer, t in _uniform_weights(cfg, depth, seed))
    runner = R.CudaModelRunner(cfg, weights, precision=C.PREC_FP32 if case["f32"] else C.PREC_BF16, num_kv_blocks=blocks,
                               max_num_seqs=case["seqs"], max_batched_tokens=sum(len(p) for p in prompts),
                               sampling=R.DEFAULT_SAMPLING if case["sampled"] else None)
    n, lens = len(prompts), np.array([len(p) for p in prompts])
    texts = np.zeros((n, lens.max() + case["steps"] + 1), dtype=np.int32)
    for i, p in enumerate(prompts):
        texts[i, :len(p)] = p
    state = {"case": case, "runner": runner, "texts": texts, "lens": lens, "tables": tables,
             "cached": [0] + [case["shared"]] * (n - 1), "temperature": [runner.temperature] * n,
             "uniforms": _draws(case, seed), "slots": list(range(n)) if runner.needs_state_slots else None}
    if case["kind"] == "decode":
        _step(state, lens, True)
    return state


# ---- one pass

def _step(s, lens, is_prefill, logits=False):
    return s["runner"].run_flat([t[:k] for t, k in zip(s["texts"], lens)], is_prefill, s["cached"] if is_prefill else None,
                                s["tables"], s["temperature"], s["uniforms"], want_logits=logits, state_slots=s["slots"])


def run(state):
    case, lens, texts = state["case"], state["lens"].copy(), state["texts"]
    if case["kind"] == "prefill":
        return {"logits": _step(state, lens, True, logits=True)[1]}
    rows, tokens, logits = np.arange(len(lens)), [], None
    for k in range(case["steps"]):
        out, logits = _step(state, lens, case["kind"] == "generate" and k == 0, logits=k == case["steps"] - 1)
        texts[rows, lens] = out
        lens += 1
        tokens.append(out)
    return {"logits": logits} if case["sampled"] else {"logits": logits, "tokens": np.stack(tokens, 1)}


# ---- what a pass cannot do without

def work(case):
    cfg = MODELS[case["model"]][0]()
    lens = _lengths(case)
    n, size = len(lens), 4 if case["f32"] else 2
    start = [case["shared"] if i else 0 for i in range(n)]
    steps = []  # (new tokens, (query, key) pairs, cached tokens read) of each step
    if case["kind"] != "decode":
        steps.append((sum(a - b for a, b in zip(lens, start)), sum((a * (a + 1) - b * (b + 1)) / 2 for a, b in zip(lens, start)),
                      case["shared"] if case["shared"] else 0))
    for k in range(len(steps), case["steps"]):
        steps.append((n, sum(lens) + n * k, sum(lens) + n * k))
    listed_model = isinstance(cfg, C.ListedModelConfig)
    head = cfg.vocab_size * cfg.hidden
    if listed_model:
        heads_dim, kv_row, layers = 32 * 64, 2 * 8 * 64, 1
        routed, state, state_flops = 0, 16 * 128 * 128 * 4, 8 * 16 * 128 * 128
        dense = sum(math.prod(s) for k, s in cfg.tensor_shapes().items() if len(s) > 1 and k not in ("embed",))
    else:
        attention = [l for l in range(cfg.num_layers) if not cfg.is_mamba(l)]
        layers, heads_dim, kv_row = len(attention), cfg.num_heads * cfg.head_dim, 2 * cfg.kv_heads() * cfg.head_dim
        specs = list(W.weight_specs(cfg))
        routed = sum(math.prod(s[2]) for s in specs if s[0] in (C.W_MOE_INPUT, C.W_MOE_OUTPUT))
        dense = sum(math.prod(s[2]) for s in specs if s[1] >= 0 and len(s[2]) > 1) - routed
        cells = cfg.mamba_num_heads * cfg.mamba_head_dim * cfg.mamba_state_size * (cfg.num_layers - layers)
        state, state_flops = 4 * cells, 5 * cells
    total_bytes = total_flops = 0.0
    for new, pairs, read in steps:
        if listed_model:  # a window of 1024
            pairs = min(pairs, 1024 * new)
            read = min(read, 1024 * n)
        share = cfg.num_experts_per_tok / cfg.num_experts if routed else 0.0
        touched = 1.0 - (1.0 - share) ** new if routed else 0.0
        total_bytes += size * (dense + touched * routed + head + layers * kv_row * (read + new)) + state * n + 4 * new
        total_flops += 2.0 * new * (dense + share * routed) + 2.0 * n * head + 4.0 * layers * heads_dim * pairs + state_flops * new
    return {"bytes": total_bytes + 4.0 * n * cfg.vocab_size, "flops": total_flops}


#: about four times the relative error against float64 of the bfloat16 path at the listed sizes
BF16_ERROR = {"gpt2": 0.013, "llama-1b": 0.022, "llama-3b": 0.016, "granite-moe": 0.006, "falcon": 0.014, "hybrid": 0.006,
              "zozonex": 0.013}


def tolerance(case):
    rel = 6e-6 if case["f32"] else BF16_ERROR[case["model"]]
    return {"rel": rel, "max": 12 * rel}


# ---- the same in float64

def _norm(x, w, b, eps, layer_norm):
    if layer_norm:
        x = x - x.mean(-1, keepdim=True)
    y = x / torch.sqrt(x.square().mean(-1, keepdim=True) + eps) * w
    return y if b is None else y + b


def _rotate(x, base):
    """x [tokens, heads, size]: halves rotated, positions from 0."""
    half = x.shape[-1] // 2
    f = base ** (-2.0 * torch.arange(half, dtype=torch.float64, device=x.device) / x.shape[-1])
    a = torch.arange(x.shape[0], dtype=torch.float64, device=x.device)[:, None, None] * f
    return torch.cat([x[..., :half] * a.cos() - x[..., half:] * a.sin(), x[..., half:] * a.cos() + x[..., :half] * a.sin()], -1)


def _attend(q, k, v, scale, window=0, sink=False):
    """One sequence: q [tokens, heads, size], k and v [tokens, K / V heads, size]."""
    t, heads = q.shape[:2]
    k, v = (z.repeat_interleave(heads // z.shape[1], 1).transpose(0, 1) for z in (k, v))
    out, q, at = [], q.transpose(0, 1), torch.arange(t, device=q.device)
    for i in range(0, t, 512):  # a band of queries at a time
        rows, stop = at[i:i + 512, None], min(t, i + 512)
        s = q[:, i:stop] @ k[:, :stop].transpose(1, 2) * scale
        seen = at[None, :stop] <= rows
        if window:
            seen = seen & (rows - at[None, :stop] < window)
        s = s.masked_fill(~seen, -math.inf)
        if sink:
            top = s.amax(-1, keepdim=True).clamp(min=0.0)
            e = (s - top).exp()
            p = e / (e.sum(-1, keepdim=True) + (-top).exp())
        else:
            p = s.softmax(-1)
        out.append(p @ v[:, :stop])
    return torch.cat(out, 1).transpose(0, 1).reshape(t, -1)


def _silu(x):
    return x * torch.sigmoid(x)


def _conv(x, w, spans):
    """Causal convolution over time of each sequence's rows; w [channels, taps], the last tap on the current row."""
    out, taps = torch.zeros_like(x), w.shape[1]
    for a, b in spans:
        for j in range(taps):
            back = taps - 1 - j
            if b - a > back:
                out[a + back:b] += x[a:b - back] * w[:, j]
    return out


def _padded(x, spans):
    """[tokens, ...] of ragged sequences -> [sequences, longest, ...]."""
    out = x.new_zeros((len(spans), max(b - a for a, b in spans)) + x.shape[1:])
    for i, (a, b) in enumerate(spans):
        out[i, :b - a] = x[a:b]
    return out


def _ragged(x, spans):
    return torch.cat([x[i, :b - a] for i, (a, b) in enumerate(spans)])


def _mamba(cfg, w, l, h, spans):
    heads, size, state, groups = cfg.mamba_num_heads, cfg.mamba_head_dim, cfg.mamba_state_size, cfg.mamba_n_groups
    inner = heads * size
    z = h @ w[C.W_MAMBA_IN_PROJ, l].T
    gate, xbc, dt = z.split([inner, inner + 2 * groups * state, heads], 1)
    xbc = _silu(_conv(xbc, w[C.W_MAMBA_CONV_W, l][:, 0], spans) + w[C.W_MAMBA_CONV_B, l])
    u, b, c = xbc.split([inner, groups * state, groups * state], 1)
    dt = torch.nn.functional.softplus(dt + w[C.W_MAMBA_DT_BIAS, l])
    decay = (-w[C.W_MAMBA_A_LOG, l].exp() * dt).exp()
    u = u.reshape(-1, heads, size)
    b, c = (_padded(m.reshape(-1, groups, state).repeat_interleave(heads // groups, 1), spans) for m in (b, c))
    du, decay = _padded(dt[..., None] * u, spans), _padded(decay, spans)
    s, ys = u.new_zeros(len(spans), heads, size, state), []
    for t in range(du.shape[1]):
        s = decay[:, t, :, None, None] * s + du[:, t, :, :, None] * b[:, t, :, None, :]
        ys.append((s * c[:, t, :, None, :]).sum(-1))
    y = (_ragged(torch.stack(ys, 1), spans) + w[C.W_MAMBA_D, l][:, None] * u).reshape(-1, inner) * _silu(gate)
    return _norm(y, w[C.W_MAMBA_NORM, l], None, 1e-5, False) @ w[C.W_MAMBA_OUT_PROJ, l].T


def _experts(cfg, w, l, h):
    top = (h @ w[C.W_MOE_ROUTER, l]).topk(cfg.num_experts_per_tok, -1)
    share, out = top.values.softmax(-1), torch.zeros_like(h)
    for e in range(cfg.num_experts):
        row, slot = (top.indices == e).nonzero(as_tuple=True)
        gate, up = (h[row] @ w[C.W_MOE_INPUT, l][e].double().T).chunk(2, 1)
        out.index_add_(0, row, share[row, slot, None] * ((_silu(gate) * up) @ w[C.W_MOE_OUTPUT, l][e].double().T))
    return out


def _uniform64(cfg, w, tokens, spans):
    """Hidden rows after the last norm; w: (weight id, layer) -> float64 tensor (experts stay in bf16)."""
    ln, heads, kv, size = cfg.norm_type == C.NORM_LAYER, cfg.num_heads, cfg.kv_heads(), cfg.head_dim
    at = torch.cat([torch.arange(b - a, device=tokens.device) for a, b in spans])
    x = w[C.W_TOKEN_EMBEDDING, -1][tokens] * (cfg.embedding_multiplier or 1.0)
    if cfg.position_type == C.POS_LEARNED:
        x = x + w[C.W_POS_EMBEDDING, -1][at]
    scale, m = cfg.attention_multiplier or size ** -0.5, cfg.residual_multiplier or 1.0
    for l in range(cfg.num_layers):
        def bias(wid):
            return w.get((wid, l), 0.0)

        h = _norm(x, w[C.W_ATTN_NORM_W, l], w.get((C.W_ATTN_NORM_B, l)), cfg.norm_eps, ln)
        if cfg.is_mamba(l):
            y = _mamba(cfg, w, l, h, spans)
        else:
            q = h @ w[C.W_Q, l] + bias(C.W_Q_BIAS)
            if cfg.attention_type == C.ATTN_MQA:
                k, v = (h @ w[C.W_KV, l]).chunk(2, 1)
            else:
                k, v = h @ w[C.W_K, l] + bias(C.W_K_BIAS), h @ w[C.W_V, l] + bias(C.W_V_BIAS)
            q, k, v = q.reshape(-1, heads, size), k.reshape(-1, kv, size), v.reshape(-1, kv, size)
            o = []
            for a, b in spans:
                qs, ks = q[a:b], k[a:b]
                if cfg.position_type == C.POS_ROPE:
                    qs, ks = _rotate(qs, cfg.rope_base), _rotate(ks, cfg.rope_base)
                o.append(_attend(qs, ks, v[a:b], scale))
            y = torch.cat(o) @ w[C.W_O, l] + bias(C.W_O_BIAS)
        if cfg.block_style == C.BLOCK_SEQUENTIAL:
            x = x + m * y
            h = _norm(x, w[C.W_FFN_NORM_W, l], w.get((C.W_FFN_NORM_B, l)), cfg.norm_eps, ln)
            y = 0.0
        if cfg.use_moe:
            f = _experts(cfg, w, l, h)
        else:
            f = h @ w[C.W_FFN_W1, l] + bias(C.W_FFN_B1)
            if cfg.activation_type == C.ACT_SWIGLU:
                f = _silu(f[:, :cfg.ffn_dim]) * f[:, cfg.ffn_dim:]
            else:
                f = torch.nn.functional.gelu(f, approximate="tanh")
            f = f @ w[C.W_FFN_W2, l] + bias(C.W_FFN_B2)
        x = x + y + m * f
    return _norm(x, w[C.W_FINAL_NORM_W, -1], w.get((C.W_FINAL_NORM_B, -1)), cfg.norm_eps, ln) / (cfg.logits_scaling or 1.0)


def _zozonex64(cfg, w, tokens, spans):
    eps, wide = cfg.norm_eps, cfg.hidden
    at = torch.cat([torch.arange(b - a, device=tokens.device) for a, b in spans]).double()[:, None]
    angle = at * 10000.0 ** (-2.0 * torch.arange(wide // 2, dtype=torch.float64, device=tokens.device) / wide)
    x = w["embed"][tokens] * cfg.embedding_scale + torch.stack([angle.sin(), angle.cos()], -1).reshape(-1, wide)
    for i, s in enumerate(cfg.layers):
        p = "l%d.mix." % i
        q, k, v = (x @ w[p + c].T for c in "qkv")
        if s.mixer == C.MIXER_DELTA:
            q, k, v = (_silu(_conv(z, w[p + c + ".conv"], spans)) for z, c in ((q, "q"), (k, "k"), (v, "v")))
            q, k = (z.reshape(-1, s.kv_heads, s.dim) for z in (q, k))
            q, k = (z / torch.sqrt(z.square().sum(-1, keepdim=True) + 1e-6) for z in (q, k))
            q, k = (_padded(z.repeat_interleave(s.heads // s.kv_heads, 1), spans) for z in (q / math.sqrt(s.dim), k))
            v = _padded(v.reshape(-1, s.heads, s.vdim), spans)
            beta = _padded(torch.sigmoid(x @ w[p + "b"].T), spans)
            g = -w[p + "A_log"].exp() * torch.nn.functional.softplus(x @ w[p + "a"].T + w[p + "dt_bias"])
            g = _padded(g.exp(), spans)
            state, o = v.new_zeros(len(spans), s.heads, s.dim, s.vdim), []
            for t in range(v.shape[1]):
                state = state * g[:, t, :, None, None]
                u = beta[:, t, :, None] * (v[:, t] - (state * k[:, t, :, :, None]).sum(2))
                state = state + k[:, t, :, :, None] * u[:, :, None, :]
                o.append((state * q[:, t, :, :, None]).sum(2))
            o = _norm(_ragged(torch.stack(o, 1), spans), w[p + "norm"], None, eps, False)
            o = o.reshape(len(x), -1) * _silu(x @ w[p + "g"].T)
        else:
            q, k = (_norm(z.reshape(-1, h, s.dim), 1.0, None, eps, False) for z, h in ((q, s.heads), (k, s.kv_heads)))
            v = v.reshape(-1, s.kv_heads, s.vdim)
            o = torch.cat([_attend(q[a:b], k[a:b], v[a:b], s.scale, s.window, True) for a, b in spans])
        x = x + _norm(o @ w[p + "o"].T, 1.0 + w["l%d.norm1" % i], None, eps, False)
        f = (x @ w["l%d.mlp.up" % i].T).clamp(min=0.0).square() @ w["l%d.mlp.down" % i].T
        x = x + _norm(f, 1.0 + w["l%d.norm2" % i], None, eps, False)
    return _norm(x, 1.0 + w["final.norm"], None, eps, False)


def exact(case, seed):
    make, depth = MODELS[case["model"]]
    cfg = make()
    if isinstance(cfg, C.ListedModelConfig):
        w = {name: t.double() for name, t in _named_weights(cfg, seed)}
        rows, head = _zozonex64, w["embed"]
    else:
        w = {(wid, layer): t if wid in (C.W_MOE_INPUT, C.W_MOE_OUTPUT) else t.double()
             for wid, layer, t in _uniform_weights(cfg, depth, seed)}
        rows, head = _uniform64, w[C.W_TOKEN_EMBEDDING, -1] if cfg.tied_embedding else w[C.W_LM_HEAD, -1].T
    texts = [torch.from_numpy(p).long().cuda() for p in _prompts(case, cfg.vocab_size, seed)]
    greedy = 0 if case["kind"] == "prefill" or case["sampled"] else case["steps"]
    # continuations start as the last token repeated and are corrected until every token is the one its prefix gives
    guess = torch.stack([t[-1:].repeat(max(greedy, 1)) for t in texts])
    while True:
        full = [torch.cat([t, g[:-1]]) for t, g in zip(texts, guess)]
        ends = np.cumsum([len(t) for t in full])
        spans = [(int(e) - len(t), int(e)) for t, e in zip(full, ends)]
        x = rows(cfg, w, torch.cat(full), spans)
        logits = torch.stack([x[b - guess.shape[1]:b] @ head.T for _, b in spans])
        tokens = logits.argmax(-1)
        if not greedy or torch.equal(tokens, guess):
            break
        guess = tokens
    out = {"logits": logits[:, -1].cpu()}
    return dict(out, tokens=tokens.cpu()) if greedy else out
