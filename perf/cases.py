"""Cases of the performance measurements: one step of one pipeline stage.

A pipeline peer keeps a range of decoder layers and its part of the paged KV cache. Per engine iteration it gets one
batch (prompt slices and decoding rows, packed by :class:`BatchBuilder`) and the hidden states of the stage before it,
and hands on its own (the last stage: logits). That step, :meth:`StageWorker.run`, is what every case times, for each
kind of decoder that the framework serves under a Hugging Face config: dense grouped-query attention, routed experts,
latent attention with block-scaled fp8 weights, latent attention over indexed keys, and the gated-delta-net hybrid.

A case:
  model          architecture (sizes of the repository's named configurations; the hybrid's are those of its layer benchmark)
  start, layers  layers ``[start, start + layers)``
  prompts, prompt, cached   prompt slices in the batch, new tokens of the longest one, tokens already in the cache
  decode, ctx    decoding rows and the longest one's context
  kv             storage of the K / V pages ("bf16" or "fp8_e4m3")
Lengths are ragged: sequence i is shorter than the longest by a remainder that depends on i.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from parallax_b200.engine.batch import BatchBuilder
from parallax_b200.engine.worker import StageWorker
from parallax_b200.models.config import config_from_hf, named_config

PAGE = 16
DEV = "cuda:0"


def _case(name, model, start, layers, prompts=0, prompt=0, cached=0, decode=0, ctx=0, kv="bf16"):
    return dict(name=name, model=model, start=start, layers=layers, prompts=prompts, prompt=prompt, cached=cached,
                decode=decode, ctx=ctx, kv=kv)


def listed():
    return [
        # a single chat on two nodes of 14 layers each: what the second node does per token (launches and latency count)
        _case("chat-one-row", "qwen3-0.6b", 14, 14, decode=1, ctx=777),
        # a micro-batch of the eight-stage pipeline that serves 512 requests, on a stage of five layers
        _case("pipeline-micro-batch", "qwen3-8b", 13, 5, decode=57, ctx=1280),
        # the headline workload: 510 decoding rows beside the prompts that replace finished requests
        _case("closed-loop-mixed", "qwen3-8b", 8, 2, prompts=2, prompt=1024, decode=510, ctx=1280),
        # one 8192-token slice of a long prompt
        _case("long-prompt-slice", "qwen3-32b", 20, 1, prompts=1, prompt=8192, cached=16384),
        # decoding with e4m3 pages, chosen where the cache is what limits the batch
        _case("e4m3-pages-decode", "qwen3-8b", 8, 2, decode=128, ctx=4096, kv="fp8_e4m3"),
        # routed experts: decoding reads almost every expert for a few rows each, prompts fill them
        _case("experts-decode", "qwen3-30b-a3b", 8, 2, decode=48, ctx=2100),
        _case("experts-prompts", "qwen3-30b-a3b", 8, 2, prompts=3, prompt=1700),
        # latent attention with fp8 weights (the dense layers at the front of the model)
        _case("latent-decode", "deepseek-v3", 1, 2, decode=64, ctx=4096),
        _case("latent-prompts", "deepseek-v3", 1, 1, prompts=2, prompt=2048),
        # latent attention over the indexer's best keys: a slice of a long prompt beside decoding rows
        _case("indexed-mixed", "deepseek-v3.2", 1, 1, prompts=1, prompt=1000, cached=5000, decode=16, ctx=8192),
        # three gated-delta-net layers and one attention layer
        _case("hybrid-prompts", "hybrid-8b", 4, 4, prompts=2, prompt=3000),
        _case("hybrid-decode", "hybrid-8b", 4, 4, decode=96, ctx=2048),
    ]


def _log(rng, lo, hi):
    """A whole number of [lo, hi], even over its logarithm, odd or even."""
    return min(hi, max(lo, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    model = rng.choice(["qwen3-0.6b", "qwen3-8b", "qwen3-8b", "qwen3-32b", "qwen3-30b-a3b", "deepseek-v3", "deepseek-v3.2",
                        "hybrid-8b"])
    kind = rng.choice(["decode", "prompts", "mixed"])
    big = {"qwen3-32b": 1, "deepseek-v3": 1, "deepseek-v3.2": 1, "hybrid-8b": 4}.get(model)
    start = {"qwen3-0.6b": 24, "deepseek-v3": 1, "deepseek-v3.2": 1, "hybrid-8b": 4}.get(model, 8)
    c = _case("", model, start, big or (4 if model == "qwen3-0.6b" else rng.choice([1, 2])))
    del c["name"]
    if kind != "decode":
        c["prompts"] = _log(rng, 1, 8)
        c["prompt"] = max(1, _log(rng, 17, 2048 if model.startswith("deepseek") else 4096) // c["prompts"])
        if rng.random() < 0.5:
            c["cached"] = _log(rng, 16, 6000)
    if kind != "prompts":
        c["decode"] = _log(rng, 1, 256)
        c["ctx"] = min(_log(rng, 16, 8192), 400000 // c["decode"])
    if not model.startswith("deepseek") and model != "hybrid-8b" and c["decode"] and not c["prompts"] and rng.random() < 0.3:
        c["kv"] = "fp8_e4m3"
    return c


# ------------------------------------------------------------------------------------------------ the batch
def _config(model):
    if model != "hybrid-8b":
        return named_config(model)
    return config_from_hf(dict(
        architectures=["Qwen3NextForCausalLM"], model_type="qwen3_next", hidden_size=4096, num_hidden_layers=32,
        num_attention_heads=32, num_key_value_heads=8, head_dim=128, intermediate_size=12288, vocab_size=1024, rope_theta=1e4,
        partial_rotary_factor=0.25, full_attention_interval=4, max_position_embeddings=16384, linear_num_key_heads=16,
        linear_num_value_heads=32, linear_key_head_dim=128, linear_value_head_dim=128, linear_conv_kernel_dim=4))


def _sequences(case):
    """(new tokens, tokens with keys after the step) of every sequence: prompts, then decoding rows."""
    p = [max(1, case["prompt"] - i * 97 % (case["prompt"] // 2 + 1)) for i in range(case["prompts"])]
    d = [max(1, case["ctx"] - i * 53 % (case["ctx"] // 4 + 1)) for i in range(case["decode"])]
    return [(n, n + case["cached"]) for n in p], d


def _plan(case, seed):
    """Index arrays of the step, with the pages of the cache in random order."""
    prompts, decode = _sequences(case)
    seqs = prompts + [(1, c) for c in decode]
    need = [-(-total // PAGE) for _n, total in seqs]
    order = np.random.RandomState(seed % (1 << 31)).permutation(sum(need)).astype(np.int32)
    table = np.zeros((len(seqs), max(need)), dtype=np.int32)
    at = 0
    for i, n in enumerate(need):
        table[i, :n] = order[at:at + n]
        at += n
    pos = np.concatenate([np.arange(total - n, total, dtype=np.int32) for n, total in seqs])
    row = np.repeat(np.arange(len(seqs)), [n for n, _t in seqs])
    slots = table[row, pos // PAGE].astype(np.int64) * PAGE + pos % PAGE
    last = np.cumsum([n for n, _t in seqs]).astype(np.int32) - 1
    return dict(prompts=prompts, decode=decode, seqs=seqs, table=table, pos=pos, slots=slots, last=last, blocks=sum(need),
                tokens=len(pos))


# ------------------------------------------------------------------------------------------------ weights and cache contents
class _Random:
    def __init__(self, seed):
        self.g = torch.Generator(device=DEV)
        self.g.manual_seed(seed)

    def normal(self, *shape, std=1.0, mean=0.0, dtype=torch.bfloat16):
        t = torch.empty(shape, device=DEV, dtype=dtype)
        return t.normal_(mean, std, generator=self.g)

    def weight(self, *shape):
        return self.normal(*shape, std=0.02)

    def fp8_weight(self, n, k):
        """A bf16 matrix as a block-scaled fp8 checkpoint holds it: e4m3 values times one power of two, whose largest
        value every 64 x 128 block has, so that every correct quantisation gives the same blocks."""
        w = self.normal(n, k, std=0.02)
        q = (w.float() * 4096).clamp_(-448, 448).to(torch.float8_e4m3fn).to(torch.bfloat16)
        q[::64, ::128] = 448.0
        return q.mul_(1 / 4096)


def _weights(cfg, case, r):
    """Checkpoint tensors of the stage's layers under their Hugging Face names."""
    H, D, Hq, Hkv, I = cfg.hidden_size, cfg.head_dim, cfg.num_attention_heads, cfg.num_key_value_heads, cfg.intermediate_size
    hybrid = cfg.model_type == "qwen3_next"
    norm = (lambda n, at=1.0: r.normal(n, std=0.1, mean=at - 1.0)) if hybrid else (lambda n, at=1.0: r.normal(n, std=0.1, mean=at))
    big = r.fp8_weight if cfg.quant_method == "fp8" else r.weight
    w = {}
    for i in range(case["start"], case["start"] + case["layers"]):
        p = f"model.layers.{i}."
        w[p + "input_layernorm.weight"], w[p + "post_attention_layernorm.weight"] = norm(H), norm(H)
        a = p + "self_attn."
        if cfg.is_mla:
            ql, L, R, nope, V = cfg.q_lora_rank, cfg.kv_lora_rank, cfg.qk_rope_head_dim, cfg.qk_nope_head_dim, cfg.v_head_dim
            w[a + "q_a_proj.weight"], w[a + "q_a_layernorm.weight"] = r.weight(ql, H), norm(ql, 2.5)
            w[a + "q_b_proj.weight"] = big(Hq * (nope + R), ql)
            w[a + "kv_a_proj_with_mqa.weight"], w[a + "kv_a_layernorm.weight"] = r.weight(L + R, H), norm(L)
            w[a + "kv_b_proj.weight"], w[a + "o_proj.weight"] = r.weight(Hq * (nope + V), L), big(H, Hq * V)
            if cfg.index_topk:
                x = a + "indexer."
                w[x + "wq_b.weight"] = r.weight(cfg.index_n_heads * cfg.index_head_dim, ql)
                w[x + "wk.weight"], w[x + "k_norm.weight"] = r.weight(cfg.index_head_dim, H), norm(cfg.index_head_dim)
                w[x + "k_norm.bias"], w[x + "weights_proj.weight"] = r.normal(cfg.index_head_dim, std=0.1), r.weight(cfg.index_n_heads, H)
        elif cfg.layer_kind(i) == "linear":
            a = p + "linear_attn."
            hk, hv, dk, dv = cfg.linear_num_key_heads, cfg.linear_num_value_heads, cfg.linear_key_head_dim, cfg.linear_value_head_dim
            c = 2 * hk * dk + hv * dv
            w[a + "in_proj_qkv.weight"], w[a + "in_proj_z.weight"] = r.weight(c, H), r.weight(hv * dv, H)
            w[a + "in_proj_b.weight"], w[a + "in_proj_a.weight"] = r.weight(hv, H), r.weight(hv, H)
            w[a + "conv1d.weight"] = r.normal(c, 1, cfg.linear_conv_kernel_dim, std=0.3)
            w[a + "A_log"] = torch.log(torch.linspace(0.02, 4.0, hv, device=DEV))      # from long memories to short ones
            w[a + "dt_bias"] = torch.linspace(-2.0, 1.0, hv, device=DEV)
            w[a + "norm.weight"], w[a + "out_proj.weight"] = r.normal(dv, std=0.1, mean=1.0), r.weight(H, hv * dv)
        else:
            # scores of a standard deviation of 2: a few dozen keys carry a softmax, as in a trained model
            w[a + "q_norm.weight"], w[a + "k_norm.weight"] = norm(D, 2.0 ** 0.5), norm(D, 2.0 ** 0.5)
            w[a + "q_proj.weight"] = r.weight(Hq * D * (2 if hybrid else 1), H)          # hybrid: per head [q | gate]
            w[a + "k_proj.weight"], w[a + "v_proj.weight"] = r.weight(Hkv * D, H), r.weight(Hkv * D, H)
            w[a + "o_proj.weight"] = r.weight(H, Hq * D)
        m = p + "mlp."
        if cfg.layer_is_moe(i):
            E, F = cfg.num_experts, cfg.moe_intermediate_size
            w[m + "gate.weight"] = r.weight(E, H)
            up, down = r.weight(2, E, F, H), r.weight(E, H, F)
            for e in range(E):
                w[m + f"experts.{e}.gate_proj.weight"], w[m + f"experts.{e}.up_proj.weight"] = up[0, e], up[1, e]
                w[m + f"experts.{e}.down_proj.weight"] = down[e]
        else:
            w[m + "gate_proj.weight"], w[m + "up_proj.weight"], w[m + "down_proj.weight"] = big(I, H), big(I, H), big(H, I)
    if case["start"] + case["layers"] == cfg.num_hidden_layers:
        w["model.norm.weight"] = norm(H)
        w["model.embed_tokens.weight"] = r.weight(cfg.vocab_size, H)                      # (tied: the head, too)
    return w


def _cached(cfg, case, plan, r):
    """Cache contents before the step, per layer: names of the layer's cache object -> tensors. The rows that the step
    writes hold other numbers until then."""
    kv = torch.float8_e4m3fn if case["kv"] == "fp8_e4m3" else torch.bfloat16
    out = []
    for i in range(case["start"], case["start"] + case["layers"]):
        kind = cfg.layer_kind(i)
        if kind == "linear":
            hv, dv, dk = cfg.linear_num_value_heads, cfg.linear_value_head_dim, cfg.linear_key_head_dim
            c = 2 * cfg.linear_num_key_heads * dk + hv * dv
            n = len(plan["seqs"])
            out.append(dict(conv_state=r.normal(n, c, cfg.linear_conv_kernel_dim - 1),
                            rec_state=r.normal(n, hv, dv, dk, std=0.05, dtype=torch.float32)))
        elif cfg.is_mla:
            k = r.normal(plan["blocks"], 1, PAGE, cfg.kv_lora_rank + cfg.qk_rope_head_dim)
            d = dict(k=k)
            if cfg.index_topk:
                d["index_k"] = r.normal(plan["blocks"], 1, PAGE, cfg.index_head_dim)
            out.append(d)
        else:
            shape = (plan["blocks"], cfg.num_key_value_heads, PAGE, cfg.head_dim)
            out.append(dict(k=r.normal(*shape, std=2.0 ** 0.5).to(kv), v=r.normal(*shape, std=1.3).to(kv)))
    return out


def _inputs(case, seed):
    cfg, plan, r = _config(case["model"]), _plan(case, seed), _Random(seed)
    # fp8 activations differ by a few per cent where a rounding falls differently: there a residual stream that outweighs one
    # layer's update, as in a trained model, so that outputs can be compared
    hidden = r.normal(plan["tokens"], cfg.hidden_size, std=8.0 if cfg.quant_method == "fp8" else 1.5)
    return cfg, plan, hidden, _weights(cfg, case, r), _cached(cfg, case, plan, r)


# ------------------------------------------------------------------------------------------------ measured
def prepare(case, seed):
    cfg, plan, hidden, weights, cached = _inputs(case, seed)
    longest = max(t for _n, t in plan["seqs"])
    worker = StageWorker(cfg, case["start"], case["start"] + case["layers"], DEV, torch.bfloat16, PAGE, num_blocks=plan["blocks"],
                         weights=weights, max_positions=longest + 8, num_linear_slots=len(plan["seqs"]),
                         kv_cache_dtype=case["kv"])
    for layer, contents in zip(worker.pool.layers, cached):
        for name, t in contents.items():
            getattr(layer, name).copy_(t)
    np_, table = len(plan["prompts"]), plan["table"]
    builder = BatchBuilder(torch.device(DEV), plan["tokens"], len(plan["seqs"]), 2 * table.shape[1])
    wide = [-(-max([t for _n, t in part], default=0) // PAGE) for part in (plan["seqs"][:np_], plan["seqs"][np_:])]
    fb = builder.build(None, plan["pos"], plan["slots"], [n for n, _t in plan["prompts"]], [t for _n, t in plan["prompts"]],
                       table[:np_, :wide[0]] if np_ else None, np.asarray(plan["decode"], dtype=np.int32),
                       table[np_:, :wide[1]] if plan["decode"] else None, plan["last"],
                       np.arange(len(plan["seqs"]), dtype=np.int32))
    return dict(worker=worker, fb=fb, hidden=hidden, builder=builder)


def run(state):
    """One step: (hidden states or logits, what the layers' caches hold afterwards)."""
    out = state["worker"].run(state["fb"], state["hidden"])
    return [out, [[t for t in (c.k, c.v, c.index_k, c.conv_state, c.rec_state) if t is not None]
                  for c in state["worker"].pool.layers]]


def work(case):
    """Weights, hidden states and cached rows once; a latent layer's prompts in the cheaper of its two forms (keys and
    values expanded per head), its decoding rows on the latent rows."""
    cfg = _config(case["model"])
    prompts, decode = _sequences(case)
    T, H, Hq, D = sum(n for n, _t in prompts) + len(decode), cfg.hidden_size, cfg.num_attention_heads, cfg.head_dim
    pairs = [sum(n * (t - n) + n * (n + 1) // 2 for n, t in prompts), sum(decode)]        # (query, key) pairs
    keys = sum(t for _n, t in prompts) + sum(decode)
    flops, size = 0.0, 2.0 * 2 * T * H
    for i in range(case["start"], case["start"] + case["layers"]):
        wide = 1.0 if cfg.quant_method == "fp8" else 2.0                                  # bytes of a large weight
        if cfg.is_mla:
            L, R, nope, V, ql = cfg.kv_lora_rank, cfg.qk_rope_head_dim, cfg.qk_nope_head_dim, cfg.v_head_dim, cfg.q_lora_rank
            small, large = H * (ql + L + R) + Hq * (nope + V) * L, Hq * ql * (nope + R) + H * Hq * V
            seen, row = pairs, L + R
            if cfg.index_topk:
                small += H * (cfg.index_head_dim + cfg.index_n_heads) + ql * cfg.index_n_heads * cfg.index_head_dim
                flops += 2.0 * sum(pairs) * cfg.index_n_heads * cfg.index_head_dim
                k = cfg.index_topk
                seen = [sum(min(t - n + j + 1, k) for n, t in prompts for j in range(n)), sum(min(c, k) for c in decode)]
                size += 2.0 * keys * cfg.index_head_dim
            flops += 2.0 * Hq * (seen[0] * (nope + R + V) + seen[1] * (2 * L + R))
            flops += 2.0 * (T * (small + large))
            size += 2.0 * small + wide * large + 2.0 * row * (min(keys, sum(seen)) if cfg.index_topk else keys)
        elif cfg.layer_kind(i) == "linear":
            hk, hv, dk, dv = cfg.linear_num_key_heads, cfg.linear_num_value_heads, cfg.linear_key_head_dim, cfg.linear_value_head_dim
            n = H * (2 * hk * dk + 3 * hv * dv + 2 * hv)
            flops += 2.0 * T * n + 6.0 * T * hv * dk * dv
            size += 2.0 * n + 4.0 * hv * dk * dv * (2 * len(decode) + len(prompts))
        else:
            n = H * D * (2 * Hq + 2 * cfg.num_key_value_heads + (Hq if cfg.model_type == "qwen3_next" else 0))
            flops += 2.0 * T * n + 4.0 * sum(pairs) * Hq * D
            size += 2.0 * n + (1.0 if case["kv"] == "fp8_e4m3" else 2.0) * 2 * keys * cfg.num_key_value_heads * D
        if cfg.layer_is_moe(i):
            E, k, one = cfg.num_experts, cfg.num_experts_per_tok, 3 * H * cfg.moe_intermediate_size
            flops += 2.0 * T * (k * one + H * E)
            size += 2.0 * one * E * (1 - (1 - k / E) ** T) + 2.0 * H * E
        else:
            flops += 2.0 * T * 3 * H * cfg.intermediate_size
            size += wide * 3 * H * cfg.intermediate_size
    if case["start"] + case["layers"] == cfg.num_hidden_layers:
        rows = len(prompts) + len(decode)
        flops += 2.0 * rows * cfg.vocab_size * H
        size += 2.0 * (H + rows) * cfg.vocab_size
    return dict(bytes=size, flops=flops)


def tolerance(case):
    """bf16 activations between the kernels of a layer (about 0.5 % of the result between two orders of the sums), with fp8
    weights e4m3 activations, too; a routed or indexed choice may fall differently on a tie."""
    return dict(rel=0.03 if case["model"].startswith("deepseek") else 0.02, max=0.9)


# ------------------------------------------------------------------------------------------------ in 64 bits
def _rms(x, w, eps):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w.double()


def _angles(pos, rot, theta):
    inv = 1.0 / (theta ** (torch.arange(0, rot, 2, dtype=torch.float64, device=DEV) / rot))
    a = pos.double()[:, None] * inv
    return a.cos(), a.sin()


def _rotate(x, pos, rot, theta, pairs):
    """Rotates the first ``rot`` columns of ``x [T, ..., D]``: neighbours (``pairs``) or halves."""
    c, s = _angles(pos, rot, theta)
    c, s = (t.view(t.shape[0], *[1] * (x.dim() - 2), -1) for t in (c, s))
    y, half = x.clone(), rot // 2
    a, b = (x[..., 0:rot:2], x[..., 1:rot:2]) if pairs else (x[..., :half], x[..., half:rot])
    if pairs:
        y[..., 0:rot:2], y[..., 1:rot:2] = a * c - b * s, a * s + b * c
    else:
        y[..., :half], y[..., half:rot] = a * c - b * s, b * c + a * s
    return y


def _mm(x, w):
    return x @ w.double().t()


def _glu(x, g, u, d):
    return _mm(torch.nn.functional.silu(_mm(x, g)) * _mm(x, u), d)


def _rows_of(cache, plan, i, total):
    """Cached rows of sequence i, ``[total, heads, columns]``."""
    pos = torch.arange(total, device=DEV)
    block = torch.from_numpy(plan["table"][i].astype(np.int64)).to(DEV)[pos // PAGE]
    return cache[block, :, pos % PAGE]


def _store(cache, rows, plan):
    s = torch.from_numpy(plan["slots"]).to(DEV)
    if cache.dtype == torch.float8_e4m3fn:
        raw = cache.view(torch.uint8)
        raw[s // PAGE, :, s % PAGE] = rows.clamp(-448, 448).float().to(cache.dtype).view(torch.uint8)
    else:
        cache[s // PAGE, :, s % PAGE] = rows.to(cache.dtype)


def _softmax_rows(scores, v, seen):
    """Rows of softmax(scores) v with the keys that ``seen [n, keys]`` allows; scores ``[heads, n, keys]``."""
    return scores.masked_fill_(~seen, -math.inf).softmax(-1) @ v


def _attend(q, k, v, n, total, scale, chosen=None):
    """``q [n, Hq, d]``, ``k``, ``v [total, Hkv, ...]`` -> ``[n, Hq, dv]``."""
    out, rep = [], q.shape[1] // k.shape[1]
    pos = torch.arange(total - n, total, device=DEV)
    step = max(1, (1 << 29) // (total * rep * (8 if chosen is not None else 4)))
    for h in range(k.shape[1]):
        qh, kh, vh = q[:, h * rep:(h + 1) * rep].transpose(0, 1), k[:, h].double(), v[:, h].double()
        parts = []
        for a in range(0, n, step):
            seen = torch.arange(total, device=DEV)[None] <= pos[a:a + step, None]
            if chosen is not None:
                seen = seen & chosen[a:a + step]
            parts.append(_softmax_rows(qh[:, a:a + step] @ kh.t() * scale, vh, seen))
        out.append(torch.cat(parts, 1).transpose(0, 1))
    return torch.cat(out, 1)


def _each(plan):
    """(index, first row, new tokens, tokens with keys) of every sequence."""
    at = 0
    for i, (n, total) in enumerate(plan["seqs"]):
        yield i, at, n, total
        at += n


def _gqa(cfg, w, a, x, c, plan, pos):
    T, D, Hq, Hkv, eps = x.shape[0], cfg.head_dim, cfg.num_attention_heads, cfg.num_key_value_heads, cfg.rms_norm_eps
    hybrid = cfg.model_type == "qwen3_next"
    q = _mm(x, w[a + "q_proj.weight"]).view(T, Hq, -1)
    q, gate = q[..., :D], q[..., D:]
    k, v = (_mm(x, w[a + n + "_proj.weight"]).view(T, Hkv, D) for n in "kv")
    one = 1.0 if hybrid else 0.0
    q = _rotate(_rms(q, w[a + "q_norm.weight"].double() + one, eps), pos, cfg.rot_dim, cfg.rope_theta, False)
    k = _rotate(_rms(k, w[a + "k_norm.weight"].double() + one, eps), pos, cfg.rot_dim, cfg.rope_theta, False)
    _store(c["k"], k, plan)
    _store(c["v"], v, plan)
    o = torch.empty_like(q)
    for i, at, n, total in _each(plan):
        # (the step's own rows come from the pages too: that they are rounded there is part of the path)
        kk, vv = _rows_of(c["k"], plan, i, total), _rows_of(c["v"], plan, i, total)
        o[at:at + n] = _attend(q[at:at + n], kk, vv, n, total, D ** -0.5)
    if hybrid:
        o = o * torch.sigmoid(gate)
    return _mm(o.reshape(T, -1), w[a + "o_proj.weight"])


def _latent(cfg, w, a, x, c, plan, pos):
    T, Hq, eps, theta = x.shape[0], cfg.num_attention_heads, cfg.rms_norm_eps, cfg.rope_theta
    L, R, nope, V = cfg.kv_lora_rank, cfg.qk_rope_head_dim, cfg.qk_nope_head_dim, cfg.v_head_dim
    qr = _rms(_mm(x, w[a + "q_a_proj.weight"]), w[a + "q_a_layernorm.weight"], eps)
    q = _mm(qr, w[a + "q_b_proj.weight"]).view(T, Hq, nope + R)
    kv = _mm(x, w[a + "kv_a_proj_with_mqa.weight"])
    row = torch.cat([_rms(kv[:, :L], w[a + "kv_a_layernorm.weight"], eps), _rotate(kv[:, L:], pos, R, theta, True)], -1)
    _store(c["k"], row[:, None], plan)
    kvb = w[a + "kv_b_proj.weight"].double().view(Hq, nope + V, L)
    q = torch.cat([torch.einsum("thd,hdl->thl", q[..., :nope], kvb[:, :nope]), _rotate(q[..., nope:], pos, R, theta, True)], -1)
    if cfg.index_topk:
        Di, x_ = cfg.index_head_dim, a + "indexer."
        iq = _rotate(_mm(qr, w[x_ + "wq_b.weight"]).view(T, -1, Di), pos, R, theta, True)
        ik = torch.nn.functional.layer_norm(_mm(x, w[x_ + "wk.weight"]), (Di,), w[x_ + "k_norm.weight"].double(),
                                            w[x_ + "k_norm.bias"].double(), 1e-5)
        _store(c["index_k"], _rotate(ik, pos, R, theta, True)[:, None], plan)
        iw = _mm(x, w[x_ + "weights_proj.weight"]) * (cfg.index_n_heads * Di) ** -0.5
    o = torch.empty((T, Hq, L), dtype=torch.float64, device=DEV)
    for i, at, n, total in _each(plan):
        rows = _rows_of(c["k"], plan, i, total)[:, 0].double()
        chosen = None
        if cfg.index_topk and total > cfg.index_topk:
            keys = _rows_of(c["index_k"], plan, i, total)[:, 0].double()
            score = torch.zeros((n, total), dtype=torch.float64, device=DEV)
            for h in range(iq.shape[1]):
                score += torch.relu(iq[at:at + n, h] @ keys.t()) * iw[at:at + n, h:h + 1]
            late = torch.arange(total, device=DEV)[None] > torch.arange(total - n, total, device=DEV)[:, None]
            best = score.masked_fill_(late, -math.inf).topk(cfg.index_topk, -1).indices
            chosen = torch.zeros((n, total), dtype=torch.bool, device=DEV).scatter_(1, best, True)
        o[at:at + n] = _attend(q[at:at + n], rows[:, None], rows[:, None, :L], n, total, (nope + R) ** -0.5, chosen)
    return _mm(torch.einsum("thl,hvl->thv", o, kvb[:, nope:]).reshape(T, -1), w[a + "o_proj.weight"])


def _delta(cfg, w, a, x, c, plan, pos):
    T = x.shape[0]
    hk, hv, dk, dv = cfg.linear_num_key_heads, cfg.linear_num_value_heads, cfg.linear_key_head_dim, cfg.linear_value_head_dim
    u, taps = _mm(x, w[a + "in_proj_qkv.weight"]), w[a + "conv1d.weight"].double()[:, 0]
    K = taps.shape[1]
    z, beta = _mm(x, w[a + "in_proj_z.weight"]).view(T, hv, dv), torch.sigmoid(_mm(x, w[a + "in_proj_b.weight"]))
    step = torch.nn.functional.softplus(_mm(x, w[a + "in_proj_a.weight"]) + w[a + "dt_bias"].double())
    decay = torch.exp(-torch.exp(w[a + "A_log"].double()) * step)
    mixed = torch.empty_like(u)
    states = c["rec_state"].double()
    for i, at, n, total in _each(plan):
        old = c["conv_state"][i].double().t() * (total > n)
        states[i] *= float(total > n)
        win = torch.cat([old, u[at:at + n]], 0)
        mixed[at:at + n] = torch.nn.functional.silu((win.unfold(0, K, 1) * taps).sum(-1))
        c["conv_state"][i] = win[-(K - 1):].t().to(torch.bfloat16)
    q, k, v = mixed.split([hk * dk, hk * dk, hv * dv], -1)
    q, k = (t.reshape(T, hk, dk) * torch.rsqrt(t.reshape(T, hk, dk).pow(2).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
    q, k = (q * dk ** -0.5).repeat_interleave(hv // hk, 1), k.repeat_interleave(hv // hk, 1)
    v, o = v.reshape(T, hv, dv), torch.empty((T, hv, dv), dtype=torch.float64, device=DEV)
    cu = np.cumsum([0] + [n for n, _t in plan["seqs"]])
    longest = max(n for n, _t in plan["seqs"])
    for j in range(longest):                                # all sequences that have a j-th new token at once
        i = torch.tensor([s for s in range(len(plan["seqs"])) if cu[s] + j < cu[s + 1]], device=DEV)
        t = torch.from_numpy(cu[:-1]).to(DEV)[i] + j
        S = states[i] * decay[t][:, :, None, None]
        d = (v[t] - torch.einsum("bhvk,bhk->bhv", S, k[t])) * beta[t][:, :, None]
        S = S + d[..., None] * k[t][:, :, None, :]
        states[i] = S
        o[t] = torch.einsum("bhvk,bhk->bhv", S, q[t])
    c["rec_state"] = states
    o = _rms(o, w[a + "norm.weight"], cfg.rms_norm_eps) * torch.nn.functional.silu(z)
    return _mm(o.reshape(T, -1), w[a + "out_proj.weight"])


def _experts(cfg, w, m, x):
    p = _mm(x, w[m + "gate.weight"]).softmax(-1)
    top, ids = p.topk(cfg.num_experts_per_tok, -1)
    top = top / top.sum(-1, keepdim=True)
    y = torch.zeros_like(x)
    for e in range(cfg.num_experts):
        t, s = (ids == e).nonzero(as_tuple=True)
        if t.numel():
            n = m + f"experts.{e}."
            one = _glu(x[t], w[n + "gate_proj.weight"], w[n + "up_proj.weight"], w[n + "down_proj.weight"])
            y.index_add_(0, t, one * top[t, s][:, None])
    return y


def exact(case, seed):
    """The same step on float64 activations, from the same weights; pages are rounded as they are stored."""
    cfg, plan, hidden, w, cached = _inputs(case, seed)
    pos = torch.from_numpy(plan["pos"]).to(DEV)
    one = 1.0 if cfg.model_type == "qwen3_next" else 0.0       # zero-centred norm weights
    h = hidden.double()
    for j, c in enumerate(cached):
        i = case["start"] + j
        p = f"model.layers.{i}."
        x = _rms(h, w[p + "input_layernorm.weight"].double() + one, cfg.rms_norm_eps)
        if cfg.layer_kind(i) == "linear":
            h = h + _delta(cfg, w, p + "linear_attn.", x, c, plan, pos)
        else:
            h = h + (_latent if cfg.is_mla else _gqa)(cfg, w, p + "self_attn.", x, c, plan, pos)
        x = _rms(h, w[p + "post_attention_layernorm.weight"].double() + one, cfg.rms_norm_eps)
        m = p + "mlp."
        if cfg.layer_is_moe(i):
            h = h + _experts(cfg, w, m, x)
        else:
            for a in range(0, x.shape[0], 4096):
                h[a:a + 4096] += _glu(x[a:a + 4096], w[m + "gate_proj.weight"], w[m + "up_proj.weight"], w[m + "down_proj.weight"])
    if case["start"] + case["layers"] == cfg.num_hidden_layers:
        rows = h[torch.from_numpy(plan["last"]).long().to(DEV)]
        h = _mm(_rms(rows, w["model.norm.weight"].double() + one, cfg.rms_norm_eps), w["model.embed_tokens.weight"])
    return [h, [[c[n].double() for n in ("k", "v", "index_k", "conv_state", "rec_state") if n in c] for c in cached]]
