"""Chained layers of the families that have something of their own in a chain (adapters, attention sinks and expert biases, block
selection, index caches) against the same layers launched one after the other."""

from contextlib import nullcontext

import numpy as np
import pytest
import torch

from parallax_b200.engine.batch import BatchBuilder
from parallax_b200.engine.worker import StageWorker
from parallax_b200.loader.lora import LoRAStack
from parallax_b200.models.config import config_from_hf, named_config

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)
PAGE = 16


def _config(name):
    if name == "gpt-oss":       # attention sinks, windows, expert biases (mxfp4 experts are expanded when they are loaded)
        return config_from_hf(dict(
            architectures=["GptOssForCausalLM"], model_type="gpt_oss", hidden_size=512, num_hidden_layers=4, num_attention_heads=8,
            num_key_value_heads=2, head_dim=64, intermediate_size=512, moe_intermediate_size=512, num_local_experts=8,
            num_experts_per_tok=2, sliding_window=128, layer_types=["sliding_attention", "full_attention"] * 2, attention_bias=True,
            vocab_size=512, rope_theta=1e4, max_position_embeddings=4096))
    return named_config("qwen3-8b" if name == "lora" else name)


@pytest.mark.parametrize("name,start", [("lora", 8), ("gpt-oss", 1), ("small-msa", 1), ("deepseek-v3.2", 1)])
def test_chained_layers_give_the_same_bits(name, start):
    from parallax_b200.ops import cuda as cu

    cfg = _config(name)
    prompts, decode = [(70, 70), (33, 50)], [300, 2300, 17, 1]         # (new tokens, context); contexts of decoding rows
    seqs = prompts + [(1, c) for c in decode]
    blocks = sum(-(-t // PAGE) for _n, t in seqs)
    table = np.zeros((len(seqs), -(-2300 // PAGE)), dtype=np.int32)
    order, at = np.random.RandomState(3).permutation(blocks).astype(np.int32), 0
    for i, (_n, t) in enumerate(seqs):
        n = -(-t // PAGE)
        table[i, :n] = order[at:at + n]
        at += n
    pos = np.concatenate([np.arange(t - n, t, dtype=np.int32) for n, t in seqs])
    row = np.repeat(np.arange(len(seqs)), [n for n, _t in seqs])
    slots = table[row, pos // PAGE].astype(np.int64) * PAGE + pos % PAGE
    last = np.cumsum([n for n, _t in seqs]).astype(np.int32) - 1
    worker = StageWorker(cfg, start, start + 2, DEV, torch.bfloat16, PAGE, num_blocks=blocks, seed=1, max_positions=2400,
                         num_linear_slots=len(seqs))
    fb = BatchBuilder(DEV, len(pos), len(seqs), 2 * table.shape[1]).build(
        None, pos, slots, [n for n, _t in prompts], [t for _n, t in prompts], table[:2, :5], np.asarray(decode, dtype=np.int32),
        table[2:], last, np.arange(len(seqs), dtype=np.int32))
    g = torch.Generator(device=DEV).manual_seed(5)
    hidden = torch.randn(len(pos), cfg.hidden_size, device=DEV, dtype=torch.bfloat16, generator=g)
    caches = [[t for t in (c.k, c.v, c.index_k, c.conv_state, c.rec_state) if t is not None] for c in worker.pool.layers]
    for layer in caches:
        for t in layer:
            t.copy_((torch.randn(t.shape, device=DEV, generator=g) * 0.5).to(t.dtype))
    kept = [[t.clone() for t in layer] for layer in caches]
    if name == "lora":
        m = worker.model
        m.lora = LoRAStack(m, 2, 16)
        for per in m.lora.layers:
            for ab in per.values():
                for t in ab:
                    t.normal_(0, 0.05, generator=g)
        m.lora.scale.fill_(0.7)
        fb.extras["lora_ids"] = (torch.arange(len(pos), device=DEV) % 3 - 1).int()

    def step():
        for layer, old in zip(caches, kept):
            for t, o in zip(layer, old):
                t.copy_(o)
        return worker.run(fb, hidden)

    worker.model.chained = lambda h: nullcontext()
    want = step()
    after = [[t.clone() for t in layer] for layer in caches]
    del worker.model.chained
    for _ in range(4):
        y = step()
        for i, (layer, old) in enumerate(zip([*caches, [y]], [*after, [want]])):
            for t, o in zip(layer, old):
                # lists of chosen keys come in any order, and sums over them in the order of the list: bf16 roundings (behind the
                # first layer's caches, which no list has touched)
                if cfg.index_topk and i > 0:
                    assert float((t.float() - o.float()).norm() / o.float().norm()) < 1e-2
                else:
                    assert torch.equal(t.view(torch.uint8), o.view(torch.uint8))
    cu.check_status(DEV)
